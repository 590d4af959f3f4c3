// Self-collisions on the device: grid binning of the tets, the point-in-tet
// query of the surface vertices, the closest rest face, and the
// DeformableDeformableCollisionConstraint projections.
//   src/simobject/XPBDMeshObject.cpp:719-762 (selfCollisionCheck)
//   src/geometry/embree/EmbreeScene.cpp:369-393, EmbreeTetMeshGeometry.cpp:20-47
//   src/geometry/DeformableMeshSDF.cpp:68-82
#include "xpbd_device.cuh"

namespace xg {

namespace {

// ---- self-collisions: detection (selfCollisionCheck, XPBDMeshObject.cpp:719-762)
// and DeformableDeformableCollisionConstraint ----

// exclusive scan of n ints in three launches (block sums, their scan, the
// blocks' scans with offsets); out[n] = total
constexpr int kScanThreads = 1024, kScanItems = 4, kScanChunk = kScanThreads * kScanItems;

__device__ __forceinline__ int block_excl_scan(int v, int* total) {
    __shared__ int wsum[kScanThreads / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) wsum[wid] = incl;
    __syncthreads();
    if (wid == 0) {
        int w = lane < kScanThreads / 32 ? wsum[lane] : 0;
        int wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += y;
        }
        if (lane < kScanThreads / 32) wsum[lane] = wi - w;  // exclusive warp offsets
    }
    __syncthreads();
    const int res = wsum[wid] + incl - v;
    if (total) {
        __shared__ int tot;
        if (threadIdx.x == kScanThreads - 1) tot = res + v;
        __syncthreads();
        *total = tot;
    }
    __syncthreads();
    return res;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_partials(const int* __restrict__ in, int n, int* __restrict__ part) {
    pdl_wait_then_release();
    const int base = blockIdx.x * kScanChunk + threadIdx.x * kScanItems;
    int s = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; i++)
        if (base + i < n) s += in[base + i];
    int total = 0;
    block_excl_scan(s, &total);
    if (threadIdx.x == 0) part[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_part_single(int* __restrict__ part, int nb) {
    pdl_wait_then_release();
    __shared__ int carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int b0 = 0; b0 < nb; b0 += kScanThreads) {
        const int i = b0 + threadIdx.x;
        const int v = i < nb ? part[i] : 0;
        int total = 0;
        const int ex = block_excl_scan(v, &total);
        if (i < nb) part[i] = carry + ex;
        __syncthreads();
        if (threadIdx.x == 0) carry += total;
        __syncthreads();
    }
    if (threadIdx.x == 0) part[nb] = carry;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_apply(const int* __restrict__ in, int n,
                                                             const int* __restrict__ part, int* __restrict__ out,
                                                             int nb) {
    pdl_wait_then_release();
    const int base = blockIdx.x * kScanChunk + threadIdx.x * kScanItems;
    int v[kScanItems], s = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        v[i] = base + i < n ? in[base + i] : 0;
        s += v[i];
    }
    int run = part[blockIdx.x] + block_excl_scan(s, nullptr);
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        if (base + i < n) out[base + i] = run;
        run += v[i];
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) out[n] = part[nb];
}

__device__ __forceinline__ int grid_cell1(float v, float o, float cell, int n) {
    float f = (v - o) / cell;
    f = fminf(fmaxf(f, 0.f), (float)(n - 1));  // NaN gives 0
    return (int)f;
}

// each tet in the cell of its centroid, or in the overflow list when its box
// is wider than a cell in some axis
__global__ void k_self_bin_count(SelfArrays a, SelfGrid g, const float4* __restrict__ x) {
    pdl_wait_then_release();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= a.T) return;
    const int4 e = a.tets[t];
    const float4 p0 = x[e.x], p1 = x[e.y], p2 = x[e.z], p3 = x[e.w];
    const float ex = fmaxf(fmaxf(p0.x, p1.x), fmaxf(p2.x, p3.x)) - fminf(fminf(p0.x, p1.x), fminf(p2.x, p3.x));
    const float ey = fmaxf(fmaxf(p0.y, p1.y), fmaxf(p2.y, p3.y)) - fminf(fminf(p0.y, p1.y), fminf(p2.y, p3.y));
    const float ez = fmaxf(fmaxf(p0.z, p1.z), fmaxf(p2.z, p3.z)) - fminf(fminf(p0.z, p1.z), fminf(p2.z, p3.z));
    int c = -1;
    if (ex <= g.cell && ey <= g.cell && ez <= g.cell) {
        const int cx = grid_cell1(0.25f * (p0.x + p1.x + p2.x + p3.x), g.ox, g.cell, g.nx);
        const int cy = grid_cell1(0.25f * (p0.y + p1.y + p2.y + p3.y), g.oy, g.cell, g.ny);
        const int cz = grid_cell1(0.25f * (p0.z + p1.z + p2.z + p3.z), g.oz, g.cell, g.nz);
        c = (cz * g.ny + cy) * g.nx + cx;
        atomicAdd(a.cell_count + c, 1);
    } else {
        a.overflow[atomicAdd(a.n_overflow, 1)] = t;
    }
    a.tet_cell[t] = c;
}

__global__ void k_self_bin_fill(SelfArrays a) {
    pdl_wait_then_release();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= a.T) return;
    const int c = a.tet_cell[t];
    if (c < 0) return;
    a.cell_tets[a.cell_off[c] + atomicAdd(a.cell_fill + c, 1)] = t;
}

// EmbreeTetMeshGeometry::isPointInTetrahedron (EmbreeTetMeshGeometry.cpp:20-47),
// float, with every product and sum rounded on its own (no contraction), as
// the host computes it
__device__ __forceinline__ bool same_side_f(const float* p, const float* a, const float* b, const float* c,
                                            const float* d) {
    const float ab0 = __fsub_rn(b[0], a[0]), ab1 = __fsub_rn(b[1], a[1]), ab2 = __fsub_rn(b[2], a[2]);
    const float ac0 = __fsub_rn(c[0], a[0]), ac1 = __fsub_rn(c[1], a[1]), ac2 = __fsub_rn(c[2], a[2]);
    const float n0 = __fsub_rn(__fmul_rn(ab1, ac2), __fmul_rn(ab2, ac1));
    const float n1 = __fsub_rn(__fmul_rn(ab2, ac0), __fmul_rn(ab0, ac2));
    const float n2 = __fsub_rn(__fmul_rn(ab0, ac1), __fmul_rn(ab1, ac0));
    const float sp = __fadd_rn(__fadd_rn(__fmul_rn(n0, __fsub_rn(p[0], a[0])), __fmul_rn(n1, __fsub_rn(p[1], a[1]))),
                               __fmul_rn(n2, __fsub_rn(p[2], a[2])));
    const float sd = __fadd_rn(__fadd_rn(__fmul_rn(n0, __fsub_rn(d[0], a[0])), __fmul_rn(n1, __fsub_rn(d[1], a[1]))),
                               __fmul_rn(n2, __fsub_rn(d[2], a[2])));
    return __fmul_rn(sp, sd) >= 0.f;
}

// EmbreeScene::tetMeshSelfCollisionQuery: the lowest-index tet holding the
// surface vertex among those that do not have it as a vertex. One warp a
// vertex: the 27 cells are nine runs of up to three neighbours in the sorted
// tet list, whose tets the lanes test 32 at a time (a chain of three dependent
// loads each; one thread a vertex walked about 150 of them, 129 us for 1,734
// vertices, now 10).
__global__ void __launch_bounds__(128) k_self_query(SelfArrays a, SelfGrid g, const float4* __restrict__ x) {
    pdl_wait_then_release();
    const int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (k >= a.n_surf) return;
    const int v = a.surf[k];
    const float4 pv = x[v];
    const float p[3] = {pv.x, pv.y, pv.z};
    int best = INT_MAX;
    auto test = [&](int t) {
        if (t >= best) return;
        const int4 e = a.tets[t];
        if (e.x == v || e.y == v || e.z == v || e.w == v) return;
        const float4 q0 = x[e.x], q1 = x[e.y], q2 = x[e.z], q3 = x[e.w];
        const float v0[3] = {q0.x, q0.y, q0.z}, v1[3] = {q1.x, q1.y, q1.z}, v2[3] = {q2.x, q2.y, q2.z},
                    v3[3] = {q3.x, q3.y, q3.z};
        if (same_side_f(p, v0, v1, v2, v3) && same_side_f(p, v0, v1, v3, v2) && same_side_f(p, v0, v2, v3, v1) &&
            same_side_f(p, v1, v2, v3, v0))
            best = t;
    };
    const int cx = grid_cell1(p[0], g.ox, g.cell, g.nx), cy = grid_cell1(p[1], g.oy, g.cell, g.ny),
              cz = grid_cell1(p[2], g.oz, g.cell, g.nz);
    // lane r < 9: the run of cells (cx - 1 .. cx + 1) of row r
    int from = 0, len = 0;
    if (lane < 9) {
        const int y = cy + lane % 3 - 1, z = cz + lane / 3 - 1;
        if (y >= 0 && y < g.ny && z >= 0 && z < g.nz) {
            const int row = (z * g.ny + y) * g.nx;
            from = a.cell_off[row + max(cx - 1, 0)];
            len = a.cell_off[row + min(cx + 1, g.nx - 1) + 1] - from;
        }
    }
    int end[9], start[9], total = 0;
#pragma unroll
    for (int r = 0; r < 9; r++) {
        const int n = __shfl_sync(0xffffffffu, len, r);
        start[r] = __shfl_sync(0xffffffffu, from, r) - total;
        total += n;
        end[r] = total;
    }
    for (int i = lane; i < total; i += 32) {
        int at = start[0];
#pragma unroll
        for (int r = 1; r < 9; r++)
            if (i >= end[r - 1]) at = start[r];
        test(a.cell_tets[at + i]);
    }
    const int no = *a.n_overflow;
    for (int i = lane; i < no; i += 32) test(a.overflow[i]);
    best = __reduce_min_sync(0xffffffffu, best);
    if (lane == 0) a.hit_tet[k] = best == INT_MAX ? -1 : best;
}

// the surface indices with a hit, ascending (one block)
__global__ void __launch_bounds__(kCompactThreads) k_self_compact(SelfArrays a) {
    __shared__ int warp_tot[kCompactThreads / 32];
    __shared__ int base;
    pdl_wait_then_release();
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    if (tid == 0) base = 0;
    __syncthreads();
    for (int b0 = 0; b0 < a.n_surf; b0 += kCompactThreads) {
        const int k = b0 + tid;
        const bool hit = k < a.n_surf && a.hit_tet[k] >= 0;
        const unsigned m = __ballot_sync(0xffffffffu, hit);
        if (lane == 0) warp_tot[wid] = __popc(m);
        __syncthreads();
        int off = base;
        for (int w = 0; w < wid; w++) off += warp_tot[w];
        if (hit) a.hit_list[off + __popc(m & ((1u << lane) - 1u))] = k;
        __syncthreads();
        if (tid == 0) {
            int t = 0;
            for (int w = 0; w < kCompactThreads / 32; w++) t += warp_tot[w];
            base += t;
        }
        __syncthreads();
    }
    if (tid == 0) *a.n_hits = base;
}

// Distance from p to triangle (a, b, c) in float: Ericson, Real-Time Collision
// Detection 5.1.5 (the method EmbreeMeshGeometry::_closestPointTriangle uses)
__device__ float point_triangle_distance_f(const float* p, const float* a, const float* b, const float* c) {
    auto dot = [](const float* u, const float* v) {
        return __fadd_rn(__fadd_rn(__fmul_rn(u[0], v[0]), __fmul_rn(u[1], v[1])), __fmul_rn(u[2], v[2]));
    };
    const float ab[3] = {__fsub_rn(b[0], a[0]), __fsub_rn(b[1], a[1]), __fsub_rn(b[2], a[2])};
    const float ac[3] = {__fsub_rn(c[0], a[0]), __fsub_rn(c[1], a[1]), __fsub_rn(c[2], a[2])};
    const float ap[3] = {__fsub_rn(p[0], a[0]), __fsub_rn(p[1], a[1]), __fsub_rn(p[2], a[2])};
    const float bp[3] = {__fsub_rn(p[0], b[0]), __fsub_rn(p[1], b[1]), __fsub_rn(p[2], b[2])};
    const float cp[3] = {__fsub_rn(p[0], c[0]), __fsub_rn(p[1], c[1]), __fsub_rn(p[2], c[2])};
    const float d1 = dot(ab, ap), d2 = dot(ac, ap), d3 = dot(ab, bp), d4 = dot(ac, bp), d5 = dot(ab, cp),
                d6 = dot(ac, cp);
    float o[3];
    if (d1 <= 0.f && d2 <= 0.f) {
        o[0] = a[0]; o[1] = a[1]; o[2] = a[2];
    } else if (d3 >= 0.f && d4 <= d3) {
        o[0] = b[0]; o[1] = b[1]; o[2] = b[2];
    } else if (d6 >= 0.f && d5 <= d6) {
        o[0] = c[0]; o[1] = c[1]; o[2] = c[2];
    } else {
        const float vc = __fsub_rn(__fmul_rn(d1, d4), __fmul_rn(d3, d2));
        const float vb = __fsub_rn(__fmul_rn(d5, d2), __fmul_rn(d1, d6));
        const float va = __fsub_rn(__fmul_rn(d3, d6), __fmul_rn(d5, d4));
        if (vc <= 0.f && d1 >= 0.f && d3 <= 0.f) {
            const float v = __fdiv_rn(d1, __fsub_rn(d1, d3));
            for (int k = 0; k < 3; k++) o[k] = __fadd_rn(a[k], __fmul_rn(v, ab[k]));
        } else if (vb <= 0.f && d2 >= 0.f && d6 <= 0.f) {
            const float v = __fdiv_rn(d2, __fsub_rn(d2, d6));
            for (int k = 0; k < 3; k++) o[k] = __fadd_rn(a[k], __fmul_rn(v, ac[k]));
        } else if (va <= 0.f && __fsub_rn(d4, d3) >= 0.f && __fsub_rn(d5, d6) >= 0.f) {
            const float v = __fdiv_rn(__fsub_rn(d4, d3), __fadd_rn(__fsub_rn(d4, d3), __fsub_rn(d5, d6)));
            for (int k = 0; k < 3; k++) o[k] = __fadd_rn(b[k], __fmul_rn(v, __fsub_rn(c[k], b[k])));
        } else {
            const float den = __fdiv_rn(1.f, __fadd_rn(__fadd_rn(va, vb), vc));
            const float v = __fmul_rn(vb, den), w = __fmul_rn(vc, den);
            for (int k = 0; k < 3; k++) o[k] = __fadd_rn(__fadd_rn(a[k], __fmul_rn(v, ab[k])), __fmul_rn(w, ac[k]));
        }
    }
    const float e0 = __fsub_rn(p[0], o[0]), e1 = __fsub_rn(p[1], o[1]), e2 = __fsub_rn(p[2], o[2]);
    return __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(e0, e0), __fmul_rn(e1, e1)), __fmul_rn(e2, e2)));
}

// the surface vertex v mapped to rest space through tet t into pm; 0 when the
// tet is degenerate
__device__ int rest_point(const SelfArrays& a, const float4* __restrict__ x, int v, int t, float* pm) {
    const int4 e = a.tets[t];
    const int ids[5] = {e.x, e.y, e.z, e.w, v};
    double xd[5][3];
    for (int i = 0; i < 5; i++) {
        const float4 q = x[ids[i]];
        xd[i][0] = q.x; xd[i][1] = q.y; xd[i][2] = q.z;
    }
    // F = Ds Q (column-major), as the host's compute_F
    const double* Q = a.Q + 9 * (size_t)t;
    double D[9], F[9];
    for (int i = 0; i < 3; i++)
        for (int r = 0; r < 3; r++) D[3 * i + r] = xd[i][r] - xd[3][r];
    for (int c = 0; c < 3; c++)
        for (int r = 0; r < 3; r++) F[3 * c + r] = D[r] * Q[3 * c] + D[3 + r] * Q[3 * c + 1] + D[6 + r] * Q[3 * c + 2];
    auto M = [&F](int r, int c) { return F[c * 3 + r]; };
    const double c00 = M(1, 1) * M(2, 2) - M(1, 2) * M(2, 1);
    const double c10 = M(1, 2) * M(2, 0) - M(1, 0) * M(2, 2);
    const double c20 = M(1, 0) * M(2, 1) - M(1, 1) * M(2, 0);
    const double det = M(0, 0) * c00 + M(0, 1) * c10 + M(0, 2) * c20;
    if (fabs(det) < 1e-8) return 0;
    const double inv = 1.0 / det;
    double Fi[9];
    Fi[0] = c00 * inv; Fi[1] = c10 * inv; Fi[2] = c20 * inv;
    Fi[3] = (M(0, 2) * M(2, 1) - M(0, 1) * M(2, 2)) * inv;
    Fi[4] = (M(0, 0) * M(2, 2) - M(0, 2) * M(2, 0)) * inv;
    Fi[5] = (M(0, 1) * M(2, 0) - M(0, 0) * M(2, 1)) * inv;
    Fi[6] = (M(0, 1) * M(1, 2) - M(0, 2) * M(1, 1)) * inv;
    Fi[7] = (M(0, 2) * M(1, 0) - M(0, 0) * M(1, 2)) * inv;
    Fi[8] = (M(0, 0) * M(1, 1) - M(0, 1) * M(1, 0)) * inv;
    const double rel[3] = {xd[4][0] - xd[3][0], xd[4][1] - xd[3][1], xd[4][2] - xd[3][2]};
    for (int r = 0; r < 3; r++)
        pm[r] = (float)(Fi[r] * rel[0] + Fi[3 + r] * rel[1] + Fi[6 + r] * rel[2] + a.X0[3 * (size_t)e.w + r]);
    return 1;
}

// DeformableMeshSDF::closestSurfaceFaceToPointInTet (DeformableMeshSDF.cpp:68-82):
// the vertex mapped to rest space through the tet it is in (F = Ds Dm^-1 in
// double, none when |det F| < 1e-8), then the closest face of the rest surface
// (float; of equally close faces the lowest index). One block a hit, one
// thread its rest point (FP64) and all of them the faces: a warp a hit took
// 122 us for 3,456 faces, all of it the chain of its own 108 rounds; now 23.
constexpr int kFaceThreads = 256;
__global__ void __launch_bounds__(kFaceThreads) k_self_face(SelfArrays a, const float4* __restrict__ x,
                                                            const int4* __restrict__ faces) {
    __shared__ float spm[3];
    __shared__ int sok, sbf[kFaceThreads / 32];
    __shared__ float sbd[kFaceThreads / 32];
    pdl_wait_then_release();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, n = *a.n_hits;
    for (int w = blockIdx.x; w < n; w += gridDim.x) {
        const int v = a.surf[a.hit_list[w]];
        if (threadIdx.x == 0) sok = rest_point(a, x, v, a.hit_tet[a.hit_list[w]], spm);
        __syncthreads();
        float bd = INFINITY;
        int bf = INT_MAX;
        if (sok) {
            const float pm[3] = {spm[0], spm[1], spm[2]};
#pragma unroll 2
            for (int f = threadIdx.x; f < a.F; f += kFaceThreads) {
                const int4 fv = faces[f];
                const float4 A = a.X0f[fv.x], B = a.X0f[fv.y], Cc = a.X0f[fv.z];
                const float qa[3] = {A.x, A.y, A.z}, qb[3] = {B.x, B.y, B.z}, qc[3] = {Cc.x, Cc.y, Cc.z};
                const float d = point_triangle_distance_f(pm, qa, qb, qc);
                if (d < bd) {
                    bd = d;
                    bf = f;
                }
            }
        }
        auto closer = [&](float od, int of) {
            if (od < bd || (od == bd && of < bf)) {
                bd = od;
                bf = of;
            }
        };
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float od = __shfl_xor_sync(0xffffffffu, bd, o);
            const int of = __shfl_xor_sync(0xffffffffu, bf, o);
            closer(od, of);
        }
        if (lane == 0) {
            sbd[wid] = bd;
            sbf[wid] = bf;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int i = 1; i < kFaceThreads / 32; i++) closer(sbd[i], sbf[i]);
            a.contact[w] = make_int2(v, bf == INT_MAX ? -1 : bf);
        }
        __syncthreads();
    }
}
// DeformableDeformableCollisionConstraint::evaluate / gradient
// (DeformableDeformableCollisionConstraint.cpp): C = (q - p1).a/|a| + 1e-5,
// a = (p2 - p1) x (p3 - p1); the gradient as the reference writes it (the
// third face vertex's term uses q - p2). g: q, p1, p2, p3 x 3
__device__ float self_contact_eval(const float* q, const float* p1, const float* p2, const float* p3, float* g) {
    const float e1[3] = {p2[0] - p1[0], p2[1] - p1[1], p2[2] - p1[2]};
    const float e2[3] = {p3[0] - p1[0], p3[1] - p1[1], p3[2] - p1[2]};
    const float av[3] = {e1[1] * e2[2] - e1[2] * e2[1], e1[2] * e2[0] - e1[0] * e2[2], e1[0] * e2[1] - e1[1] * e2[0]};
    const float an = sqrtf(av[0] * av[0] + av[1] * av[1] + av[2] * av[2]);
    const float u1[3] = {q[0] - p1[0], q[1] - p1[1], q[2] - p1[2]};
    const float u2[3] = {q[0] - p2[0], q[1] - p2[1], q[2] - p2[2]};
    const float C = (u1[0] * av[0] + u1[1] * av[1] + u1[2] * av[2]) / an + 1e-5f;
    const float an3 = an * an * an;
    float r1[3], r2[3];
    const float ad1 = av[0] * u1[0] + av[1] * u1[1] + av[2] * u1[2];
    const float ad2 = av[0] * u2[0] + av[1] * u2[1] + av[2] * u2[2];
    for (int k = 0; k < 3; k++) {
        r1[k] = u1[k] / an - av[k] * ad1 / an3;
        r2[k] = u2[k] / an - av[k] * ad2 / an3;
    }
    auto cross = [](const float* x, const float* y, float* r) {
        r[0] = x[1] * y[2] - x[2] * y[1];
        r[1] = x[2] * y[0] - x[0] * y[2];
        r[2] = x[0] * y[1] - x[1] * y[0];
    };
    float t[3];
    for (int k = 0; k < 3; k++) g[k] = av[k] / an;
    const float d32[3] = {p3[0] - p2[0], p3[1] - p2[1], p3[2] - p2[2]};
    cross(r1, d32, t);
    for (int k = 0; k < 3; k++) g[3 + k] = -av[k] / an + t[k];
    const float d13[3] = {p1[0] - p3[0], p1[1] - p3[1], p1[2] - p3[2]};
    cross(r1, d13, t);
    for (int k = 0; k < 3; k++) g[6 + k] = t[k];
    const float d21[3] = {p2[0] - p1[0], p2[1] - p1[1], p2[2] - p1[2]};
    cross(r2, d21, t);
    for (int k = 0; k < 3; k++) g[9 + k] = t[k];
    return C;
}

// ConstraintProjector::project (ConstraintProjector.hpp:111-172) of self
// contact j on the vertices xs (surface vertex, face): skipped when C > 0;
// alpha~ = 1e-8/dt^2 (or /dt)
__device__ bool self_update(const SelfArrays& a, int j, bool first, float at, const float4 xs[4], float d[4][3],
                            Flags* flags) {
    float lam = first ? 0.f : a.lam[j];
    float p[4][3];
    for (int i = 0; i < 4; i++) {
        p[i][0] = xs[i].x; p[i][1] = xs[i].y; p[i][2] = xs[i].z;
    }
    float g[12];
    const float C = self_contact_eval(p[0], p[1], p[2], p[3], g);
    bool ok = false;
    if (!(C > 0.f)) {
        float L = at;
        for (int i = 0; i < 4; i++)
            L += fabsf(xs[i].w) * (g[3 * i] * g[3 * i] + g[3 * i + 1] * g[3 * i + 1] + g[3 * i + 2] * g[3 * i + 2]);
        const float dl = (-C - at * lam) / L;
        if (!isfinite(dl)) {
            atomicAdd(&flags->nonfinite, 1ull);
        } else {
            lam += dl;
            for (int i = 0; i < 4; i++)
                for (int k = 0; k < 3; k++) d[i][k] = fabsf(xs[i].w) * g[3 * i + k] * dl;
            ok = true;
        }
    }
    a.lam[j] = lam;
    return ok;
}

__device__ __forceinline__ int4 self_ids(const SelfArrays& a, int j, const int4* __restrict__ faces) {
    const int2 ct = a.contact[j];
    if (ct.y < 0) return make_int4(-1, -1, -1, -1);
    const int4 fv = faces[ct.y];
    return make_int4(ct.x, fv.x, fv.y, fv.z);
}

// After a detection: the Gauss-Seidel contacts in rounds that keep the effect
// of detection order. In each round every contact that is left bids for its
// four vertices with its number; one that holds all four has no earlier
// contact left on any of them and goes into the round. Contacts of one round
// share no vertex, and of two on a common vertex the earlier one is in the
// earlier round. One block; the bids lie in shared memory, by each vertex's
// lowest (contact, corner) number, or beyond kPlanShared contacts in owner[].
// owner is all 0x7f bytes before.
// A vertex of many contacts takes a round for each of them, in which all that are
// left bid again: 10,201 contacts, 9,460 of them on one face, took 226 ms to plan
// and lost by it (four sweeps 41.0 ms in rounds, 34.0 one by one). So there is no
// plan (n_rounds -1, the projection walks the list) where a vertex has more than
// plan_rounds(n) contacts or the rounds get to be more. Two cubes pressed
// together take about 2 sqrt(n).
constexpr int kPlanThreads = 1024, kPlanShared = 4096, kPlanMost = 32 * kPlanThreads;
constexpr int kNoOwner = 0x7f7f7f7f;
__host__ __device__ constexpr int plan_rounds(int n) { return n < 256 ? 64 : (n < 2048 ? n / 4 : 512); }
__global__ void __launch_bounds__(kPlanThreads) k_self_plan(SelfArrays a, const int4* __restrict__ faces) {
    extern __shared__ int bids[];  // [4 kPlanShared] bids, [4 kPlanShared] the vertices' numbers
    __shared__ int placed, left, most;
    pdl_wait_then_release();
    const int n = *a.n_hits, tid = threadIdx.x, limit = plan_rounds(n);
    if (n > kPlanMost) {  // more than a thread's 32 bits: the projection walks them one by one
        if (tid == 0) *a.n_rounds = -1;
        return;
    }
    const bool small = n <= kPlanShared;
    volatile int* const owner = a.owner;
    unsigned mine = 0;  // contacts tid + 1024 b that are left
    if (tid == 0) placed = most = 0;
    for (int b = 0; tid + kPlanThreads * b < n; b++) {
        const int j = tid + kPlanThreads * b;
        const int4 id = self_ids(a, j, faces);
        if (id.x < 0) continue;
        mine |= 1u << b;
        if (small) {
            const int v[4] = {id.x, id.y, id.z, id.w};
            for (int k = 0; k < 4; k++) atomicMin(a.owner + v[k], 4 * j + k);
        }
    }
    __syncthreads();
    if (small) {
        for (int i = tid; i < 4 * n; i += kPlanThreads) bids[i] = kNoOwner;
        for (unsigned m = mine; m; m &= m - 1) {
            const int j = tid + kPlanThreads * (__ffs((int)m) - 1);
            const int4 id = self_ids(a, j, faces);
            const int v[4] = {id.x, id.y, id.z, id.w};
            for (int k = 0; k < 4; k++) bids[4 * kPlanShared + 4 * j + k] = owner[v[k]];
        }
        __syncthreads();
        for (unsigned m = mine; m; m &= m - 1) {
            const int4 id = self_ids(a, tid + kPlanThreads * (__ffs((int)m) - 1), faces);
            owner[id.x] = kNoOwner; owner[id.y] = kNoOwner; owner[id.z] = kNoOwner; owner[id.w] = kNoOwner;
        }
        __syncthreads();
    }
    volatile int* const own = small ? bids : a.owner;
    auto each = [&](unsigned set, auto&& f) {
        for (unsigned m = set; m; m &= m - 1) {
            const int b = __ffs((int)m) - 1, j = tid + kPlanThreads * b;
            int at[4];
            if (small) {
                for (int k = 0; k < 4; k++) at[k] = bids[4 * kPlanShared + 4 * j + k];
            } else {
                const int4 id = self_ids(a, j, faces);
                at[0] = id.x; at[1] = id.y; at[2] = id.z; at[3] = id.w;
            }
            f(b, j, at);
        }
    };
    // the contacts of the vertex that has most, counted down from kNoOwner
    each(mine, [&](int, int, const int* at) {
        for (int k = 0; k < 4; k++) atomicSub((int*)own + at[k], 1);
    });
    __syncthreads();
    each(mine, [&](int, int, const int* at) {
        for (int k = 0; k < 4; k++)
            if (kNoOwner - own[at[k]] > limit) most = limit + 1;
    });
    __syncthreads();
    if (most > limit) {
        if (tid == 0) *a.n_rounds = -1;
        return;
    }
    each(mine, [&](int, int, const int* at) {
        for (int k = 0; k < 4; k++) own[at[k]] = kNoOwner;
    });
    __syncthreads();
    int round = 0;
    for (;;) {
        if (tid == 0) {
            a.round_off[round] = placed;
            left = 0;
        }
        each(mine, [&](int, int j, const int* at) {
            for (int k = 0; k < 4; k++) atomicMin((int*)own + at[k], j);
        });
        __syncthreads();
        unsigned ready = 0;
        each(mine, [&](int b, int j, const int* at) {
            if (own[at[0]] == j && own[at[1]] == j && own[at[2]] == j && own[at[3]] == j) ready |= 1u << b;
        });
        __syncthreads();
        each(ready, [&](int, int j, const int* at) {
            for (int k = 0; k < 4; k++) own[at[k]] = kNoOwner;
            const int i = atomicAdd(&placed, 1);
            a.plan[i] = j;
            a.plan_ids[i] = self_ids(a, j, faces);
        });
        mine &= ~ready;
        if (mine) left = 1;
        __syncthreads();
        round++;
        if (!left || round == limit) break;
        __syncthreads();
    }
    if (tid == 0) {
        a.round_off[round] = placed;
        *a.n_rounds = left ? -1 : round;
    }
}

// Gauss-Seidel: the contacts as in detection (vertex) order, by the rounds of
// k_self_plan, one block. (One thread walking the list took 264 us for two
// 12^3 cubes in contact, four dependent loads and 0.4 us of arithmetic a
// contact; the rounds 48 us.) Without a plan one thread walks it.
constexpr int kSelfGsThreads = 128;
__device__ __forceinline__ void self_contact_gs(const SelfArrays& a, int j, const int4& ids, float4* __restrict__ x,
                                                bool first, float at, Flags* flags) {
    const float4 xs[4] = {x[ids.x], x[ids.y], x[ids.z], x[ids.w]};
    float d[4][3];
    if (!self_update(a, j, first, at, xs, d, flags)) return;
    const int v[4] = {ids.x, ids.y, ids.z, ids.w};
    if (v[0] != v[1] && v[0] != v[2] && v[0] != v[3] && v[1] != v[2] && v[1] != v[3] && v[2] != v[3]) {
        for (int i = 0; i < 4; i++)
            x[v[i]] = make_float4(xs[i].x + d[i][0], xs[i].y + d[i][1], xs[i].z + d[i][2], xs[i].w);
    } else {
        for (int i = 0; i < 4; i++) {
            const float4 c = x[v[i]];  // a vertex may repeat: add to the current value
            x[v[i]] = make_float4(c.x + d[i][0], c.y + d[i][1], c.z + d[i][2], c.w);
        }
    }
}

// Without a plan: one by one, one thread. Such lists have many contacts on one
// face, whose vertices stay in registers from one contact to the next; the next
// one's surface vertex is on its way meanwhile (a face or vertex that this
// contact moves is read after it). 10,201 contacts: 0.83 us each, 0.86 with every
// vertex read again.
__device__ void walk_contacts(const SelfArrays& a, const int4* __restrict__ faces, float4* __restrict__ x, bool first,
                              float at, Flags* flags) {
    const int n = *a.n_hits;
    const int4 none = make_int4(-1, -1, -1, -1);
    int4 ids = n > 0 ? self_ids(a, 0, faces) : none;
    float4 xs[4] = {};
    if (ids.x >= 0) { xs[0] = x[ids.x]; xs[1] = x[ids.y]; xs[2] = x[ids.z]; xs[3] = x[ids.w]; }
    for (int j = 0; j < n; j++) {
        const int4 next = j + 1 < n ? self_ids(a, j + 1, faces) : none;
        float4 nx = xs[0];
        if (next.x >= 0) nx = x[next.x];
        bool kept = ids.x >= 0;  // xs holds the face's current positions
        float d[4][3];
        if (ids.x >= 0 && self_update(a, j, first, at, xs, d, flags)) {
            const int v[4] = {ids.x, ids.y, ids.z, ids.w};
            kept = v[0] != v[1] && v[0] != v[2] && v[0] != v[3] && v[1] != v[2] && v[1] != v[3] && v[2] != v[3];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float4 c = kept ? xs[i] : x[v[i]];  // a vertex may repeat: add to the current value
                xs[i] = make_float4(c.x + d[i][0], c.y + d[i][1], c.z + d[i][2], c.w);
                x[v[i]] = xs[i];
            }
        }
        if (next.x >= 0) {
            if (!(kept && next.y == ids.y && next.z == ids.z && next.w == ids.w)) {
                xs[1] = x[next.y]; xs[2] = x[next.z]; xs[3] = x[next.w];
            }
            const bool moved = next.x == ids.x || next.x == ids.y || next.x == ids.z || next.x == ids.w;
            xs[0] = moved ? x[next.x] : nx;
        }
        ids = next;
    }
}

__global__ void __launch_bounds__(kSelfGsThreads) k_self_contacts_gs(SelfArrays a, const int4* __restrict__ faces,
                                                                     float4* __restrict__ x, bool first, float at,
                                                                     Flags* flags) {
    pdl_wait_then_release();
    const int rounds = *a.n_rounds;
    if (rounds < 0) {
        if (threadIdx.x == 0) walk_contacts(a, faces, x, first, at, flags);
        return;
    }
    // a round's first contacts are loaded while the one before runs
    int lo = rounds > 0 ? a.round_off[0] : 0, hi = rounds > 0 ? a.round_off[1] : 0;
    int i = lo + threadIdx.x, j = 0;
    int4 ids = make_int4(0, 0, 0, 0);
    if (i < hi) {
        j = a.plan[i];
        ids = a.plan_ids[i];
    }
    for (int r = 0; r < rounds; r++) {
        const int nhi = r + 1 < rounds ? a.round_off[r + 2] : hi;
        const int ni = hi + threadIdx.x;
        int nj = 0;
        int4 nids = make_int4(0, 0, 0, 0);
        if (r + 1 < rounds && ni < nhi) {
            nj = a.plan[ni];
            nids = a.plan_ids[ni];
        }
        if (i < hi) self_contact_gs(a, j, ids, x, first, at, flags);
        for (int k = i + kSelfGsThreads; k < hi; k += kSelfGsThreads)
            self_contact_gs(a, a.plan[k], a.plan_ids[k], x, first, at, flags);
        __syncthreads();
        i = ni;
        hi = nhi;
        j = nj;
        ids = nids;
    }
}

// Jacobi: every contact from the same positions, updates summed into dx
__global__ void k_self_contacts_jacobi(SelfArrays a, const int4* __restrict__ faces, const float4* __restrict__ x,
                                       float4* __restrict__ dx, bool first, float at, Flags* flags) {
    pdl_wait_then_release();
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= *a.n_hits) return;
    const int4 ids = self_ids(a, j, faces);
    if (ids.x < 0) return;
    const float4 xs[4] = {x[ids.x], x[ids.y], x[ids.z], x[ids.w]};
    float d[4][3];
    if (!self_update(a, j, first, at, xs, d, flags)) return;
    const int v[4] = {ids.x, ids.y, ids.z, ids.w};
    for (int i = 0; i < 4; i++) add_vec4(dx + v[i], d[i][0], d[i][1], d[i][2]);
}

}  // namespace

void launch_self_detect(const Launch& s, const SelfArrays& a, const SelfGrid& g, const float4* x, const int4* faces,
                        bool jacobi) {
    if (a.n_surf <= 0 || a.T <= 0) return;
    const int ncells = g.nx * g.ny * g.nz;
    cudaMemsetAsync(a.cell_count, 0, sizeof(int) * (size_t)ncells, s.s);
    cudaMemsetAsync(a.cell_fill, 0, sizeof(int) * (size_t)ncells, s.s);
    cudaMemsetAsync(a.n_overflow, 0, sizeof(int), s.s);
    go(k_self_bin_count, nblk(a.T, 256), 256, s, a, g, x);
    const int nb = (ncells + kScanChunk - 1) / kScanChunk;
    go(k_scan_partials, nb, kScanThreads, s, (const int*)a.cell_count, ncells, a.scan_part);
    go(k_scan_part_single, 1, kScanThreads, s, a.scan_part, nb);
    go(k_scan_apply, nb, kScanThreads, s, (const int*)a.cell_count, ncells, (const int*)a.scan_part, a.cell_off, nb);
    go(k_self_bin_fill, nblk(a.T, 256), 256, s, a);
    go(k_self_query, nblk(32 * (long long)a.n_surf, 128), 128, s, a, g, x);
    go(k_self_compact, 1, kCompactThreads, s, a);
    go(k_self_face, a.n_surf < 1024 ? a.n_surf : 1024, kFaceThreads, s, a, x, faces);
    if (!jacobi) {
        cudaMemsetAsync(a.owner, 0x7f, sizeof(int) * (size_t)a.V, s.s);
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(1);
        cfg.blockDim = dim3(kPlanThreads);
        cfg.dynamicSmemBytes = 8 * sizeof(int) * kPlanShared;
        cfg.stream = s.s;
        cudaLaunchKernelEx(&cfg, k_self_plan, a, faces);
    }
}

cudaError_t self_prepare_kernels() {
    return cudaFuncSetAttribute(k_self_plan, cudaFuncAttributeMaxDynamicSharedMemorySize, 8 * sizeof(int) * kPlanShared);
}

void launch_self_contacts(const Launch& s, const SelfArrays& a, const int4* faces, float4* x, float4* dx,
                          bool jacobi, bool first, float alpha_tilde, Flags* flags) {
    if (a.n_surf <= 0) return;
    if (jacobi) go(k_self_contacts_jacobi, nblk(a.n_surf, 128), 128, s, a, faces, (const float4*)x, dx, first,
                   alpha_tilde, flags);
    else go(k_self_contacts_gs, 1, kSelfGsThreads, s, a, faces, x, first, alpha_tilde, flags);
}

}  // namespace xg
