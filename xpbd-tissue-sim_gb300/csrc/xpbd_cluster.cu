// Gauss-Seidel on chip: a whole substep of a small mesh in one launch of one
// thread-block cluster per instance. Vertices, multipliers and the patches'
// topology live in shared memory for the whole solve, a colour ends at a
// cluster (or, with one block, a block) barrier, and a vertex that two blocks
// hold is written into the other's copy over distributed shared memory. Same patches, colours, order and arithmetic as the colour launches
// and the versioned sweep (xpbd_kernels.cu); the results agree bit for bit.
//
// Measured on GB300, per substep against the versioned sweep with its launches
// around it: the 5,000-tet cube at 10 sweeps 187 -> 105 us (one block, 1.09 us a
// colour), the 50,000-tet beam at 20 sweeps with a sphere's contacts 680 -> 400
// us (10 blocks, 1.5 us). Tried for the exchange between blocks and slower, per
// colour of 126 patches a block: a cluster barrier with the stores in the
// projecting lanes 2.1 us, vertices counted on an mbarrier (st.async) 2.9 us.
#include "xpbd_device.cuh"

namespace xg {

namespace {

__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ unsigned mapa(unsigned addr, unsigned rank) {
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}

// A block's vertex: the position and a fourth word in one 128-bit word. The
// first nb vertices of a block are held by one other block of the cluster too;
// their fourth word is the vertex's version, and the inverse mass, which no
// sweep changes, lies beside (sw). The others' is the inverse mass. Shared
// vertices are read and written by one scalar .b128 access, which the PTX
// memory model makes single-copy atomic: a reader that sees the due version
// has the three coordinates written with it.
struct alignas(16) VertWord {
    unsigned long long xy, zf;  // x | y << 32, z | fourth << 32
};
__device__ __forceinline__ unsigned long long pack2(float lo, unsigned hi) {
    return (unsigned long long)__float_as_uint(lo) | (unsigned long long)hi << 32;
}
__device__ __forceinline__ VertWord ld_vert(const VertWord* p) {
    VertWord v;
    asm volatile(
        "{\n\t.reg .b128 q;\n\tld.relaxed.cluster.shared::cta.b128 q, [%2];\n\tmov.b128 {%0, %1}, q;\n\t}"
        : "=l"(v.xy), "=l"(v.zf)
        : "r"(smem_u32(p))
        : "memory");
    return v;
}
__device__ __forceinline__ void st_vert(VertWord* p, const VertWord& v) {
    asm volatile(
        "{\n\t.reg .b128 q;\n\tmov.b128 q, {%1, %2};\n\tst.relaxed.cluster.shared::cta.b128 [%0], q;\n\t}" ::"r"(
            smem_u32(p)),
        "l"(v.xy), "l"(v.zf)
        : "memory");
}
__device__ __forceinline__ void st_vert_cluster(unsigned addr, const VertWord& v) {  // shared::cluster address
    asm volatile(
        "{\n\t.reg .b128 q;\n\tmov.b128 q, {%1, %2};\n\tst.relaxed.cluster.shared::cluster.b128 [%0], q;\n\t}" ::"r"(
            addr),
        "l"(v.xy), "l"(v.zf)
        : "memory");
}
__device__ __forceinline__ void red_or_cluster(unsigned addr, unsigned bits) {  // shared::cluster address
    asm volatile("red.relaxed.cluster.shared::cluster.or.b32 [%0], %1;" ::"r"(addr), "r"(bits) : "memory");
}

template <bool MULTI>
struct BlockVerts {
    VertWord* sv;
    const float* sw;   // [nb] the shared vertices' inverse masses
    const unsigned* rem;  // [nb] their other copy: rank << 12 | index
    int nb;
    __device__ __forceinline__ bool shared(int l) const { return MULTI && l < nb; }
    // vertex l into p; whether it is due (a block's own vertices always are)
    __device__ __forceinline__ bool look(int l, int due, float4& p) const {
        if (!MULTI) {
            p = *reinterpret_cast<const float4*>(sv + l);
            return true;
        }
        const VertWord v = ld_vert(sv + l);
        const unsigned f = (unsigned)(v.zf >> 32);
        p = make_float4(__uint_as_float((unsigned)v.xy), __uint_as_float((unsigned)(v.xy >> 32)),
                        __uint_as_float((unsigned)v.zf), __uint_as_float(f));
        if (shared(l)) p.w = sw[l];
        return !shared(l) || (int)f >= due;
    }
    __device__ __forceinline__ void put(int l, const float4& p, int ver) const {
        if (!MULTI) *reinterpret_cast<float4*>(sv + l) = p;
        else st_vert(sv + l, VertWord{pack2(p.x, __float_as_uint(p.y)),
                                      pack2(p.z, shared(l) ? (unsigned)ver : __float_as_uint(p.w))});
    }
    // a shared vertex into its other copy
    __device__ __forceinline__ void send(int l) const {
        if (!shared(l)) return;
        const VertWord v = ld_vert(sv + l);
        const unsigned m = rem[l];
        st_vert_cluster(mapa(smem_u32(sv) + 16u * (m & 0xfffu), m >> 12), v);
    }
};

// One lane's patch: the projections, their order and the near-degenerate and
// non-finite rules are those of the other sweep kernels. Combined form
// (WHICH 2): one straight FP32 pass, redone from the patch's state before the
// task (still in shared memory, nothing is stored before the end) with the
// per-tet FP64 guard when a tet needs it. WHICH 0 / 1: one constraint, the
// guard per tet. HEX: the canonical grid-hex layout, vertices in registers;
// else in the lane's scratch column.
// due: the versions at which its shared vertices are ready. Returns false when
// the wait for one gave up.
template <int WHICH, bool HEX, bool MULTI>
__device__ __forceinline__ bool cluster_patch(const TetArrays& t, const BlockVerts<MULTI>& bv, const int4& vi,
                                              const int (&due)[kMaxPatchVerts], const int4& meta, const int* __restrict__ slot, const float4* __restrict__ q0,
                                              const float4* __restrict__ q1, const float4* __restrict__ q2,
                                              float2* __restrict__ sl, float4* __restrict__ scratch, int sstride,
                                              unsigned polls, Flags* flags) {
    const int ntets = HEX ? kMaxPatchTets : (meta.y & 0xff);
    const int nverts = HEX ? kMaxPatchVerts : (meta.y >> 8);
    const int vw[4] = {vi.x, vi.y, vi.z, vi.w};
    int l8[kMaxPatchVerts];
#pragma unroll
    for (int k = 0; k < kMaxPatchVerts; k++) l8[k] = (vw[k >> 1] >> (16 * (k & 1))) & 0xffff;
    float4 pv[kMaxPatchVerts] = {};
    auto vget = [&](int l) -> float4 { return HEX ? pv[l] : scratch[l * sstride]; };
    auto vset = [&](int l, const float4& p) {
        if (HEX) pv[l] = p;
        else scratch[l * sstride] = p;
    };
    unsigned pending = 0;
#pragma unroll
    for (int k = 0; k < kMaxPatchVerts; k++) {
        if (k >= nverts) continue;
        float4 p;
        if (!bv.look(l8[k], due[k], p)) pending |= 1u << k;
        vset(k, p);
    }
    if (MULTI) {
        // every corner again in one go (the loads overlap), the pending ones taken
        for (unsigned n = 0; pending; n++) {
            if (n > polls) return false;
            VertWord v[kMaxPatchVerts];
#pragma unroll
            for (int k = 0; k < kMaxPatchVerts; k++) v[k] = ld_vert(bv.sv + l8[k]);
#pragma unroll
            for (int k = 0; k < kMaxPatchVerts; k++) {
                if ((pending & (1u << k)) && (int)(v[k].zf >> 32) >= due[k]) {
                    vset(k, make_float4(__uint_as_float((unsigned)v[k].xy), __uint_as_float((unsigned)(v[k].xy >> 32)),
                                        __uint_as_float((unsigned)v[k].zf), vget(k).w));
                    pending &= ~(1u << k);
                }
            }
        }
    }
    const unsigned long long loc =
        HEX ? kHexLocA : ((unsigned long long)(unsigned)meta.z | ((unsigned long long)(unsigned)meta.w << 32));
    float2 lam0[kMaxPatchTets];
#pragma unroll
    for (int i = 0; i < kMaxPatchTets; i++) lam0[i] = i < ntets ? sl[i] : make_float2(0.f, 0.f);
    bool careful = false;
#pragma unroll
    for (int i = 0; i < kMaxPatchTets; i++) {
        if (!HEX && i >= ntets) break;
        TetState<float> st;
        unpack_static(q0[i], q1[i], q2[i], st);
        int l[4];
        float4 xp[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            l[q] = (int)((loc >> (12 * i + 3 * q)) & 7ull);
            xp[q] = vget(l[q]);
            st.p[q][0] = xp[q].x; st.p[q][1] = xp[q].y; st.p[q][2] = xp[q].z;
            st.w[q] = fabsf(xp[q].w);
        }
        float2 lam = lam0[i];
        float d[4][3];
        bool ok = true;
        if (WHICH == 2) {
            float r0, r1, dl0, dl1, J;
            tet_project_combined_fast(st, lam.x, lam.y, r0, r1, dl0, dl1, d, J);
            careful |= !(fabsf(J) >= kDegenerateJ && isfinite(dl0) && isfinite(dl1));
            lam.x += dl0;
            lam.y += dl1;
        } else {
            float J, r, dl;
            const float lw = WHICH == 0 ? lam.x : lam.y;
            tet_project_single(st, WHICH, lw, r, dl, d, J);
            if (fabsf(J) < kDegenerateJ) {
                const Fp64Out o = project_single_fp64(t, __ldg(slot) + i, xp[0], xp[1], xp[2], xp[3], WHICH, lw);
                dl = o.dl0;
#pragma unroll
                for (int a = 0; a < 4; a++)
#pragma unroll
                    for (int k = 0; k < 3; k++) d[a][k] = o.d[3 * a + k];
                atomicAdd(&flags->degenerate, 1ull);
            }
            ok = isfinite(dl);
            if (!ok) atomicAdd(&flags->nonfinite, 1ull);
            else if (WHICH == 0) lam.x += dl;
            else lam.y += dl;
        }
        if (ok) {
#pragma unroll
            for (int q = 0; q < 4; q++) vset(l[q], moved(xp[q], d[q]));
        }
        sl[i] = lam;
    }
    if (WHICH == 2 && careful) {
#pragma unroll
        for (int k = 0; k < kMaxPatchVerts; k++) {
            if (k >= nverts) continue;
            float4 p;
            bv.look(l8[k], 0, p);
            vset(k, p);
        }
#pragma unroll
        for (int i = 0; i < kMaxPatchTets; i++) {
            if (!HEX && i >= ntets) break;
            TetState<float> st;
            unpack_static(q0[i], q1[i], q2[i], st);
            int l[4];
            float4 xp[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                l[q] = (int)((loc >> (12 * i + 3 * q)) & 7ull);
                xp[q] = vget(l[q]);
                st.p[q][0] = xp[q].x; st.p[q][1] = xp[q].y; st.p[q][2] = xp[q].z;
                st.w[q] = fabsf(xp[q].w);
            }
            float2 lam = lam0[i];
            float d[4][3];
            double rsq;
            if (project_one<false>(st, t, __ldg(slot) + i, xp, lam, d, rsq, flags)) {
#pragma unroll
                for (int q = 0; q < 4; q++) vset(l[q], moved(xp[q], d[q]));
            }
            sl[i] = lam;
        }
    }
#pragma unroll
    for (int k = 0; k < kMaxPatchVerts; k++)
        if (k < nverts) bv.put(l8[k], vget(k), due[k] + 1);
    return true;
}

// One substep (or its sweeps alone). What bounds it is the chain of iters x
// colours phases, each five dependent projections; the versioned sweep adds an
// L2 round trip (a poll after the neighbour's store) to every phase, this
// kernel a shared-memory access and a barrier. Warps 0-3 project (one on each
// scheduler, at most one patch a lane and colour), warp 4 stages the next
// colour's tet records by bulk copies, and every warp takes part in moving the
// positions and multipliers in and out. The colours here are those of
// build_cluster, which halves a colour that has more patches than lanes.
// A phase ends at a barrier of those warps. With several blocks (MULTI) that
// barrier stays inside the block; a vertex that two blocks hold carries a
// version, and its readers poll their own copy until the version is due (the
// versioned sweep's rule: per iteration one version for each patch, and each
// face with active contacts, around the vertex). Warps 5-7 send what a
// colour wrote to the other copy, by distributed-shared-memory stores, while the
// next colour is projected. Each version goes out at most once, by its own
// colour: a vertex that the next colour has already moved on is left to that
// colour (this block was its next writer, so the other block does not wait for
// the version in between), because a second send of one version could land on a
// newer one that the receiver has written since.
// No vertex lies in more than two blocks (ClusterPartition::crowded), and that
// is what orders a copy's versions without a fence: it is written by its own
// block and by one other. The own block writes version n + 1 after it read n
// from the copy itself, or wrote n; the other's sends are ordered among
// themselves by its phase barriers. With a third block, A's store of n into C
// and B's of n + 1 (made after A's store of n into B) would race.
template <bool SEPARATE, bool CONTACTS, bool MULTI>
__global__ void __launch_bounds__(kClusterThreads, 1)
    k_sweep_cluster(ClusterArrays a, ClusterShape s, TetArrays t, ClusterIo io, int iters, bool first_zero,
                    ContactArrays ca, Flags* flags) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) unsigned long long bar[2], tbar;
    __shared__ int4 srg[kMaxClusterColours];             // this block's patches per colour
    __shared__ int sne[kMaxClusterColours];              // its colours that have patches
    __shared__ int ssoff[kMaxClusterColours + 1];        // MULTI: its vertices to send per colour
    __shared__ int soff[kMaxFlowFaceColours + 1];        // its active faces per face colour
    __shared__ unsigned long long s_faces;               // face colours active in this block
    __shared__ int s_stop;                               // a wait for staged records ran out
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, wid = tid >> 5;
    constexpr int cw = kClusterLanes / 32, producer = cw;  // projecting warps, the record stager
    // the vertices come first: at the same place in every block
    VertWord* sv = reinterpret_cast<VertWord*>(smem);
    float4* rec = reinterpret_cast<float4*>(sv + s.max_nv);
    int4* tv = reinterpret_cast<int4*>(rec + (s.resident ? 3 : 6) * (size_t)s.rec_cap);
    int4* tm = tv + s.max_p;
    int4* td = tm + s.max_p;  // MULTI
    unsigned* rem = reinterpret_cast<unsigned*>(td + (MULTI ? s.max_p : 0));  // MULTI
    unsigned long long* smask = reinterpret_cast<unsigned long long*>(rem + (MULTI ? s.max_nb : 0));  // MULTI, CONTACTS
    float* sw = reinterpret_cast<float*>(smask + (MULTI ? s.max_nb : 0));  // MULTI
    uint2* ssend = reinterpret_cast<uint2*>(sw + (MULTI ? s.max_nb : 0));  // MULTI
    float2* slam = reinterpret_cast<float2*>(ssend + (MULTI ? s.max_send : 0));
    float4* scratch = reinterpret_cast<float4*>(slam + s.max_t);
    const int4 pa = __ldg(a.part + 2 * blockIdx.x), pb = __ldg(a.part + 2 * blockIdx.x + 1);
    const int v0 = pa.x, nv = pa.y, nb = pa.z, p0 = pa.w, np = pb.x, b0 = pb.y, ntets = pb.z, t0 = pb.w;
    // the block's tables and records: static, so they load before the wait on the previous kernel
    for (int c = tid; c < s.ncol; c += nt) srg[c] = __ldg(a.range + (size_t)blockIdx.x * s.ncol + c);
    if (MULTI)
        for (int c = tid; c <= s.ncol; c += nt) ssoff[c] = __ldg(a.send_off + (size_t)blockIdx.x * (s.ncol + 1) + c);
    if (tid == 0) {
        s_stop = 0;
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        mbar_init(&tbar, 1);
        const unsigned bytes = 16u * (unsigned)((MULTI ? 3 : 2) * np);
        mbar_arrive_expect_tx(&tbar, bytes);
        if (np) {
            tma_load_1d(tv, a.vidx + p0, 16u * (unsigned)np, &tbar);
            tma_load_1d(tm, a.meta + p0, 16u * (unsigned)np, &tbar);
            if (MULTI) tma_load_1d(td, a.ver + p0, 16u * (unsigned)np, &tbar);
        }
    }
    __syncthreads();
    if (MULTI) {
        for (int i = tid; i < nb; i += nt) rem[i] = __ldg(a.remote + b0 + i);
        for (int i = tid; i < ssoff[s.ncol] - ssoff[0]; i += nt) ssend[i] = __ldg(a.send + ssoff[0] + i);
    }
    int nne = 0;  // colours with patches here, in order
    for (int c = 0; c < s.ncol; c++) {
        if (srg[c].y > 0) {
            if (tid == 0) sne[nne] = c;
            nne++;
        }
    }
    auto copy_records = [&](int c, float4* dst, unsigned long long* b) {  // one thread
        const int4 rg = srg[c];
        const unsigned bytes = 16u * (unsigned)rg.z;
        const size_t at = (size_t)t0 + rg.w;
        mbar_arrive_expect_tx(b, 3u * bytes);
        tma_load_1d(dst, a.rec + at, bytes, b);
        tma_load_1d(dst + s.rec_cap, a.rec + a.nrec + at, bytes, b);
        tma_load_1d(dst + 2 * s.rec_cap, a.rec + 2 * a.nrec + at, bytes, b);
    };
    __syncthreads();
    if (wid == producer && lane == 0 && nne > 0) {
        if (s.resident) {  // the block's records whole
            const unsigned bytes = 16u * (unsigned)ntets;
            mbar_arrive_expect_tx(&bar[0], 3u * bytes);
            for (int k = 0; k < 3; k++) tma_load_1d(rec + k * s.rec_cap, a.rec + k * a.nrec + t0, bytes, &bar[0]);
        } else {
            copy_records(sne[0], rec, &bar[0]);
        }
    }
    pdl_wait_then_release();
    // positions (predicted here when io.predict), four to a thread in flight
    for (int i0 = tid; i0 < nv; i0 += 4 * nt) {
        int e[4];
        float4 p[4], v[4];
#pragma unroll
        for (int u = 0; u < 4; u++) e[u] = i0 + u * nt < nv ? __ldg(a.verts + v0 + i0 + u * nt) : 0;
#pragma unroll
        for (int u = 0; u < 4; u++) {
            if (i0 + u * nt >= nv) continue;
            const int g = e[u] & 0x7fffffff;
            if (io.xv) {
                const VerRec r = io.xv[io.vperm[g]];
                p[u] = make_float4(__uint_as_float((unsigned)r.x), __uint_as_float((unsigned)r.y),
                                   __uint_as_float((unsigned)r.z), __uint_as_float((unsigned)r.w));
            } else {
                p[u] = io.x[g];
            }
            if (io.predict && !io.gdz) v[u] = io.vel[g];
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
            if (i0 + u * nt >= nv) continue;
            const int g = e[u] & 0x7fffffff;
            float4 q = p[u];
            if (io.predict) {
                if (e[u] < 0) io.prev[g] = q;
                if (io.gdz) q = make_float4(q.x, q.y, q.z + __ldg(io.gdz + g), q.w);
                else q = make_float4(q.x + io.dt * v[u].x, q.y + io.dt * v[u].y, (q.z + io.dt * v[u].z) + io.dz, q.w);
            }
            const int l = i0 + u * nt;
            const bool sh = MULTI && l < nb;  // version 0
            sv[l] = VertWord{pack2(q.x, __float_as_uint(q.y)), pack2(q.z, sh ? 0u : __float_as_uint(q.w))};
            if (sh) sw[l] = q.w;
        }
    }
    // without its tables a thread neither projects nor touches the multipliers
    const bool tables = mbar_wait_bounded(&tbar, 0, kWaitLimit);
    bool ok = tables;
    if (first_zero) {
        for (int i = tid; i < ntets; i += nt) slam[i] = make_float2(0.f, 0.f);
    } else if (tables) {
        for (int i = tid; i < np; i += nt) {
            const int4 m = tm[i];
            const int slot = __ldg(a.slot + p0 + i);
            for (int k = 0; k < (m.y & 0xff); k++) slam[m.x + k] = t.lam[slot + k];
        }
    }
    if (CONTACTS) {
        // the active faces of this block, and (MULTI) for each shared vertex
        // the colours of the active faces around it in the cluster, which add
        // to its versions
        const int nf = s.nfcol;
        if (tid == 0) s_faces = 0ull;
        for (int c = tid; c <= nf; c += nt) soff[c] = a.act_off[(size_t)blockIdx.x * (nf + 1) + c];
        if (MULTI)
            for (int i = tid; i < nb; i += nt) smask[i] = 0ull;
        __syncthreads();
        for (int c = tid; c < nf; c += nt)
            if (soff[c + 1] > soff[c]) atomicOr(&s_faces, 1ull << c);
        if (MULTI) {
            cluster_sync_all();  // the masks are zero in every block
            for (int c = 0; c < nf; c++)
                for (int j = soff[c] + tid; j < soff[c + 1]; j += nt) {
                    const int4 fl = __ldg(a.faces + a.act_faces[j]);
                    const int l[3] = {fl.x, fl.y, fl.z};
                    for (int q = 0; q < 3; q++) {
                        if (l[q] >= nb) continue;
                        const unsigned at = smem_u32(smask) + 4u * (unsigned)(c >> 5), bit = 1u << (c & 31);
                        red_or_cluster(mapa(at + 8u * (unsigned)l[q], blockIdx.x % s.csize), bit);
                        const unsigned m = rem[l[q]];
                        red_or_cluster(mapa(at + 8u * (m & 0xfffu), m >> 12), bit);
                    }
                }
        }
    }
    if (MULTI) cluster_sync_all();
    else __syncthreads();
    if (s.resident && nne > 0) ok = mbar_wait_bounded(&bar[0], 0, kWaitLimit) && ok;
    const int passes = SEPARATE ? 2 : 1;
    const int total = iters * passes * nne;  // this block's colours with records to stage
    // A wait that gave up: the warp skips the work from then on (a neighbour's
    // waits then give up in turn) but still meets its block at the barriers.
    ok = __all_sync(0xffffffffu, ok) != 0;
    auto phase_end = [&]() {
        asm volatile("bar.sync 1, %0;" ::"r"(MULTI ? kClusterThreads : 32 * (cw + 1)) : "memory");
    };
    const BlockVerts<MULTI> bv{sv, sw, rem, nb};
    int staged = nne > 0 ? 1 : 0;  // copies issued (the producer's first lane counts them)
    if (MULTI || wid <= producer) {
        int seq = 0;
        for (int it = 0; it < iters; it++) {
            for (int pc = 0; pc < passes * s.ncol; pc++) {
                const int pass = SEPARATE && pc >= s.ncol ? 1 : 0, c = pc - pass * s.ncol;
                const int4 rg = srg[c];
                const int n = rg.y;
                if (wid == producer) {
                    // The next colour's records into the other buffer, whose readers passed the last
                    // barrier, and before it waited for the copy that this one follows; after a wait
                    // that ran out nothing is staged any more.
                    if (!s.resident && n > 0) {
                        if (lane == 0 && seq + 1 < total && !*(volatile int*)&s_stop) {
                            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                            copy_records(sne[(seq + 1) % nne], rec + ((seq + 1) & 1) * 3 * (size_t)s.rec_cap,
                                         &bar[(seq + 1) & 1]);
                            staged = seq + 2;
                        }
                        seq++;
                    }
                } else if (wid < cw && n > 0) {
                    // equal consecutive shares of the colour for the warps
                    const int per = (n + cw - 1) / cw, q = wid * per + lane;
                    const bool on = lane < per && q < n;
                    int4 vi = make_int4(0, 0, 0, 0), meta = vi;
                    if (on) {
                        vi = tv[rg.x + q];
                        meta = tm[rg.x + q];
                    }
                    const float4* buf = rec;
                    int rsub = 0;
                    if (!s.resident) {
                        // a warp that skips its work still waits for the copy: the buffer is written again
                        const bool landed =
                            __all_sync(0xffffffffu, mbar_wait_bounded(&bar[seq & 1], (seq >> 1) & 1, kWaitLimit)) != 0;
                        if (!landed) s_stop = 1;
                        ok = ok && landed;
                        buf = rec + (seq & 1) * 3 * (size_t)s.rec_cap;
                        rsub = rg.w;
                        seq++;
                    }
                    const unsigned long long loc =
                        (unsigned long long)(unsigned)meta.z | ((unsigned long long)(unsigned)meta.w << 32);
                    const bool hex =
                        __all_sync(0xffffffffu, !on || (meta.y == (5 | (8 << 8)) && loc == kHexLocA)) != 0;
                    int due[kMaxPatchVerts] = {};
                    if (MULTI && on) {
                        const int4 dv = td[rg.x + q];
                        const int dw[4] = {dv.x, dv.y, dv.z, dv.w};
                        const int vw[4] = {vi.x, vi.y, vi.z, vi.w};
#pragma unroll
                        for (int k = 0; k < kMaxPatchVerts; k++) {
                            const int h = (dw[k >> 1] >> (16 * (k & 1))) & 0xffff;  // deg << 8 | pre
                            int per_it = passes * (h >> 8);
                            const int l = (vw[k >> 1] >> (16 * (k & 1))) & 0xffff;
                            if (CONTACTS && l < nb) per_it += __popcll(smask[l]);
                            due[k] = it * per_it + pass * (h >> 8) + (h & 0xff);
                        }
                    }
                    if (on && ok) {
                        const float4* b0r = buf + (meta.x - rsub);
                        const int* slot = a.slot + p0 + rg.x + q;
#define XG_PATCH(W, H) ok = cluster_patch<W, H, MULTI>(t, bv, vi, due, meta, slot, b0r, b0r + s.rec_cap, b0r + 2 * s.rec_cap, \
                                                  slam + meta.x, scratch + tid, 32 * cw, s.polls, flags)
                        if (SEPARATE) {
                            if (pass == 0) { if (hex) XG_PATCH(0, true); else XG_PATCH(0, false); }
                            else { if (hex) XG_PATCH(1, true); else XG_PATCH(1, false); }
                        } else {
                            if (hex) XG_PATCH(2, true); else XG_PATCH(2, false);
                        }
#undef XG_PATCH
                    }
                    if (MULTI) ok = __all_sync(0xffffffffu, ok) != 0;
                }
                phase_end();
                if (MULTI && wid > producer)
                    for (int i = ssoff[c] - ssoff[0] + tid - 32 * (producer + 1); i < ssoff[c + 1] - ssoff[0];
                         i += kClusterThreads - 32 * (producer + 1)) {
                        const uint2 m = ssend[i];  // (local index << 16 | rank << 12 | index there, deg << 8 | pre)
                        const int l = (int)(m.x >> 16), deg = (int)(m.y >> 8);
                        int per_it = passes * deg;
                        if (CONTACTS) per_it += __popcll(smask[l]);
                        const VertWord v = ld_vert(sv + l);
                        if ((int)(v.zf >> 32) == it * per_it + pass * deg + (int)(m.y & 0xffu) + 1)
                            st_vert_cluster(mapa(smem_u32(sv) + 16u * (m.x & 0xfffu), (m.x >> 12) & 15u), v);
                    }
            }
            if (CONTACTS) {
                // static contacts: face colours in order, a face's contacts in slot
                // order. A contact's thread sends its vertices itself, so the last
                // colour's sends are done first.
                if (MULTI && s_faces) phase_end();
                for (unsigned long long m = s_faces; m; m &= m - 1) {
                    const int c = __ffsll((long long)m) - 1;
                    if (wid < cw) {
                        for (int j = soff[c] + tid; ok && j < soff[c + 1]; j += 32 * cw) {
                            const int f = a.act_faces[j];
                            const int4 fl = __ldg(a.faces + f);
                            const int l[3] = {fl.x, fl.y, fl.z};
                            const int dw[3] = {fl.w & 0xff, (fl.w >> 8) & 0xff, (fl.w >> 16) & 0xff};  // patches
                            float4 xs[3];
                            int due[3] = {};
                            unsigned pending = 0;
#pragma unroll
                            for (int q = 0; q < 3; q++) {
                                if (bv.shared(l[q])) {
                                    const unsigned long long m2 = smask[l[q]];
                                    due[q] = it * (passes * dw[q] + __popcll(m2)) + passes * dw[q] +
                                             __popcll(m2 & ((1ull << c) - 1));
                                }
                                if (!bv.look(l[q], due[q], xs[q])) pending |= 1u << q;
                            }
                            if (MULTI) {
                                for (unsigned n = 0; pending && ok; n++) {
                                    if (n > s.polls) ok = false;
#pragma unroll
                                    for (int q = 0; q < 3; q++) {
                                        float4 p;
                                        if ((pending & (1u << q)) && bv.look(l[q], due[q], p)) {
                                            xs[q] = p;
                                            pending &= ~(1u << q);
                                        }
                                    }
                                }
                                if (!ok) break;
                            }
                            for (int k = 0; k < ca.S; k++) {
                                const int slot = k * ca.F + f;
                                if (ca.bary[slot].w != 1.f) continue;  // empty, or against a free rigid body
                                float lam = it == 0 ? 0.f : ca.lam[slot];
                                float d[3][3];
                                if (contact_update(ca, slot, xs, d, lam)) {
#pragma unroll
                                    for (int q = 0; q < 3; q++) xs[q] = moved(xs[q], d[q]);
                                }
                                ca.lam[slot] = lam;
                            }
                            // moved or not, the next version
#pragma unroll
                            for (int q = 0; q < 3; q++) {
                                bv.put(l[q], xs[q], due[q] + 1);
                                bv.send(l[q]);
                            }
                        }
                        if (MULTI) ok = __all_sync(0xffffffffu, ok) != 0;
                    }
                    phase_end();
                }
            }
        }
    }
    // a copy or a neighbour's vertex that never came: counted; the work after it
    // was skipped, and the copies get a last bounded chance: no block leaves with
    // one into it in flight
    if (!__syncthreads_and(ok)) {
        if (tid == 0) {
            atomicAdd(&flags->timeouts, 1ull);
            mbar_wait_bounded(&tbar, 0, kWaitLimit);
        }
        if (wid == producer && lane == 0)
            for (int k = staged > 1 ? staged - 2 : 0; k < staged; k++)  // the last in each buffer
                mbar_wait_bounded(&bar[k & 1], (k >> 1) & 1, kWaitLimit);
    }
    if (MULTI) cluster_sync_all();  // the other blocks' last stores are here
    // owners write the vertices back; every block its multipliers
    for (int i0 = tid; i0 < nv; i0 += 4 * nt) {
        int e[4];
        float4 p[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            e[u] = i0 + u * nt < nv ? __ldg(a.verts + v0 + i0 + u * nt) : 0;
            if (e[u] < 0 && io.finalize) p[u] = io.x[e[u] & 0x7fffffff];  // the position before the substep
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
            if (e[u] >= 0) continue;
            const int g = e[u] & 0x7fffffff;
            const int l = i0 + u * nt;
            float4 xx;
            bv.look(l, 0, xx);
            if (io.xv) {
                io.xv[io.vperm[g]] = VerRec{__float_as_uint(xx.x), __float_as_uint(xx.y), __float_as_uint(xx.z),
                                            __float_as_uint(xx.w)};
                continue;
            }
            if (io.finalize) {
                if (p[u].w < 0.f) xx = p[u];
                if (io.write_vel)
                    io.vel[g] = make_float4((xx.x - p[u].x) / io.dt, (xx.y - p[u].y) / io.dt, (xx.z - p[u].z) / io.dt,
                                            0.f);
            }
            io.x[g] = xx;
        }
    }
    for (int i = tid; tables && i < np; i += nt) {
        const int4 m = tm[i];
        const int slot = __ldg(a.slot + p0 + i);
        for (int k = 0; k < (m.y & 0xff); k++) t.lam[slot + k] = slam[m.x + k];
    }
}

template <typename K>
cudaError_t prepare(K* k, const ClusterShape& s) {
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kClusterSmemMax);
    if (e == cudaSuccess && s.csize > 8) e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return e;
}

void cluster_config(const Launch& L, const ClusterShape& s, cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr) {
    cfg.gridDim = dim3((unsigned)s.ncta);
    cfg.blockDim = dim3((unsigned)s.threads);
    cfg.dynamicSmemBytes = s.smem;
    cfg.stream = L.s;
    int n = 0;
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = L.pdl ? 1 : 0;
    if (s.csize > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = (unsigned)s.csize;
        attr[n].val.clusterDim.y = 1;
        attr[n++].val.clusterDim.z = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = (unsigned)n;
}

}  // namespace

#define XG_CLUSTER_EACH(DO)                                                               \
    do {                                                                                  \
        const bool _m = s.csize > 1;                                                      \
        if (separate) {                                                                   \
            if (contacts) { if (_m) DO((k_sweep_cluster<true, true, true>)); else DO((k_sweep_cluster<true, true, false>)); } \
            else { if (_m) DO((k_sweep_cluster<true, false, true>)); else DO((k_sweep_cluster<true, false, false>)); }        \
        } else {                                                                          \
            if (contacts) { if (_m) DO((k_sweep_cluster<false, true, true>)); else DO((k_sweep_cluster<false, true, false>)); } \
            else { if (_m) DO((k_sweep_cluster<false, false, true>)); else DO((k_sweep_cluster<false, false, false>)); }        \
        }                                                                                 \
    } while (0)

// Prepares the kernel for this shape; returns how many clusters of it the
// device holds at once (0: it cannot run). The blocks of a cluster share a GPC:
// a GB300 holds 8 clusters of eleven blocks, not 13.
int sweep_cluster_fits(const ClusterShape& s, bool separate, bool contacts) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    cluster_config(Launch{nullptr, false}, s, cfg, attr);
    cudaError_t e = cudaSuccess;
    int n = 0;
#define XG_DO(K)                                                                       \
    do {                                                                               \
        e = prepare(K, s);                                                             \
        if (e == cudaSuccess) {                                                        \
            if (s.csize > 1) e = cudaOccupancyMaxActiveClusters(&n, K, &cfg);          \
            else e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, K, s.threads, s.smem); \
        }                                                                              \
    } while (0)
    XG_CLUSTER_EACH(XG_DO);
#undef XG_DO
    int dev = 0, sms = 1;
    if (e == cudaSuccess && s.csize == 1) {
        e = cudaGetDevice(&dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    }
    if (e != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n * sms;
}

cudaError_t launch_sweep_cluster(const Launch& L, const ClusterArrays& a, const ClusterShape& s, const TetArrays& t,
                                 const ClusterIo& io, int iters, bool first_zero, bool separate, bool contacts,
                                 const ContactArrays& ca, Flags* flags) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    cluster_config(L, s, cfg, attr);
    cudaError_t e = cudaSuccess;
#define XG_DO(K) e = cudaLaunchKernelEx(&cfg, K, a, s, t, io, iters, first_zero, ca, flags)
    XG_CLUSTER_EACH(XG_DO);
#undef XG_DO
    return e;
}

}  // namespace xg
