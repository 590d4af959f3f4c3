// Position transfers between the caller's host arrays and the device: the
// conversion kernels read and write the host array directly when the GPU
// addresses pageable host memory.
#include "xpbd_device.cuh"

namespace xg {

namespace {

// ---- host arrays the device addresses directly (coherent pageable memory
// on a Grace-Blackwell system): 3 values per vertex, converted here ----
// A block moves its 256 vertices' 3 x 256 values through shared memory, so the
// host side is read and written in whole 16-byte pieces covering full cache
// lines (when the block's run of the array is 16-byte aligned).
constexpr int kHostIoThreads = 256;

template <typename H>
__global__ void __launch_bounds__(kHostIoThreads) k_xyz_from_host(float4* __restrict__ x, const H* __restrict__ h,
                                                                  int V, bool keep_w) {
    __shared__ __align__(16) H buf[3 * kHostIoThreads];
    const int tid = threadIdx.x, v0 = blockIdx.x * kHostIoThreads;
    const int n = min(kHostIoThreads, V - v0), nv = 3 * n;
    const H* src = h + 3 * (size_t)v0;
    constexpr int kPer16 = 16 / (int)sizeof(H);
    if (((uintptr_t)src & 15) == 0) {
        for (int i = tid; i < nv / kPer16; i += kHostIoThreads)
            reinterpret_cast<uint4*>(buf)[i] = __ldcv(reinterpret_cast<const uint4*>(src) + i);
        for (int i = nv / kPer16 * kPer16 + tid; i < nv; i += kHostIoThreads) buf[i] = src[i];
    } else {
        for (int i = tid; i < nv; i += kHostIoThreads) buf[i] = src[i];
    }
    __syncthreads();
    if (tid < n) {
        const int i = v0 + tid;
        const float w = keep_w ? x[i].w : 0.f;  // inverse mass and fixed sign stay
        x[i] = make_float4((float)buf[3 * tid], (float)buf[3 * tid + 1], (float)buf[3 * tid + 2], w);
    }
}

template <typename H>
__global__ void __launch_bounds__(kHostIoThreads) k_xyz_to_host(H* __restrict__ h, const float4* __restrict__ x,
                                                                int V) {
    __shared__ __align__(16) H buf[3 * kHostIoThreads];
    const int tid = threadIdx.x, v0 = blockIdx.x * kHostIoThreads;
    const int n = min(kHostIoThreads, V - v0), nv = 3 * n;
    if (tid < n) {
        const float4 p = x[v0 + tid];
        buf[3 * tid] = (H)p.x;
        buf[3 * tid + 1] = (H)p.y;
        buf[3 * tid + 2] = (H)p.z;
    }
    __syncthreads();
    H* dst = h + 3 * (size_t)v0;
    constexpr int kPer16 = 16 / (int)sizeof(H);
    if (((uintptr_t)dst & 15) == 0) {
        for (int i = tid; i < nv / kPer16; i += kHostIoThreads)
            reinterpret_cast<uint4*>(dst)[i] = reinterpret_cast<const uint4*>(buf)[i];
        for (int i = nv / kPer16 * kPer16 + tid; i < nv; i += kHostIoThreads) dst[i] = buf[i];
    } else {
        for (int i = tid; i < nv; i += kHostIoThreads) dst[i] = buf[i];
    }
}

// The network's rows (16 floats) as BF16 and their targets (2 floats), read from
// host arrays the device addresses: eight values a thread, in 16-byte pieces
// where the arrays are aligned to them. (Rounding on one host core, a fresh
// device buffer and a pageable copy took 0.5 of the 0.64 ms of a loss and
// gradient call on 65,536 rows.)
__global__ void __launch_bounds__(256) k_rows_from_host(__nv_bfloat16* __restrict__ X, const float* __restrict__ hX,
                                                        float* __restrict__ Y, const float* __restrict__ hY,
                                                        long long n) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < 2 * n) {
        float v[8];
        const float* p = hX + 8 * i;
        if (((uintptr_t)hX & 15) == 0) {
            const float4 a = __ldcv(reinterpret_cast<const float4*>(p)), b = __ldcv(reinterpret_cast<const float4*>(p) + 1);
            v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
            v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
        } else {
            for (int k = 0; k < 8; k++) v[k] = __ldcv(p + k);
        }
        __nv_bfloat162 h[4];
#pragma unroll
        for (int k = 0; k < 4; k++) h[k] = __floats2bfloat162_rn(v[2 * k], v[2 * k + 1]);
        reinterpret_cast<uint4*>(X)[i] = *reinterpret_cast<const uint4*>(h);
        if (Y && i < n) {
            Y[2 * i] = __ldcv(hY + 2 * i);
            Y[2 * i + 1] = __ldcv(hY + 2 * i + 1);
        }
    }
}

}  // namespace

void launch_rows_from_host(cudaStream_t s, __nv_bfloat16* X, const float* hX, float* Y, const float* hY, long long n) {
    if (n > 0) k_rows_from_host<<<nblk(2 * n, 256), 256, 0, s>>>(X, hX, Y, hY, n);
}

void launch_xyz_from_host(cudaStream_t s, float4* x, const double* h, int V, bool keep_w) {
    if (V > 0) k_xyz_from_host<double><<<nblk(V, kHostIoThreads), kHostIoThreads, 0, s>>>(x, h, V, keep_w);
}
void launch_xyz_from_host(cudaStream_t s, float4* x, const float* h, int V, bool keep_w) {
    if (V > 0) k_xyz_from_host<float><<<nblk(V, kHostIoThreads), kHostIoThreads, 0, s>>>(x, h, V, keep_w);
}
void launch_xyz_to_host(cudaStream_t s, double* h, const float4* x, int V) {
    if (V > 0) k_xyz_to_host<double><<<nblk(V, kHostIoThreads), kHostIoThreads, 0, s>>>(h, x, V);
}
void launch_xyz_to_host(cudaStream_t s, float* h, const float4* x, int V) {
    if (V > 0) k_xyz_to_host<float><<<nblk(V, kHostIoThreads), kHostIoThreads, 0, s>>>(h, x, V);
}

}  // namespace xg
