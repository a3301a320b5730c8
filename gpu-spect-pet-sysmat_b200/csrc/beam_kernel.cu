// Beam masks and multiplexing (MPXI) of a photoelectric sysmat, on the device.
//
// The reference computes these after the fact on the CPU, from a memory-mapped
// .sysmat file (PEGen_RayTracing_CircularHole/extract_beam_prop_masks.py:52-87,
// compute_mpxi_3d.py:45-52): per (rotation, crystal) row the beam mask is
// "entry > 0.05 * row max" (threshold 1.0 for an all-zero row), with the row's
// sum and mask size as beam properties; per rotation, MPXI(voxel) counts the
// rows whose mask holds the voxel.  Here the same quantities come from the
// sysmat where it already lives, in HBM:
//
//  beam_fused_kernel  rows of up to kFusedVoxels voxels: the row lives in shared
//                     memory between the passes.  Each thread copies its own voxels
//                     (cp.async, one or two rows ahead), reduces max (exact) and sum
//                     (double), and after the block's one barrier per row writes the
//                     mask and adds to its own voxels' counts (16 bits, shared memory);
//                     the counts leave in one integer atomicAdd per voxel at the end,
//                     exact and independent of order.  HBM-bound: 4 bytes read and 1
//                     written per entry, nothing twice.  6400 x 16384 with mask and
//                     MPXI through beam_held_kernel (its comment): 99 to 108
//                     us from one GPU to another, 4.9 to 5.3 TB/s; two passes over global
//                     memory took 171 us.
//  beam_rows_kernel   longer rows.  One CTA per row (grid-stride): pass A reduces max
//                     and sum with 128-bit loads; pass B re-reads the row (from L2) and
//                     writes the int8 mask with 32-bit stores and counts it.
//  beam_mpxi_kernel   longer rows.  4 voxels per thread, rows split over gridDim.y;
//                     counts in registers, read from the mask when it was written (1
//                     byte per entry) or else from the sysmat and the row thresholds;
//                     one integer atomicAdd per (thread, voxel) at the end.
//
// The threshold is the product frac * max rounded to single precision, as numpy forms it
// for a float32 row and a Python float.
#include <algorithm>
#include <cstdint>
#include <type_traits>

#include <cuda_runtime.h>

#include "common.h"

namespace smb {
namespace {

constexpr int kBeamThreads = 256;
constexpr int kBeamWarps = kBeamThreads / 32;

struct RowReduce {
    float mx[kBeamWarps];
    double sum[kBeamWarps];
    int cnt[kBeamWarps];
    float thr;
};

__device__ __forceinline__ float row_threshold(float mx, float frac) {
    return mx > 0.0f ? __fmul_rn(frac, mx) : 1.0f;
}

// Longest row beam_fused_kernel takes: two copies of it and the counts in 227 KB, of which
// the block's own variables take 1 KB.
constexpr int kFusedVoxels = 23000;
constexpr int kFusedBytes = 226 * 1024;
static_assert(sizeof(float) * kFusedVoxels * 5 / 2 <= kFusedBytes, "two copies and the counts fit");

__device__ __forceinline__ void copy_async(float* dst, const float* src, bool wide) {
    const unsigned to = (unsigned)__cvta_generic_to_shared(dst);
    if (wide) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(to), "l"(src) : "memory");
}

// VEC: rows, masks and their pitches allow 16-byte loads and 4-byte mask stores.
template <bool VEC, int STAGES>
__global__ void __launch_bounds__(1024) beam_fused_kernel(const float* __restrict__ A, long long rows, int V, long long ld,
                                                         float frac, float* __restrict__ row_max,
                                                         double* __restrict__ row_sum, int* __restrict__ row_count,
                                                         signed char* __restrict__ mask, long long ldm,
                                                         unsigned* __restrict__ mpxi) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ float s_max[2][32];
    __shared__ double s_sum[2][32];
    __shared__ int s_cnt[2][32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, T = blockDim.x, warps = T >> 5;
    const int Vp = (V + 3) & ~3, n4 = VEC ? V >> 2 : 0;   // voxels [4 n4, V) go one by one
    float* buf = reinterpret_cast<float*>(smem_raw);
    unsigned short* cnt = reinterpret_cast<unsigned short*>(buf + (size_t)STAGES * Vp);
    if (mpxi) {   // every thread clears, counts and adds up its own voxels
        for (int i = tid; i < n4; i += T) reinterpret_cast<ushort4*>(cnt)[i] = make_ushort4(0, 0, 0, 0);
        for (int i = 4 * n4 + tid; i < V; i += T) cnt[i] = 0;
    }
    // rows of this block: blockIdx.x, + gridDim.x, ...; every thread copies the voxels it later reads
    auto fetch = [&](long long r, int stage) {
        if (r < rows) {
            const float* src = A + r * ld;
            float* dst = buf + (size_t)stage * Vp;
#pragma unroll 4
            for (int i = tid; i < n4; i += T) copy_async(dst + 4 * i, src + 4 * i, true);
#pragma unroll 4
            for (int i = 4 * n4 + tid; i < V; i += T) copy_async(dst + i, src + i, false);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int s = 0; s < STAGES - 1; ++s) fetch(blockIdx.x + (long long)s * gridDim.x, s);
    long long prev = -1;
    int par = 0, stage = 0;
    for (long long r = blockIdx.x; r < rows; r += gridDim.x, par ^= 1) {
        fetch(r + (long long)(STAGES - 1) * gridDim.x, stage == 0 ? STAGES - 1 : stage - 1);
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 1) : "memory");
        const float* row = buf + (size_t)stage * Vp;
        // ---- max and sum
        float mx = -INFINITY;
        double s = 0.0;
#pragma unroll 4
        for (int i = tid; i < n4; i += T) {
            const float4 v = reinterpret_cast<const float4*>(row)[i];
            mx = fmaxf(fmaxf(mx, fmaxf(v.x, v.y)), fmaxf(v.z, v.w));
            s += ((double)v.x + (double)v.y) + ((double)v.z + (double)v.w);
        }
#pragma unroll 4
        for (int i = 4 * n4 + tid; i < V; i += T) {
            const float v = row[i];
            mx = fmaxf(mx, v);
            s += (double)v;
        }
        for (int o = 16; o > 0; o >>= 1) {
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            s += __shfl_xor_sync(0xffffffffu, s, o);
        }
        if (lane == 0) {
            s_max[par][warp] = mx;
            s_sum[par][warp] = s;
        }
        __syncthreads();
        mx = lane < warps ? s_max[par][lane] : -INFINITY;
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        const float thr = row_threshold(mx, frac);
        if (warp == 0) {
            // this row's sum and, its barrier being past, the previous row's count
            double t = lane < warps ? s_sum[par][lane] : 0.0;
            int c = prev >= 0 && lane < warps ? s_cnt[par ^ 1][lane] : 0;
            for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            c = __reduce_add_sync(0xffffffffu, c);
            if (lane == 0) {
                row_max[r] = mx;
                row_sum[r] = t;
                if (prev >= 0) row_count[prev] = c;
            }
        }
        // ---- mask, its size, counts per voxel.  A thread's voxels are its own, so it tests its
        // own bits: most see no beam and skip the counts.  Two loops, as the test costs 5000 x
        // 20000 without MPXI 4 %.
        int c = 0;
        signed char* mrow = mask ? mask + r * ldm : nullptr;
        auto take = [&](auto counting) {
#pragma unroll 4
            for (int i = tid; i < n4; i += T) {
                const float4 v = reinterpret_cast<const float4*>(row)[i];
                const int b0 = v.x > thr, b1 = v.y > thr, b2 = v.z > thr, b3 = v.w > thr, n = b0 + b1 + b2 + b3;
                c += n;
                if (mrow) __stcs(reinterpret_cast<int*>(mrow) + i, b0 | b1 << 8 | b2 << 16 | b3 << 24);
                if (counting.value && n) {
                    ushort4 u = reinterpret_cast<ushort4*>(cnt)[i];
                    u.x += b0; u.y += b1; u.z += b2; u.w += b3;
                    reinterpret_cast<ushort4*>(cnt)[i] = u;
                }
            }
#pragma unroll 4
            for (int i = 4 * n4 + tid; i < V; i += T) {
                const int b = row[i] > thr;
                c += b;
                if (mrow) mrow[i] = (signed char)b;
                if (counting.value && b) cnt[i] += b;
            }
        };
        if (mpxi) take(std::true_type{});
        else take(std::false_type{});
        c = __reduce_add_sync(0xffffffffu, c);
        if (lane == 0) s_cnt[par][warp] = c;
        prev = r;
        stage = stage + 1 == STAGES ? 0 : stage + 1;
    }
    __syncthreads();
    if (warp == 0) {
        const int c = __reduce_add_sync(0xffffffffu, lane < warps ? s_cnt[par ^ 1][lane] : 0);
        if (lane == 0) row_count[prev] = c;
    }
    if (mpxi) {
        for (int i = tid; i < n4; i += T) {
            const ushort4 u = reinterpret_cast<const ushort4*>(cnt)[i];
            const unsigned n[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (n[k]) atomicAdd(mpxi + 4 * i + k, n[k]);
        }
        for (int i = 4 * n4 + tid; i < V; i += T)
            if (cnt[i]) atomicAdd(mpxi + i, (unsigned)cnt[i]);
    }
}

// Rows of 8192 to kHeldVoxels voxels, aligned: a thread holds its 32 voxels in registers
// from the reduction to the mask, and as soon as it has taken them from shared memory it
// starts copying the same voxels of the next row there.  One copy of the row is enough, so
// two blocks share an SM and one reduces while the other writes: 6400 x 16384 with mask
// and MPXI in 99 us, against 127 us for beam_fused_kernel (one block per SM, bound by
// the chain of its reductions) and 171 us for the two passes over global memory.
constexpr int kHeldThreads = 512, kHeld = 8;   // float4 per thread
constexpr int kHeldVoxels = kHeldThreads * 4 * kHeld;
constexpr int kHeldBytes = sizeof(float) * kHeldVoxels + 16;

__global__ void __launch_bounds__(kHeldThreads, 2) beam_held_kernel(const float* __restrict__ A, long long rows, int V, long long ld,
                                                          float frac, float* __restrict__ row_max,
                                                          double* __restrict__ row_sum, int* __restrict__ row_count,
                                                          signed char* __restrict__ mask, long long ldm,
                                                          unsigned* __restrict__ mpxi) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ float s_max[2][32];
    __shared__ double s_sum[2][32];
    __shared__ int s_cnt[2][32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int T = kHeldThreads, warps = T / 32;
    const int n4 = V >> 2, tail = V & 3;                    // thread t < tail also takes voxel 4 n4 + t
    float4* buf = reinterpret_cast<float4*>(smem_raw);
    float* buf_tail = reinterpret_cast<float*>(buf + n4);
    // counts of this thread's voxels: four bytes per word, the mask word added row by row
    // and moved out before a byte can overflow
    unsigned cnt[kHeld], cnt_tail = 0u;
#pragma unroll
    for (int j = 0; j < kHeld; ++j) cnt[j] = 0u;
    auto flush = [&] {
#pragma unroll
        for (int j = 0; j < kHeld; ++j) {
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (const unsigned n = cnt[j] >> (8 * e) & 255u) atomicAdd(mpxi + 4 * (tid + j * T) + e, n);
            cnt[j] = 0u;
        }
        if (cnt_tail) atomicAdd(mpxi + 4 * n4 + tid, cnt_tail);
        cnt_tail = 0u;
    };
    int held_rows = 0;
    auto fetch = [&](long long r) {                         // this thread's voxels of row r
        const float* src = A + r * ld + 4 * tid;
        float* dst = reinterpret_cast<float*>(buf + tid);
#pragma unroll
        for (int j = 0; j < kHeld; ++j)
            if (tid + j * T < n4) copy_async(dst + 4 * j * T, src + 4 * j * T, true);
        if (tid < tail) copy_async(buf_tail + tid, A + r * ld + 4 * n4 + tid, false);
    };
    fetch(blockIdx.x);
    long long prev = -1;
    int par = 0;
    for (long long r = blockIdx.x; r < rows; r += gridDim.x, par ^= 1) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        // ---- take the row; max and sum
        float4 v[kHeld];
        float last = -INFINITY, mx = -INFINITY;
        double s = 0.0;
#pragma unroll
        for (int j = 0; j < kHeld; ++j) {
            const int i = tid + j * T;
            v[j] = make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);   // never in the mask, nor the maximum
            if (i < n4) {
                v[j] = buf[i];
                s += ((double)v[j].x + (double)v[j].y) + ((double)v[j].z + (double)v[j].w);
            }
        }
        if (tid < tail) {
            last = buf_tail[tid];
            s += (double)last;
        }
        if (r + gridDim.x < rows) fetch(r + gridDim.x);
        mx = fmaxf(mx, last);
#pragma unroll
        for (int j = 0; j < kHeld; ++j) mx = fmaxf(fmaxf(mx, fmaxf(v[j].x, v[j].y)), fmaxf(v[j].z, v[j].w));
        for (int o = 16; o > 0; o >>= 1) {
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            s += __shfl_xor_sync(0xffffffffu, s, o);
        }
        if (lane == 0) {
            s_max[par][warp] = mx;
            s_sum[par][warp] = s;
        }
        __syncthreads();
        mx = lane < warps ? s_max[par][lane] : -INFINITY;
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        const float thr = row_threshold(mx, frac);
        if (warp == 0) {
            // this row's sum and, its barrier being past, the previous row's count
            double t = lane < warps ? s_sum[par][lane] : 0.0;
            int c = prev >= 0 && lane < warps ? s_cnt[par ^ 1][lane] : 0;
            for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            c = __reduce_add_sync(0xffffffffu, c);
            if (lane == 0) {
                row_max[r] = mx;
                row_sum[r] = t;
                if (prev >= 0) row_count[prev] = c;
            }
        }
        // ---- mask, its size, counts per voxel
        int c = 0;
        unsigned* mrow = mask ? reinterpret_cast<unsigned*>(mask + r * ldm) + tid : nullptr;
#pragma unroll
        for (int j = 0; j < kHeld; ++j) {
            const unsigned bits = (unsigned)(v[j].x > thr) | (unsigned)(v[j].y > thr) << 8 | (unsigned)(v[j].z > thr) << 16 |
                                  (unsigned)(v[j].w > thr) << 24;
            c += __popc(bits);
            cnt[j] += bits;
            if (mrow && tid + j * T < n4) __stcs(mrow + j * T, bits);
        }
        if (tid < tail) {
            const unsigned b = last > thr;
            c += b;
            cnt_tail += b;
            if (mask) mask[r * ldm + 4 * n4 + tid] = (signed char)b;
        }
        if (++held_rows == 255) {
            if (mpxi) flush();
            held_rows = 0;
        }
        c = __reduce_add_sync(0xffffffffu, c);
        if (lane == 0) s_cnt[par][warp] = c;
        prev = r;
    }
    __syncthreads();
    if (warp == 0) {
        const int c = __reduce_add_sync(0xffffffffu, lane < warps ? s_cnt[par ^ 1][lane] : 0);
        if (lane == 0) row_count[prev] = c;
    }
    if (mpxi) flush();
}

template <bool VEC>
__global__ void __launch_bounds__(kBeamThreads) beam_rows_kernel(const float* __restrict__ A, long long rows,
                                                                  long long V, long long ld, float frac,
                                                                  float* __restrict__ row_max,
                                                                  double* __restrict__ row_sum,
                                                                  int* __restrict__ row_count,
                                                                  signed char* __restrict__ mask, long long ldm) {
    __shared__ RowReduce R;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (long long r = blockIdx.x; r < rows; r += gridDim.x) {
        const float* row = A + r * ld;
        // ---- pass A: max and sum
        float mx = -INFINITY;
        double s = 0.0;
        long long i0 = 0;
        if (VEC) {
            const float4* row4 = reinterpret_cast<const float4*>(row);
            const long long n4 = V >> 2;
            for (long long i = tid; i < n4; i += kBeamThreads) {
                const float4 v = __ldg(row4 + i);
                mx = fmaxf(fmaxf(mx, fmaxf(v.x, v.y)), fmaxf(v.z, v.w));
                s += ((double)v.x + (double)v.y) + ((double)v.z + (double)v.w);
            }
            i0 = n4 << 2;
        }
        for (long long i = i0 + tid; i < V; i += kBeamThreads) {
            const float v = __ldg(row + i);
            mx = fmaxf(mx, v);
            s += (double)v;
        }
        for (int o = 16; o > 0; o >>= 1) {
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            s += __shfl_xor_sync(0xffffffffu, s, o);
        }
        if (lane == 0) {
            R.mx[warp] = mx;
            R.sum[warp] = s;
        }
        __syncthreads();
        if (tid == 0) {
            float m = R.mx[0];
            double t = R.sum[0];
            for (int w = 1; w < kBeamWarps; ++w) {
                m = fmaxf(m, R.mx[w]);
                t += R.sum[w];
            }
            R.thr = row_threshold(m, frac);
            row_max[r] = m;
            row_sum[r] = t;
        }
        __syncthreads();
        const float thr = R.thr;
        // ---- pass B: mask and its size
        int c = 0;
        signed char* mrow = mask ? mask + r * ldm : nullptr;
        if (VEC) {
            const float4* row4 = reinterpret_cast<const float4*>(row);
            const long long n4 = V >> 2;
            for (long long i = tid; i < n4; i += kBeamThreads) {
                const float4 v = __ldg(row4 + i);
                const int b0 = v.x > thr, b1 = v.y > thr, b2 = v.z > thr, b3 = v.w > thr;
                c += b0 + b1 + b2 + b3;
                if (mrow) reinterpret_cast<char4*>(mrow)[i] = make_char4(b0, b1, b2, b3);
            }
        }
        for (long long i = i0 + tid; i < V; i += kBeamThreads) {
            const int b = __ldg(row + i) > thr;
            c += b;
            if (mrow) mrow[i] = (signed char)b;
        }
        for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
        if (lane == 0) R.cnt[warp] = c;
        __syncthreads();
        if (tid == 0) {
            int t = 0;
            for (int w = 0; w < kBeamWarps; ++w) t += R.cnt[w];
            row_count[r] = t;
        }
        __syncthreads();
    }
}

// MPXI: thread owns voxels 4t..4t+3; block (x, y) counts rows [y * rpb, (y + 1) * rpb).
template <bool FROM_MASK, bool VEC>
__global__ void __launch_bounds__(kBeamThreads) beam_mpxi_kernel(const float* __restrict__ A, long long ld,
                                                                  const signed char* __restrict__ mask,
                                                                  long long ldm, const float* __restrict__ row_max,
                                                                  float frac, long long rows, long long V,
                                                                  long long rows_per_block,
                                                                  unsigned* __restrict__ mpxi) {
    const long long c0 = 4 * ((long long)blockIdx.x * kBeamThreads + threadIdx.x);
    if (c0 >= V) return;
    const long long r0 = (long long)blockIdx.y * rows_per_block;
    const long long r1 = r0 + rows_per_block < rows ? r0 + rows_per_block : rows;
    const int nc = V - c0 >= 4 ? 4 : (int)(V - c0);
    unsigned u[4] = {0u, 0u, 0u, 0u};
    for (long long r = r0; r < r1; ++r) {
        if (FROM_MASK) {
            const signed char* m = mask + r * ldm + c0;
            if (VEC && nc == 4) {
                const char4 b = *reinterpret_cast<const char4*>(m);
                u[0] += b.x; u[1] += b.y; u[2] += b.z; u[3] += b.w;
            } else {
                for (int k = 0; k < nc; ++k) u[k] += m[k];
            }
        } else {
            const float thr = row_threshold(__ldg(row_max + r), frac);
            const float* a = A + r * ld + c0;
            if (VEC && nc == 4) {
                const float4 v = __ldg(reinterpret_cast<const float4*>(a));
                u[0] += v.x > thr; u[1] += v.y > thr; u[2] += v.z > thr; u[3] += v.w > thr;
            } else {
                for (int k = 0; k < nc; ++k) u[k] += __ldg(a + k) > thr;
            }
        }
    }
    for (int k = 0; k < nc; ++k)
        if (u[k]) atomicAdd(mpxi + c0 + k, u[k]);
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
bool aligned4(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 3u) == 0; }

}  // namespace
}  // namespace smb

using namespace smb;

extern "C" int sm_beam_metrics(const float* sysmat, int64_t rows, int64_t voxels, int64_t ld, float frac,
                               float* row_max, double* row_sum, int32_t* row_count, int8_t* mask, int64_t ld_mask,
                               uint32_t* mpxi, void* stream_ptr) {
    if (!sysmat || !row_max || !row_sum || !row_count) return fail(SM_ERR_INVALID, "null argument");
    if (rows < 1 || voxels < 1) return fail(SM_ERR_INVALID, "rows (%lld) and voxels (%lld) must be >= 1",
                                            (long long)rows, (long long)voxels);
    if (ld < voxels) return fail(SM_ERR_INVALID, "ld = %lld is smaller than %lld voxels", (long long)ld, (long long)voxels);
    if (mask && ld_mask < voxels)
        return fail(SM_ERR_INVALID, "ld_mask = %lld is smaller than %lld voxels", (long long)ld_mask, (long long)voxels);
    if (!(frac >= 0.0f) || !(frac < INFINITY)) return fail(SM_ERR_INVALID, "frac = %g must be finite and >= 0", frac);
    cudaStream_t stream = (cudaStream_t)stream_ptr;
    int sms = 148, dev = 0;
    SM_CUDA(cudaGetDevice(&dev));
    SM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const bool vec = (ld % 4 == 0) && aligned16(sysmat) && (!mask || ((ld_mask % 4 == 0) && aligned4(mask)));
    signed char* m = reinterpret_cast<signed char*>(mask);
    unsigned* out = reinterpret_cast<unsigned*>(mpxi);
    if (mpxi) SM_CUDA(cudaMemsetAsync(mpxi, 0, sizeof(uint32_t) * (size_t)voxels, stream));
    // Unaligned rows beyond 2048 voxels: copies of 4 bytes cost more than reading the row twice
    // (3000 x 5000: 46 us against 40).
    if (voxels <= (vec ? kFusedVoxels : 2048)) {
        const int V = (int)voxels;
        const size_t row = sizeof(float) * (size_t)((V + 3) & ~3);
        const bool held = vec && V >= 8192 && V <= kHeldVoxels;
        // 16 to 32 voxels a thread (short rows 8 to 16: more blocks hide their barriers);
        // three rows of shared memory where they fit, else two
        int threads = 32;
        while (threads < 1024 && threads * (V < 2048 ? 16 : 32) < V) threads *= 2;
        const int stages = 3 * row + row / 2 + 1024 <= kFusedBytes ? 3 : 2;
        size_t smem = stages * row + row / 2;
        if (held) {
            threads = kHeldThreads;
            smem = row + 16;
        }
        // `most`: the kernel's largest row.  The attribute is the kernel's, not the launch's: a
        // value of this call's own would fail the launch of a thread with longer rows.
        auto launch = [&](auto kernel, int most) -> cudaError_t {
            cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
            int per_sm = 0;
            if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
            if (e != cudaSuccess) return e;
            // Resident blocks, at most 16 per SM: each adds its counts to the same voxels at
            // the end (rows of 64 voxels: 37 us with 32 per SM).  No more rows to a block than
            // its 16-bit counts hold.
            long long grid = (long long)sms * std::max(1, std::min(per_sm, 16));
            grid = std::max(std::min(grid, (long long)rows), ((long long)rows + 65534) / 65535);
            kernel<<<(unsigned)grid, threads, smem, stream>>>(sysmat, rows, V, ld, frac, row_max, row_sum, row_count, m,
                                                              ld_mask, out);
            return cudaGetLastError();
        };
        if (held) SM_CUDA(launch(beam_held_kernel, kHeldBytes));
        else SM_CUDA(vec ? (stages == 3 ? launch(beam_fused_kernel<true, 3>, kFusedBytes) : launch(beam_fused_kernel<true, 2>, kFusedBytes))
                    : (stages == 3 ? launch(beam_fused_kernel<false, 3>, kFusedBytes) : launch(beam_fused_kernel<false, 2>, kFusedBytes)));
        return SM_OK;
    }
    const long long grid1 = rows < (long long)sms * 8 ? rows : (long long)sms * 8;
    if (vec)
        beam_rows_kernel<true><<<(unsigned)grid1, kBeamThreads, 0, stream>>>(sysmat, rows, voxels, ld, frac, row_max,
                                                                             row_sum, row_count, m, ld_mask);
    else
        beam_rows_kernel<false><<<(unsigned)grid1, kBeamThreads, 0, stream>>>(sysmat, rows, voxels, ld, frac, row_max,
                                                                              row_sum, row_count, m, ld_mask);
    SM_CUDA(cudaGetLastError());
    if (!mpxi) return SM_OK;
    const long long threads = (voxels + 3) / 4;
    const long long gx = (threads + kBeamThreads - 1) / kBeamThreads;
    long long gy = ((long long)sms * 8 + gx - 1) / gx;
    if (gy > rows) gy = rows;
    if (gy > 65535) gy = 65535;
    if (gx > 0x7fffffffLL) return fail(SM_ERR_CAPACITY, "%lld voxels exceed the launch grid", (long long)voxels);
    const long long rpb = (rows + gy - 1) / gy;
    gy = (rows + rpb - 1) / rpb;
    const dim3 grid2((unsigned)gx, (unsigned)gy);
    if (mask) {
        if (vec)
            beam_mpxi_kernel<true, true><<<grid2, kBeamThreads, 0, stream>>>(sysmat, ld, m, ld_mask, row_max, frac, rows,
                                                                            voxels, rpb, out);
        else
            beam_mpxi_kernel<true, false><<<grid2, kBeamThreads, 0, stream>>>(sysmat, ld, m, ld_mask, row_max, frac,
                                                                             rows, voxels, rpb, out);
    } else {
        if (vec)
            beam_mpxi_kernel<false, true><<<grid2, kBeamThreads, 0, stream>>>(sysmat, ld, m, ld_mask, row_max, frac,
                                                                             rows, voxels, rpb, out);
        else
            beam_mpxi_kernel<false, false><<<grid2, kBeamThreads, 0, stream>>>(sysmat, ld, m, ld_mask, row_max, frac,
                                                                              rows, voxels, rpb, out);
    }
    SM_CUDA(cudaGetLastError());
    return SM_OK;
}
