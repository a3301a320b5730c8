// BF16 GEMM on the sm_100a tensor cores (tcgen05.mma, accumulators in TMEM),
// for the scatter surrogate: C[M x N] (fp32) = alpha_row[m] * sum_k A[m][k] B[n][k]
// (+ bias[n]) (+ C when accumulating).
//
// A and B are bf16 with arbitrary strides: A[m][k] at a[m * a_ms + k * a_ks],
// B[n][k] at b[n * b_ns + k * b_ks].
//
// One persistent CTA per SM walks 128 x BN tiles of C (BN 256, 128 or 64), m
// fastest so that the CTAs at work share their B tiles in L2.  Its warps split the
// work: one loads operands by TMA, one issues the MMAs, four write results, and -
// only for operands TMA cannot take - sixteen load through registers:
//  * operands are staged 64 k at a time in a ring of 128-byte-swizzled K-major
//    tiles (192 KB); a K-contiguous operand with 16-byte aligned base and row
//    pitch comes by TMA (out-of-range rows and k read as zero), any other through
//    the loader warps, coalesced along k or along the rows, whichever is contiguous;
//  * one thread issues four 128 x BN x 16 MMAs per chunk; their commit frees the
//    ring slot.  Two TMEM accumulators alternate, so a tile's epilogue overlaps the
//    next tile's MMAs;
//  * the epilogue warps read 32 columns of their 32 TMEM lanes, pass them through
//    shared memory, and store whole 128-byte rows.
// What bounds it: for the surrogate's shapes (K = 256) the fp32 result, then the chain
// of a tile's four chunks: 2048 x 131072 x 256 takes 224 us back to back and 269 us on
// inputs that are not in L2 (a plain fill of the result 144 us, the same walk storing an eighth of the
// columns 140 us), the version before, one CTA per tile with loads, MMAs and stores in
// turn, 2072 us.  With rows off
// 16 bytes (1491 x 3906 x 975) 110 us against 203; both operands row-contiguous
// (1000 x 20000 x 512) 201 us against 460.
//
// Every wait is bounded (wait_limit polls, set process-wide by
// sm_tc_wait_limit): a wait that runs out sets the error word, the roles stop and
// skip their epilogue.  Any role may be the one that fails, so only once all have
// stopped are the copies and MMAs still in flight waited for (bounded by the default
// limit); then the CTA frees its TMEM and returns.
#include <atomic>
#include <cstdint>

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "gemm_tc.h"
#include "tc_common.cuh"

namespace smb {
namespace {

using namespace tc;
constexpr int kStoreWarps = 4;
constexpr int kWarpTma = 0, kWarpMma = 1, kWarpStore = 2, kWarpLoad = kWarpStore + kStoreWarps;   // first warp of each role
constexpr int kLoadWarps = 16;
constexpr int kRowBytes = 2 * kChunkK;       // a staged row: 64 bf16, one swizzle span

// KEEP: B's whole tile (k <= 256) stays in shared memory while the CTA walks along m.
constexpr int kKeepChunks = 4;
template <int BN, bool KEEP>
struct Ring {
    static constexpr int kStages = KEEP ? 4 : (BN == 256 ? 4 : (BN == 128 ? 6 : 8));
    static constexpr int kSlotsB = KEEP ? kKeepChunks : kStages;
    static constexpr int kBytesA = kTileM * kRowBytes, kBytesB = BN * kRowBytes;
};

template <int BN, bool KEEP>
struct __align__(1024) GemmSmem {
    static constexpr int kStages = Ring<BN, KEEP>::kStages;
    unsigned char a[kStages][Ring<BN, KEEP>::kBytesA];
    unsigned char b[Ring<BN, KEEP>::kSlotsB][Ring<BN, KEEP>::kBytesB];
    float out[kStoreWarps][32][36];                    // per epilogue warp: 32 rows x 32 columns, padded
    unsigned long long landed[kStages];      // TMA bytes arrived
    unsigned long long loaded[kStages];      // loader warps done
    unsigned long long empty[kStages];       // MMAs have read the slot
    unsigned long long kept, unkept;         // KEEP: B's tile arrived; MMAs have read it for the last time
    unsigned long long acc_full[2], acc_empty[2], drain;
    uint32_t tmem_base;
    int failed;
};

// Shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t swizzled_desc(uint32_t addr) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | (uint64_t)1 << 16 | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 |
           (uint64_t)2 << 61;
}

__device__ __forceinline__ void arrive(unsigned long long* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void arrive_expect(unsigned long long* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ void commit(unsigned long long* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void tma_load(void* dst, const CUtensorMap* map, int k, int row, unsigned long long* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            smem_u32(dst)),
        "l"(map), "r"(k), "r"(row), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ void tmem_load32(uint32_t taddr, float v[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int e = 0; e < 32; ++e) v[e] = __uint_as_float(r[e]);
}

// Rows [r0, r0 + rows) x k [k0, k0 + 64) of a strided operand into a swizzled tile, by
// one of kLoadWarps warps; rows beyond `rows_total` and k beyond `k_total` are zero.
__device__ __forceinline__ void load_rows(unsigned char* dst, int rows, const __nv_bfloat16* src, long long rs,
                                          long long ks, int r0, int rows_total, int k0, int k_total, int warp, int lane) {
    if (ks == 1) {
        // lane = two consecutive k of a row, eight rows in flight.  A row that starts off
        // a 4-byte boundary is read one element early and shifted across the lanes; the word
        // holds the row's first element too, so it lies in the operand's memory whatever the
        // stride.
        const char* bytes = reinterpret_cast<const char*>(src);
        const unsigned base_off = (unsigned)(reinterpret_cast<uintptr_t>(src) >> 1) & 1u, odd = (unsigned)rs & 1u;
        const bool full = k0 + kChunkK <= k_total;
        for (int r = warp * 8; r < rows; r += kLoadWarps * 8) {
            const char* p = bytes + 2 * ((long long)(r0 + r) * rs + k0) + 4 * lane;
            unsigned char* to = dst + r * kRowBytes + (lane & 3) * 4;
            uint32_t v[8];
            if (full && r0 + r + 8 <= rows_total && !(base_off && r0 + r == 0 && k0 == 0)) {
                uint32_t last[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const bool off = base_off ^ (odd & i & 1u);
                    v[i] = __ldg(reinterpret_cast<const uint32_t*>(p + 2 * i * rs - (off ? 2 : 0)));
                    last[i] = 0u;
                    if (off && lane == 31) last[i] = __ldg(reinterpret_cast<const unsigned short*>(p + 2 * i * rs + 2));
                }
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (base_off ^ (odd & i & 1u)) {
                        const uint32_t next = __shfl_down_sync(0xffffffffu, v[i], 1);
                        v[i] = __funnelshift_r(v[i], lane == 31 ? last[i] : next, 16);
                    }
            } else {
                const int k = k0 + 2 * lane;
                for (int i = 0; i < 8; ++i) {
                    uint32_t w = 0u;
                    if (r0 + r + i < rows_total) {
                        const unsigned short* q = reinterpret_cast<const unsigned short*>(p + 2 * i * rs);
                        if (k < k_total) w = __ldg(q);
                        if (k + 1 < k_total) w |= (uint32_t)__ldg(q + 1) << 16;
                    }
                    v[i] = w;
                }
            }
#pragma unroll
            for (int i = 0; i < 8; ++i)
                *reinterpret_cast<uint32_t*>(to + i * kRowBytes + (((lane >> 2) ^ i) << 4)) = v[i];
        }
    } else {
        // lane = row, eight k at a time
        for (int u = warp; u < rows / 32 * 8; u += kLoadWarps) {
            const int r = (u >> 3) * 32 + lane, c = u & 7, k = k0 + 8 * c;
            uint32_t v[4] = {0u, 0u, 0u, 0u};
            if (r0 + r < rows_total) {
                const unsigned short* p = reinterpret_cast<const unsigned short*>(src) + (long long)(r0 + r) * rs + (long long)k * ks;
#pragma unroll
                for (int e = 0; e < 8; ++e)
                    if (k + e < k_total) v[e >> 1] |= (uint32_t)__ldg(p + e * ks) << (16 * (e & 1));
            }
            *reinterpret_cast<uint4*>(dst + r * kRowBytes + ((c ^ (r & 7)) << 4)) = make_uint4(v[0], v[1], v[2], v[3]);
        }
    }
}

// A CTA's walk over the tiles: panels of gridDim.x tiles along n, every m of a panel
// before the next one, so a CTA keeps its n (and B's tile) down a whole panel.  Stepped
// without divisions but in the last, narrower panel: the MMA thread takes these steps
// between its tiles.
template <int BN>
struct Walk {
    int tiles_m, tiles_n, first, width, m, col;   // the panel's first n tile and width; the tile in it
    bool more;
    __device__ __forceinline__ Walk(const GemmArgs& g)
        : tiles_m((g.m + kTileM - 1) / kTileM), tiles_n((g.n + BN - 1) / BN), first(0), m(0), col((int)blockIdx.x), more(true) {
        width = min((int)gridDim.x, tiles_n);
        place(col);
    }
    // the tile `at` places after the panel's start, in this panel or a later one
    __device__ __forceinline__ void place(int at) {
        while (more && (long long)at >= (long long)width * tiles_m) {
            at -= width * tiles_m;
            first += (int)gridDim.x;
            more = first < tiles_n;
            width = min((int)gridDim.x, tiles_n - first);
        }
        if (more) {
            m = at / width;
            col = at - m * width;
        }
    }
    __device__ __forceinline__ void next() {
        if (width == (int)gridDim.x && m + 1 < tiles_m) ++m;
        else place(m * width + col + (int)gridDim.x);
    }
    __device__ __forceinline__ int m0() const { return m * kTileM; }
    __device__ __forceinline__ int n0() const { return (first + col) * BN; }
};

// TA, TB: operand A / B comes by TMA.
template <int BN, bool TA, bool TB, bool KEEP>
__global__ void __launch_bounds__(32 * (kWarpLoad + (TA && TB ? 0 : kLoadWarps)), 1)
gemm_bf16_tc_kernel(const __grid_constant__ GemmArgs g, const __grid_constant__ CUtensorMap map_a,
                    const __grid_constant__ CUtensorMap map_b, uint32_t wait_limit) {
    static_assert(!KEEP || (TA && TB), "B is kept by TMA");
    using R = Ring<BN, KEEP>;
    extern __shared__ unsigned char smem_raw[];
    GemmSmem<BN, KEEP>& S = *reinterpret_cast<GemmSmem<BN, KEEP>*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int chunks = (g.k + kChunkK - 1) / kChunkK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < R::kStages; ++s) {
            mbar_init(&S.landed[s], 1);
            mbar_init(&S.loaded[s], kLoadWarps);
            mbar_init(&S.empty[s], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&S.acc_full[i], 1);
            mbar_init(&S.acc_empty[i], kStoreWarps);
        }
        mbar_init(&S.drain, 1);
        mbar_init(&S.kept, 1);
        mbar_init(&S.unkept, 1);
        S.failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kWarpMma) tmem_alloc(&S.tmem_base, 2 * BN);
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = S.tmem_base;
    volatile int* failed = &S.failed;
    auto wait = [&](unsigned long long* bar, uint32_t phase) {
        if (*failed) return false;
        if (mbar_wait(bar, phase, wait_limit)) return true;
        *failed = 1;
        return false;
    };

    uint32_t it = 0, keeps = 0;   // this role's chunks and kept B tiles so far
    if (warp == kWarpTma) {
        if ((TA || TB) && lane == 0) {
            int kept_n = -1;
            bool ok = true;
            for (Walk<BN> at(g); at.more && ok; at.next()) {
                if (KEEP && at.n0() != kept_n) {
                    if (!(ok = wait(&S.unkept, (keeps + 1) & 1u))) break;
                    arrive_expect(&S.kept, chunks * R::kBytesB);
                    for (int c = 0; c < chunks; ++c) tma_load(S.b[c], &map_b, c * kChunkK, at.n0(), &S.kept);
                    kept_n = at.n0();
                    ++keeps;
                }
                for (int c = 0; c < chunks; ++c, ++it) {
                    const int s = it % R::kStages;
                    if (!(ok = wait(&S.empty[s], (it / R::kStages + 1) & 1u))) break;
                    arrive_expect(&S.landed[s], (TA ? R::kBytesA : 0) + (TB && !KEEP ? R::kBytesB : 0));
                    if (TA) tma_load(S.a[s], &map_a, c * kChunkK, at.m0(), &S.landed[s]);
                    if (TB && !KEEP) tma_load(S.b[s], &map_b, c * kChunkK, at.n0(), &S.landed[s]);
                }
            }
        }
    } else if (warp == kWarpMma) {
        if (lane == 0) {
            const uint32_t idesc = instr_desc(BN);
            uint32_t n = 0;
            int kept_n = -1;
            bool ok = true;
            for (Walk<BN> at(g); at.more && ok; ++n) {
                const uint32_t acc = tmem + (n & 1u) * BN;
                if (!(ok = wait(&S.acc_empty[n & 1u], ((n >> 1) + 1) & 1u))) break;
                if (KEEP) {
                    if (at.n0() != kept_n && !(ok = wait(&S.kept, keeps++ & 1u))) break;
                    kept_n = at.n0();
                }
                asm volatile("tcgen05.fence::after_thread_sync;");
                for (int c = 0; c < chunks; ++c, ++it) {
                    const int s = it % R::kStages;
                    const uint32_t phase = (it / R::kStages) & 1u;
                    if (TA || TB) ok = wait(&S.landed[s], phase);
                    if (!(TA && TB) && ok) ok = wait(&S.loaded[s], phase);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;");
                    const uint32_t a = smem_u32(S.a[s]), b = smem_u32(S.b[KEEP ? c : s]);
#pragma unroll
                    for (int j = 0; j < kChunkK / 16; ++j) {
                        const uint64_t da = swizzled_desc(a + 32u * j), db = swizzled_desc(b + 32u * j);
                        const uint32_t accumulate = (c > 0 || j > 0) ? 1u : 0u;
                        asm volatile(
                            "{\n\t.reg .pred p;\n\t"
                            "setp.ne.b32 p, %4, 0;\n\t"
                            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}"
                            :
                            : "r"(acc), "l"(da), "l"(db), "r"(idesc), "r"(accumulate), "r"(0u), "r"(0u), "r"(0u), "r"(0u));
                    }
                    commit(&S.empty[s]);
                }
                if (ok) commit(&S.acc_full[n & 1u]);
                at.next();
                if (KEEP && ok && at.more && at.n0() != kept_n) commit(&S.unkept);
            }
        }
    } else if (warp < kWarpLoad) {
        const int part = warp & 3;                     // TMEM lanes 32 part .. 32 part + 31
        static_assert(kStoreWarps == 4, "a store warp for each 32 TMEM lanes");
        float(*out)[36] = S.out[warp - kWarpStore];
        const bool vec = g.ldc % 4 == 0 && (reinterpret_cast<uintptr_t>(g.c) & 15u) == 0 &&
                         (!g.bias || (reinterpret_cast<uintptr_t>(g.bias) & 15u) == 0);
        uint32_t n = 0;
        for (Walk<BN> at(g); at.more; at.next(), ++n) {
            const int m0 = at.m0() + 32 * part, n0 = at.n0();
            if (!__all_sync(0xffffffffu, wait(&S.acc_full[n & 1u], (n >> 1) & 1u))) break;
            asm volatile("tcgen05.fence::after_thread_sync;");
            const float scale = g.row_scale && m0 + lane < g.m ? g.row_scale[m0 + lane] : g.alpha;
            const int cols = min(BN, g.n - n0);
            for (int c0 = 0; c0 < cols; c0 += 32) {
                float v[32];
                tmem_load32(tmem + (n & 1u) * BN + ((uint32_t)(32 * part) << 16) + (uint32_t)c0, v);
#pragma unroll
                for (int e = 0; e < 32; e += 4)
                    *reinterpret_cast<float4*>(&out[lane][e]) = make_float4(v[e] * scale, v[e + 1] * scale, v[e + 2] * scale, v[e + 3] * scale);
                __syncwarp();
                const int r0 = lane >> 3, col = n0 + c0 + (lane & 7) * 4;   // rows r0, r0 + 4, ...
                float4 w[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) w[i] = *reinterpret_cast<const float4*>(&out[r0 + 4 * i][(lane & 7) * 4]);
                float* p = g.c + (long long)(m0 + r0) * g.ldc + col;
                const long long step = 4 * g.ldc;
                if (vec && m0 + 32 <= g.m && c0 + 32 <= cols) {
                    // a whole 32 x 32 block: no test per row, one warp per scheduler has nobody to hide it
                    if (g.bias && g.epilogue != 1) {
                        const float4 o = __ldg(reinterpret_cast<const float4*>(g.bias + col));
#pragma unroll
                        for (int i = 0; i < 8; ++i) w[i] = make_float4(w[i].x + o.x, w[i].y + o.y, w[i].z + o.z, w[i].w + o.w);
                    }
                    if (g.accumulate || g.epilogue == 1) {
                        float4 o[8];
#pragma unroll
                        for (int i = 0; i < 8; ++i) o[i] = *reinterpret_cast<const float4*>(p + i * step);
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            w[i] = g.epilogue == 1
                                       ? make_float4(o[i].x * __expf(w[i].x), o[i].y * __expf(w[i].y), o[i].z * __expf(w[i].z), o[i].w * __expf(w[i].w))
                                       : make_float4(w[i].x + o[i].x, w[i].y + o[i].y, w[i].z + o[i].z, w[i].w + o[i].w);
                    }
#pragma unroll
                    for (int i = 0; i < 8; ++i) __stcs(reinterpret_cast<float4*>(p + i * step), w[i]);
                } else {
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float x[4] = {w[i].x, w[i].y, w[i].z, w[i].w};
                        if (m0 + r0 + 4 * i < g.m)
#pragma unroll
                            for (int e = 0; e < 4; ++e)
                                if (col + e < g.n) {
                                    float* q = p + i * step + e;
                                    if (g.epilogue == 1) *q = *q * __expf(x[e]);
                                    else {
                                        float y = x[e];
                                        if (g.bias) y += g.bias[col + e];
                                        if (g.accumulate) y += *q;
                                        *q = y;
                                    }
                                }
                    }
                }
                __syncwarp();
            }
            asm volatile("tcgen05.fence::before_thread_sync;");
            __syncwarp();
            if (lane == 0) arrive(&S.acc_empty[n & 1u]);
        }
    } else if (!(TA && TB)) {
        bool ok = true;
        for (Walk<BN> at(g); at.more && ok; at.next()) {
            for (int c = 0; c < chunks; ++c, ++it) {
                const int s = it % R::kStages;
                if (!(ok = __all_sync(0xffffffffu, wait(&S.empty[s], (it / R::kStages + 1) & 1u)))) break;
                if (!TA) load_rows(S.a[s], kTileM, g.a, g.a_ms, g.a_ks, at.m0(), g.m, c * kChunkK, g.k, warp - kWarpLoad, lane);
                if (!TB) load_rows(S.b[s], BN, g.b, g.b_ns, g.b_ks, at.n0(), g.n, c * kChunkK, g.k, warp - kWarpLoad, lane);
                // generic-proxy stores must be visible to the tensor core's async proxy
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) arrive(&S.loaded[s]);
            }
        }
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (*failed) {   // no role sets it any more, so all take this branch or none
        if (threadIdx.x == 0 && g.error) atomicOr(g.error, 1);
        if (warp == kWarpTma && lane == 0) {   // copies land before the CTA goes
            if (keeps) mbar_wait(&S.kept, (keeps - 1) & 1u, kWaitLimit);
            for (uint32_t i = it < (uint32_t)R::kStages ? 0u : it - R::kStages; i < it; ++i)
                mbar_wait(&S.landed[i % R::kStages], (i / R::kStages) & 1u, kWaitLimit);
        }
        if (warp == kWarpMma && lane == 0) {   // MMAs finish before the tensor memory goes
            commit(&S.drain);
            mbar_wait(&S.drain, 0, kWaitLimit);
        }
        __syncwarp();
        __syncthreads();
    }
    if (warp == kWarpMma) {
        asm volatile("tcgen05.fence::after_thread_sync;");
        tmem_dealloc(tmem, 2 * BN);
    }
}

std::atomic<uint32_t> g_wait_limit{kWaitLimit};

// cuTensorMapEncodeTiled through the runtime (the library does not link libcuda).
using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                              const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                              CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeFn tensor_map_encoder() {
    static const EncodeFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult st;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &st) != cudaSuccess ||
            st != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            p = nullptr;
        }
        return reinterpret_cast<EncodeFn>(p);
    }();
    return fn;
}

// A [rows][k] bf16 operand in boxes of box_rows x 64 k; false when TMA cannot take it
// (k not contiguous, base or row pitch off the 16 bytes the copy needs).
bool make_map(const __nv_bfloat16* p, long long rs, long long ks, int rows, int k, int box_rows, CUtensorMap* map) {
    if (ks != 1 || rs < k || (rs * 2) % 16 != 0 || (reinterpret_cast<uintptr_t>(p) & 15u) != 0) return false;
    const EncodeFn encode = tensor_map_encoder();
    if (!encode) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)rows}, pitch[1] = {(cuuint64_t)rs * 2};
    const cuuint32_t box[2] = {(cuuint32_t)kChunkK, (cuuint32_t)box_rows}, step[2] = {1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<__nv_bfloat16*>(p), dims, pitch, box, step,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int BN, bool TA, bool TB, bool KEEP>
cudaError_t launch(const GemmArgs& g, const CUtensorMap& a, const CUtensorMap& b, int sms, cudaStream_t stream) {
    const auto kernel = gemm_bf16_tc_kernel<BN, TA, TB, KEEP>;
    const int smem = (int)sizeof(GemmSmem<BN, KEEP>) + 1024;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    const long long tiles = (long long)((g.m + kTileM - 1) / kTileM) * ((g.n + BN - 1) / BN);
    const int threads = 32 * (kWarpLoad + (TA && TB ? 0 : kLoadWarps));
    kernel<<<(unsigned)(tiles < sms ? tiles : sms), threads, smem, stream>>>(g, a, b, g_wait_limit.load());
    return cudaGetLastError();
}

template <int BN>
cudaError_t launch_width(const GemmArgs& g, int sms, cudaStream_t stream) {
    CUtensorMap a{}, b{};
    const bool ta = make_map(g.a, g.a_ms, g.a_ks, g.m, g.k, kTileM, &a);
    const bool tb = make_map(g.b, g.b_ns, g.b_ks, g.n, g.k, BN, &b);
    // Short products over several m tiles: the ring would read B's tile from L2 again for each
    // (2048 x 131072 x 256: 2.6 GB through L2 in 240 us; kept, 1.7 GB).
    if (BN == 256 && ta && tb && g.k <= kKeepChunks * kChunkK && g.m > kTileM)
        return launch<256, true, true, true>(g, a, b, sms, stream);
    if (ta) return tb ? launch<BN, true, true, false>(g, a, b, sms, stream) : launch<BN, true, false, false>(g, a, b, sms, stream);
    return tb ? launch<BN, false, true, false>(g, a, b, sms, stream) : launch<BN, false, false, false>(g, a, b, sms, stream);
}

}  // namespace

uint32_t gemm_wait_limit(int64_t polls) {
    const uint32_t prev = g_wait_limit.load();
    if (polls < 0) g_wait_limit.store(kWaitLimit);
    else g_wait_limit.store(polls > 0xffffffffLL ? 0xffffffffu : (uint32_t)polls);
    return prev;
}

cudaError_t gemm_bf16_tc(const GemmArgs& args, cudaStream_t stream) {
    if (args.m <= 0 || args.n <= 0 || args.k <= 0) return cudaSuccess;
    int dev = 0, sms = 148;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    // The width of the shortest walk: waves of tiles times the width of one, plus a share of 64
    // columns for what does not shrink with it (A's loads, the chain load - MMA - store).
    const long long rows = (args.m + kTileM - 1) / kTileM;
    auto walk = [&](int bn) { return (rows * ((args.n + bn - 1) / bn) + sms - 1) / sms * (bn + 64); };
    if (walk(256) <= walk(128) && walk(256) <= walk(64)) return launch_width<256>(args, sms, stream);
    if (walk(128) <= walk(64)) return launch_width<128>(args, sms, stream);
    return launch_width<64>(args, sms, stream);
}

}  // namespace smb
