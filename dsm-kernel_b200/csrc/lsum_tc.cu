// Split-precision l-sum contraction on the sm_100a tensor cores.
//
// Persistent, warp-specialised kernel, one CTA per SM:
//   warp 0      TMA producer: per stage, the hi and lo pieces of a 128 x BK
//               A tile and of a 128 x BK B tile (four bulk tensor loads,
//               one mbarrier with the byte count)
//   warp 1      MMA issuer: per stage and 16-order step, three
//               tcgen05.mma (hi*hi, hi*lo, lo*hi) into the current chunk
//               accumulator; tcgen05.commit frees the stage and hands
//               finished chunk accumulators over
//   warps 2..9  epilogue: tcgen05.ld of the chunk accumulators (two warps
//               per 32-lane quarter, 64 columns each), FP64 sum of the
//               chunks, row x column scaling, column-major or row-major stores
// Accuracy: the tensor cores add each step into the FP32 accumulator with a
// rounding relative to the accumulator's magnitude, so a long order sum
// loses bits in proportion to its length.  The products therefore go into
// short chunks (chunk stages of BK orders) whose partial sums the epilogue
// adds in FP64.  The cross terms (2^-11 smaller than hi*hi) share the chunk
// accumulator: each stage issues them before its hi*hi products, so in a
// one-stage chunk they are summed while the accumulator is still small.  Tensor
// memory (512 columns): four chunk buffers of 128 columns, so the epilogue
// drains a pair while the MMAs fill the other pair, across tile boundaries
// too.  TC_REVERSE runs the orders from high to low.
// Every wait is bounded: after about a second a role raises the CTA's abort
// flag, all roles leave their loops, the issued copies and MMAs are waited
// for (again bounded), the tensor memory is freed and the error word is set.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <mutex>

#include "lsum_tc.cuh"

namespace dsm {
namespace tc {

namespace {

constexpr int EPI_THREADS = 256;                 // warps 2..9
constexpr int NTHREADS = 64 + EPI_THREADS;
constexpr uint32_t TMEM_COLS = 512;
constexpr int SMEM_STAGES = 192 * 1024;         // operand stages
constexpr int NHB = 4;                          // chunk buffers in tensor memory

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ unsigned long long gtimer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ void mbar_init(uint64_t* b, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* b, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(b)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* b) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(b)) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint64_t* b, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(b)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait.  Gives up when another role has aborted or after the limit
// (then it aborts the CTA itself).
__device__ __forceinline__ bool mbar_wait(uint64_t* b, uint32_t parity, volatile int* abort_flag,
                                          unsigned long long limit_ns) {
    const unsigned long long t0 = gtimer();
    for (uint32_t n = 0;; ++n) {
        if (mbar_try(b, parity)) return true;
        if ((n & 63) == 63) {
            if (*abort_flag) return false;
            if (gtimer() - t0 > limit_ns) {
                *abort_flag = 1;
                return false;
            }
        }
    }
}
// Bounded wait used while draining after an abort (ignores the flag).
__device__ __forceinline__ void mbar_drain(uint64_t* b, uint32_t parity, unsigned long long limit_ns) {
    const unsigned long long t0 = gtimer();
    while (!mbar_try(b, parity))
        if (gtimer() - t0 > limit_ns) return;
}

__device__ __forceinline__ void tma_a(const CUtensorMap* m, void* dst, uint64_t* bar, int x, int y, int z, int w) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], "
        "[%2];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z), "r"(w)
        : "memory");
}
__device__ __forceinline__ void tma_b(const CUtensorMap* m, void* dst, uint64_t* bar, int x, int y, int z) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], "
        "[%2];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
        : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Shared-memory matrix descriptor of an order-major tile whose rows are
// BK*2 bytes, swizzled as the TMA wrote them (64B or 128B pattern), 8-row
// groups at 8*BK*2 bytes.
template <int BK>
__device__ __forceinline__ uint64_t sdesc(uint32_t addr) {
    constexpr uint64_t layout = BK == 32 ? 4 : 2;   // SWIZZLE_64B : SWIZZLE_128B
    constexpr uint64_t sbo = (8 * BK * 2) >> 4;
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | (1ull << 16) | (sbo << 32) | (1ull << 46) | (layout << 61);
}

__device__ __forceinline__ void mma_f16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void tmem_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}
// Tile t of a launch: its problem p, row tile mt and column tile nt.  A CTA
// visits its tiles in increasing order, so p only moves forward from the
// previous tile's problem (the caller keeps it, starting at 0).
__device__ __forceinline__ void decode(const Problem* ps, int np, int t, int& p, int& mt, int& nt) {
    while (p + 1 < np && ps[p + 1].tile0 <= t) ++p;
    const int loc = t - ps[p].tile0;
    mt = loc / ps[p].tiles_n;
    nt = loc - mt * ps[p].tiles_n;
}

template <int BK>
__global__ void __launch_bounds__(NTHREADS, 1)
    k_lsum_tc(const __grid_constant__ Maps maps, const Problem* __restrict__ probs, int np, int ntiles,
              uint32_t idesc, uint32_t flags, int chunk, int* __restrict__ err, unsigned long long wait_ns) {
    constexpr int A_BYTES = BM * BK * 2, B_BYTES = BN * BK * 2;
    constexpr int STAGE = 2 * A_BYTES + 2 * B_BYTES;
    constexpr int STAGES = SMEM_STAGES / STAGE;
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t full[STAGES], empty[STAGES], hfull[NHB], hempty[NHB], fin;
    __shared__ uint32_t tmem_sh;
    __shared__ int abort_sh;
    __shared__ Problem ps[MAXP];

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool reverse = (flags & TC_REVERSE) != 0;
    unsigned char* base = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    volatile int* abort_flag = &abort_sh;

    for (int i = threadIdx.x; i < np; i += NTHREADS) ps[i] = probs[i];
    if (threadIdx.x == 0) {
        abort_sh = 0;
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < NHB; ++b) {
            mbar_init(&hfull[b], 1);
            mbar_init(&hempty[b], EPI_THREADS);
        }
        mbar_init(&fin, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&maps.a[0])) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&maps.b[0])) : "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_sh)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_sh;
    // tensor memory: chunk accumulators [0..NHB) at columns [0, NHB BN)

    if (warp == 0) {
        if (lane == 0) {  // ---------------------------------------- producer
            int it = 0, p = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x) {
                int mt, nt;
                decode(ps, np, t, p, mt, nt);
                const Problem& P = ps[p];
                const int kbn = P.kb ? max(0, min(P.kb[mt], P.kblocks)) : P.kblocks;  // this row tile's order blocks
                for (int kb = 0; kb < kbn; ++kb, ++it) {
                    const int s = it % STAGES;
                    const uint32_t ph = (it / STAGES) & 1;
                    if (!mbar_wait(&empty[s], ph ^ 1, abort_flag, wait_ns)) {
                        ok = false;
                        break;
                    }
                    // test hook: CTA 0 issues nothing for its first stage
                    if ((flags & TC_TEST_STALL) && blockIdx.x == 0 && it == 0) continue;
                    unsigned char* sp = base + s * STAGE;
                    const int x = (reverse ? kbn - 1 - kb : kb) * BK;
                    mbar_expect_tx(&full[s], STAGE);
                    tma_a(&maps.a[P.amap], sp, &full[s], x, P.row0 + mt * BM, P.z, 0);
                    tma_a(&maps.a[P.amap], sp + A_BYTES, &full[s], x, P.row0 + mt * BM, P.z, 1);
                    tma_b(&maps.b[P.bmap], sp + 2 * A_BYTES, &full[s], x, nt * BN, 0);
                    tma_b(&maps.b[P.bmap], sp + 2 * A_BYTES + B_BYTES, &full[s], x, nt * BN, 1);
                }
            }
            // every issued copy has landed before the CTA may exit
            for (int s = 0; s < STAGES && s < it; ++s) {
                const int last = s + ((it - 1 - s) / STAGES) * STAGES;
                mbar_drain(&full[s], (last / STAGES) & 1, wait_ns);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {  // ---------------------------------------- MMA issuer
            int it = 0, cc = 0, p = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x) {
                int mt, nt;
                decode(ps, np, t, p, mt, nt);
                const int kbn = ps[p].kb ? max(0, min(ps[p].kb[mt], ps[p].kblocks)) : ps[p].kblocks;
                const int ch = chunk > 0 ? chunk : max(kbn, 1);
                // the last column tile of a contraction runs with N cut to
                // its columns (a multiple of 16): no MMA time on padding
                const int nrem = ps[p].N - nt * BN;
                const uint32_t ncols = (uint32_t)min(BN, (nrem + 15) & ~15);
                const uint32_t idt = (idesc & ~(0x3Fu << 17)) | ((ncols >> 3) << 17);
                uint32_t dh = tmem;
                int hb = 0;
                for (int kb = 0; kb < kbn; ++kb, ++it) {
                    const bool cfirst = kb % ch == 0;
                    if (cfirst) {
                        hb = cc % NHB;
                        if (!mbar_wait(&hempty[hb], ((cc / NHB) & 1) ^ 1, abort_flag, wait_ns)) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                        dh = tmem + (uint32_t)(hb * BN);
                    }
                    const int s = it % STAGES;
                    if (!mbar_wait(&full[s], (it / STAGES) & 1, abort_flag, wait_ns)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t ah = smem_u32(base + s * STAGE), al = ah + A_BYTES;
                    const uint32_t bh = ah + 2 * A_BYTES, bl = bh + B_BYTES;
                    // the cross terms first: while the accumulator holds only
                    // them (2^-11 of hi*hi), their roundings are that much smaller
#pragma unroll
                    for (int j = 0; j < BK / 16; ++j) {
                        const uint32_t o = 32u * j;
                        mma_f16(dh, sdesc<BK>(ah + o), sdesc<BK>(bl + o), idt, (cfirst && j == 0) ? 0u : 1u);
                        mma_f16(dh, sdesc<BK>(al + o), sdesc<BK>(bh + o), idt, 1u);
                    }
#pragma unroll
                    for (int j = 0; j < BK / 16; ++j) {
                        const uint32_t o = 32u * j;
                        mma_f16(dh, sdesc<BK>(ah + o), sdesc<BK>(bh + o), idt, 1u);
                    }
                    mma_commit(&empty[s]);
                    if (kb % ch == ch - 1 || kb == kbn - 1) {
                        mma_commit(&hfull[hb]);
                        ++cc;
                    }
                }
            }
            // all issued MMAs complete before tensor memory is released
            mma_commit(&fin);
            mbar_drain(&fin, 0, wait_ns);
        }
    } else {  // ------------------------------------------------------ epilogue
        // two warps per tensor-memory lane quarter, each owning 64 columns;
        // the chunks are summed in FP64 registers
        const int q = warp & 3, half = (warp - 2) >> 2;
        const uint32_t lanes = (uint32_t)(q * 32) << 16;
        int cc = 0, p = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x) {
            int mt, nt;
            decode(ps, np, t, p, mt, nt);
            const Problem& P = ps[p];
            const int kbn = P.kb ? max(0, min(P.kb[mt], P.kblocks)) : P.kblocks, ch = chunk > 0 ? chunk : max(kbn, 1);
            const int nch = (kbn + ch - 1) / ch;
            double acc[64];
#pragma unroll
            for (int j = 0; j < 64; ++j) acc[j] = 0.0;
            // chunks in pairs: the two FP32 chunk sums are added in FP32
            // (one rounding, unbiased) before the FP64 accumulation, which
            // halves the conversions and FP64 additions
            for (int c = 0; c + 1 < nch; c += 2, cc += 2) {
                const int hb0 = cc % NHB, hb1 = (cc + 1) % NHB;
                bool got = mbar_wait(&hfull[hb0], (cc / NHB) & 1, abort_flag, wait_ns);
                got = got && mbar_wait(&hfull[hb1], ((cc + 1) / NHB) & 1, abort_flag, wait_ns);
                if (!__all_sync(0xffffffffu, got)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t ta0 = tmem + lanes + (uint32_t)(hb0 * BN + half * 64);
                const uint32_t ta1 = tmem + lanes + (uint32_t)(hb1 * BN + half * 64);
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                    uint32_t r0[16], r1[16];
                    tmem_ld16(ta0 + 16 * g, r0);
                    tmem_ld16(ta1 + 16 * g, r1);
                    tmem_wait();
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        acc[g * 16 + j] += (double)(__uint_as_float(r0[j]) + __uint_as_float(r1[j]));
                }
                tc_fence_before();
                mbar_arrive(&hempty[hb0]);
                mbar_arrive(&hempty[hb1]);
            }
            if (ok && (nch & 1)) {  // the odd last chunk
                const int hb = cc % NHB;
                const bool got = mbar_wait(&hfull[hb], (cc / NHB) & 1, abort_flag, wait_ns);
                if (!__all_sync(0xffffffffu, got)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t ta = tmem + lanes + (uint32_t)(hb * BN + half * 64);
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                    uint32_t r0[16];
                    tmem_ld16(ta + 16 * g, r0);
                    tmem_wait();
#pragma unroll
                    for (int j = 0; j < 16; ++j) acc[g * 16 + j] += (double)__uint_as_float(r0[j]);
                }
                tc_fence_before();
                mbar_arrive(&hempty[hb]);
                ++cc;
            }
            if (!ok) break;
            const int m = mt * BM + q * 32 + lane;
            const bool mv = m < P.M;
            const double rs = mv ? (double)P.sa[m] : 0.0;
            if (P.rowmajor) {  // a row's 64 columns: 16-byte stores where a whole group of 32 lies within N
                float* Cr = P.C + (long long)m * P.ldc;
#pragma unroll
                for (int g = 0; g < 2; ++g) {
                    const int n0 = nt * BN + half * 64 + g * 32;
                    if (!mv) continue;
                    if (n0 + 32 <= P.N) {
#pragma unroll
                        for (int j = 0; j < 32; j += 4) {
                            float4 v;
                            v.x = (float)(acc[g * 32 + j] * rs * (double)P.sb[n0 + j]);
                            v.y = (float)(acc[g * 32 + j + 1] * rs * (double)P.sb[n0 + j + 1]);
                            v.z = (float)(acc[g * 32 + j + 2] * rs * (double)P.sb[n0 + j + 2]);
                            v.w = (float)(acc[g * 32 + j + 3] * rs * (double)P.sb[n0 + j + 3]);
                            *reinterpret_cast<float4*>(Cr + n0 + j) = v;
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < 32; ++j)
                            if (n0 + j < P.N) Cr[n0 + j] = (float)(acc[g * 32 + j] * rs * (double)P.sb[n0 + j]);
                    }
                }
            } else {
                float* Cm = P.C + m;
#pragma unroll
                for (int g = 0; g < 2; ++g) {
                    const int n0 = nt * BN + half * 64 + g * 32;
                    if (mv) {
#pragma unroll
                        for (int j = 0; j < 32; ++j) {
                            const int n = n0 + j;
                            if (n < P.N)
                                Cm[(long long)n * P.ldc] =
                                    (float)(acc[g * 32 + j] * rs * (double)P.sb[n]);
                        }
                    }
                }
            }
        }
    }

    __syncthreads();
    if (warp == 0) {
        __syncwarp();
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS)
                     : "memory");
    }
    if (threadIdx.x == 0 && abort_sh) atomicExch(err, 1);
}

// ------------------------------------------------------------ piece split
// x = s (hi + lo): s = 2^e with the row (column) maximum scaled into
// [2^14, 2^15), below the fp16 limit with a factor-two margin.  The scale is
// exact, so hi + lo carries ~22 (fp16) or ~16 (bf16) significant bits.
__device__ __forceinline__ int piece_exp(double mx) {
    if (!(mx > 0.0)) return 0;
    int e = ilogb(mx) - 14;
    return max(-126, min(127, e));
}
__device__ __forceinline__ void split2(double x, int fmt, uint16_t& hi, uint16_t& lo) {
    if (fmt == PIECE_BF16) {
        __nv_bfloat16 h = __double2bfloat16(x);
        __nv_bfloat16 l = __double2bfloat16(x - (double)__bfloat162float(h));
        hi = __bfloat16_as_ushort(h);
        lo = __bfloat16_as_ushort(l);
    } else {
        __half h = __double2half(x);
        __half l = __double2half(x - (double)__half2float(h));
        hi = __half_as_ushort(h);
        lo = __half_as_ushort(l);
    }
}

// the same split for two FP32 values already scaled by 2^-e: the residual
// x - hi has at most 13 (fp16) or 16 (bf16) significant bits, so it is exact
// in FP32 and each piece is one rounding of an exact value, as in split2
__device__ __forceinline__ void split2x(float x, float y, int fmt, uint32_t& hi, uint32_t& lo) {
    if (fmt == PIECE_BF16) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
        const __nv_bfloat162 l = __floats2bfloat162_rn(x - __low2float(h), y - __high2float(h));
        hi = *reinterpret_cast<const uint32_t*>(&h);
        lo = *reinterpret_cast<const uint32_t*>(&l);
    } else {
        const __half2 h = __floats2half2_rn(x, y);
        const __half2 l = __floats2half2_rn(x - __low2float(h), y - __high2float(h));
        hi = *reinterpret_cast<const uint32_t*>(&h);
        lo = *reinterpret_cast<const uint32_t*>(&l);
    }
}
__device__ __forceinline__ void split2x(double x, double y, int fmt, uint32_t& hi, uint32_t& lo) {
    uint16_t h0, h1, l0, l1;
    split2(x, fmt, h0, l0);
    split2(y, fmt, h1, l1);
    hi = (uint32_t)h0 | ((uint32_t)h1 << 16);
    lo = (uint32_t)l0 | ((uint32_t)l1 << 16);
}

// up to three row sets (|m| = 0, 1, 2) of a run of frequencies in one launch
struct SplitSet {
    const void* A;
    int n, rows, block0;  // rows in all, rows of a frequency, first block
    uint16_t* P;
    size_t stride;        // between the two pieces
    float* sa;
    int* lnz;
    const int* rowrec;
    int rf;               // rows of the first row group (row tiles start at 0 and here)
};
struct SplitArgs {
    SplitSet s[3];
    int ns, lcap, kcap, bk, fmt, R1;
    const int *nord, *zf;
};

// One warp per row, four orders per lane and load.  The row's first NC groups
// of 128 orders stay in registers between its maximum (which sets the scale)
// and the pieces; longer rows are read twice.
//
// Bound: the bytes of the rows read and the pieces written.  Read twice, with
// a launch per |m| and a power of two applied per element by ldexp, the
// slices' rows took 1.24 ms (8 slices of up to 1024, FP32) and 0.94 ms (16 SH
// slices of up to 256, FP64, one order a lane); now 0.94 and 0.73, of which
// the row tiles' order blocks (k_tile_orders) are 0.05.  Zeros past a tile's
// blocks are not written (more than half of the P-SV rows' orders with the
// depth cut): 1.04 -> 0.94.
constexpr int SPLIT_THREADS = 128;
template <class T>
struct Vec4 {
    T x[4];
};
template <class T, int NC>
__global__ void __launch_bounds__(SPLIT_THREADS) k_split_rows(const SplitArgs a) {
    int si = 0;
    while (si + 1 < a.ns && (int)blockIdx.x >= a.s[si + 1].block0) ++si;
    const SplitSet& S = a.s[si];
    const int row = ((int)blockIdx.x - S.block0) * (SPLIT_THREADS / 32) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (row >= S.n) return;
    const int w = row / S.rows;
    const int K = a.nord ? min(a.nord[w], a.lcap) : a.lcap;
    // orders at or above Kr are known to be zero: not read
    const int Kr = a.zf ? min(K, a.zf[w * a.R1 + S.rowrec[row - w * S.rows]]) : K;
    // order blocks the row's tile can have (k_tile_orders, from rows that are
    // zero where their receivers are): pieces past them are not read
    const int kbl = (K + a.bk - 1) / a.bk;
    int kb = kbl;
    if (a.zf) {
        const int rw = row - w * S.rows, g0 = rw < S.rf ? 0 : S.rf, g1 = rw < S.rf ? S.rf : S.rows;
        const int t0 = g0 + (rw - g0) / BM * BM;
        int far = 0;
#pragma unroll
        for (int i = 0; i < BM / 32; ++i) {
            const int r = min(t0 + 32 * i + lane, g1 - 1);
            far = max(far, a.zf[w * a.R1 + S.rowrec[r]]);
        }
        far = min(K, __reduce_max_sync(0xffffffffu, far));
        kb = min(kbl, (far + a.bk - 1) / a.bk);
        kb += kb > 0 && ((kbl - kb) & 1);
    }
    const int nv = min(a.kcap, kb * a.bk) / 4;
    const T* A = static_cast<const T*>(S.A) + (size_t)row * a.lcap;
    auto load = [&](int v) {
        Vec4<T> r;
        const int i = 4 * v;
#pragma unroll
        for (int c = 0; c < 4; ++c) r.x[c] = (T)0;
        if (v < nv && i < Kr) {
            const T* p = A + i;
            if (sizeof(T) == 4) {
                const float4 q = *reinterpret_cast<const float4*>(p);
                r.x[0] = q.x; r.x[1] = q.y; r.x[2] = q.z; r.x[3] = q.w;
            } else {
                const double2 q0 = *reinterpret_cast<const double2*>(p), q1 = *reinterpret_cast<const double2*>(p + 2);
                r.x[0] = q0.x; r.x[1] = q0.y; r.x[2] = q1.x; r.x[3] = q1.y;
            }
#pragma unroll
            for (int c = 0; c < 4; ++c)
                if (i + c >= Kr) r.x[c] = (T)0;
        }
        return r;
    };
    T mx = (T)0;
    int last = 0;  // one past the last nonzero order
    auto look = [&](const Vec4<T>& r, int v) {
        const int i = 4 * v;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            mx = sizeof(T) == 4 ? (T)fmaxf((float)mx, fabsf((float)r.x[c])) : (T)fmax((double)mx, fabs((double)r.x[c]));
            if (r.x[c] != (T)0) last = max(last, i + c + 1);
        }
    };
    Vec4<T> keep[NC];
#pragma unroll
    for (int t = 0; t < NC; ++t) keep[t] = load(lane + 32 * t);
#pragma unroll
    for (int t = 0; t < NC; ++t) look(keep[t], lane + 32 * t);
#pragma unroll 4
    for (int v = lane + 32 * NC; v < nv; v += 32) look(load(v), v);
    for (int o = 16; o > 0; o >>= 1) {
        const T y = __shfl_xor_sync(0xffffffffu, mx, o);
        mx = sizeof(T) == 4 ? (T)fmaxf((float)mx, (float)y) : (T)fmax((double)mx, (double)y);
    }
    last = __reduce_max_sync(0xffffffffu, last);
    const int e = piece_exp((double)mx);
    if (lane == 0) {
        S.sa[row] = __int_as_float((127 + e) << 23);
        if (S.lnz) S.lnz[row] = last;
    }
    const T down = sizeof(T) == 4 ? (T)ldexpf(1.0f, -e) : (T)scalbn(1.0, -e);  // exact: e <= 127
    uint16_t* P = S.P + (size_t)row * a.kcap;
    auto put = [&](const Vec4<T>& r, int v) {
        if (v >= nv) return;
        uint2 hi, lo;
        split2x(r.x[0] * down, r.x[1] * down, a.fmt, hi.x, lo.x);
        split2x(r.x[2] * down, r.x[3] * down, a.fmt, hi.y, lo.y);
        uint16_t* q = P + 4 * v;
        *reinterpret_cast<uint2*>(q) = hi;
        *reinterpret_cast<uint2*>(q + S.stride) = lo;
    };
#pragma unroll
    for (int t = 0; t < NC; ++t) put(keep[t], lane + 32 * t);
#pragma unroll 4
    for (int v = lane + 32 * NC; v < nv; v += 32) put(load(v), v);
}

template <class T>
void launch_split(SplitArgs& a, int nblk, cudaStream_t st) {
    // registers for the rows' usual length: FP32 rows of up to 1024 orders in
    // 8 vectors a lane, longer in 16; FP64 vectors are twice as large
    if (sizeof(T) == 4 && a.lcap > 1024) k_split_rows<T, 16><<<nblk, SPLIT_THREADS, 0, st>>>(a);
    else k_split_rows<T, 8><<<nblk, SPLIT_THREADS, 0, st>>>(a);
    DSM_CUDA(cudaGetLastError());
}

// A warp per row tile, TO_Y blocks of TO_W warps per problem.
constexpr int TO_W = 8, TO_Y = 4;
__global__ void k_tile_orders(const Problem* __restrict__ probs, int bk) {
    const Problem& P = probs[blockIdx.x];
    if (!P.kb || !P.lz) return;
    const int lane = threadIdx.x & 31, M = P.M, mtiles = (M + BM - 1) / BM;
    const int* __restrict__ lz = P.lz;
    for (int mt = blockIdx.y * TO_W + (threadIdx.x >> 5); mt < mtiles; mt += TO_Y * TO_W) {
        int last = 0;
#pragma unroll
        for (int r = mt * BM + lane; r < (mt + 1) * BM; r += 32)
            if (r < M) last = max(last, lz[r]);
        last = __reduce_max_sync(0xffffffffu, last);
        // blocks are summed in pairs from the top: a tile keeps the pairs of
        // the whole contraction, so zero blocks left out change no result
        int kb = min(P.kblocks, (last + bk - 1) / bk);
        if (kb > 0 && ((P.kblocks - kb) & 1)) ++kb;
        if (lane == 0) P.kb[mt] = kb;
    }
}

PFN_cuTensorMapEncodeTiled_v12000 encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    });
    if (!fn) throw Error(DSM_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    return fn;
}

CUtensorMapDataType dtype(int piece_fmt) {
    return piece_fmt == PIECE_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
}

void check(CUresult r, const char* what) {
    if (r != CUDA_SUCCESS) throw Error(DSM_ERR_CUDA, std::string("tensor map for ") + what + " rejected (" +
                                                         std::to_string((int)r) + ")");
}

}  // namespace

void encode_a(CUtensorMap* m, const void* base, int piece_fmt, int kcap, int rows, int nfreq, int bk) {
    if (kcap % bk) throw Error(DSM_ERR_INVALID, "order capacity of the split fields is not a multiple of BK");
    cuuint64_t dims[4] = {(cuuint64_t)kcap, (cuuint64_t)rows, (cuuint64_t)nfreq, 2};
    cuuint64_t strides[3] = {(cuuint64_t)kcap * 2, (cuuint64_t)kcap * 2 * rows, (cuuint64_t)kcap * 2 * rows * nfreq};
    cuuint32_t box[4] = {(cuuint32_t)bk, BM, 1, 1};
    cuuint32_t es[4] = {1, 1, 1, 1};
    check(encoder()(m, dtype(piece_fmt), 4, const_cast<void*>(base), dims, strides, box, es,
                    CU_TENSOR_MAP_INTERLEAVE_NONE,
                    bk == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE),
          "the split fields");
}

void encode_b(CUtensorMap* m, const void* base, int piece_fmt, int kcap, int cols, int bk) {
    if (kcap % bk) throw Error(DSM_ERR_INVALID, "order capacity of the split bases is not a multiple of BK");
    cuuint64_t dims[3] = {(cuuint64_t)kcap, (cuuint64_t)cols, 2};
    cuuint64_t strides[2] = {(cuuint64_t)kcap * 2, (cuuint64_t)kcap * 2 * cols};
    cuuint32_t box[3] = {(cuuint32_t)bk, BN, 1};
    cuuint32_t es[3] = {1, 1, 1};
    check(encoder()(m, dtype(piece_fmt), 3, const_cast<void*>(base), dims, strides, box, es,
                    CU_TENSOR_MAP_INTERLEAVE_NONE,
                    bk == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE),
          "the split bases");
}

void split_fields(const SplitRows* sets, int nsets, int in_bytes, int nf, int lcap, const int* d_nord,
                  int kcap, int F, int piece_fmt, int bk, cudaStream_t st, const int* zf, int R1) {
    if (kcap % bk || lcap % 4)
        throw Error(DSM_ERR_INVALID, "order capacity of the split fields is not a multiple of BK");
    SplitArgs a{};
    int nblk = 0;
    for (int k = 0; k < nsets; ++k) {
        const SplitRows& r = sets[k];
        if (r.rows <= 0 || nf <= 0) continue;
        a.s[a.ns++] = SplitSet{r.A, nf * r.rows, r.rows, nblk, r.P, (size_t)F * r.rows * kcap, r.sa, r.lnz, r.rowrec, r.rf};
        nblk += (nf * r.rows + SPLIT_THREADS / 32 - 1) / (SPLIT_THREADS / 32);
    }
    if (a.ns == 0) return;
    a.lcap = lcap;
    a.kcap = kcap;
    a.bk = bk;
    a.fmt = piece_fmt;
    a.R1 = R1;
    a.nord = d_nord;
    a.zf = zf;
    if (in_bytes == 4) launch_split<float>(a, nblk, st);
    else launch_split<double>(a, nblk, st);
}

void split_bases(const double* B, int cols, int lcap, uint16_t* P, float* sb, int kcap, int piece_fmt,
                 cudaStream_t st) {
    const SplitRows r{B, cols, P, sb, nullptr, nullptr, cols};
    split_fields(&r, 1, 8, 1, lcap, nullptr, kcap, 1, piece_fmt, kcap, st, nullptr, 0);
}

void tile_orders(const Problem* d_probs, int np, int bk, cudaStream_t st) {
    if (np <= 0) return;
    k_tile_orders<<<dim3(np, TO_Y), 32 * TO_W, 0, st>>>(d_probs, bk);
    DSM_CUDA(cudaGetLastError());
}

void launch(const Maps& maps, const Problem* d_probs, int np, int ntiles, int piece_fmt, int bk, uint32_t flags,
            int chunk, int* d_err, int nsm, cudaStream_t st, unsigned long long wait_ns) {
    if (np <= 0 || ntiles <= 0) return;
    if (np > MAXP) throw Error(DSM_ERR_INVALID, "too many contractions in one launch");
    // kind::f16 instruction descriptor: FP32 accumulator, both operands of
    // the piece type and order-major, N = BN, M = BM
    const uint32_t fmt = piece_fmt == PIECE_BF16 ? 1u : 0u;
    const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(BN >> 3) << 17) |
                           ((uint32_t)(BM >> 4) << 24);
    const int grid = std::min(ntiles, nsm);
    const size_t smem = SMEM_STAGES + 1024;
    // the shared-memory attribute is set on every launch: it belongs to the
    // current device, and contexts of several devices or host threads
    // launch here (a host call of about a microsecond)
    if (bk == 32) {
        DSM_CUDA(cudaFuncSetAttribute(k_lsum_tc<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        k_lsum_tc<32><<<grid, NTHREADS, smem, st>>>(maps, d_probs, np, ntiles, idesc, flags, chunk, d_err, wait_ns);
    } else if (bk == 64) {
        DSM_CUDA(cudaFuncSetAttribute(k_lsum_tc<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        k_lsum_tc<64><<<grid, NTHREADS, smem, st>>>(maps, d_probs, np, ntiles, idesc, flags, chunk, d_err, wait_ns);
    } else {
        throw Error(DSM_ERR_INVALID, "BK must be 32 or 64");
    }
    DSM_CUDA(cudaGetLastError());
}

}  // namespace tc
}  // namespace dsm
