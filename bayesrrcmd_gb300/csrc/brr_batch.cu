// Batched Gibbs sweeps of C chains on shared genotypes, with the dot products
// and the residual updates on the tensor cores (tcgen05, kind::f16).
//
// Reference semantics per chain: BayesRBase::processColumn over the dense
// kernel (src/BayesRBase.cpp:287-392, src/densebayesrkernel.cpp:10-20), every
// chain visiting the markers in one shared order (any scan order is a valid
// Gibbs sweep; the per-marker draws u, z stay per chain).
//
// Layout.  Individuals are cut into G slices (one CTA each, a multiple of 16
// individuals per slice).  Every CTA holds:
//   g   : a block's genotypes (32 markers) over its slice, FP16, [marker t][individual i]
//         in the no-swizzle K-major core-matrix layout (8 rows x 16 bytes);
//   E   : all chains' residuals over the slice as exact fixed point
//         E = eps * 2^40, four balanced 11-bit limbs per value, FP16, rows
//         r = 4*chain + limb, stored MN-major (8 consecutive rows in 16 bytes);
//   W   : a block's update coefficients, FP16 limbs, [row r][marker t].
// Tensor-core products (all partial sums are integers below 2^24, exact in FP32):
//   dots   D1[r][t] = sum_i E[r][i] * g[t][i]      (M = 128 rows per tile, N = 32)
//   update D2[i][r] = sum_t g[t][i] * W[r][t]      (M = 128 individuals, N = rows)
// The integer pair products P of every block's markers with its own and the block
// before are formed ahead of the sweep (launch_batch_pairs): they are the same for
// all chains.
//
// Two roles per CTA that meet only through L2, one block apart:
//   workers (12 warps) wait until block b is resolved, apply E_i += sum_p W_p g_p[i] -
//     sum_p C_p through D2, renormalise the limbs, then form the dot products of block
//     b + 2 and add them, as exact integers, to the global accumulators;
//   resolvers (one warp per chain) wait for the dot products of block b, which miss the
//     update of block b - 1, add that block's exact integer moves
//     sum_p W_p P[p][t] - C S_t, and resolve the 32 markers in order: lane t holds marker
//     t's num_t = sigma_t (dot_t - colmean_t * sum(E)) 2^-40 + beta_old (N-1) (FP64, then
//     a double-float pair).  A marker without effect whose num^2 lies below its
//     certified threshold stays in component 0; the others are decided one by one, in
//     FP32 with a rigorous error bound and in FP64 whenever the bound cannot certify
//     the decision, and a change moves the later markers' num by
//     dBeta sigma_p sigma_t (P[p][t] - colmean_t S_p).
//     W_p = round(dBeta sigma_p 2^40), C_p = round(dBeta sigma_p colmean_p 2^40).
// beta, component and P(component 0) are written by marker afterwards (k_batch_finish).
//
// 64 chains, N = 50,000, M = 40,000 in the burn-in, per block of 32 markers: 75k clk when
// the phases followed one another on all warps (decode and dots 12.6k, publication 9k
// with 32 sectors per atomic instruction, resolve 37k, update 18k), 27k with the roles
// apart: the workers' update 12.8k (two thirds of its instructions are the
// limbs' FP32 carries), dots 4.1k, publication 2.3k, decoding 1k.  Packed f32x2
// carries need as many instructions for the register pairs as they save (16.6k).
// Every wait is bounded (timeout -> error word, the CTAs leave, TMEM freed).
#include <cuda_fp16.h>

#include "brr_internal.h"
#include "brr_device.cuh"
#include "brr_pick.cuh"
#include "brr_stream.h"

namespace brr {
namespace {

constexpr int kBT = 512;               // threads per CTA
constexpr int kBW = kBT / 32;
constexpr int kResWarps = 4;           // warps 0-3 resolve the CTA's chains
constexpr int kWorkers = kBT - 32 * kResWarps;   // the others own the slice: dot products and residual updates
constexpr int kGroups = kWorkers / 128;          // groups of four warps (a warp reaches one quarter of TMEM's lanes)
constexpr int kTileWords = (batch_tile_bytes(kBatchMaxChains) / 16 + kWorkers - 1) / kWorkers;
constexpr int kCodeWords = 4;          // 32-bit code words of a marker block per worker thread, at most
constexpr int kTmemCols = 512;
constexpr int kCounterGap = 16;        // words between the four arrival counters
constexpr long long kLimbHalf = 1024;  // balanced limbs in [-1024, 1023]
constexpr unsigned kMinSmemPerCta = 116u * 1024u;

__device__ __forceinline__ unsigned smem_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor, no swizzle: start address, leading-dimension
// byte offset (the stride between core matrices along K) and stride-dimension
// byte offset (the stride between core matrices along M or N).
__device__ __forceinline__ uint64_t smem_desc(unsigned addr, unsigned lbo, unsigned sbo)
{
    uint64_t d = (uint64_t)((addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46;
    return d;
}

// Instruction descriptor of kind::f16 with FP16 operands and FP32 accumulation.
__device__ __forceinline__ uint32_t idesc_f16(int M, int N, bool a_mn)
{
    return (1u << 4) | ((a_mn ? 1u : 0u) << 15) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void umma_f16(unsigned d_tmem, uint64_t a, uint64_t b, uint32_t idesc, unsigned accumulate)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
                 "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
                 : "memory");
}

__device__ __forceinline__ void umma_commit(uint64_t *mbar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(mbar))
                 : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// 32 consecutive TMEM columns of this warp's 32 lanes.
__device__ __forceinline__ void tmem_ld32(unsigned taddr, float (&v)[32])
{
    uint32_t r[32];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
                 "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
                   "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]),
                   "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]),
                   "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int k = 0; k < 32; ++k)
        v[k] = __uint_as_float(r[k]);
}

__device__ __forceinline__ void mbar_init1(uint64_t *m)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(m)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ bool mbar_done(uint64_t *m, unsigned parity)
{
    unsigned ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok)
                 : "r"(smem_addr(m)), "r"(parity)
                 : "memory");
    return ok != 0;
}

__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *m, unsigned parity, uint64_t timeout_ns)
{
    if (mbar_done(m, parity))
        return true;
    const uint64_t t0 = global_timer_ns();
    unsigned spins = 0;
    while (!mbar_done(m, parity)) {
        if ((++spins & 63u) == 0 && global_timer_ns() - t0 > timeout_ns)
            return false;
    }
    return true;
}

__device__ __forceinline__ bool counter_wait(const unsigned long long *c, unsigned long long target, const int *err,
                                             uint64_t timeout_ns)
{
    if (ld_acquire_u64(c) >= target)
        return true;
    const uint64_t t0 = global_timer_ns();
    unsigned spins = 0;
    while (ld_acquire_u64(c) < target) {
        if ((++spins & 255u) == 0) {
            if (*(volatile const int *)err != kDevOk || global_timer_ns() - t0 > timeout_ns)
                return false;
        }
    }
    return true;
}

// Balanced radix-2^11 digits of x: x = sum_l d_l 2^(11 l), d_l in [-1024, 1023].
// Returns false when x needs more than four digits.
__device__ __forceinline__ bool split4(long long x, int (&d)[kBatchLimbs])
{
#pragma unroll
    for (int l = 0; l < kBatchLimbs - 1; ++l) {
        const long long r = ((x + kLimbHalf) & 2047) - kLimbHalf;
        d[l] = (int)r;
        x = (x - r) >> 11;
    }
    d[kBatchLimbs - 1] = (int)x;
    return x >= -kLimbHalf && x < kLimbHalf;
}

__device__ __forceinline__ long long join4(const int (&d)[kBatchLimbs])
{
    long long x = d[kBatchLimbs - 1];
#pragma unroll
    for (int l = kBatchLimbs - 2; l >= 0; --l)
        x = x * 2048 + d[l];
    return x;
}

// v / 2048 to the nearest integer (halves to even), of an integer-valued float
// |v| < 2^21: the carry that brings a limb into [-1024, 1024].  One FMA rounds it as
// the sum with 1.5 * 2^23, whose unit is 1.
__device__ __forceinline__ float limb_carry(float v)
{
    return __fsub_rn(__fmaf_rn(v, 1.f / 2048.f, 12582912.f), 12582912.f);
}

// Row of limb l of chain c in E, D1 and W.
__device__ __forceinline__ int limb_row(int c, int l) { return 4 * c + l; }

__device__ __forceinline__ unsigned short h_bits(int v) { return __half_as_ushort(__int2half_rn(v)); }
__device__ __forceinline__ int h_int(unsigned short b) { return __half2int_rn(__ushort_as_half(b)); }

struct BatchPlan {
    unsigned off_g, off_e, off_w, off_p, total;
    unsigned sbo_g;      // stride between 8-marker groups of g (= kext/8 * 128)
    unsigned lbo_e;      // stride between 8-individual groups of E (= R/8 * 128)
};

__host__ __device__ inline BatchPlan batch_plan(int C, int kext)
{
    BatchPlan p;
    const unsigned R = 4u * (unsigned)C;
    p.sbo_g = (unsigned)(kext / 8) * 128u;
    p.lbo_e = (R / 8u) * 128u;
    p.off_g = 0;
    p.off_e = p.off_g + 32u * (unsigned)kext * 2u;
    p.off_w = p.off_e + R * (unsigned)kext * 2u;
    p.off_p = p.off_w + (unsigned)batch_tile_bytes(C);
    p.total = p.off_p + 64u * kBatchBlock * 4u;
    p.total = (p.total + 127u) & ~127u;
    // every CTA allocates all 512 TMEM columns and waits on the others, so
    // no two CTAs may share an SM: at least half the SM's shared memory each
    if (p.total < kMinSmemPerCta)
        p.total = kMinSmemPerCta;
    return p;
}

__device__ __forceinline__ void worker_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kWorkers) : "memory"); }
__device__ __forceinline__ void resolver_sync() { asm volatile("bar.sync 2, %0;" ::"n"(32 * kResWarps) : "memory"); }

__device__ __forceinline__ long long warp_sum(long long v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// PROF: the variant that counts phase cycles on CTA 0 (the plain variant reads
// no clock, whose reads would constrain the scheduling of every CTA's code).
template <int KM, bool PROF>
__global__ void __launch_bounds__(kBT, 1) k_sweep_batch(BatchArgs a)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t s_mbar;
    __shared__ unsigned s_tmem;
    __shared__ int s_wstop[2], s_rstop[2];   // a wait ran out in block b (b & 1): workers, resolvers
    __shared__ unsigned s_moved[2];          // chains with a change in the block

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int s = blockIdx.x;
    const int C = a.C, R = 4 * C, MT = R / 128;
    const int kext = a.kext;
    const int lo = a.slice_lo[s];
    const int ns = a.slice_lo[s + 1] - lo;
    const BatchPlan pl = batch_plan(C, kext);
    uint8_t *g_t = smem + pl.off_g;
    uint8_t *e_t = smem + pl.off_e;
    const int nblocks = (int)((a.M + kBatchBlock - 1) / kBatchBlock);
    const double inv2f = 1.0 / (double)(1ll << kBatchFrac);
    // arrivals of the CTAs' dot products and of the resolved chains, for even and odd
    // blocks apart: both run up to one block ahead
    unsigned long long *cnt1 = a.counter, *cnt2 = a.counter + 2 * kCounterGap;
    long long *prof = (PROF && s == 0) ? a.prof : nullptr;
    long long ph[8] = {0, 0, 0, 0, 0, 0, 0, 0};

    if (tid == 0) {
        s_wstop[0] = s_wstop[1] = s_rstop[0] = s_rstop[1] = 0;
        mbar_init1(&s_mbar);
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&s_tmem)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }

    // ---- residuals of all chains over the slice, with the updateMu shift, as limbs
    for (int idx = tid; idx < (C / 2) * kext; idx += kBT) {
        const int i = idx % kext, cp = idx / kext;
        uint32_t w[4];
        bool ok = true;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int c = 2 * cp + h;
            long long x = 0;
            if (i < ns)
                x = a.E[(size_t)c * a.N + lo + i] + a.dmu[c];
            int d[kBatchLimbs];
            ok = split4(x, d) && ok;
            w[2 * h] = (uint32_t)h_bits(d[0]) | ((uint32_t)h_bits(d[1]) << 16);
            w[2 * h + 1] = (uint32_t)h_bits(d[2]) | ((uint32_t)h_bits(d[3]) << 16);
        }
        if (!ok)
            atomicCAS(a.err, kDevOk, kDevRange);
        *reinterpret_cast<uint4 *>(e_t + (i >> 3) * pl.lbo_e + cp * 128 + (i & 7) * 16) = make_uint4(w[0], w[1], w[2], w[3]);
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = s_tmem;

    if (warp >= kResWarps) {
        // ================= workers: dot products and residual updates of the slice
        uint8_t *w_t = smem + pl.off_w;
        const float *s_cl = reinterpret_cast<const float *>(w_t + R * 64);   // the constants' limbs, in the rows' order
        const int wt = tid - 32 * kResWarps, ww = warp - kResWarps, q4 = warp & 3, wg = ww >> 2;
        const int KS = kext / 16;                       // K steps of the dot GEMM; code words per marker
        const int NT = (kext + 127) / 128;              // individual tiles of the update GEMM
        int CW = R;                                     // rows of the update per TMEM pass
        while (NT * CW > kTmemCols)
            CW /= 2;
        const unsigned ug = smem_addr(g_t), ue = smem_addr(e_t), uw = smem_addr(w_t);
        unsigned mphase = 0;
        bool late = false;   // a tensor-core wait ran out

        // code words of block b: this thread's marker is lane, its words ww, ww + 12, ...
        auto load_codes = [&](int b, uint32_t (&w)[kCodeWords]) {
            const int64_t q = (int64_t)b * kBatchBlock + lane;
            const bool in = q < a.M;
            const uint32_t *src =
                reinterpret_cast<const uint32_t *>(a.codes + (size_t)(in ? a.order[q] : 0u) * a.col_stride + lo / 4);
#pragma unroll
            for (int k = 0; k < kCodeWords; ++k) {
                const int x = ww + k * (kWorkers / 32), left = ns - 16 * x;   // individuals of the slice in the word
                uint32_t v = 0xFFFFFFFFu;                                     // genotype 0
                if (in && left > 0) {
                    v = __ldg(src + x);
                    if (left < 16)
                        v |= 0xFFFFFFFFu << (2 * left);
                }
                w[k] = v;
            }
        };
        // the block's genotypes as FP16 (2.0, 1.0, 0.0: one byte each)
        auto decode = [&](const uint32_t (&w)[kCodeWords]) {
#pragma unroll
            for (int k = 0; k < kCodeWords; ++k) {
                const int x = ww + k * (kWorkers / 32);
                if (x < KS) {
                    uint32_t o[8];
#pragma unroll
                    for (int h = 0; h < 8; ++h) {
                        const unsigned c = (w[k] >> (4 * h)) & 15u;
                        o[h] = __byte_perm(0x003C0040u, 0u, 0x0404u | ((c & 3u) << 4) | ((c & 12u) << 10));
                    }
                    uint8_t *dst = g_t + (lane >> 3) * pl.sbo_g + x * 256 + (lane & 7) * 16;
                    *reinterpret_cast<uint4 *>(dst) = make_uint4(o[0], o[1], o[2], o[3]);
                    *reinterpret_cast<uint4 *>(dst + 128) = make_uint4(o[4], o[5], o[6], o[7]);
                }
            }
        };
        auto wait_mma = [&]() {
            if (!late && !mbar_wait_bounded(&s_mbar, mphase & 1u, a.timeout_ns)) {
                atomicCAS(a.err, kDevOk, kDevTimeout);
                late = true;
            }
            ++mphase;
            tc_fence_after();
        };
        auto before_mma = [&]() {
            fence_async_smem();
            tc_fence_before();
            worker_sync();
            tc_fence_after();
        };
        // dot products of the block in g with the residuals, added to the accumulators of block b
        auto dots = [&](int b) {
            long long t0 = prof ? clock64() : 0;
            before_mma();
            if (wt == 0) {
                // one thread issues: the descriptors move by constants (start address, 16-byte units)
                const uint32_t id_dot = idesc_f16(128, 32, true);
                for (int mt = 0; mt < MT; ++mt) {
                    uint64_t da = smem_desc(ue + mt * 2048, pl.lbo_e, 128), db = smem_desc(ug, 128, pl.sbo_g);
                    umma_f16(tmem + (unsigned)(mt * 32), da, db, id_dot, 0);
#pragma unroll 4
                    for (int ks = 1; ks < KS; ++ks) {
                        da += pl.lbo_e >> 3;
                        db += 16;
                        umma_f16(tmem + (unsigned)(mt * 32), da, db, id_dot, 1);
                    }
                }
                umma_commit(&s_mbar);
            }
            wait_mma();
            if (prof)
                ph[0] += clock64() - t0, t0 = clock64();
            // lanes 4k..4k+3 hold the limbs of one chain and leave with eight markers of it
            // each.  A warp's 32 lanes add to 32 consecutive words at a time:
            // 8 sectors of the L2 instead of 32.
            if (ww < MT * 4) {
                const int mt = ww >> 2;
                float f[32];
                tmem_ld32(tmem + ((unsigned)(q4 * 32) << 16) + (unsigned)(mt * 32), f);
                const int l = lane & 3;
                const int r = mt * 128 + q4 * 32 + lane;
                const bool up2 = (l & 2) != 0, up1 = (l & 1) != 0;
                long long k16[16];
#pragma unroll
                for (int k = 0; k < 16; ++k) {
                    const float send = up2 ? f[k] : f[k + 16], keep = up2 ? f[k + 16] : f[k];
                    const float other = __shfl_xor_sync(0xffffffffu, send, 2);
                    // limbs l and l ^ 2 of the same chain and marker
                    k16[k] = (long long)(int)keep * (1ll << (11 * l)) + (long long)(int)other * (1ll << (11 * (l ^ 2)));
                }
                unsigned long long *acc = a.acc + ((size_t)(b & 1) * kBatchCopies + s % kBatchCopies) * C * kBatchBlock + r;
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const long long send = up1 ? k16[k] : k16[k + 8];
                    const long long keep = up1 ? k16[k + 8] : k16[k];
                    const long long v = keep + __shfl_xor_sync(0xffffffffu, send, 1);
                    red_add_u64(acc + (size_t)k * R, (unsigned long long)v);
                }
            }
            tc_fence_before();
            worker_sync();
            if (wt == 0)
                red_release_add_u64(cnt1 + (b & 1) * kCounterGap, 1ull);
            if (prof)
                ph[1] += clock64() - t0;
        };

        uint32_t cur[kCodeWords], nxt[kCodeWords];
        load_codes(0, cur);
        load_codes(1, nxt);
        decode(cur);
        dots(0);
        if (nblocks > 1) {
            decode(nxt);
            dots(1);
            decode(cur);
        }
#pragma unroll
        for (int k = 0; k < kCodeWords; ++k)
            cur[k] = nxt[k];
        for (int b = 0; b < nblocks; ++b) {
            load_codes(b + 2, nxt);
            long long t0 = prof ? clock64() : 0;
            if (late)
                s_wstop[b & 1] = 1;
            if (wt == 0 && !counter_wait(cnt2 + (b & 1) * kCounterGap, (unsigned long long)C * (unsigned)(b / 2 + 1), a.err,
                                         a.timeout_ns)) {
                atomicCAS(a.err, kDevOk, kDevTimeout);
                s_wstop[b & 1] = 1;
            }
            worker_sync();   // orders the acquire before the loads below
            if (prof)
                ph[7] += clock64() - t0, t0 = clock64();
            if (s_wstop[b & 1])
                break;
            // ---- update coefficients, laid out by the resolvers as the operand tile
            const uint4 *wsrc = reinterpret_cast<const uint4 *>(a.wt + (size_t)(b & 1) * batch_tile_bytes(C));
            const int wn = batch_tile_bytes(C) / 16;
            uint4 wv[kTileWords];
#pragma unroll
            for (int k = 0; k < kTileWords; ++k)
                if (wt + k * kWorkers < wn)
                    wv[k] = __ldcg(wsrc + wt + k * kWorkers);
            if (wt < C) {
                const unsigned m = __ballot_sync(0xffffffffu, __ldcg(a.moved + (b & 1) * kBatchMaxChains + wt) != 0);
                if (lane == 0)
                    s_moved[ww] = m;
            }
#pragma unroll
            for (int k = 0; k < kTileWords; ++k)
                if (wt + k * kWorkers < wn)
                    reinterpret_cast<uint4 *>(w_t)[wt + k * kWorkers] = wv[k];
            before_mma();

            // ---- residual update D2[i][4c+l] = sum_t g[t][i] W[4c+l][t], all tiles of 128
            // individuals times CW rows (chains) per TMEM pass
            const uint32_t id_upd = idesc_f16(128, CW, true);
            float top = 0.f;   // of the highest limbs, in [-1024, 1023]
            for (int r0 = 0; r0 < R; r0 += CW) {
                if (wt == 0) {
                    for (int it = 0; it < NT; ++it)
#pragma unroll
                        for (int ks = 0; ks < 2; ++ks)
                            umma_f16(tmem + (unsigned)(it * CW),
                                     smem_desc(ug + it * 2048 + ks * 2 * pl.sbo_g, pl.sbo_g, 128),
                                     smem_desc(uw + r0 * 64 + ks * 256, 128, 512), id_upd, ks > 0);
                    umma_commit(&s_mbar);
                }
                wait_mma();
                // pieces of eight chains of a tile dealt to the groups of four warps
                int it = wg, c0 = r0 / 4;                 // tile, first chain
                for (const int ce = (r0 + CW) / 4;; it += kGroups) {
                    while (it >= NT) {
                        it -= NT;
                        c0 += 8;
                    }
                    if (c0 >= ce)
                        break;
                    const int i = it * 128 + q4 * 32 + lane;
                    if (i - lane >= ns || !((s_moved[c0 >> 5] >> (c0 & 31)) & 255u))
                        continue;
                    float f[32];
                    tmem_ld32(tmem + ((unsigned)(q4 * 32) << 16) + (unsigned)(it * CW + 4 * c0 - r0), f);
                    if (i >= ns)   // past the slice the genotypes are 0 and the constants are not
                        continue;
                    uint8_t *ep = e_t + (i >> 3) * pl.lbo_e + (c0 >> 1) * 128 + (i & 7) * 16;
                    const float4 *kp = reinterpret_cast<const float4 *>(s_cl + 4 * c0);
#pragma unroll
                    for (int half = 0; half < 2; ++half) {
                        // limbs + update - constant, renormalised with carries, all in FP32
                        // on exact integers (|values| < 2^17), four chains side by side
                        float v[4][4];
#pragma unroll
                        for (int cc = 0; cc < 4; cc += 2) {
                            const uint4 w4 = *reinterpret_cast<const uint4 *>(ep + (4 * half + cc) * 64);
                            const uint32_t w[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
                            for (int x = 0; x < 4; ++x) {
                                const float2 e2 = __half22float2(*reinterpret_cast<const __half2 *>(&w[x]));
                                const float4 k4 = kp[4 * half + cc + (x >> 1)];
                                const float *d = &f[16 * half + 4 * cc + 2 * x];
                                v[cc + (x >> 1)][2 * (x & 1)] = __fsub_rn(__fadd_rn(e2.x, d[0]), (x & 1) ? k4.z : k4.x);
                                v[cc + (x >> 1)][2 * (x & 1) + 1] = __fsub_rn(__fadd_rn(e2.y, d[1]), (x & 1) ? k4.w : k4.y);
                            }
                        }
#pragma unroll
                        for (int l = 0; l < 3; ++l)
#pragma unroll
                            for (int cc = 0; cc < 4; ++cc) {
                                const float k = limb_carry(v[cc][l]);
                                v[cc][l] = __fmaf_rn(-2048.f, k, v[cc][l]);
                                v[cc][l + 1] = __fadd_rn(v[cc][l + 1], k);
                            }
#pragma unroll
                        for (int cc = 0; cc < 4; cc += 2) {
                            uint32_t w[4];
#pragma unroll
                            for (int x = 0; x < 4; ++x) {
                                const __half2 n2 =
                                    __floats2half2_rn(v[cc + (x >> 1)][2 * (x & 1)], v[cc + (x >> 1)][2 * (x & 1) + 1]);
                                w[x] = *reinterpret_cast<const uint32_t *>(&n2);
                            }
                            top = fmaxf(top, fmaxf(fabsf(v[cc][3] + 0.5f), fabsf(v[cc + 1][3] + 0.5f)));
                            *reinterpret_cast<uint4 *>(ep + (4 * half + cc) * 64) = make_uint4(w[0], w[1], w[2], w[3]);
                        }
                    }
                }
                if (r0 + CW < R) {   // the next pass overwrites the accumulators
                    tc_fence_before();
                    worker_sync();
                    tc_fence_after();
                }
            }
            if (!(top <= 1023.5f))
                atomicCAS(a.err, kDevOk, kDevRange);
            if (prof)
                ph[3] += clock64() - t0;
            if (b + 2 < nblocks) {
                decode(nxt);
                dots(b + 2);
            }
            if (b + 1 < nblocks)
                decode(cur);
#pragma unroll
            for (int k = 0; k < kCodeWords; ++k)
                cur[k] = nxt[k];
        }
    } else if (s < C) {
        // ================= resolvers: one warp per chain, lane t holds marker t of the block
        int *s_p = reinterpret_cast<int *>(smem + pl.off_p);   // [64][32]: rows of the last block, then of this one
        const int nk = (C - s - a.G * warp + kResWarps * a.G - 1) / (kResWarps * a.G);   // chains of this warp
        // pair products of the markers of block b with those of blocks b - 1 and b
        auto load_pairs = [&](int b) {
            const int *src = a.pairs[b == 0 ? 0 : (b & 1) ^ 1] + (size_t)(b == 0 ? 0 : (b - 1) >> 1) * 4096;
            for (int idx = tid; idx < 64 * 8; idx += 32 * kResWarps) {
                const int row = idx >> 3, x = (idx & 7) * 4;
                if (b > 0)
                    cp_async16(s_p + row * 32 + x, src + row * 64 + 32 + x);
                else if (row >= 32)
                    cp_async16(s_p + row * 32 + x, src + (row - 32) * 64 + x);
            }
            cp_async_commit();
        };
        long long Wl = 0, Csum = 0, sumE = 0;
        for (int b = 0; b < nblocks; ++b) {
            load_pairs(b);
            for (int k = 0; k < nk || k == 0; ++k) {
                const int c = s + a.G * (warp + kResWarps * k);
                const int64_t q = (int64_t)b * kBatchBlock + lane;
                const bool in = q < a.M && nk > 0;
                BatchRec rc{};
                ChainRec cr{};
                cr.s0 = INFINITY;
                if (in) {
                    rc = a.rec[q];
                    cr = a.crec[(size_t)c * a.M + q];
                }
                if (nk > 0 && (nk > 1 || b == 0)) {
                    const long long *st = a.wx + (size_t)c * (kBatchBlock + 1);
                    Wl = b ? st[lane] : 0;
                    Csum = b ? st[kBatchBlock] : 0;
                    sumE = a.sumE[c];
                }
                const double base = fma(rc.sB, (double)sumE, cr.bN1);
                const long long Si = rc.S;
                const float Sf = (float)rc.S;
                if (k == 0) {
                    // every CTA's dot products, and the pair products
                    const long long tw = prof ? clock64() : 0;
                    if (lane == 0 && !counter_wait(cnt1 + (b & 1) * kCounterGap,
                                                   (unsigned long long)(a.G + a.phantom) * (unsigned)(b / 2 + 1), a.err,
                                                   a.timeout_ns)) {
                        atomicCAS(a.err, kDevOk, kDevTimeout);
                        s_rstop[b & 1] = 1;
                    }
                    cp_async_wait_all();
                    resolver_sync();
                    if (prof)
                        ph[4] += clock64() - tw;
                    if (s_rstop[b & 1])
                        break;
                }
                if (nk == 0)
                    break;
                const long long tl = prof ? clock64() : 0;
                long long dot = 0;
                unsigned long long *acc = a.acc + (size_t)(b & 1) * kBatchCopies * C * kBatchBlock +
                                          (size_t)(lane & 7) * R + limb_row(c, lane >> 3);
#pragma unroll
                for (int cp = 0; cp < kBatchCopies; ++cp)
                    dot += (long long)ld_relaxed_u64(acc + (size_t)cp * C * kBatchBlock);
#pragma unroll
                for (int cp = 0; cp < kBatchCopies; ++cp)
                    acc[(size_t)cp * C * kBatchBlock] = 0ull;
                // the dots were formed before the last block's update: its exact integer moves
                for (unsigned m = __ballot_sync(0xffffffffu, Wl != 0); m; m &= m - 1u) {
                    const int p = __ffs(m) - 1;
                    dot += __shfl_sync(0xffffffffu, Wl, p) * (long long)s_p[p * 32 + lane];
                }
                dot -= Csum * Si;
                // num from the exact integer dot and residual total, in FP64; then carried
                // as a double-float pair through the block's changes: after marker p
                // changes, num_t moves by dBeta_p x_p.x_t = dBeta_p sigma_p sigma_t (P[p][t] - colmean_t S_p)
                float nh, nl;
                df_from_double(fma(rc.sA, (double)dot, base), nh, nl);
                float sx = num_sq(nh, nl);
                const size_t crow = (size_t)c * a.n_groups;
                float bnh = 0.f, bnl = 0.f, uh = 0.f, ul = 0.f;
                int fcomp = 0, steps = 0;
                int grp = 0, K = a.gK[0];
                float2 fk = reinterpret_cast<const float2 *>(a.gcf + crow * kMaxK * 2)[lane & (kMaxK - 1)];
                // A marker may change when its old effect is not zero or num^2 is past the range
                // where component 0 is certain; only those are worked out, in order
                for (int pos = 0; pos < 32; ++steps) {
                    const unsigned m = __ballot_sync(0xffffffffu, lane >= pos && sx > cr.s0);
                    if (!m)
                        break;
                    const int p = __ffs(m) - 1;
                    pos = p + 1;
                    // r = P - colmean_t S_p, g = sigma_t r, ahead of the decision
                    const float Sp = __shfl_sync(0xffffffffu, Sf, p);
                    const float qh = __fmul_rn(rc.mh, Sp);
                    const float ql = __fmaf_rn(rc.ml, Sp, __fmaf_rn(rc.mh, Sp, -qh));
                    float rh = (float)s_p[(32 + p) * 32 + lane], rl = 0.f, gh, gl;
                    df_add(rh, rl, -qh, -ql);
                    df_mul(rc.sh, rc.sl, rh, rl, gh, gl);
                    if (a.n_groups > 1) {
                        grp = __shfl_sync(0xffffffffu, rc.group, p);
                        K = a.gK[grp];
                        fk = reinterpret_cast<const float2 *>(a.gcf + (crow + grp) * kMaxK * 2)[lane & (kMaxK - 1)];
                    }
                    int comp = pick_lanes<KM>(lane, __shfl_sync(0xffffffffu, sx, p), __shfl_sync(0xffffffffu, cr.uf, p),
                                              fk, K);
                    bool fbd = false;   // decided by the FP64 sampler
                    double fb_beta = 0.0;
                    if (comp == -2) {
                        // 700 guards possibly active or u near a boundary
                        if (lane == p) {
                            float w;
                            const float *gcf = a.gcf + (crow + grp) * kMaxK * 2;
                            if (!pick_margin<KM>(sx, cr.uf, gcf, K, comp, w) && !pick_f32<KM>(nh, nl, cr.uf, gcf, K, comp, w)) {
                                const Pick pk = pick_marker<false, KM>((double)nh + (double)nl, cr.u, cr.z, 0.0,
                                                                       a.gconst + (crow + grp) * kMaxK * 4, K);
                                comp = pk.comp;
                                fb_beta = pk.beta;
                                fbd = true;
                            }
                        }
                        comp = __shfl_sync(0xffffffffu, comp, p);
                    }
                    if (lane == p)
                        fcomp = comp;
                    if (comp <= 0 && __shfl_sync(0xffffffffu, cr.s0, p) != kHasEffect)
                        continue;
                    // the new effect and dBeta sigma_p, on marker p's lane
                    float ah = 0.f, al = 0.f;
                    if (comp > 0) {
                        const float4 k4 = a.gdf[(crow + grp) * kMaxK + comp];   // {sdk hi, lo, invden hi, lo}
                        float xh, xl;
                        df_mul(cr.zh, cr.zl, k4.x, k4.y, ah, al);
                        df_mul(nh, nl, k4.z, k4.w, xh, xl);
                        df_add(ah, al, xh, xl);
                        if (fbd)
                            df_from_double(fb_beta, ah, al);
                    } else if (comp < 0) {
                        ah = cr.boh;
                        al = cr.bol;
                    }
                    float dh = cr.boh, dl = cr.bol, vh, vl;
                    df_add(dh, dl, -ah, -al);
                    df_mul(dh, dl, rc.sh, rc.sl, vh, vl);
                    if (lane == p) {
                        bnh = ah;
                        bnl = al;
                        uh = vh;
                        ul = vl;
                    }
                    vh = __shfl_sync(0xffffffffu, vh, p);
                    vl = __shfl_sync(0xffffffffu, vl, p);
                    if (lane > p) {
                        float xh, xl;
                        df_mul(vh, vl, gh, gl, xh, xl);
                        df_add(nh, nl, xh, xl);
                        sx = num_sq(nh, nl);
                    }
                }
                // exact fixed-point coefficients W = round(dBeta sigma 2^40) and
                // round(dBeta sigma colmean 2^40) of the changed markers
                const float two40 = (float)(1ll << kBatchFrac);
                float ch, cl;
                df_mul(uh, ul, rc.mh, rc.ml, ch, cl);
                Wl = __float2ll_rn(__fmul_rn(uh, two40)) + __float2ll_rn(__fmul_rn(ul, two40));
                const long long Cl = __float2ll_rn(__fmul_rn(ch, two40)) + __float2ll_rn(__fmul_rn(cl, two40));
                int d[kBatchLimbs];
                bool ok = split4(Wl, d);
                uint8_t *tile = a.wt + (size_t)(b & 1) * batch_tile_bytes(C);
#pragma unroll
                for (int l = 0; l < kBatchLimbs; ++l) {
                    const int n = limb_row(c, l);
                    *reinterpret_cast<unsigned short *>(tile + (n >> 3) * 512 + (lane >> 3) * 128 + (n & 7) * 16 +
                                                        (lane & 7) * 2) = h_bits(d[l]);
                }
                const bool moved = __any_sync(0xffffffffu, Wl != 0 || Cl != 0);
                Csum = 0;
                if (moved)
                    Csum = warp_sum(Cl);
                ok = split4(Csum, d) && ok;
                if (lane == 0) {
#pragma unroll
                    for (int l = 0; l < kBatchLimbs; ++l)
                        *reinterpret_cast<float *>(tile + R * 64 + 4 * limb_row(c, l)) = (float)d[l];
                    a.moved[(b & 1) * kBatchMaxChains + c] = moved ? 1 : 0;
                }
                if (!ok)
                    atomicCAS(a.err, kDevOk, kDevRange);
                __syncwarp();
                if (lane == 0)
                    red_release_add_u64(cnt2 + (b & 1) * kCounterGap, 1ull);
                // ---- off the chain: the residual total, what the outputs are made from, the
                // state of several chains
                if (moved)
                    sumE += warp_sum(Wl * Si - (long long)a.N * Cl);
                if (in) {
                    const size_t at = (size_t)c * a.M + q;
                    a.pos[at] = make_float4(nh, nl, bnh, bnl);
                    a.pcomp[at] = (signed char)fcomp;
                }
                if (nk > 1) {
                    long long *st = a.wx + (size_t)c * (kBatchBlock + 1);
                    st[lane] = Wl;
                    if (lane == 0) {
                        st[kBatchBlock] = Csum;
                        a.sumE[c] = sumE;
                    }
                } else if (b == nblocks - 1 && lane == 0) {
                    a.sumE[c] = sumE;
                }
                if (prof) {
                    ph[5] += clock64() - tl;
                    ph[6] += steps;
                }
            }
            if (s_rstop[b & 1])
                break;
            resolver_sync();   // the pair products are read
        }
    }
    if (prof && (tid == 0 || tid == 32 * kResWarps)) {
        // workers: dots, publication, update, wait for the resolvers; resolvers: the others
        for (int k = 0; k < 8; ++k)
            if ((k < 2 || k == 3 || k == 7) == (tid != 0))
                prof[k] = k == 2 ? ph[4] + ph[5] : ph[k];
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();

    // ---- residuals back to HBM; per-slice sum(E) and sum(eps^2) per chain, a warp per pair of chains.
    // The squares are summed in the order that does not depend on who sums: eight
    // groups of 32 individuals apart by 256, a butterfly per group, the groups in turn.
    for (int cp = warp; cp < C / 2; cp += kBW) {
        long long se[2] = {0, 0};
        double total[2] = {0.0, 0.0};
        for (int g = 0; g < 8; ++g) {
            double sq[2] = {0.0, 0.0};
            for (int i = 32 * g + lane; i < ns; i += 256) {
                const uint4 w4 = *reinterpret_cast<const uint4 *>(e_t + (i >> 3) * pl.lbo_e + cp * 128 + (i & 7) * 16);
                const uint32_t w[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    int d[kBatchLimbs];
#pragma unroll
                    for (int l = 0; l < kBatchLimbs; ++l)
                        d[l] = h_int((unsigned short)(w[2 * h + (l >> 1)] >> (16 * (l & 1))));
                    const long long x = join4(d);
                    a.E[(size_t)(2 * cp + h) * a.N + lo + i] = x;
                    se[h] += x;
                    const double e = (double)x * inv2f;
                    sq[h] = fma(e, e, sq[h]);
                }
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1)
                    sq[h] += __shfl_xor_sync(0xffffffffu, sq[h], o);
                total[h] += sq[h];
            }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            se[h] = warp_sum(se[h]);
            if (lane == 0) {
                double *pp = a.part + ((size_t)s * C + 2 * cp + h) * 2;
                pp[0] = __longlong_as_double(se[h]);
                pp[1] = total[h];
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
}

// One thread per chain and sweep position: the marker's draws, the words of its old
// effect and draw that the resolve works with, and the threshold below which it is certain
// to stay in component 0.
template <int KM>
__global__ void __launch_bounds__(256) k_batch_draws(uint32_t seed, uint32_t chain0, uint32_t it, int64_t M, int64_t N,
                                                     const uint32_t *__restrict__ order,
                                                     const double *__restrict__ beta, const int32_t *__restrict__ group,
                                                     int n_groups, const double *__restrict__ gconst,
                                                     const int32_t *__restrict__ gK, ChainRec *__restrict__ crec)
{
    const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int c = blockIdx.y;
    if (q >= M)
        return;
    const uint32_t j = order[q];
    ChainRec r;
    marker_draws(StreamKey{seed, chain0 + (uint32_t)c}, it, j, &r.u, &r.z);
    const double bold = beta[(size_t)c * M + j];
    const int g = group[j];
    r.bN1 = bold * ((double)N - 1.0);
    df_from_double(bold, r.boh, r.bol);
    df_from_double(r.z, r.zh, r.zl);
    r.uf = __double2float_rn(r.u);
    r.s0 = bold != 0.0 ? kHasEffect
                       : certain_zero<KM>(r.uf, gconst + ((size_t)c * n_groups + g) * kMaxK * 4, gK[g]);
    crec[(size_t)c * M + q] = r;
}

__global__ void k_batch_gather(const uint32_t *__restrict__ order, int64_t M, const double *__restrict__ scale,
                               const int64_t *__restrict__ counts, const int32_t *__restrict__ group,
                               BatchRec *__restrict__ rec)
{
    const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= M)
        return;
    const uint32_t j = order[q];
    const double sigma = scale[2 * j], colmean = scale[2 * j + 1], inv2f = 1.0 / (double)(1ll << kBatchFrac);
    BatchRec r;
    r.sA = sigma * inv2f;
    r.sB = -sigma * colmean * inv2f;
    df_from_double(sigma, r.sh, r.sl);
    df_from_double(colmean, r.mh, r.ml);
    r.S = (int32_t)(counts[4 * (size_t)j + 1] + 2 * counts[4 * (size_t)j + 2]);
    r.group = group[j];
    r.j = j;
    r.pad = 0;
    rec[q] = r;
}

// Per chain: beta, component and P(component 0) by marker from the resolve's records
// by sweep position, component counts per group and the exact fixed-point sum of the
// squared non-zero betas per group over the markers whose component was drawn
// (src/BayesRBase.cpp:200-202, :348-366).  P(component 0) is the FP32 sampler's where
// that one could certify the decision, else the FP64 one's.  A sweep that ended with a
// status has not written all of pos and pcomp: the chains keep what they had.
template <int KM>
__global__ void __launch_bounds__(256) k_batch_finish(int64_t M, const int *__restrict__ err,
                                                      const BatchRec *__restrict__ rec,
                                                      const ChainRec *__restrict__ crec, const float4 *__restrict__ pos,
                                                      const signed char *__restrict__ pcomp, int n_groups,
                                                      const double *__restrict__ gconst, const float *__restrict__ gcf,
                                                      const int32_t *__restrict__ gK, double *__restrict__ beta,
                                                      double *__restrict__ acum, int32_t *__restrict__ comp,
                                                      unsigned long long *__restrict__ out)
{
    __shared__ unsigned long long sv[kMaxGroups * kMaxK];
    __shared__ unsigned long long sb[kMaxGroups][2];
    if (*err != kDevOk)
        return;
    const int c = blockIdx.y;
    unsigned long long *o = out + (size_t)c * (n_groups * kMaxK + 2 * n_groups);
    for (int i = threadIdx.x; i < n_groups * kMaxK; i += blockDim.x)
        sv[i] = 0ull;
    for (int i = threadIdx.x; i < n_groups; i += blockDim.x)
        sb[i][0] = sb[i][1] = 0ull;
    __syncthreads();
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < M; q += (int64_t)gridDim.x * blockDim.x) {
        const size_t at = (size_t)c * M + q;
        const uint32_t j = rec[q].j;
        const int g = rec[q].group, k = pcomp[at], K = gK[g];
        const float4 v = pos[at];
        const size_t crow = (size_t)c * n_groups + g, cj = (size_t)c * M + j;
        const float uf = crec[at].uf;
        const float *f = gcf + crow * kMaxK * 2;
        float a0, w;
        int c2;
        const bool cert = pick_margin<KM>(num_sq(v.x, v.y), uf, f, K, c2, w);
        const bool guarded = pick_f32<KM>(v.x, v.y, uf, f, K, c2, a0);
        acum[cj] = cert || guarded ? (double)a0
                                   : pick_marker<false, KM>((double)v.x + (double)v.y, crec[at].u, 0.0, 0.0,
                                                            gconst + crow * kMaxK * 4, K).acum0;
        if (k < 0)
            continue;   // no component chosen: the marker keeps its state
        const double bn = k == 0 ? 0.0 : (double)v.z + (double)v.w;
        beta[cj] = bn;
        comp[cj] = k;
        atomicAdd(&sv[g * kMaxK + k], 1ull);
        if (k >= 1) {
            __int128 x;
            fx_from_double(bn * bn, x);
            const Fx fx = fx_split(x);
            atomicAdd(&sb[g][0], (unsigned long long)fx.hi);
            atomicAdd(&sb[g][1], fx.lo);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n_groups * kMaxK; i += blockDim.x)
        if (sv[i])
            atomicAdd(&o[i], sv[i]);
    for (int i = threadIdx.x; i < n_groups; i += blockDim.x) {
        atomicAdd(&o[n_groups * kMaxK + 2 * i], sb[i][0]);
        atomicAdd(&o[n_groups * kMaxK + 2 * i + 1], sb[i][1]);
    }
}

template <int KM>
cudaError_t launch_batch_km(const BatchArgs &a, cudaStream_t st)
{
    const size_t smem = batch_smem_bytes(a.C, a.kext);
    const void *f = a.prof ? (const void *)k_sweep_batch<KM, true> : (const void *)k_sweep_batch<KM, false>;
    cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess)
        return e;
    BatchArgs args = a;
    void *params[] = {&args};
    return cudaLaunchCooperativeKernel(f, dim3((unsigned)a.G), dim3(kBT), params, smem, st);
}

}  // namespace

size_t batch_smem_bytes(int C, int kext) { return batch_plan(C, kext).total; }

int batch_max_ctas_per_sm(int C, int kext, size_t smem)
{
    if (kext / 16 > kCodeWords * (kWorkers / 32))
        return 0;   // a worker's code words
    int n = 1 << 30;
    const void *fs[4] = {(const void *)k_sweep_batch<4, false>, (const void *)k_sweep_batch<16, false>,
                         (const void *)k_sweep_batch<4, true>, (const void *)k_sweep_batch<16, true>};
    for (const void *f : fs) {
        int m = 0;
        if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&m, f, kBT, smem) != cudaSuccess) {
            cudaGetLastError();
            return 0;
        }
        n = m < n ? m : n;
    }
    (void)C;
    return n;
}

cudaError_t launch_batch_gather(const uint32_t *order, int64_t M, const double *scale, const int64_t *counts,
                                const int32_t *group, BatchRec *rec, cudaStream_t st)
{
    k_batch_gather<<<(unsigned)((M + 255) / 256), 256, 0, st>>>(order, M, scale, counts, group, rec);
    return cudaGetLastError();
}

cudaError_t launch_batch_draws(uint32_t seed, uint32_t chain0, uint32_t it, const BatchArgs &a, int kmax,
                               const int32_t *group, ChainRec *crec, cudaStream_t st)
{
    const dim3 grid((unsigned)((a.M + 255) / 256), (unsigned)a.C);
    if (kmax <= 4)
        k_batch_draws<4><<<grid, 256, 0, st>>>(seed, chain0, it, a.M, a.N, a.order, a.beta, group, a.n_groups, a.gconst,
                                               a.gK, crec);
    else
        k_batch_draws<kMaxK><<<grid, 256, 0, st>>>(seed, chain0, it, a.M, a.N, a.order, a.beta, group, a.n_groups,
                                                   a.gconst, a.gK, crec);
    return cudaGetLastError();
}

cudaError_t launch_batch_finish(const BatchArgs &a, int kmax, unsigned long long *out, cudaStream_t st)
{
    const dim3 grid((unsigned)((a.M + 255) / 256 < 64 ? (a.M + 255) / 256 : 64), (unsigned)a.C);
    auto go = [&](auto f) {
        f<<<grid, 256, 0, st>>>(a.M, a.err, a.rec, a.crec, a.pos, a.pcomp, a.n_groups, a.gconst, a.gcf, a.gK, a.beta, a.acum,
                                a.comp, out);
    };
    if (kmax <= 4)
        go(k_batch_finish<4>);
    else if (kmax <= 8)
        go(k_batch_finish<8>);
    else
        go(k_batch_finish<kMaxK>);
    return cudaGetLastError();
}

cudaError_t launch_sweep_batch(const BatchArgs &a, int kmax, cudaStream_t st)
{
    if (kmax <= 4)
        return launch_batch_km<4>(a, st);
    if (kmax <= 8)
        return launch_batch_km<8>(a, st);
    return launch_batch_km<16>(a, st);
}

}  // namespace brr
