// Whole-round Gibbs sweep (sm_103a): every round resolves all its markers.
//
// Replaces BayesRBase::processColumn (src/BayesRBase.cpp:287-392) driven once
// per marker by AnalysisGraph::exec (src/sequential.cpp:23-26,
// src/limitsequencegraph.cpp:46-55) for dense (src/densebayesrkernel.cpp:10-20),
// ragged (src/raggedbayesrkernel.cpp:10-35, src/SparseBayesRRG.cpp:76-92) and
// Eigen markers (src/eigenbayesrkernel.cpp:10-20), in both sweep forms and for
// the asynchronous schedule (src/BayesRBase.cpp:394-524).
//
// What bounds a sweep is its chain: marker t's draw needs the residual left by
// marker t - 1.  The restart sweep (brr_sweep.cu) ends a round at the first
// marker that changes the residual; here a round of B markers is resolved
// whole, because marker p's change dBeta moves the later markers' num by
// dBeta G[p][t], and G, the markers' products with each other, does not depend on
// the residual: k_pair_sums forms its exact integer sums for all rounds of a
// sweep before the sweep starts.
//
// Residual.  Each CTA owns a slice of individuals.  Its residual is exact fixed
// point E = eps 2^s (int64; s from the largest |eps| at the sweep start, 3 bits
// of headroom below 2^62), so sums do not depend on their order and an update
// adds the nearest integer of dBeta x 2^s.  The grid is one for all individuals,
// where a stored value (FP64, or a pair of FP32 words) has a spacing of its own, so
// it has to be no coarser than the spacing at a typical value, the mean of |eps|:
// 2^-s <= 2^(floor(log2 mean) - 53) in the FP64 form, 2^(... - 49) in the FP32C form.
// With normal residuals of variance 1 the largest of 100,000 is 4.5, 2^-s is 2^-56 and
// 2^-54 would do; one bit of headroom instead of three allows for a largest |eps| of
// 128 to 256 means (FP32C: 2,048 to 4,096).  Where no grid is fine enough (an outlier further out, values that
// are not finite), and where a value outgrows the headroom during the sweep, the
// sweep ends with the range status and the host runs the restart sweep instead; the
// residual in memory is only replaced by a sweep that ended well.
//
// Dot products run on the tensor cores: E in seven balanced 10-bit limbs stored
// as FP16 planes (|limb| <= 512) times the genotypes 0, 1, 2 in FP16 with FP32
// accumulation; every partial sum is an integer below 2^24, so they are exact.
// FP64 arithmetic would bound a round (two FP64 operations per SM clock: 64
// markers x 660 individuals take 21k clocks); the 176 mma.sync of the same
// block take about 0.4k.  mma.sync and not tcgen05: the tile is 64 markers x 8
// limb columns x one slice, far below a tcgen05 tile, and its operands are
// decoded in registers straight from the 2-bit codes.
//
// Exchange: the partial sums of a round as two 64-bit integers per marker, added
// in L2 with the count of arrivals in their top byte (no barrier), or stored into
// the other CTAs' shared memory of one thread-block cluster (k_round_cl).
//
// Sampling: one warp walks the chain, markers t and 32 + t on lane t, identically
// in every CTA, and only decides components, by the certified FP32 samplers of
// brr_pick.cuh (FP64 where they cannot certify); num, beta and the corrections
// are FP64, on a warp that follows it.  P(component 0) is left to k_round_finish,
// one thread per marker over the whole GPU, from the stored num.
#include "brr_cluster.cuh"
#include "brr_device.cuh"
#include "brr_internal.h"
#include "brr_mma.cuh"
#include "brr_pick.cuh"

namespace brr {

namespace {

constexpr int kRT = 512;                 // threads per CTA
constexpr int kRW = kRT / 32;
// Accumulators in L2: two alternating buffers of up to kAccCopies copies, each
// four rows (low and high word of the markers' sums and of their sums over the
// missing genotypes) of 65 words (64 markers and the slice totals) in 72.  A row is
// contiguous so that a warp's reductions touch 8 sectors; CTA s adds into copy
// s mod copies, because the reductions on one sector serialise.
//
// The words count their own arrivals: a CTA adds 2^56 + bias + value, with every
// round's biased sum below 2^56, and a reader that knows the word's last complete
// value waits until the difference carries the expected count in its top
// byte.  So the sums need neither a barrier counter (whose release would wait for
// the sums to reach L2, an arrival and a poll more: 2.5k clocks of a round) nor
// clearing.  Two buffers are enough: a CTA publishes round r + 2 after it has read
// round r + 1, to which every CTA has contributed after reading round r.
constexpr int kAccRow = 72;
constexpr int kAccCopies = 2;
constexpr int kAccCopyWords = 4 * kAccRow;
constexpr int kRoundAccStride = kAccCopies * kAccCopyWords;
constexpr int kCountShift = 56;
constexpr unsigned long long kAccBias = 1ull << 47;   // |value| < 2^47 of one CTA, 255 CTAs below 2^56
constexpr unsigned long long kAccMask = (1ull << kCountShift) - 1;
constexpr long long kLow30 = (1ll << 30) - 1;
constexpr long long kNoChange = 0x7FF8000000000001ll;   // a NaN that no arithmetic returns

struct RoundPlan {
    size_t E, planes, codes, rec, gram, ids, part, gconst, gk, gcf, gdf, xch, prev, total;
    int plane_stride;                    // bytes
    int code_stride;                     // bytes of one ring slot: an odd number of 16-byte chunks
};

__host__ __device__ inline size_t al16(size_t x) { return (x + 15) & ~(size_t)15; }

// 16-byte words of one CTA's exchange record in a cluster: the markers' sums and
// the slice total, then the sums over the missing genotypes.
__host__ __device__ inline int xch_words(int B) { return 2 * (B < 16 ? 16 : B) + 1; }

// Packed upper triangle of a round's pair products: row p holds t = p+1 .. B-1.
__host__ __device__ inline int gram_entries_per_block(int B) { return B * (B - 1) / 2; }

__host__ __device__ inline RoundPlan round_plan(int slice_max, int B, int n_groups, int cluster, bool pairs,
                                                bool missing)
{
    RoundPlan p;
    const int chunks = slice_max / kChunk;
    p.plane_stride = limb_plane_stride(slice_max);
    p.code_stride = 16 * (chunks | 1);
    const int B16 = B < 16 ? 16 : B;
    size_t o = 0;
    p.E = o;
    o += (size_t)8 * slice_max;
    p.planes = o;
    o += al16((size_t)kLimbPlanes * p.plane_stride);
    p.codes = o;
    o += (size_t)2 * B16 * p.code_stride;
    p.rec = o;
    o += (size_t)2 * B16 * sizeof(RoundRec);
    p.gram = o;
    if (pairs)
        o += (size_t)2 * al16((size_t)8 * gram_entries_per_block(B16));
    p.ids = o;
    o += al16((size_t)4 * B16 * 4);
    p.part = o;
    o += (size_t)kRW * 16 * 8 * 4 * (missing ? 2 : 1);
    p.gconst = o;
    o += al16((size_t)n_groups * kMaxK * 4 * sizeof(double));
    p.gk = o;
    o += al16((size_t)n_groups * sizeof(int32_t));
    p.gcf = o;
    o += al16((size_t)n_groups * kMaxK * 2 * sizeof(float));
    p.gdf = o;
    o += (size_t)n_groups * kMaxK * sizeof(float4);
    p.xch = o;
    o += (size_t)2 * cluster * xch_words(B) * 16;
    p.prev = o;
    if (!cluster)
        o += (size_t)2 * kAccCopyWords * kAccCopies * sizeof(unsigned long long);
    p.total = al16(o);
    return p;
}

__device__ __forceinline__ double pow2d(int e) { return __longlong_as_double((long long)(1023 + e) << 52); }

// A double as a float pair h + l (h truncated, l the next 24 bits) with integer
// operations: the FP64 pipe takes 64 clocks per warp instruction, and a
// conversion through it four of them.
__device__ __forceinline__ void split_double(double v, float &h, float &l)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    const int e = (int)((b >> 52) & 0x7FF);
    const unsigned sign = (unsigned)(b >> 32) & 0x80000000u;
    if (e < 960) {   // below 2^-63: as zero
        h = l = 0.f;
        return;
    }
    h = __uint_as_float(sign | ((unsigned)(e - 896) << 23) | ((unsigned)(b >> 29) & 0x7FFFFFu));
    l = __uint2float_rn((unsigned)b & 0x1FFFFFFFu) * __uint_as_float(sign | ((unsigned)(e - 948) << 23));
}

// v as the FP32 value next to it towards zero, by integer operations (an FP64
// instruction takes 64 clocks); below 2^-126 zero.
__device__ __forceinline__ float double_hi(double v)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    const unsigned top = (unsigned)(b >> 32);
    return (top & 0x7FF00000u) < (897u << 20)
               ? 0.f
               : __uint_as_float((top & 0x80000000u) | (((unsigned)(b >> 29) + 0x40000000u) & 0x7FFFFFFFu));
}

__device__ __forceinline__ bool nonzero(double v) { return ((unsigned long long)__double_as_longlong(v) << 1) != 0ull; }

// The guarded FP32 sampler's decision on num as a pair of FP32 words, -2 where it cannot
// certify one.
template <int KM>
__device__ __noinline__ int decide_pair(float nh, float nl, float uf, const float *gcf, int K)
{
    int comp;
    float a0;
    return pick_f32<KM>(nh, nl, uf, gcf, K, comp, a0) ? comp : -2;
}

// A decision the margin sampler cannot certify: the guarded FP32 sampler, else
// FP64 on the marker's FP64 num (a pair of FP32 words holds 48 bits of it, which
// moves P(component 0) by up to 1e-12 of itself).  Out of line: about one marker in a
// thousand.
template <int KM>
__device__ __noinline__ int decide_slow(double num, double u, const double *gc, const float *gcf, int K)
{
    float nh, nl, a0;
    int comp;
    df_from_double(num, nh, nl);
    if (!pick_f32<KM>(nh, nl, __double2float_rn(u), gcf, K, comp, a0))
        comp = pick_marker<true, KM>(num, u, 0.0, 0.0, gc, K).comp;
    return comp;
}

// A question to the FP64 warp and its answer.  Out of line with decide_slow: an inlined
// load that orders others made the chain's loop 4 % slower on 2,000 x 5,000.
__device__ __noinline__ double ask_fp64_warp(volatile int *ask, const volatile double *told, int question, int *err)
{
    *ask = question;
    unsigned spins = 0;
    while (*ask != 0 && ++spins < (1u << 28))
        ;
    if (ld_acquire_shared(ask) != 0u)   // orders the answer after the word
        atomicCAS(err, kDevOk, kDevTimeout);
    return *told;
}

// --------------------------------------------------------------------------
// The sweep of one chain over its G CTAs; sidx is this CTA's slice.
template <int KM, bool PROF, bool CL>
__device__ __forceinline__ void round_body(const SweepArgs &a, const int sidx)
{
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ double s_num[kMaxSpec];
    __shared__ double s_beta[kMaxSpec];
    __shared__ int s_comp[kMaxSpec];
    __shared__ float2 s_ndf[kMaxSpec];    // num as a float pair
    __shared__ uint32_t s_nz[2][2];       // pair rounds: bits of the rows of the pair products in shared memory
    __shared__ double s_Td;               // dense: the residual total
    __shared__ float2 s_Tf;               // the residual total or the running sum as a float pair
    __shared__ volatile int s_ask;        // the chain's question to the FP64 warp: events before it << 8, marker + 1
    __shared__ volatile double s_told;    // and its answer: the marker's num
    __shared__ volatile int s_ev[kMaxSpec + 1];   // changes of the round in order, for the FP64 warp
    // beta_old - beta_new of the changes from the FP64 warp, kNoChange until then: the word
    // is the value, so its reader needs no other
    __shared__ volatile long long s_dB[kMaxSpec];
    __shared__ int s_ci[kMaxSpec];
    __shared__ __align__(16) long long s_d[kMaxSpec][4];
    __shared__ long long s_T[2];          // dense: the residual total, T = s_T[1] 2^30 + s_T[0]
    __shared__ double s_es;               // sparse: the running residual sum
    __shared__ double s_red[kRW][2];
    __shared__ float s_sum[kRW];
    __shared__ int s_nchg, s_fin, s_abort;
    __shared__ unsigned long long s_acc[kMaxSpec + 1][4];   // one CTA: the round's sums
    __shared__ __align__(8) uint64_t s_xbar[2];

    const bool solo = !CL && a.G == 1 && a.phantom == 0;
    const bool dense = a.rkind == BRR_KIND_DENSE;
    const bool pairs = a.rmode == kRoundPairs;
    // sums over the missing genotypes enter num for dense and Eigen markers
    const bool msum = a.has_missing && (dense || a.eigen);
    const int B = a.B;
    const unsigned Rm = 2u * (unsigned)(B < 16 ? 16 : B) - 1u;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (a.t_out && sidx == 0 && tid == 0)
        a.t_out[0] = global_timer_ns();
    const int lo = a.slice_lo[sidx];
    const int ns = a.slice_lo[sidx + 1] - lo;
    const int nchunk = (ns + kChunk - 1) / kChunk;
    const int64_t byte_lo = lo / 4;
    const RoundPlan plan = round_plan(a.slice_max, B, a.n_groups, CL ? a.G : 0, pairs, a.has_missing);
    long long *E = reinterpret_cast<long long *>(smem + plan.E);
    unsigned char *planes = smem + plan.planes;
    unsigned char *codes = smem + plan.codes;
    const RoundRec *rec = reinterpret_cast<const RoundRec *>(smem + plan.rec);
    const int gn = gram_entries_per_block(B);
    const size_t gslot = al16((size_t)8 * gram_entries_per_block(B < 16 ? 16 : B));
    uint32_t *ids = reinterpret_cast<uint32_t *>(smem + plan.ids);
    float *part = reinterpret_cast<float *>(smem + plan.part);
    double *gconst = reinterpret_cast<double *>(smem + plan.gconst);
    int32_t *gk = reinterpret_cast<int32_t *>(smem + plan.gk);
    float *gcf = reinterpret_cast<float *>(smem + plan.gcf);
    ulonglong2 *xch = reinterpret_cast<ulonglong2 *>(smem + plan.xch);
    float4 *gdf = reinterpret_cast<float4 *>(smem + plan.gdf);
    const int xrow = xch_words(B), B16 = B < 16 ? 16 : B;
    const int ncopy = a.G >= 24 ? kAccCopies : 1;

    // ---- prefetch machinery (ring positions modulo powers of two)
    const unsigned M32 = (unsigned)a.M;
    const unsigned Im = 2u * Rm + 1u;
    unsigned ids_issued = 0, code_issued = 0;
    int gram_issued = 0;
    constexpr int kPT = kRT - 128;   // prefetching threads: the warps without a part in the resolve
    const int ptid = tid - 128;
    auto issue_ids = [&](unsigned upto) {
        upto = min(upto, M32);
        for (unsigned q = ids_issued + ptid; q < upto; q += kPT)
            cp_async4(&ids[q & Im], &a.order[q]);
        ids_issued = max(ids_issued, upto);
    };
    // chunk c of marker q by thread: c varies fastest over cw consecutive threads
    int cw = 1;
    while (cw < nchunk && cw < 32)
        cw *= 2;
    auto issue_codes = [&](unsigned upto) {   // records and codes; their ids have landed
        upto = min(upto, M32);
        if (upto <= code_issued)
            return;
        const unsigned n = upto - code_issued;
        constexpr unsigned kRecWords = sizeof(RoundRec) / 16;
        for (unsigned e = ptid; e < n * kRecWords; e += kPT) {
            const unsigned q = code_issued + e / kRecWords, c = e % kRecWords;
            cp_async16(smem + plan.rec + (size_t)(q & Rm) * sizeof(RoundRec) + 16 * c,
                       reinterpret_cast<const unsigned char *>(&a.rrec[q]) + 16 * c);
        }
        for (unsigned q = code_issued + (unsigned)ptid / cw; q < upto; q += kPT / cw) {
            const uint8_t *src = a.codes + (int64_t)ids[q & Im] * a.col_stride + byte_lo;
            unsigned char *dst = codes + (size_t)(q & Rm) * plan.code_stride;
            for (int c = ptid & (cw - 1); c < nchunk; c += cw)
                cp_async16(dst + 16 * c, src + 16 * c);
        }
        code_issued = upto;
    };
    const int nblocks = (int)((a.M + B - 1) / B);
    // pair products: only the rows of markers that are sure or likely to change are
    // fetched, ahead of their round; another marker's row is read from L2 when it
    // changes.  All rows would be 16 KB per CTA and round, half of what 152 CTAs then read
    // from L2 during the exchange.  (Fetching the rows of the markers that may change
    // once their num is known, during the round, was 0.2 % faster at 2,000 x 5,000 and 0.8 %
    // slower at 100,000 x 100,000, before the loads that its arrival needs to be ordered,
    // which cost 5 % and 1 %.)
    auto issue_gram = [&](int upto) {
        if (!pairs)
            return;
        upto = min(upto, nblocks);
        for (; gram_issued < upto; ++gram_issued) {
            const unsigned q0 = (unsigned)gram_issued * (unsigned)B;
            uint32_t w0 = a.rnz[q0 >> 5] >> (q0 & 31u), w1 = B > 32 ? a.rnz[(q0 >> 5) + 1] : 0u;
            if (B < 32)
                w0 &= (1u << B) - 1u;
            if (ptid == 0) {
                s_nz[gram_issued & 1][0] = w0;
                s_nz[gram_issued & 1][1] = w1;
            }
            const double *src = a.rgram + (size_t)gram_issued * gn;
            double *dst = reinterpret_cast<double *>(smem + plan.gram + (gram_issued & 1) * gslot);
            for (int p = warp - 4; p < B; p += kRW - 4) {
                if (!(((p < 32 ? w0 : w1) >> (p & 31)) & 1u))
                    continue;
                const int base = p * (2 * B - p - 1) / 2;
                for (int t = lane; t < B - 1 - p; t += 32)
                    cp_async8(dst + base + t, src + base + t);
            }
        }
    };

    if (warp >= 4)
        issue_ids(3u * B);
    cp_async_commit();

    // ---- prologue: constants, the residual's scale, the residual
    for (int i = tid; i < a.n_groups * kMaxK * 4; i += kRT)
        gconst[i] = a.gconst[i];
    for (int i = tid; i < a.n_groups; i += kRT)
        gk[i] = a.gK[i];
    for (int i = tid; i < a.n_groups * kMaxK; i += kRT) {
        const int k = i % kMaxK;
        const double *row = a.gconst + (size_t)(i / kMaxK) * kMaxK * 4;
        gcf[2 * i] = k == 0 ? 0.f : __double2float_rn(row[4 * k] - row[0]);
        gcf[2 * i + 1] = k == 0 ? 0.f : __double2float_rn(row[4 * k + 2]);
        float4 v;   // beta = z sd_k + num / den_k of a non-zero component
        df_from_double(row[4 * k + 3], v.x, v.y);
        df_from_double(row[4 * k + 1], v.z, v.w);
        gdf[i] = v;
    }
    for (int i = tid; i <= kMaxSpec; i += kRT)
        s_ev[i] = 0;
    if (tid == 0)
        s_ask = 0;
    if (!CL)
        for (int i = tid; i < 2 * kRoundAccStride; i += kRT)
            reinterpret_cast<unsigned long long *>(smem + plan.prev)[i] = 0ull;
    for (int i = tid; i < (kMaxSpec + 1) * 4; i += kRT)
        (&s_acc[0][0])[i] = 0ull;
    {
        unsigned long long mx = 0ull;
        float sa = 0.f;
        for (int i = tid; i < a.n_emax; i += kRT) {
            const unsigned long long b = magnitude_bits(a.emax[i]);
            mx = b > mx ? b : mx;
            sa += float_below(a.emax[a.n_emax + i]);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long b = __shfl_xor_sync(0xffffffffu, mx, o);
            mx = b > mx ? b : mx;
            sa += __shfl_xor_sync(0xffffffffu, sa, o);
        }
        if (lane == 0) {
            s_red[warp][0] = __longlong_as_double((long long)mx);
            s_sum[warp] = sa;
        }
    }
    if (tid == 0) {
        s_abort = 0;
        s_es = a.epsSum;
        s_T[0] = s_T[1] = 0;
        s_Td = 0.0;
        float th, tl;
        df_from_double(a.epsSum, th, tl);
        s_Tf = make_float2(th, tl);
        if (CL) {
            cl_bar_init(&s_xbar[0]);
            cl_bar_init(&s_xbar[1]);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
    }
    cp_async_wait_all();
    __syncthreads();
    if (warp >= 4) {
        issue_codes(2u * B);
        issue_gram(1);
        cp_async_commit();
    }
    // the residual's scale, the same in every CTA
    int sc;
    bool coarse;
    {
        unsigned long long mx = 0ull;
        float sa = 0.f;
        for (int w = 0; w < kRW; ++w) {
            const unsigned long long b = magnitude_bits(s_red[w][0]);
            mx = b > mx ? b : mx;
            sa += s_sum[w];
        }
        // bounds of the residual after mu_new is subtracted: its largest magnitude, below
        // 2^e2, and its mean magnitude
        const double emax = fabs(a.mu_new) + __longlong_as_double((long long)mx);
        const float mean = __fdividef(sa, (float)a.N) - float_below(a.mu_new);
        const int e2 = (int)(magnitude_bits(emax) >> 52) - 1022;
        const int need = (a.form == BRR_FORM_FP64 ? 53 : 49) - ((int)(__float_as_uint(mean) >> 23) - 127);
        const int most = min(61 - e2, 100);   // E below 2^61: one bit of headroom
        sc = max(min(59 - e2, most), min(need, most));
        coarse = !(mean > 0.f && mean < INFINITY) || sc < need;
        if (coarse)
            sc = 0;
    }
    const double up = pow2d(sc), down = pow2d(-sc);
    bool range = coarse;
    for (int i = tid; i < a.slice_max; i += kRT) {
        const int ind = limb_individual(i);
        long long v = 0;
        if (ind < ns) {
            if (a.form == BRR_FORM_FP64) {
                v = __double2ll_rn(__dsub_rn(a.eps[lo + ind], a.mu_new) * up);
            } else {
                float h = a.eps_hi[lo + ind], l = a.eps_lo[lo + ind], mh, ml;
                df_from_double(-a.mu_new, mh, ml);
                df_add(h, l, mh, ml);
                v = __double2ll_rn((double)h * up) + __double2ll_rn((double)l * up);
            }
        }
        E[i] = v;
    }
    __syncthreads();
    {
        long long tl = 0, th = 0;
        for (int i = tid; i < plan.plane_stride / 4; i += kRT)
            reinterpret_cast<unsigned *>(planes + (size_t)3 * plan.plane_stride)[i] = 0u;
        for (int pr = tid; pr < a.slice_max / 2; pr += kRT) {
            const longlong2 e = reinterpret_cast<const longlong2 *>(E)[pr];
            put_limbs(planes, plan.plane_stride, pr, e.x, e.y);
            tl += (e.x & kLow30) + (e.y & kLow30);
            th += (e.x >> 30) + (e.y >> 30);
        }
        if (dense) {
            // the slice's total, published with the first round
            atomicAdd(reinterpret_cast<unsigned long long *>(&s_T[0]), (unsigned long long)tl);
            atomicAdd(reinterpret_cast<unsigned long long *>(&s_T[1]), (unsigned long long)th);
        }
    }
    if (CL)
        cl_sync_all();   // every CTA's mbarriers exist before the first store into it

    const double Nm1 = (double)a.N - 1.0;
    const bool prof = PROF && sidx == 0 && tid == 0;
    long long ph[5] = {0, 0, 0, 0, 0};
    long long tp = prof ? clock64() : 0;
    // an entry of an event list of the CTA; its writer always ends the list, so the
    // limit is not reached
    auto wait_event = [&](const volatile int *e) {
        int v;
        unsigned spins = 0;
        while ((v = *e) == 0 && ++spins < (1u << 28))
            ;
        if (v == 0)
            atomicCAS(a.err, kDevOk, kDevTimeout);
        return v;
    };
    auto mark = [&](int k) {
        if (prof) {
            const long long t = clock64();
            ph[k] += t - tp;
            tp = t;
        }
    };
    // counting variant: the parts of the exchange and resolve, on the first lane of their warps
    const bool wprof = PROF && sidx == 0 && lane == 0;
    long long wt = 0;
    auto wstart = [&]() {
        if (wprof)
            wt = clock64();
    };
    auto wmark = [&](int k) {
        if (wprof) {
            const long long t = clock64();
            atomicAdd(reinterpret_cast<unsigned long long *>(a.prof + k), (unsigned long long)(t - wt));
            wt = t;
        }
    };
    // tensor tiles of 16 markers; the warps of a tile split the chunks
    const int nmt = B <= 16 ? 1 : B / 16;
    const int nkg = kRW / nmt;
    const int mt = warp % nmt, kg = warp / nmt;
    const int fg = lane >> 2, fq = lane & 3;   // fragment row / column group

    unsigned start = coarse ? M32 : 0u;
    long long r = 0;
    int turn = 0;   // r mod G: the CTA that writes the round's outputs
    while (start < M32) {
        cp_async_wait_all();
        __syncthreads();
        if (tid < kMaxSpec)
            s_dB[tid] = kNoChange;
        // pair rounds stay inside a block of B positions, whose products they use: blk, from
        // position off (not 0 after a change whose row was not formed)
        const unsigned blk = start / (unsigned)B;
        const int off = pairs ? (int)(start - blk * (unsigned)B) : 0;
        const int nb = (int)min((unsigned)(a.rmode == kRoundAsync ? a.async_batch : B - off), M32 - start);
        mark(0);

        // ---- partial dot products over the slice
        {
            const unsigned char *ra = codes + (size_t)((start + mt * 16 + fg) & Rm) * plan.code_stride + 4 * fq;
            const unsigned char *rbp = codes + (size_t)((start + mt * 16 + fg + 8) & Rm) * plan.code_stride + 4 * fq;
            const unsigned char *pb = planes + (size_t)fg * plan.plane_stride + 32 * fq;
            float c[4] = {0.f, 0.f, 0.f, 0.f}, cm[4] = {0.f, 0.f, 0.f, 0.f};
            for (int ch = kg; ch < nchunk; ch += nkg) {
                const unsigned w0 = *reinterpret_cast<const unsigned *>(ra + 16 * ch);
                const unsigned w1 = *reinterpret_cast<const unsigned *>(rbp + 16 * ch);
                const uint4 x = *reinterpret_cast<const uint4 *>(pb + 128 * ch);
                const uint4 y = *reinterpret_cast<const uint4 *>(pb + 128 * ch + 16);
                mma_chunk(c, w0, w1, kGenoTable, x, y);
                if (msum)
                    mma_chunk(cm, w0, w1, kMissTable, x, y);
            }
            float2 *dst = reinterpret_cast<float2 *>(part + ((size_t)(kg * nmt + mt) * 16 + fg) * 8) + fq;
            dst[0] = make_float2(c[0], c[1]);
            dst[32] = make_float2(c[2], c[3]);
            if (msum) {
                dst += kRW * 16 * 4;
                dst[0] = make_float2(cm[0], cm[1]);
                dst[32] = make_float2(cm[2], cm[3]);
            }
        }
        __syncthreads();

        // ---- publication: thread m the low word (limbs 0-2) of marker m's sum, thread
        // 64 + m the high word, threads 128 and 192 on those of its sum over the missing
        // genotypes, threads 256 and 257 (first round) the slice total
        {
            const int m = tid & 63, which = tid >> 6;
            const bool total = which == 4 && m < 2 && r == 0 && dense;
            if ((m < nb && (which < 2 || (which < 4 && msum))) || total) {
                const int word = total ? m : which & 1, half = total ? 0 : which >> 1;
                long long v;
                if (total) {
                    v = m == 0 ? s_T[0] & kLow30 : s_T[1] + (s_T[0] >> 30);
                } else {
                    v = limb_sum(part + (size_t)half * kRW * 16 * 8, m, word, nkg, nmt * 32);
                }
                if (CL) {
                    reinterpret_cast<long long *>(
                        xch + ((size_t)(r & 1) * a.G + sidx) * xrow + (total ? B16 : half * (B16 + 1) + m))[word] = v;
                } else if (solo) {
                    s_acc[total ? kMaxSpec : m][2 * half + word] = (unsigned long long)v;
                } else {
                    red_add_u64(a.acc + (size_t)(r & 1) * kRoundAccStride + (sidx % ncopy) * kAccCopyWords +
                                    (2 * half + word) * kAccRow + (total ? kMaxSpec : m),
                                (1ull << kCountShift) + kAccBias + (unsigned long long)v);
                }
            }
        }
        __syncthreads();
        if (CL) {
            // this CTA's records into the other CTAs' shared memory, one warp per
            // destination, one 16-byte store per record
            const int rows = nb + (msum ? nb : 0) + (r == 0 && dense ? 1 : 0);
            const ulonglong2 *own = xch + ((size_t)(r & 1) * a.G + sidx) * xrow;
            for (int d = warp; d < a.G; d += kRW) {
                if (d == sidx)
                    continue;
                const unsigned dst = cl_map(cl_addr(own), (unsigned)d), bar = cl_map(cl_addr(&s_xbar[r & 1]), (unsigned)d);
                for (int w = lane; w < rows; w += 32) {
                    const int at = w < nb ? w : (msum && w < 2 * nb) ? B16 + 1 + w - nb : B16;
                    const ulonglong2 v = own[at];
                    cl_push16(dst + 16u * (unsigned)at, v.x, v.y, bar);
                }
            }
        }
        mark(1);

        // ---- exchange and resolve.  Warps 2 and 3 wait for the sums (bounded),
        // form num and take every marker's first decision; warp 0 walks the
        // chain of changes in double-float; warp 1 follows it in FP64; the others
        // fetch the next round's markers.
        wstart();
        if (warp == 2 || warp == 3) {
            const int m = tid - 64;
            // the part of num that does not wait, c + at T (in the first round of dense
            // markers T comes with the sums)
            const RoundRec &rc = rec[(start + (m < nb ? m : 0)) & Rm];
            float ch = rc.cf[0], cl = rc.cf[1];
            auto add_T = [&](float th, float tl) {
                float xh, xl;
                df_mul(rc.atf[0], rc.atf[1], th, tl, xh, xl);
                df_add(ch, cl, xh, xl);
            };
            if (!dense || r > 0)
                add_T(s_Tf.x, s_Tf.y);
            if (CL) {
                if (m == 0)
                    cl_expect(&s_xbar[r & 1],
                              (unsigned)((a.G - 1) * 16 * (nb + (msum ? nb : 0) + (r == 0 && dense ? 1 : 0)) +
                                         a.phantom * 32));
                if (lane == 0 && !cl_wait(&s_xbar[r & 1], (unsigned)(r >> 1) & 1u, a.timeout_ns)) {
                    atomicCAS(a.err, kDevOk, kDevTimeout);
                    s_abort = 1;
                }
                __syncwarp();
            }
            if (warp == 2)
                wmark(6);
            // sums over all CTAs of marker slot's residual products (half 0) or of its
            // residual over the missing genotypes (half 1); in L2, waits for them
            // (bounded)
            auto fetch = [&](int slot, int half, long long &L, long long &H) {
                L = H = 0;
                if (CL) {
                    const ulonglong2 *x2 =
                        xch + (size_t)(r & 1) * a.G * xrow + (slot == kMaxSpec ? B16 : half * (B16 + 1) + slot);
                    for (int s = 0; s < a.G; ++s) {
                        const ulonglong2 w = x2[(size_t)s * xrow];
                        L += (long long)w.x;
                        H += (long long)w.y;
                    }
                } else if (solo) {
                    L = (long long)s_acc[slot][2 * half];
                    H = (long long)s_acc[slot][2 * half + 1];
                } else {
                    const int off = (int)(r & 1) * kRoundAccStride + 2 * half * kAccRow + slot;
                    const unsigned long long *acc = a.acc + off;
                    // the words' last complete values
                    unsigned long long *prev = reinterpret_cast<unsigned long long *>(smem + plan.prev) + off;
                    unsigned long long w[kAccCopies][2] = {};
                    uint64_t t0 = 0;
                    for (unsigned spins = 0;; ++spins) {
                        bool all = true;
#pragma unroll
                        for (int c = 0; c < kAccCopies; ++c)
                            if (c < ncopy) {
                                w[c][0] = ld_relaxed_u64(acc + c * kAccCopyWords);
                                w[c][1] = ld_relaxed_u64(acc + c * kAccCopyWords + kAccRow);
                            }
#pragma unroll
                        for (int c = 0; c < kAccCopies; ++c)
                            if (c < ncopy) {
                                // CTAs of this copy (and the arrivals a timeout test never sees)
                                const unsigned n = (unsigned)((a.G - c + ncopy - 1) / ncopy + (c == 0 ? a.phantom : 0));
#pragma unroll
                                for (int k = 0; k < 2; ++k) {
                                    const unsigned long long p = prev[c * kAccCopyWords + k * kAccRow];
                                    all = all && (unsigned)((w[c][k] - p) >> kCountShift) == n;
                                }
                            }
                        if (all)
                            break;
                        if ((spins & 255u) == 255u) {
                            const uint64_t now = global_timer_ns();
                            if (t0 == 0)
                                t0 = now;
                            if (*(volatile int *)a.err == kDevTimeout || now - t0 > a.timeout_ns) {
                                atomicCAS(a.err, kDevOk, kDevTimeout);
                                s_abort = 1;
                                break;
                            }
                        }
                    }
#pragma unroll
                    for (int c = 0; c < kAccCopies; ++c)
                        if (c < ncopy) {
                            const unsigned long long n = (unsigned long long)((a.G - c + ncopy - 1) / ncopy);
#pragma unroll
                            for (int k = 0; k < 2; ++k) {
                                unsigned long long &p = prev[c * kAccCopyWords + k * kAccRow];
                                const long long v = (long long)((w[c][k] - p) & kAccMask) - (long long)(n * kAccBias);
                                (k ? H : L) += v;
                                if (slot != kMaxSpec)   // read once, by every thread
                                    p = w[c][k];
                            }
                        }
                }
            };
            if (r == 0 && dense) {
                long long TL, TH;
                fetch(kMaxSpec, 0, TL, TH);
                float th, tl;
                fixed_to_df(TH, TL, -sc, th, tl);
                add_T(th, tl);
                if (m == 0) {
                    s_T[0] = TL & kLow30;
                    s_T[1] = TH + (TL >> 30);
                    s_Td = fixed_to_double(TH, TL, -sc);
                    s_Tf = make_float2(th, tl);
                }
            }
            long long L = 0, H2 = 0, mL = 0, mH = 0;
            if (m < nb) {
                fetch(m, 0, L, H2);
                if (msum)
                    fetch(m, 1, mL, mH);
                if (warp == 2)
                    wmark(7);
                // num in double-float
                float sh, sl, nh, nl;
                fixed_to_df(H2, L, -sc, sh, sl);
                df_mul(rc.sf[0], rc.sf[1], sh, sl, nh, nl);
                if (msum) {
                    float th, tl;
                    fixed_to_df(mH, mL, -sc, sh, sl);
                    df_mul(rc.amf[0], rc.amf[1], sh, sl, th, tl);
                    df_add(nh, nl, th, tl);
                }
                df_add(nh, nl, ch, cl);
                s_ndf[m] = make_float2(nh, nl);
                if (warp == 2)
                    wmark(8);
            }
            __syncwarp();
            asm volatile("bar.sync 1, 96;" ::: "memory");
            // num in FP64, for the warp that follows the chain
            if (m < nb) {
                const double at = -(rc.s * rc.m);
                double num = fma(at, dense ? s_Td : s_es, rc.beta_old * Nm1);
                num = fma(rc.s, fixed_to_double(H2, L, -sc), num);
                if (msum)
                    num = fma(dense ? fma(rc.s, rc.m, rc.x) : -at, fixed_to_double(mH, mL, -sc), num);
                s_num[m] = num;
            }
            __syncwarp();
            asm volatile("bar.sync 2, 96;" ::: "memory");
            if (warp == 3) {
                // the moves of every change per 2-bit code, as the FP64 warp finishes them
                for (int u = 0;; ++u) {
                    const int ev = wait_event(&s_ev[u]);
                    if (ev <= 0)
                        break;
                    const RoundRec &rp = rec[(start + ((ev - 1) & 63)) & Rm];
                    // (genotype - mean) scale; missing genotypes apart
                    const double x = up * (lane == 1 ? (dense ? rp.x : 0.0)
                                                     : __dmul_rn(__dsub_rn(lane == 0 ? 2.0 : lane == 2 ? 1.0 : 0.0, rp.m), rp.s));
                    long long dB;
                    unsigned spins = 0;
                    while ((dB = s_dB[u]) == kNoChange && ++spins < (1u << 28))
                        ;
                    if (dB == kNoChange)
                        atomicCAS(a.err, kDevOk, kDevTimeout);
                    if (lane < 4) {
                        const double d = __dmul_rn(__longlong_as_double(dB), x);   // up is a power of two
                        // |d| < 2^62, by its exponent
                        const bool ok = ((unsigned)__double2hiint(d) & 0x7FF00000u) < (1085u << 20);
                        range = range || !ok;
                        s_d[u][lane] = ok ? __double2ll_rn(d) : 0ll;
                    }
                }
            }
        } else if (warp == 0) {
            // lane t holds markers t and 32 + t.  The loop below runs once per marker that
            // may change, on one warp, from instructions that the other phases have
            // pushed out of the nearest instruction cache: its length is its cost.  It only
            // decides: num is carried in FP32 with a bound er on its error, which widens
            // the certificates of the decisions; where they fail, the FP64 warp is
            // asked for the marker's num.  (With num as a pair of FP32 words a change took
            // 1.17k clk, so 0.97k; dense 2,000 x 5,000 in the burn-in, 27 changes a round: 1.63
            // and 1.46 ms per sweep.)
            float s0[2], bo[2], zf[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int t = lane + 32 * h;
                const RoundRec &rc = rec[(start + (t < nb ? t : 0)) & Rm];
                // num^2 above which the marker may change: always with an old effect
                bo[h] = double_hi(rc.beta_old);
                zf[h] = double_hi(rc.z);
                s0[h] = !(t < nb) ? INFINITY : nonzero(rc.beta_old) ? -1.f : rc.s0;
                s_comp[t] = 0;
            }
            const double *gr = reinterpret_cast<const double *>(smem + plan.gram + (blk & 1u) * gslot);
            const double *grow = a.rgram + (size_t)blk * gn;
            const uint32_t *nz = s_nz[blk & 1u];
            __syncwarp();
            asm volatile("bar.sync 1, 96;" ::: "memory");
            mark(2);
            wstart();
            float x[2], er[2], sx[2];   // num, its error, the square of its largest magnitude
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float2 v = s_ndf[lane + 32 * h];
                x[h] = v.x;
                er[h] = __fmaf_rn(1e-10f, fabsf(v.x), 1.01f * fabsf(v.y));
                sx[h] = (fabsf(x[h]) + er[h]) * (fabsf(x[h]) + er[h]);
            }
            // A marker may change when its old effect is not zero or num^2 is not in
            // the range where component 0 is certain (s0; P(component 0) falls as
            // num^2 grows).  Only such a marker's component is worked out, when the
            // chain reaches it; the markers before it stay in component 0.
            int nchg = 0, fin = nb, pos = 0;
            // num of marker p after the changes so far, from the FP64 warp, on one lane
            auto ask_num = [&](int p) { return ask_fp64_warp(&s_ask, &s_told, (nchg << 8) | (p + 1), a.err); };
            if (a.rmode == kRoundAsync) {
                // every marker is decided on the residual before the batch
#pragma unroll 1
                for (int h = 0; h < 2; ++h) {
                    const int t = lane + 32 * h;
                    int comp = 0;
                    const bool c = (h ? sx[1] : sx[0]) > (h ? s0[1] : s0[0]) && t < nb;
                    const RoundRec &rc = rec[(start + (c ? t : 0)) & Rm];
                    const unsigned g = rc.gm & 255u;
                    if (c)
                        comp = decide_pair<KM>(s_ndf[t].x, s_ndf[t].y, rc.uf, gcf + (size_t)g * kMaxK * 2, gk[g]);
                    for (unsigned m = __ballot_sync(0xffffffffu, comp == -2); m; m &= m - 1u) {
                        if (lane == __ffs(m) - 1)
                            comp = decide_slow<KM>(ask_num(t), a.u[rc.j], gconst + (size_t)g * kMaxK * 4,
                                                   gcf + (size_t)g * kMaxK * 2, gk[g]);
                        __syncwarp();
                    }
                    const bool b = c && (comp > 0 || rc.beta_old != 0.0);
                    const unsigned kb = __ballot_sync(0xffffffffu, b);
                    if (c)
                        s_comp[t] = comp;
                    if (b)
                        s_ev[nchg + __popc(kb & ((1u << lane) - 1u))] = 1 + t + ((comp + 1) << 8);
                    nchg += __popc(kb);
                }
                pos = 64;
            }
            while (pos < 64 && !s_abort) {
                const unsigned k0 = __ballot_sync(0xffffffffu, lane >= pos && sx[0] > s0[0]);
                const unsigned k1 = __ballot_sync(0xffffffffu, lane + 32 >= pos && sx[1] > s0[1]);
                if (!(k0 | k1))
                    break;
                const int p = k0 ? __ffs(k0) - 1 : 31 + __ffs(k1);
                const bool hi = p >= 32, own = lane == (p & 31);
                pos = p + 1;
                // row p of the pair products, ahead of dBeta
                double gv0 = 0.0, gv1 = 0.0;
                bool last = !pairs;
                if (pairs) {
                    const int q = off + p;
                    const bool here = ((nz[q >> 5] >> (q & 31)) & 1u) != 0u;
                    last = !here && !a.rall;
                    const double *row = (here ? gr : grow) + q * (2 * B - q - 1) / 2 - p - 1;
                    if (!last && lane > p && lane < nb)
                        gv0 = row[lane];
                    if (!last && lane + 32 > p && lane + 32 < nb)
                        gv1 = row[lane + 32];
                }
                const RoundRec &rc = rec[(start + p) & Rm];
                const unsigned g = rc.gm & 255u;
                const float xp = hi ? x[1] : x[0], ep = hi ? er[1] : er[0];
                const float px = __shfl_sync(0xffffffffu, xp, p & 31), pe = __shfl_sync(0xffffffffu, ep, p & 31);
                // D_k moves by 2 h_k |num| er: 5e6 = 2 / 4e-7, in units of the samplers' own error
                int comp = pick_lanes<KM>(lane, px * px, rc.uf,
                                          reinterpret_cast<const float2 *>(gcf + (size_t)g * kMaxK * 2)[lane & (kMaxK - 1)],
                                          gk[g], 5e6f * pe * (fabsf(px) + pe));
                if (comp == -2) {
                    if (own)
                        comp = decide_slow<KM>(ask_num(p), a.u[rc.j], gconst + (size_t)g * kMaxK * 4,
                                               gcf + (size_t)g * kMaxK * 2, gk[g]);
                    comp = __shfl_sync(0xffffffffu, comp, p & 31);
                }
                if (own)
                    s_comp[p] = comp;
                if (comp <= 0 && !nonzero(rc.beta_old))
                    continue;
                if (own)
                    s_ev[nchg] = 1 + p + ((comp + 1) << 8);
                ++nchg;
                if (last) {
                    fin = p + 1;   // a restart round ends at its first change, a pair round at one without a row
                    break;
                }
                // beta_old - beta_new and its error, on the owner's lane.  With the truncation of
                // G the roundings come to 3.0e-7 of the old effect, 4.8e-7 of z sd and 3.6e-7 of
                // num / den; those of er itself, 2e-7 of it a change, stay inside the 1 % that its
                // first term has over
                float d = hi ? bo[1] : bo[0], e = fabsf(d);
                if (comp > 0) {
                    const float4 k4 = gdf[g * kMaxK + comp];   // {sdk hi, lo, invden hi, lo}
                    const float zs = (hi ? zf[1] : zf[0]) * k4.x, xi = xp * k4.z;
                    d -= zs + xi;
                    e = __fmaf_rn(ep, k4.z, 5e-7f * (e + fabsf(zs) + fabsf(xi)));
                } else {
                    e *= 3e-7f;
                    if (comp < 0)
                        d = e = 0.f;
                }
                d = __shfl_sync(0xffffffffu, d, p & 31);
                e = __shfl_sync(0xffffffffu, e, p & 31);
                // the later markers' num; 7e-8 |num|: its rounding
                const float g0 = double_hi(gv0), g1 = double_hi(gv1);
                x[0] = __fmaf_rn(d, g0, x[0]);
                x[1] = __fmaf_rn(d, g1, x[1]);
                er[0] = __fmaf_rn(7e-8f, fabsf(x[0]), __fmaf_rn(e, fabsf(g0), er[0]));
                er[1] = __fmaf_rn(7e-8f, fabsf(x[1]), __fmaf_rn(e, fabsf(g1), er[1]));
                sx[0] = (fabsf(x[0]) + er[0]) * (fabsf(x[0]) + er[0]);
                sx[1] = (fabsf(x[1]) + er[1]) * (fabsf(x[1]) + er[1]);
            }
            __syncwarp();
            if (lane == 0) {
                s_nchg = nchg;
                s_fin = fin;
                __threadfence_block();
                s_ev[nchg] = -1;
            }
            wmark(10);
            if (wprof)
                atomicAdd(reinterpret_cast<unsigned long long *>(a.prof + 14), (unsigned long long)nchg);
        } else if (warp == 1) {
            // num, beta and the corrections in FP64, one change behind the chain
            const double *gr = reinterpret_cast<const double *>(smem + plan.gram + (blk & 1u) * gslot);
            const double *grow = a.rgram + (size_t)blk * gn;
            const uint32_t *nz = s_nz[blk & 1u];
            __syncwarp();
            asm volatile("bar.sync 2, 96;" ::: "memory");
            wstart();
            double num[2] = {lane < nb ? s_num[lane] : 0.0, lane + 32 < nb ? s_num[lane + 32] : 0.0};
            if (lane < nb)
                s_beta[lane] = 0.0;   // a marker without a change has beta 0
            if (lane + 32 < nb)
                s_beta[lane + 32] = 0.0;
            __syncwarp();
            int nchg = 0;
            for (;; ++nchg) {
                int ev;
                unsigned spins = 0;
                while ((ev = s_ev[nchg]) == 0 && ++spins < (1u << 28)) {
                    const int ask = s_ask;
                    if (ask != 0 && ((ask - 1) & 31) == lane && ask >> 8 == nchg) {
                        s_told = ((ask - 1) & 32) ? num[1] : num[0];
                        __threadfence_block();
                        s_ask = 0;
                    }
                }
                if (ev == 0)
                    atomicCAS(a.err, kDevOk, kDevTimeout);
                if (ev <= 0)
                    break;
                const int p = (ev - 1) & 63, comp = (ev - 1) / 256 - 1;
                double dB = 0.0;
                if (lane == (p & 31)) {
                    const RoundRec &rc = rec[(start + p) & Rm];
                    const double *gc = gconst + ((size_t)(rc.gm & 255u) * kMaxK + max(comp, 0)) * 4;
                    const double x = p < 32 ? num[0] : num[1];
                    // (src/BayesRBase.cpp:346-364)
                    const double b = comp > 0 ? __dadd_rn(__dmul_rn(rc.z, gc[3]), __dmul_rn(x, gc[1]))
                                              : comp == 0 ? 0.0 : rc.beta_old;
                    dB = rc.beta_old - b;
                    s_beta[p] = b;
                    s_dB[nchg] = __double_as_longlong(dB);
                    s_ci[nchg] = p;
                }
                if (!pairs)
                    continue;
                dB = __shfl_sync(0xffffffffu, dB, p & 31);
                const int q = off + p;
                const bool here = ((nz[q >> 5] >> (q & 31)) & 1u) != 0u;
                if (!here && !a.rall)
                    continue;   // the round ends here
                const double *row = (here ? gr : grow) + q * (2 * B - q - 1) / 2 - p - 1;
                if (p < 31 && lane > p && lane < nb)
                    num[0] = fma(dB, row[lane], num[0]);
                if (nb > 32 && lane + 32 > p && lane + 32 < nb)
                    num[1] = fma(dB, row[lane + 32], num[1]);
            }
            if (lane < nb)
                s_num[lane] = num[0];
            if (lane + 32 < nb)
                s_num[lane + 32] = num[1];
            wmark(11);
        } else {
            issue_ids(start + 3u * B);
            issue_codes(start + 2u * B);
            issue_gram((int)blk + 2);
            cp_async_commit();
            if (warp == 4)
                wmark(13);
        }
        __syncthreads();
        mark(3);
        if (s_abort)
            break;

        // ---- outputs of the round, the running sums, the residual update
        const int nchg = s_nchg, fin = s_fin;
        if (tid < fin && turn == sidx) {
            const RoundRec &rc = rec[(start + tid) & Rm];
            const int c = s_comp[tid];
            a.beta_out[rc.j] = s_beta[tid];
            a.num_out[rc.j] = s_num[tid];
            a.comp_out[rc.j] = c;
        }
        if (tid <= nchg)
            s_ev[tid] = 0;
        if (nchg) {
            if (dense && warp == kRW - 1) {
                // the residual total, exactly: individuals per code times the code's move
                long long tl = 0, th = 0;
                for (int u = lane; u < nchg; u += 32) {
                    const RoundRec &rc = rec[(start + s_ci[u]) & Rm];
                    const long long nm = rc.gm >> 8, n2 = rc.n2, n1 = rc.n1, n0 = a.N - nm - n2 - n1;
                    const long long d0 = s_d[u][0], d1 = s_d[u][1], d2 = s_d[u][2], d3 = s_d[u][3];
                    tl += (d0 & kLow30) * n2 + (d1 & kLow30) * nm + (d2 & kLow30) * n1 + (d3 & kLow30) * n0;
                    th += (d0 >> 30) * n2 + (d1 >> 30) * nm + (d2 >> 30) * n1 + (d3 >> 30) * n0;
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    tl += __shfl_xor_sync(0xffffffffu, tl, o);
                    th += __shfl_xor_sync(0xffffffffu, th, o);
                }
                if (lane == 0) {
                    tl += s_T[0];
                    th += s_T[1] + (tl >> 30);
                    tl &= kLow30;
                    s_T[0] = tl;
                    s_T[1] = th;
                    s_Td = fixed_to_double(th, tl, -sc);
                    float fh, fl;
                    split_double(s_Td, fh, fl);
                    s_Tf = make_float2(fh, fl);
                }
            } else if (!dense && tid == kRT - 1) {
                double es = s_es;
                for (int u = 0; u < nchg; ++u) {
                    const RoundRec &rc = rec[(start + s_ci[u]) & Rm];
                    es += __longlong_as_double(s_dB[u]) * ((rc.x - rc.m * (double)a.N) * rc.s);
                }
                s_es = es;
                float fh, fl;
                split_double(es, fh, fl);
                s_Tf = make_float2(fh, fl);
            }
            long long top = 0;
            for (int pr = tid; pr < 32 * nchunk; pr += kRT) {
                longlong2 e = reinterpret_cast<const longlong2 *>(E)[pr];
                const int sh = limb_pair_shift(pr);
                for (int u = 0; u < nchg; ++u) {
                    const unsigned w = *reinterpret_cast<const unsigned *>(
                                           codes + (size_t)((start + s_ci[u]) & Rm) * plan.code_stride + 4 * (pr >> 3)) >> sh;
                    e.x += s_d[u][w & 3u];
                    e.y += s_d[u][(w >> 8) & 3u];
                    top |= (e.x ^ (e.x << 1)) | (e.y ^ (e.y << 1));
                }
                // individuals past the slice's end keep a zero residual
                const int ind = 16 * (pr >> 3) + (sh >> 1);
                if (ind >= ns)
                    e.x = 0;
                if (ind + 4 >= ns)
                    e.y = 0;
                reinterpret_cast<longlong2 *>(E)[pr] = e;
                put_limbs(planes, plan.plane_stride, pr, e.x, e.y);
            }
            if (top < 0)
                range = true;
        }
        mark(4);
        start += (unsigned)fin;
        ++r;
        turn = turn + 1 == a.G ? 0 : turn + 1;
    }
    if (range)
        atomicCAS(a.err, kDevOk, kDevRange);
    if (prof) {
        for (int k = 0; k < 5; ++k)
            a.prof[k] = ph[k];
        a.prof[5] = r;
    }
    cp_async_wait_all();
    __syncthreads();

    // ---- epilogue: the residual to its output buffer, per-slice sums
    double s1 = 0.0, s2 = 0.0;
    for (int i = tid; i < a.slice_max; i += kRT) {
        const int ind = limb_individual(i);
        if (ind >= ns)
            continue;
        double e = (double)E[i] * down;
        if (a.form == BRR_FORM_FP64) {
            a.eps_out[lo + ind] = e;
        } else {
            float h, l;
            df_from_double(e, h, l);
            a.eps_hi_out[lo + ind] = h;
            a.eps_lo_out[lo + ind] = l;
            e = (double)h + (double)l;
        }
        s1 += e;
        s2 = fma(e, e, s2);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        s1 += __shfl_xor_sync(0xffffffffu, s1, o);
        s2 += __shfl_xor_sync(0xffffffffu, s2, o);
    }
    if (lane == 0) {
        s_red[warp][0] = s1;
        s_red[warp][1] = s2;
    }
    __syncthreads();
    if (tid == 0) {
        double t1 = 0.0, t2 = 0.0;
        for (int q = 0; q < kRW; ++q) {
            t1 += s_red[q][0];
            t2 += s_red[q][1];
        }
        a.part[2 * sidx] = t1;
        a.part[2 * sidx + 1] = t2;
        if (sidx == 0) {
            a.stats_out[0] = s_es;
            *a.rounds_out = r;
            if (a.t_out)
                a.t_out[1] = global_timer_ns();
        }
    }
    if (CL)
        cl_sync_all();   // no CTA exits while another may still store into its shared memory
}

template <int KM, bool PROF>
__global__ void __launch_bounds__(kRT, 1) k_round(SweepArgs a)
{
    round_body<KM, PROF, false>(a, (int)blockIdx.x);
}

// The sweep as one thread-block cluster of G CTAs (the whole grid).
template <int KM, bool PROF>
__global__ void __launch_bounds__(kRT, 1) k_round_cl(SweepArgs a)
{
    round_body<KM, PROF, true>(a, (int)cl_rank());
}

// Several independent chains of different sizes in one cooperative launch:
// CTAs [cta_start[i], cta_start[i+1]) run instance i's sweep over its slices;
// the instances share no data, so one chain's progress never waits on another's.
template <int KM>
__global__ void __launch_bounds__(kRT, 1) k_round_multi(const __grid_constant__ MultiSweepArgs m)
{
    int i = 0;
    while (i + 1 < m.n && (int)blockIdx.x >= m.cta_start[i + 1])
        ++i;
    round_body<KM, false, false>(m.inst[i], (int)blockIdx.x - m.cta_start[i]);
}

// --------------------------------------------------------------------------
// Records in sweep order, and the bits of the markers that are sure to change (an
// old effect) or likely to (component 0 not certain at num^2 = `likely`).
template <int KM>
__global__ void k_round_gather(const uint32_t *__restrict__ order, int64_t M, int64_t N, int kind,
                               const double *__restrict__ table, const double *__restrict__ scale,
                               const int64_t *__restrict__ counts, const double *__restrict__ beta,
                               const double *__restrict__ u, const double *__restrict__ z,
                               const int32_t *__restrict__ group, const double *__restrict__ gconst,
                               const int32_t *__restrict__ gK, float likely, RoundRec *rec, uint32_t *nz)
{
    const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    bool set = false;
    if (q < M) {
        const uint32_t j = order[q];
        const int g = group[j];
        RoundRec r;
        r.beta_old = beta[j];
        r.uf = __double2float_rn(u[j]);
        r.z = z[j];
        r.s0 = certain_zero<KM>(r.uf, gconst + (size_t)g * kMaxK * 4, gK[g]);
        r.j = j;
        r.gm = (uint32_t)g | ((uint32_t)counts[4 * (int64_t)j + 3] << 8);
        r.n1 = (uint32_t)counts[4 * (int64_t)j + 1];
        r.n2 = (uint32_t)counts[4 * (int64_t)j + 2];
        if (kind == BRR_KIND_DENSE) {
            r.s = scale[2 * (int64_t)j];
            r.m = scale[2 * (int64_t)j + 1];
            r.x = table[4 * (int64_t)j + 1];
        } else {
            r.s = 1.0 / table[4 * (int64_t)j + 1];
            r.m = table[4 * (int64_t)j];
            r.x = table[4 * (int64_t)j + 3];
        }
        const double at = -(r.s * r.m);
        df_from_double(r.s, r.sf[0], r.sf[1]);
        df_from_double(at, r.atf[0], r.atf[1]);
        df_from_double(r.beta_old * ((double)N - 1.0), r.cf[0], r.cf[1]);
        df_from_double(kind == BRR_KIND_DENSE ? fma(r.s, r.m, r.x) : -at, r.amf[0], r.amf[1]);
        rec[q] = r;
        set = r.beta_old != 0.0 || r.s0 < likely;
    }
    const unsigned w = __ballot_sync(0xffffffffu, set);
    if ((threadIdx.x & 31) == 0)
        nz[q >> 5] = w;   // the grid covers whole warps past M: at most 7 words more
}

// Markers p of block b whose row of pair products is formed: all of them, or
// those sure or likely to change (the bits nz).
__device__ __forceinline__ unsigned long long block_rows(const uint32_t *nz, int64_t b, int B, int rows, bool all)
{
    unsigned long long m = rows == 64 ? ~0ull : (1ull << rows) - 1ull;
    if (!all) {
        const int64_t q = b * B;
        unsigned long long w = nz[q >> 5] >> (q & 31);
        if (B > 32)
            w |= (unsigned long long)nz[(q >> 5) + 1] << 32;
        m &= w;
    }
    return m;
}

// Integer pair sums over all individuals for the rounds of a sweep: row p of block
// b (p's rank r among the block's rows), column t: sums[mode][b][r][t] with mode 0:
// genotype x genotype, 1: missing at p x genotype at t, 2: genotype at p x missing
// at t, 3: missing at both (MISS: 0 the first alone, 1 the first two, 2 all).
// One CTA per (block, part of the individuals, 16 rows): the block's markers are the
// 16-row operand of m16n8k16 FP16 mma.sync (exact: integers below 2^24 in FP32),
// the CTA's rows p the 8-column one, both decoded in registers from the staged codes.
// Bound by the decoding (24 instructions per 16 genotypes), which is why only the
// rows that a sweep is likely to need are formed on large problems: N = M = 100,000
// after the burn-in (4-5 rows of 64) 2.67 ms for all rows on or above the diagonal.
// (E4M3 operands take 254 registers: mma.sync converts them to FP16 on this GPU.)
constexpr int kPairSeg = 512;                       // bytes of a marker per stage (2,048 individuals)
constexpr int kPairRow = kPairSeg + 16;             // row pitch in shared memory: conflict-free word reads
constexpr int kPairStages = 3;
constexpr int kPairCols = 16;                       // rows p per CTA

template <int NT, int MISS>
__global__ void __launch_bounds__(256, 1) k_pair_sums(const uint32_t *__restrict__ order, int64_t M, int B,
                                                      const uint8_t *__restrict__ codes, int64_t col_stride,
                                                      const uint32_t *__restrict__ nz, int all, int *__restrict__ out,
                                                      int64_t mode_stride)
{
    constexpr int R16 = NT / 16;                    // 16-marker tiles
    constexpr int NM = MISS == 0 ? 1 : MISS == 1 ? 2 : 4;
    constexpr int kStage = NT * kPairRow;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ uint32_t s_id[NT];
    __shared__ int s_row[kPairCols];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int fg = lane >> 2, fq = lane & 3;
    const int64_t b = blockIdx.x, q0 = b * B;
    const int rows = (int)imin64(B, M - q0);
    const unsigned long long mask = block_rows(nz, b, B, rows, all != 0);
    const int r0 = blockIdx.z * kPairCols, nrow = min(kPairCols, __popcll(mask) - r0);
    if (nrow <= 0)
        return;
    if (tid < rows)
        s_id[tid] = order[q0 + tid];
    if (tid < B && ((mask >> tid) & 1ull)) {
        const int k = __popcll(mask & ((1ull << tid) - 1ull)) - r0;
        if (k >= 0 && k < kPairCols)
            s_row[k] = tid;
    }
    // genotype 0 (code 3) everywhere; the copies overwrite what the markers have
    for (int i = tid; i < kPairStages * kStage / 16; i += 256)
        reinterpret_cast<uint4 *>(smem)[i] = make_uint4(~0u, ~0u, ~0u, ~0u);
    __syncthreads();
    const int nseg = (int)((col_stride + kPairSeg - 1) / kPairSeg);
    const int first = (int)((int64_t)nseg * blockIdx.y / gridDim.y), last = (int)((int64_t)nseg * (blockIdx.y + 1) / gridDim.y);
    // a warp copies 512 contiguous bytes of a marker at a time
    auto issue = [&](int seg) {
        unsigned char *st = smem + (seg % kPairStages) * kStage;
        const int64_t at = (int64_t)seg * kPairSeg + 16 * lane;
        for (int m = warp; m < rows; m += 8) {
            if (at < col_stride)
                cp_async16(st + m * kPairRow + 16 * lane, codes + (int64_t)s_id[m] * col_stride + at);
            else   // past the markers' end, in a buffer that held an earlier segment
                *reinterpret_cast<uint4 *>(st + m * kPairRow + 16 * lane) = make_uint4(~0u, ~0u, ~0u, ~0u);
        }
    };
    for (int k = 0; k < kPairStages - 1; ++k) {
        if (first + k < last)
            issue(first + k);
        cp_async_commit();
    }
    const bool two = nrow > 8;
    const int c0 = s_row[min(fg, nrow - 1)], c1 = s_row[min(fg + 8, nrow - 1)];
    float acc[NM][R16][2][4] = {};
    for (int seg = first; seg < last; ++seg) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kPairStages - 2) : "memory");
        __syncthreads();   // segment seg has landed; every warp is done with segment seg - 1
        if (seg + kPairStages - 1 < last)
            issue(seg + kPairStages - 1);
        cp_async_commit();
        // this warp's 256 individuals of the segment, 64 at a time
        const unsigned char *src = smem + (seg % kPairStages) * kStage + 64 * warp + 4 * fq;
#pragma unroll 1
        for (int k = 0; k < 4; ++k, src += 16) {
            unsigned bw[2];
            bw[0] = *reinterpret_cast<const unsigned *>(src + c0 * kPairRow);
            bw[1] = *reinterpret_cast<const unsigned *>(src + c1 * kPairRow);
            unsigned bg[2][8], bm[2][8];
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const int sh = 2 * (e & 3) + 16 * (e >> 2) - 4;   // pair e's codes to bits 4 and 12
                    const unsigned x = sh < 0 ? bw[n] << (sh < 0 ? -sh : 0) : bw[n] >> (sh < 0 ? 0 : sh);
                    const unsigned sel = (x & 0x3030u) | 0x0404u;
                    bg[n][e] = __byte_perm(kGenoTable, 0u, sel);
                    bm[n][e] = MISS ? __byte_perm(kMissTable, 0u, sel) : 0u;
                }
#pragma unroll
            for (int ri = 0; ri < R16; ++ri) {
                const unsigned w0 = *reinterpret_cast<const unsigned *>(src + (16 * ri + fg) * kPairRow);
                const unsigned w1 = *reinterpret_cast<const unsigned *>(src + (16 * ri + 8 + fg) * kPairRow);
#pragma unroll
                for (int s = 0; s < 4; ++s) {
                    const int sa = 4 * (s & 1) + 16 * (s >> 1) - 4, sb = sa + 2;   // pairs 2 s and 2 s + 1
                    const unsigned e00 = ((sa < 0 ? w0 << 4 : w0 >> (sa < 0 ? 0 : sa)) & 0x3030u) | 0x0404u;
                    const unsigned e10 = ((sa < 0 ? w1 << 4 : w1 >> (sa < 0 ? 0 : sa)) & 0x3030u) | 0x0404u;
                    const unsigned e01 = ((sb < 0 ? w0 << 2 : w0 >> (sb < 0 ? 0 : sb)) & 0x3030u) | 0x0404u;
                    const unsigned e11 = ((sb < 0 ? w1 << 2 : w1 >> (sb < 0 ? 0 : sb)) & 0x3030u) | 0x0404u;
                    const unsigned a0 = __byte_perm(kGenoTable, 0u, e00), a1 = __byte_perm(kGenoTable, 0u, e10);
                    const unsigned a2 = __byte_perm(kGenoTable, 0u, e01), a3 = __byte_perm(kGenoTable, 0u, e11);
                    mma_f16(acc[0][ri][0], a0, a1, a2, a3, bg[0][2 * s], bg[0][2 * s + 1]);
                    if (two)
                        mma_f16(acc[0][ri][1], a0, a1, a2, a3, bg[1][2 * s], bg[1][2 * s + 1]);
                    if (MISS >= 1) {
                        mma_f16(acc[NM > 1 ? 1 : 0][ri][0], a0, a1, a2, a3, bm[0][2 * s], bm[0][2 * s + 1]);
                        if (two)
                            mma_f16(acc[NM > 1 ? 1 : 0][ri][1], a0, a1, a2, a3, bm[1][2 * s], bm[1][2 * s + 1]);
                    }
                    if (MISS >= 2) {
                        const unsigned m0 = __byte_perm(kMissTable, 0u, e00), m1 = __byte_perm(kMissTable, 0u, e10);
                        const unsigned m2 = __byte_perm(kMissTable, 0u, e01), m3 = __byte_perm(kMissTable, 0u, e11);
                        mma_f16(acc[NM > 2 ? 2 : 0][ri][0], m0, m1, m2, m3, bg[0][2 * s], bg[0][2 * s + 1]);
                        mma_f16(acc[NM > 2 ? 3 : 0][ri][0], m0, m1, m2, m3, bm[0][2 * s], bm[0][2 * s + 1]);
                        if (two) {
                            mma_f16(acc[NM > 2 ? 2 : 0][ri][1], m0, m1, m2, m3, bg[1][2 * s], bg[1][2 * s + 1]);
                            mma_f16(acc[NM > 2 ? 3 : 0][ri][1], m0, m1, m2, m3, bm[1][2 * s], bm[1][2 * s + 1]);
                        }
                    }
                }
            }
        }
    }
    // the warps' sums through shared memory (the stages are done with)
    cp_async_wait_all();
    __syncthreads();
    int *s_sum = reinterpret_cast<int *>(smem);      // [NM][kPairCols][NT]
    for (int i = tid; i < NM * kPairCols * NT; i += 256)
        s_sum[i] = 0;
    __syncthreads();
#pragma unroll
    for (int m = 0; m < NM; ++m)
#pragma unroll
        for (int ri = 0; ri < R16; ++ri)
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    atomicAdd(&s_sum[(m * kPairCols + 8 * n + 2 * fq + (e & 1)) * NT + 16 * ri + fg + 8 * (e >> 1)],
                              (int)acc[m][ri][n][e]);
    __syncthreads();
    for (int m = 0; m < NM; ++m)
        for (int i = tid; i < nrow * NT; i += 256) {
            int *dst = out + m * mode_stride + ((size_t)b * NT + r0) * NT + i;
            if (gridDim.y > 1)
                atomicAdd(dst, s_sum[m * kPairCols * NT + i]);
            else
                *dst = s_sum[m * kPairCols * NT + i];
        }
}

template <int NT, int MISS>
cudaError_t pair_sums(const uint32_t *order, int64_t M, int B, const uint8_t *codes, int64_t col_stride,
                      const uint32_t *nz, int all, int *sums, int64_t stride, dim3 grid, cudaStream_t st)
{
    constexpr int smem = kPairStages * NT * kPairRow;
    static_assert(smem >= 4 * kPairCols * NT * 4, "the warps' sums take the stages' place");
    const cudaError_t e = cudaFuncSetAttribute((const void *)k_pair_sums<NT, MISS>,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess)
        return e;
    k_pair_sums<NT, MISS><<<grid, 256, smem, st>>>(order, M, B, codes, col_stride, nz, all, sums, stride);
    return cudaGetLastError();
}

template <int NT>
cudaError_t pair_sums(const uint32_t *order, int64_t M, int B, const uint8_t *codes, int64_t col_stride,
                      const uint32_t *nz, int all, int *sums, int64_t stride, int modes, dim3 grid, cudaStream_t st)
{
    return modes == 1   ? pair_sums<NT, 0>(order, M, B, codes, col_stride, nz, all, sums, stride, grid, st)
           : modes == 2 ? pair_sums<NT, 1>(order, M, B, codes, col_stride, nz, all, sums, stride, grid, st)
                        : pair_sums<NT, 2>(order, M, B, codes, col_stride, nz, all, sums, stride, grid, st);
}

// G[p][t], the move of marker t's num per unit of beta_old - beta_new at marker
// p, from the integer sums: an exact integer numerator (64 bits hold 16 N^3 up to
// N = 800,000, else 128) times the two markers' scales, so nothing cancels in
// floating point.  The numerators are over the markers' counts of present
// genotypes (dense), over N (ragged) or N^2 (Eigen); the per-marker quotients are
// formed once per block, because an FP64 division costs about ten FP64 operations.
template <class I>
__global__ void k_pair_gram(const uint32_t *__restrict__ order, int64_t M, int64_t N, int B, int NT, int kind,
                            int eigen, int missing, int64_t pad, const double *__restrict__ table,
                            const double *__restrict__ scale, const int64_t *__restrict__ counts,
                            const uint32_t *__restrict__ nz, int all, const int *__restrict__ sums,
                            int64_t mode_stride, double *__restrict__ G)
{
    __shared__ int64_t s_q[kMaxSpec], s_m[kMaxSpec];   // genotype sum, missing count
    __shared__ double s_s[kMaxSpec];
    __shared__ int s_row[kMaxSpec];
    const int64_t b = blockIdx.x;
    const int gn = gram_entries_per_block(B);
    const int rows = (int)imin64(B, M - b * B);
    const unsigned long long mask = block_rows(nz, b, B, rows, all != 0);
    for (int p = threadIdx.x; p < rows; p += blockDim.x) {
        const int64_t j = order[b * B + p];
        s_q[p] = counts[4 * j + 1] + 2 * counts[4 * j + 2];
        s_m[p] = counts[4 * j + 3];
        s_s[p] = kind == BRR_KIND_DENSE ? scale[2 * j] / (double)(N - s_m[p]) : 1.0 / table[4 * j + 1];
        if ((mask >> p) & 1ull)
            s_row[__popcll(mask & ((1ull << p) - 1ull))] = p;
    }
    __syncthreads();
    const double over = kind == BRR_KIND_DENSE ? 1.0 : eigen ? 1.0 / ((double)N * (double)N) : 1.0 / (double)N;
    const int nrow = __popcll(mask);
    for (int e = threadIdx.x; e < nrow * B; e += blockDim.x) {
        const int rk = e / B, p = s_row[rk], t = e % B;
        if (p >= t)
            continue;
        double v = 0.0;
        if (t < rows) {
            const I sp = s_q[p], st = s_q[t], mp = s_m[p], mt = s_m[t];
            const int *w = sums + ((size_t)b * NT + rk) * NT + t;
            const I P = w[0], Nn = N;
            I num;
            if (kind == BRR_KIND_DENSE && !missing) {
                // N P - q_p q_t over N, the second N in s_s
                num = (Nn * P - sp * st) * Nn;
            } else {
                const I Gmp = missing ? w[mode_stride] : 0;    // genotypes of t over those missing at p
                I Gmt = 0, MM = 0;
                if (missing && (kind == BRR_KIND_DENSE || eigen)) {
                    Gmt = w[2 * mode_stride];
                    MM = w[3 * mode_stride] - pad;
                }
                if (kind == BRR_KIND_DENSE) {
                    const I np = Nn - mp, nt = Nn - mt;
                    num = np * nt * P - np * st * (sp - Gmt) - sp * nt * (st - Gmp) + sp * st * (Nn - mp - mt + MM);
                } else if (!eigen) {
                    num = Nn * P + sp * Gmp - sp * st;
                } else {
                    num = Nn * Nn * P - Nn * sp * (st - Gmp) + Nn * st * Gmt - st * sp * (mt - MM) - st * sp * mp;
                }
            }
            v = (double)num * over * (s_s[p] * s_s[t]);
        }
        G[(size_t)b * gn + p * (2 * B - p - 1) / 2 + (t - p - 1)] = v;
    }
}

// The effects, components and chosen flags of a sweep that ended well, and P(component 0)
// of every marker at its final num (src/BayesRBase.cpp:346; acum null: left as it
// was; acum_given: num holds it).  A sweep with a status leaves the chain as it was.
template <int KM>
__global__ void k_round_finish(int64_t M, int form, const int *__restrict__ err, const double *__restrict__ beta_out,
                               const int32_t *__restrict__ comp_out, const double *__restrict__ num,
                               bool acum_given, const double *__restrict__ u, const int32_t *__restrict__ group,
                               const double *__restrict__ gconst, const int32_t *__restrict__ gK,
                               double *__restrict__ beta, int32_t *__restrict__ comp, uint8_t *__restrict__ chosen,
                               double *__restrict__ acum)
{
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= M || *err != kDevOk)
        return;
    const int c = comp_out[j];
    beta[j] = beta_out[j];
    chosen[j] = c >= 0 ? 1 : 0;
    if (c >= 0)
        comp[j] = c;
    if (!acum)
        return;
    if (acum_given) {
        acum[j] = num[j];
        return;
    }
    const int g = group[j];
    const double *gc = gconst + (size_t)g * kMaxK * 4;
    if (form == BRR_FORM_FP64) {
        acum[j] = pick_marker<false, KM>(num[j], u[j], 0.0, 0.0, gc, gK[g]).acum0;
        return;
    }
    float gcf[2 * KM];
#pragma unroll
    for (int k = 0; k < KM; ++k) {
        gcf[2 * k] = k == 0 ? 0.f : __double2float_rn(gc[4 * k] - gc[0]);
        gcf[2 * k + 1] = k == 0 ? 0.f : __double2float_rn(gc[4 * k + 2]);
    }
    float h, l, a0;
    int picked;
    df_from_double(num[j], h, l);
    if (pick_f32<KM>(h, l, __double2float_rn(u[j]), gcf, gK[g], picked, a0))
        acum[j] = (double)a0;
    else
        acum[j] = pick_marker<true, KM>(num[j], u[j], 0.0, 0.0, gc, gK[g]).acum0;
}

const void *round_fn(int km, bool prof, bool cl)
{
    if (cl)
        return km <= 4 ? (prof ? (const void *)k_round_cl<4, true> : (const void *)k_round_cl<4, false>)
                       : (prof ? (const void *)k_round_cl<kMaxK, true> : (const void *)k_round_cl<kMaxK, false>);
    return km <= 4 ? (prof ? (const void *)k_round<4, true> : (const void *)k_round<4, false>)
                   : (prof ? (const void *)k_round<kMaxK, true> : (const void *)k_round<kMaxK, false>);
}

cudaError_t round_attrs(const void *f, size_t smem, bool cl)
{
    cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess && cl)
        e = cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return e;
}

cudaLaunchConfig_t round_config(int G, size_t smem, cudaStream_t st, cudaLaunchAttribute *attr, bool cl)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)G);
    cfg.blockDim = dim3(kRT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    if (cl) {
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)G;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
    } else {
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

}  // namespace

// --------------------------------------------------------------------------
// Launchers.

size_t round_smem_bytes(const SweepArgs &a)
{
    return round_plan(a.slice_max, a.B, a.n_groups, a.cluster, a.rmode == kRoundPairs, a.has_missing != 0).total;
}

size_t round_smem_limit(int dev)
{
    const void *fs[10] = {(const void *)k_round_multi<4>, (const void *)k_round_multi<kMaxK>};
    int n = 2, optin = 0;
    for (int km : {4, kMaxK})
        for (int v = 0; v < 4; ++v)
            fs[n++] = round_fn(km, (v & 1) != 0, (v & 2) != 0);
    size_t used = 0;
    for (const void *f : fs) {
        cudaFuncAttributes fa{};
        if (cudaFuncGetAttributes(&fa, f) != cudaSuccess) {
            cudaGetLastError();
            return 0;
        }
        used = fa.sharedSizeBytes > used ? fa.sharedSizeBytes : used;
    }
    if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return (size_t)optin - used;
}

// CTAs that can be resident at once: per SM without a cluster, else 1 when a
// cluster of G CTAs can be scheduled (0: none).
int round_fits(int G, size_t smem, bool cluster)
{
    int n = 1 << 30;
    for (int km : {4, kMaxK})
        for (bool prof : {false, true}) {
            const void *f = round_fn(km, prof, cluster);
            cudaLaunchAttribute attr[1];
            const cudaLaunchConfig_t cfg = round_config(G, smem, nullptr, attr, cluster);
            int m = 0;
            const cudaError_t e =
                round_attrs(f, smem, cluster) != cudaSuccess ? cudaErrorInvalidValue
                : cluster ? cudaOccupancyMaxActiveClusters(&m, f, &cfg)
                          : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&m, f, kRT, smem);
            if (e != cudaSuccess) {
                cudaGetLastError();
                return 0;
            }
            n = m < n ? m : n;
        }
    return n;
}

cudaError_t launch_round(const SweepArgs &a, size_t smem, cudaStream_t st)
{
    const bool cl = a.cluster > 0;
    const void *f = round_fn(a.kmax, a.prof != nullptr, cl);
    cudaError_t e = round_attrs(f, smem, cl);
    if (e != cudaSuccess)
        return e;
    cudaLaunchAttribute attr[1];
    const cudaLaunchConfig_t cfg = round_config(a.G, smem, st, attr, cl);
    SweepArgs args = a;
    void *params[] = {&args};
    return cudaLaunchKernelExC(&cfg, f, params);
}

// Sets the kernel's shared-memory attribute too, which must happen outside a
// stream capture of launch_round_multi.
int round_multi_ctas_per_sm(int kmax, size_t smem)
{
    const void *f = kmax <= 4 ? (const void *)k_round_multi<4> : (const void *)k_round_multi<kMaxK>;
    int n = 0;
    if (round_attrs(f, smem, false) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, f, kRT, smem) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

cudaError_t launch_round_multi(int kmax, const MultiSweepArgs &m, size_t smem, cudaStream_t st)
{
    cudaLaunchAttribute attr[1];
    const cudaLaunchConfig_t cfg = round_config(m.cta_start[m.n], smem, st, attr, false);
    MultiSweepArgs args = m;
    void *params[] = {&args};
    return cudaLaunchKernelExC(&cfg, kmax <= 4 ? (const void *)k_round_multi<4> : (const void *)k_round_multi<kMaxK>,
                               params);
}

cudaError_t launch_round_gather(const uint32_t *order, int64_t M, int64_t N, int kind, int kmax, const double *table,
                                const double *scale, const int64_t *counts, const double *beta, const double *u,
                                const double *z, const int32_t *group, const double *gconst, const int32_t *gK,
                                float likely, RoundRec *rec, uint32_t *nz, cudaStream_t st)
{
    const unsigned nb = (unsigned)((M + 255) / 256);
    if (kmax <= 4)
        k_round_gather<4><<<nb, 256, 0, st>>>(order, M, N, kind, table, scale, counts, beta, u, z, group, gconst, gK, likely, rec, nz);
    else
        k_round_gather<kMaxK><<<nb, 256, 0, st>>>(order, M, N, kind, table, scale, counts, beta, u, z, group, gconst, gK,
                                                  likely, rec, nz);
    return cudaGetLastError();
}

static int pair_tile(int B) { return B <= 16 ? 16 : B; }

int round_pair_modes(int kind, int eigen, int missing)
{
    return !missing ? 1 : (kind == BRR_KIND_DENSE || eigen) ? 4 : 2;
}

void round_pair_sizes(int64_t M, int B, int modes, size_t *sum_words, size_t *gram_doubles)
{
    const int64_t nb = (M + B - 1) / B;
    const int NT = pair_tile(B);
    *sum_words = (size_t)modes * nb * NT * NT;
    *gram_doubles = (size_t)nb * gram_entries_per_block(B) + 2;
}

cudaError_t launch_round_pairs(const uint32_t *order, int64_t M, int64_t N, int B, int kind, int eigen, int missing,
                               const uint8_t *codes, int64_t col_stride, const double *table, const double *scale,
                               const int64_t *counts, const uint32_t *nz, int all, int *sums, double *gram, int sms,
                               cudaStream_t st)
{
    const int64_t nb = (M + B - 1) / B;
    const int NT = pair_tile(B);
    const int modes = round_pair_modes(kind, eigen, missing);
    const int64_t stride = nb * NT * NT;
    // few blocks: the individuals are split over more CTAs, at least one segment each
    const int64_t split = imax64(1, imin64((2 * sms + nb - 1) / nb, (col_stride + kPairSeg - 1) / kPairSeg));
    cudaError_t e = cudaSuccess;
    if (split > 1)
        e = cudaMemsetAsync(sums, 0, sizeof(int) * (size_t)stride * modes, st);
    const dim3 grid((unsigned)nb, (unsigned)split, (unsigned)((B + kPairCols - 1) / kPairCols));
    if (e == cudaSuccess)
        e = NT == 16   ? pair_sums<16>(order, M, B, codes, col_stride, nz, all, sums, stride, modes, grid, st)
            : NT == 32 ? pair_sums<32>(order, M, B, codes, col_stride, nz, all, sums, stride, modes, grid, st)
                       : pair_sums<64>(order, M, B, codes, col_stride, nz, all, sums, stride, modes, grid, st);
    if (e != cudaSuccess)
        return e;
    const int64_t pad = 4 * col_stride - N;   // individuals past the last have missing codes
    if (N <= 800000)
        k_pair_gram<int64_t><<<(unsigned)nb, 256, 0, st>>>(order, M, N, B, NT, kind, eigen, missing, pad, table, scale,
                                                           counts, nz, all, sums, stride, gram);
    else
        k_pair_gram<__int128><<<(unsigned)nb, 256, 0, st>>>(order, M, N, B, NT, kind, eigen, missing, pad, table, scale,
                                                            counts, nz, all, sums, stride, gram);
    return cudaGetLastError();
}

size_t batch_pair_words(int64_t M) { return (size_t)((M + 63) / 64) * 64 * 64; }

cudaError_t launch_batch_pairs(const uint32_t *order, int64_t M, const uint8_t *codes, int64_t col_stride, int *sums0,
                               int *sums1, int sms, cudaStream_t st)
{
    for (int half = 0; half < 2; ++half) {
        const int64_t m = M - 32 * half;
        if (m < 1)
            break;
        const int64_t nb = (m + 63) / 64;
        int *sums = half ? sums1 : sums0;
        const int64_t split = imax64(1, imin64((2 * sms + nb - 1) / nb, (col_stride + kPairSeg - 1) / kPairSeg));
        cudaError_t e = cudaSuccess;
        if (split > 1)
            e = cudaMemsetAsync(sums, 0, sizeof(int) * (size_t)nb * 4096, st);
        if (e == cudaSuccess)
            e = pair_sums<64, 0>(order + 32 * half, m, 64, codes, col_stride, nullptr, 1, sums, nb * 4096,
                                 dim3((unsigned)nb, (unsigned)split, 64 / kPairCols), st);
        if (e != cudaSuccess)
            return e;
    }
    return cudaSuccess;
}

cudaError_t launch_round_finish(const SweepArgs &a, const int32_t *group, bool acum_given, cudaStream_t st)
{
    const unsigned nb = (unsigned)((a.M + 127) / 128);
    double *acum = a.async_batch > 0 ? nullptr : a.acum;   // processColumnAsync leaves acum as it was
    const auto f = a.kmax <= 4 ? k_round_finish<4> : k_round_finish<kMaxK>;
    f<<<nb, 128, 0, st>>>(a.M, a.form, a.err, a.beta_out, a.comp_out, a.num_out, acum_given, a.u, group, a.gconst,
                          a.gK, a.beta, a.comp, a.chosen, acum);
    return cudaGetLastError();
}

}  // namespace brr
