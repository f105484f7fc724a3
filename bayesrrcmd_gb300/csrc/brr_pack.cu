// Device packer: PLINK BED payload -> device marker store.
//
// Replaces the per-genotype MarkerBuilder calls of the reference preprocess
// (src/preprocessgraph.cpp:24-60 drives DenseMarkerBuilder /
// RaggedSparseMarkerBuilder::processAllele once per genotype).  Here the 2-bit
// codes stay 2-bit in HBM (one column per marker, padded to 16-byte chunks of
// 64 individuals), per-marker genotype counts are reduced on the device and
// the standardisation table or ragged statistics are derived from the counts.
#include "brr_device.cuh"
#include "brr_internal.h"
#include "brr_stream.h"

namespace brr {

// Decode of one 2-bit field (src/preprocessgraph.cpp:43-56): allele1 = !bit0,
// allele2 = !bit1; (0,1) is missing (src/densemarkerbuilder.cpp:30).
//   code 0 -> g = 2, code 1 -> missing, code 2 -> g = 1, code 3 -> g = 0.

// Genotype counts of the 16 codes in a word whose low 2 * n bits are valid, by
// population counts: g = 1, g = 2, missing.
struct CodeCounts {
    int c1, c2, cm;
};
__device__ __forceinline__ void count_codes(unsigned w, unsigned valid, CodeCounts &c)
{
    const unsigned m = valid & 0x55555555u, l = w & m, h = (w >> 1) & m;
    c.c1 += __popc(h & ~l);
    c.cm += __popc(l & ~h);
    c.c2 += __popc(m & ~(l | h));
}
// Mask of the first n codes of a word.
__device__ __forceinline__ unsigned code_mask(int64_t n)
{
    return n <= 0 ? 0u : n >= 16 ? 0xFFFFFFFFu : (1u << (2 * n)) - 1u;
}

// One warp per marker, a lane per 16 bytes of its column: the payload's bytes start
// at any address, so a lane reads the five aligned words around its 16 bytes and
// shifts them into place; the few lanes whose words would leave the payload read
// bytes.  Bits past the last individual become missing codes.  Bound by HBM: a byte
// at a time took 374 us for N = 20,011 x M = 20,000 (100 MB in and out), this 50 us.
__global__ void __launch_bounds__(kThreads) k_pack_counts(const uint8_t *__restrict__ bed, int64_t N,
                                                          int64_t M, uint8_t *__restrict__ codes,
                                                          int64_t col_stride, int64_t *__restrict__ counts)
{
    const int64_t cb = (N + 3) >> 2, chunks = col_stride / 16;
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (kThreads / 32);
    const uint8_t *const end = bed + M * cb;
    for (int64_t j = (int64_t)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5); j < M; j += warps) {
        const uint8_t *src = bed + j * cb;
        uint4 *dst = reinterpret_cast<uint4 *>(codes + j * col_stride);
        CodeCounts c{0, 0, 0};
#pragma unroll 2
        for (int64_t k = lane; k < chunks; k += 32) {
            const uint8_t *at = src + 16 * k;
            const uint32_t *al = reinterpret_cast<const uint32_t *>((uintptr_t)at & ~(uintptr_t)3);
            unsigned w[4];
            if (reinterpret_cast<const uint8_t *>(al) >= bed && reinterpret_cast<const uint8_t *>(al + 5) <= end) {
                unsigned x[5];
#pragma unroll
                for (int q = 0; q < 5; ++q)
                    x[q] = __ldg(al + q);
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    w[q] = __funnelshift_r(x[q], x[q + 1], 8u * (unsigned)((uintptr_t)at & 3));
            } else {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    w[q] = 0u;
                    for (int e = 0; e < 4; ++e)
                        if (16 * k + 4 * q + e < cb)
                            w[q] |= (unsigned)at[4 * q + e] << (8 * e);
                }
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const unsigned v = code_mask(N - 64 * k - 16 * q);
                count_codes(w[q], v, c);
                w[q] = (w[q] & v) | (0x55555555u & ~v);
            }
            dst[k] = make_uint4(w[0], w[1], w[2], w[3]);
        }
        const int c1 = __reduce_add_sync(0xffffffffu, c.c1), c2 = __reduce_add_sync(0xffffffffu, c.c2),
                  cm = __reduce_add_sync(0xffffffffu, c.cm);
        if (lane < 4)
            counts[4 * j + lane] = lane == 0 ? N - c1 - c2 - cm : lane == 1 ? c1 : lane == 2 ? c2 : cm;
    }
}

// Totals over the markers of the counts of g = 1, g = 2 and missing.
__global__ void __launch_bounds__(kThreads) k_count_totals(const int64_t *__restrict__ counts, int64_t M,
                                                           unsigned long long *__restrict__ tot)
{
    long long t[3] = {0, 0, 0};
    for (int64_t j = (int64_t)blockIdx.x * kThreads + threadIdx.x; j < M; j += (int64_t)gridDim.x * kThreads)
#pragma unroll
        for (int k = 0; k < 3; ++k)
            t[k] += counts[4 * j + 1 + k];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            t[k] += __shfl_xor_sync(0xffffffffu, t[k], o);
        if ((threadIdx.x & 31) == 0 && t[k])
            atomicAdd(&tot[k], (unsigned long long)t[k]);
    }
}

// Dense standardisation table from the counts (src/densemarkerbuilder.cpp:43-60):
// missing -> mean of non-missing, centre by the column mean, scale to squared
// norm N-1.  The column holds four distinct values, so mean, column mean and
// squared norm follow from the counts; every operation is a separately rounded
// IEEE operation so the table is bit-identical to the CPU restatement.
__global__ void k_dense_tables(const int64_t *__restrict__ counts, int64_t N, int64_t M,
                               double *__restrict__ lut, double *__restrict__ scale, double *__restrict__ colsum,
                               int *bad)
{
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= M)
        return;
    const int64_t n0 = counts[4 * j], n1 = counts[4 * j + 1], n2 = counts[4 * j + 2], nm = counts[4 * j + 3];
    if (nm >= N) {
        atomicMin(bad, (int)j);
        return;
    }
    const double S = (double)(n1 + 2 * n2);
    const double mean = __ddiv_rn(S, __dsub_rn((double)N, (double)nm));
    const double colmean = __ddiv_rn(__dadd_rn(S, __dmul_rn((double)nm, mean)), (double)N);
    const double c0 = __dsub_rn(0.0, colmean), c1 = __dsub_rn(1.0, colmean);
    const double c2 = __dsub_rn(2.0, colmean), cm = __dsub_rn(mean, colmean);
    const double sqn = __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn((double)n0, __dmul_rn(c0, c0)),
                                                     __dmul_rn((double)n1, __dmul_rn(c1, c1))),
                                           __dmul_rn((double)n2, __dmul_rn(c2, c2))),
                                 __dmul_rn((double)nm, __dmul_rn(cm, cm)));
    if (!(sqn > 0.0)) {
        atomicMin(bad, (int)j);
        return;
    }
    const double sigma = __ddiv_rn(1.0, __dsqrt_rn(__ddiv_rn(sqn, __dsub_rn((double)N, 1.0))));
    lut[4 * j + 0] = __dmul_rn(c2, sigma);
    lut[4 * j + 1] = __dmul_rn(cm, sigma);
    lut[4 * j + 2] = __dmul_rn(c1, sigma);
    lut[4 * j + 3] = __dmul_rn(c0, sigma);
    scale[2 * j + 0] = sigma;
    scale[2 * j + 1] = colmean;
    // sum of the standardised column (zero up to rounding)
    colsum[j] = (double)n0 * lut[4 * j + 3] + (double)n1 * lut[4 * j + 2] + (double)n2 * lut[4 * j + 0] +
                (double)nm * lut[4 * j + 1];
}

// Ragged statistics (src/sparsemarker.cpp:8-19, src/raggedsparsemarkerbuilder.cpp:43-55):
// mean over N including missing, sd from the sum and sum of squares.
__global__ void k_ragged_stats(const int64_t *__restrict__ counts, int64_t N, int64_t M, int eigen,
                               double *__restrict__ stats, int *bad)
{
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= M)
        return;
    const int64_t n1 = counts[4 * j + 1], n2 = counts[4 * j + 2];
    double Zsum = (double)(n1 + 2 * n2);
    double sqrdZ = (double)(n1 + 4 * n2);
    const double Nd = (double)N;
    const double mean = __ddiv_rn(Zsum, Nd);
    if (eigen) {
        // src/eigensparsemarkerbuilder.cpp:46-56: the missing genotypes enter
        // sqrdZ and Zsum at the mean before the sd is formed
        const double nm = (double)counts[4 * j + 3];
        sqrdZ = __dadd_rn(sqrdZ, __dmul_rn(__dmul_rn(mean, mean), nm));
        Zsum = __dadd_rn(Zsum, __dmul_rn(mean, nm));
    }
    const double var = __ddiv_rn(__dadd_rn(__dsub_rn(sqrdZ, __dmul_rn(__dmul_rn(2.0, mean), Zsum)),
                                           __dmul_rn(__dmul_rn(Nd, mean), mean)),
                                 __dsub_rn(Nd, 1.0));
    const double sd = __dsqrt_rn(var);
    stats[4 * j + 0] = mean;
    stats[4 * j + 1] = sd;
    stats[4 * j + 2] = sqrdZ;
    stats[4 * j + 3] = Zsum;
    // src/raggedsparsemarker.cpp:68-77: a marker without ones and twos is invalid.
    if (n1 + n2 == 0 || !(sd > 0.0))
        atomicMin(bad, (int)j);
}

// Per (marker, slice) counts of ones / twos / missing for the slice-major ragged
// layout: a thread per slice, 64 individuals (16 bytes: slices begin on chunks) at a
// time.  N = 20,011 x M = 20,000, 152 slices: 382 us an individual at a time, 34 us so.
__global__ void __launch_bounds__(kThreads) k_ragged_slice_counts(const uint8_t *__restrict__ codes,
                                                                  int64_t col_stride, int64_t M, int G,
                                                                  const int32_t *__restrict__ slice_lo,
                                                                  int32_t *__restrict__ cnt3)
{
    const int64_t MG = M * (int64_t)G;
    // M G fits 31 bits
    for (unsigned e = blockIdx.x * kThreads + threadIdx.x; e < (unsigned)MG; e += gridDim.x * kThreads) {
        const unsigned j = e / (unsigned)G, s = e - j * (unsigned)G;
        const int lo = slice_lo[s], hi = slice_lo[s + 1];
        const uint4 *col = reinterpret_cast<const uint4 *>(codes + (int64_t)j * col_stride + (lo >> 2));
        CodeCounts c{0, 0, 0};
        for (int i = lo; i < hi; i += 64) {
            const uint4 w = __ldg(col++);
            count_codes(w.x, code_mask(hi - i), c);
            count_codes(w.y, code_mask(hi - i - 16), c);
            count_codes(w.z, code_mask(hi - i - 32), c);
            count_codes(w.w, code_mask(hi - i - 48), c);
        }
        cnt3[e] = c.c1;
        cnt3[MG + 1 + e] = c.c2;
        cnt3[2 * (MG + 1) + e] = c.cm;
    }
}

// Fill slice-local indices in ascending order (src/raggedsparsemarkerbuilder.cpp:25-41
// appends in decode order, i.e. ascending individual index), from the set bits of the
// genotypes that are not 0.  A warp takes 32 consecutive (marker, slice) pairs, whose
// lists lie one behind the other: they are put together in shared memory and leave as
// contiguous stores, because a store per entry costs a sector of the L2 each.  Pairs
// with more entries than the buffer holds are stored one by one.  N = 20,011 x
// M = 20,000 (80 M entries): 780 us an individual at a time, 544 us from the set
// bits with a store per entry, 314 us this way.
constexpr int kFillEntries = 4608;      // per warp

__global__ void __launch_bounds__(kThreads) k_ragged_fill(const uint8_t *__restrict__ codes, int64_t col_stride,
                                                          int64_t M, int G, const int32_t *__restrict__ slice_lo,
                                                          const int32_t *__restrict__ off0,
                                                          const int32_t *__restrict__ off1,
                                                          const int32_t *__restrict__ off2,
                                                          uint16_t *__restrict__ idx0, uint16_t *__restrict__ idx1,
                                                          uint16_t *__restrict__ idx2)
{
    extern __shared__ uint16_t s_fill[];
    const unsigned MG = (unsigned)(M * (int64_t)G);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint16_t *const buf = s_fill + warp * kFillEntries;
    const int32_t *const off[3] = {off0, off1, off2};
    uint16_t *const idx[3] = {idx0, idx1, idx2};
    const unsigned step = gridDim.x * kThreads;
    for (unsigned e0 = blockIdx.x * kThreads + 32 * warp; e0 < MG; e0 += step) {
        const unsigned e = e0 + lane < MG ? e0 + lane : MG, e1 = e0 + 32 < MG ? e0 + 32 : MG;
        int32_t first[3], count[3];
        uint16_t *at[3];
        int32_t total = 0;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            first[k] = off[k][e0];
            count[k] = off[k][e1] - first[k];
            total += count[k];
        }
        const bool staged = total <= kFillEntries;
        uint16_t *seg = buf;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const int32_t o = off[k][e];
            at[k] = staged ? seg + (o - first[k]) : idx[k] + o;
            seg += count[k];
        }
        if (e < MG) {
            const unsigned j = e / (unsigned)G, s = e - j * (unsigned)G;
            const int lo = slice_lo[s], n = slice_lo[s + 1] - lo;
            const uint4 *col = reinterpret_cast<const uint4 *>(codes + (int64_t)j * col_stride + (lo >> 2));
            for (int i = 0; i < n; i += 64) {
                const uint4 v = __ldg(col++);
                const unsigned w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const unsigned in = code_mask(n - i - 16 * q) & 0x55555555u, l = w[q] & in, h = (w[q] >> 1) & in;
                    for (unsigned r = in & ~(l & h); r; r &= r - 1u) {
                        const int p = __ffs(r) - 1;
                        const uint16_t li = (uint16_t)(i + 16 * q + (p >> 1));
                        if ((h >> p) & 1u)
                            *at[0]++ = li;
                        else if ((l >> p) & 1u)
                            *at[2]++ = li;
                        else
                            *at[1]++ = li;
                    }
                }
            }
        }
        if (staged) {
            __syncwarp();
            const uint16_t *src = buf;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                for (int32_t x = lane; x < count[k]; x += 32)
                    idx[k][first[k] + x] = src[x];
                src += count[k];
            }
            __syncwarp();
        }
    }
}

// Exclusive scans of several int32 arrays of n elements one behind the other, in
// three passes (tile scan, scan of tile sums in one CTA per array, add).  Tiles of
// 1024 elements; tile_sums: as many words per array as there are tiles.
constexpr int kScanTile = 1024;

__global__ void __launch_bounds__(kThreads) k_scan_tiles(int32_t *data, int64_t n, int32_t *tile_sums)
{
    data += n * blockIdx.y;
    tile_sums += (int64_t)gridDim.x * blockIdx.y;
    __shared__ int32_t sh[kScanTile];
    __shared__ int32_t wsum[kThreads / 32];
    const int64_t base = (int64_t)blockIdx.x * kScanTile;
    for (int k = threadIdx.x; k < kScanTile; k += blockDim.x)
        sh[k] = (base + k < n) ? data[base + k] : 0;
    __syncthreads();
    // each thread scans 4 consecutive elements
    const int t = threadIdx.x;
    int32_t v0 = sh[4 * t], v1 = sh[4 * t + 1], v2 = sh[4 * t + 2], v3 = sh[4 * t + 3];
    const int32_t tot = v0 + v1 + v2 + v3;
    int32_t x = tot;
    const int l = t & 31, w = t >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (l >= o)
            x += y;
    }
    if (l == 31)
        wsum[w] = x;
    __syncthreads();
    int32_t wpre = 0;
    for (int q = 0; q < w; ++q)
        wpre += wsum[q];
    const int32_t excl = wpre + x - tot;
    sh[4 * t] = excl;
    sh[4 * t + 1] = excl + v0;
    sh[4 * t + 2] = excl + v0 + v1;
    sh[4 * t + 3] = excl + v0 + v1 + v2;
    __syncthreads();
    for (int k = threadIdx.x; k < kScanTile; k += blockDim.x)
        if (base + k < n)
            data[base + k] = sh[k];
    if (threadIdx.x == blockDim.x - 1) {
        int32_t s = 0;
        for (int q = 0; q < (int)(blockDim.x >> 5); ++q)
            s += wsum[q];
        tile_sums[blockIdx.x] = s;
    }
}

__global__ void __launch_bounds__(1024) k_scan_sums(int32_t *tile_sums, int64_t ntiles)
{
    __shared__ int32_t wsum[32];
    tile_sums += ntiles * blockIdx.x;
    const int t = threadIdx.x, l = t & 31, w = t >> 5;
    int32_t run = 0;
    for (int64_t q0 = 0; q0 < ntiles; q0 += 1024) {
        const int32_t v = q0 + t < ntiles ? tile_sums[q0 + t] : 0;
        int32_t x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (l >= o)
                x += y;
        }
        if (l == 31)
            wsum[w] = x;
        __syncthreads();
        int32_t pre = 0, all = 0;
        for (int k = 0; k < 32; ++k) {
            pre += k < w ? wsum[k] : 0;
            all += wsum[k];
        }
        if (q0 + t < ntiles)
            tile_sums[q0 + t] = run + pre + x - v;
        run += all;
        __syncthreads();
    }
}

__global__ void k_scan_add(int32_t *data, int64_t n, const int32_t *tile_sums, int64_t ntiles)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n)
        data[n * blockIdx.y + i] += tile_sums[ntiles * blockIdx.y + i / kScanTile];
}

cudaError_t launch_pack_counts(const uint8_t *bed, int64_t N, int64_t M, uint8_t *codes, int64_t col_stride,
                               int64_t *counts, cudaStream_t st)
{
    const int blocks = (int)imin64((M + 7) / 8, 152 * 8);
    k_pack_counts<<<blocks, kThreads, 0, st>>>(bed, N, M, codes, col_stride, counts);
    return cudaGetLastError();
}

cudaError_t launch_dense_tables(const int64_t *counts, int64_t N, int64_t M, double *lut, double *scale,
                                double *colsum, int *bad, cudaStream_t st)
{
    k_dense_tables<<<(unsigned)((M + 255) / 256), 256, 0, st>>>(counts, N, M, lut, scale, colsum, bad);
    return cudaGetLastError();
}

cudaError_t launch_ragged_stats(const int64_t *counts, int64_t N, int64_t M, int eigen, double *stats, int *bad,
                                cudaStream_t st)
{
    k_ragged_stats<<<(unsigned)((M + 255) / 256), 256, 0, st>>>(counts, N, M, eigen, stats, bad);
    return cudaGetLastError();
}

cudaError_t launch_ragged_slice_counts(const uint8_t *codes, int64_t col_stride, int64_t M, int G,
                                       const int32_t *slice_lo, int32_t *cnt3, cudaStream_t st)
{
    const int blocks = (int)imin64((M * G + kThreads - 1) / kThreads, 152 * 32);
    k_ragged_slice_counts<<<blocks, kThreads, 0, st>>>(codes, col_stride, M, G, slice_lo, cnt3);
    return cudaGetLastError();
}

cudaError_t launch_count_totals(const int64_t *counts, int64_t M, unsigned long long *tot, cudaStream_t st)
{
    const cudaError_t e = cudaMemsetAsync(tot, 0, 3 * sizeof *tot, st);
    if (e != cudaSuccess)
        return e;
    k_count_totals<<<(unsigned)imin64((M + kThreads - 1) / kThreads, 152), kThreads, 0, st>>>(counts, M, tot);
    return cudaGetLastError();
}

int64_t scan_tiles(int64_t n) { return (n + kScanTile - 1) / kScanTile; }

cudaError_t launch_exclusive_scans_i32(int32_t *data, int64_t n, int arrays, int32_t *tmp, cudaStream_t st)
{
    const int64_t ntiles = scan_tiles(n);
    const unsigned y = (unsigned)arrays;
    k_scan_tiles<<<dim3((unsigned)ntiles, y), kThreads, 0, st>>>(data, n, tmp);
    k_scan_sums<<<y, 1024, 0, st>>>(tmp, ntiles);
    k_scan_add<<<dim3((unsigned)((n + 255) / 256), y), 256, 0, st>>>(data, n, tmp, ntiles);
    return cudaGetLastError();
}

cudaError_t launch_ragged_fill(const uint8_t *codes, int64_t col_stride, int64_t M, int G, const int32_t *slice_lo,
                               const int32_t *off0, const int32_t *off1, const int32_t *off2, uint16_t *idx0,
                               uint16_t *idx1, uint16_t *idx2, cudaStream_t st)
{
    const int blocks = (int)imin64((M * G + kThreads - 1) / kThreads, 152 * 32);
    const int smem = kThreads / 32 * kFillEntries * (int)sizeof(uint16_t);
    const cudaError_t e = cudaFuncSetAttribute((const void *)k_ragged_fill, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess)
        return e;
    k_ragged_fill<<<blocks, kThreads, smem, st>>>(codes, col_stride, M, G, slice_lo, off0, off1, off2, idx0, idx1, idx2);
    return cudaGetLastError();
}

}  // namespace brr

namespace brr {

// Seeded synthetic genotypes written directly as a BED payload: marker j has
// allele frequency p_j = p_lo + (p_hi - p_lo) * U, genotypes are two
// Bernoulli(p_j) draws, missing at rate `miss`.  Every byte is a function of
// (seed, j, byte index) through the same Philox stream as the sampler.
__global__ void k_synth_bed(uint8_t *__restrict__ out, int64_t N, int64_t M, uint32_t seed, double p_lo,
                            double p_hi, double miss, double beta_a, double beta_b)
{
    const int64_t cb = (N + 3) >> 2;
    for (int64_t j = blockIdx.x; j < M; j += gridDim.x) {
        float p;
        if (beta_a > 0.0) {
            // p ~ Beta(a, b) = X / (X + Y), X ~ Gamma(a), Y ~ Gamma(b), clipped to [p_lo, p_hi]
            __shared__ double s_p;
            if (threadIdx.x == 0) {
                double x = 1.0, y = 1.0;
                const StreamKey k{seed, 0x5EEDu};
                gamma_draw(k, (uint32_t)j, 12u, 0u, beta_a, &x);
                gamma_draw(k, (uint32_t)j, 12u, 1u, beta_b, &y);
                s_p = fmin(fmax(x / (x + y), p_lo), p_hi);
            }
            __syncthreads();
            p = (float)s_p;
            __syncthreads();
        } else {
            const U4 pb = philox4x32_10((uint32_t)j, 0u, 9u, 0u, seed, 0x5EEDu);
            p = (float)(p_lo + (p_hi - p_lo) * u53(pb.x, pb.y));
        }
        const uint32_t t1 = (uint32_t)fminf(4294967040.f, p * 4294967296.f);
        const uint32_t tm = (uint32_t)fminf(4294967040.f, (float)miss * 4294967296.f);
        for (int64_t b = threadIdx.x; b < cb; b += blockDim.x) {
            const U4 r = philox4x32_10((uint32_t)j, (uint32_t)b, 10u, 0u, seed, 0x5EEDu);
            const U4 q = philox4x32_10((uint32_t)j, (uint32_t)b, 11u, 0u, seed, 0x5EEDu);
            const uint32_t ra[4] = {r.x, r.y, r.z, r.w};
            const uint32_t qa[4] = {q.x, q.y, q.z, q.w};
            unsigned byte = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                // two allele draws from the two halves of one 32-bit word (16 bits each)
                const unsigned a1 = (ra[k] & 0xFFFFu) < (t1 >> 16);
                const unsigned a2 = (ra[k] >> 16) < (t1 >> 16);
                const unsigned gv = a1 + a2;
                unsigned code = gv == 2 ? 0u : (gv == 1 ? 2u : 3u);
                if (qa[k] < tm)
                    code = 1u;
                if (b * 4 + k >= N)
                    code = 0u;
                byte |= code << (2 * k);
            }
            out[j * cb + b] = (uint8_t)byte;
        }
        // keep every marker polymorphic: individual 0 heterozygous, 1 homozygous
        if (threadIdx.x == 0 && N >= 2) {
            unsigned v = out[j * cb];
            v = (v & ~0x0Fu) | 2u | (3u << 2);
            out[j * cb] = (uint8_t)v;
        }
    }
}

cudaError_t launch_synth_bed(uint8_t *out, int64_t N, int64_t M, uint32_t seed, double p_lo, double p_hi,
                             double miss, cudaStream_t st, double beta_a, double beta_b)
{
    const int blocks = (int)imin64(M, 152 * 32);
    k_synth_bed<<<blocks, kThreads, 0, st>>>(out, N, M, seed, p_lo, p_hi, miss, beta_a, beta_b);
    return cudaGetLastError();
}

}  // namespace brr
