// Genotype x residual products on the tensor cores, shared by the sweep kernels
// (sm_103a): the 2-bit codes decoded in registers to FP16 operands and the
// fixed-point residual as FP16 limb planes in shared memory.
//
// The residual E (int64, |E| < 2^62) is held as seven balanced 10-bit limbs, E =
// sum l_k 2^(10 k) with l_k in [-512, 511] (the last one smaller), each a plane of
// FP16 values; a genotype (0, 1, 2) times a limb summed over up to 8,192 individuals
// is an integer below 2^24, so FP32 accumulation is exact.  The limbs are the 8
// columns of an m16n8k16 tile (columns l0 l1 l2 0 l3 l4 l5 l6) and 16 markers its
// rows.
//
// Positions: the 16 individuals of a 32-bit code word are stored in the order the
// decoding leaves them in, pairs (0,4) (1,5) (2,6) (3,7) (8,12) (9,13) (10,14) (11,15).
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace brr {

constexpr int kLimbs = 7;
constexpr int kLimbPlanes = 8;

// Bytes of one limb plane: 16 beyond a multiple of 128, so that the eight columns of a
// fragment load hit different banks.
__host__ __device__ inline int limb_plane_stride(int slice_max) { return 2 * slice_max + 16; }

// Individual (within the slice) at position i.
__device__ __forceinline__ int limb_individual(int i)
{
    return (i & ~15) + (((i >> 1) & 3) | (((i >> 3) & 1) << 3) | ((i & 1) << 2));
}

// Shift that brings the code of the first individual of pair pr (positions 2 pr and
// 2 pr + 1) of a code word to bit 0; the second one is 8 bits above it.
__device__ __forceinline__ int limb_pair_shift(int pr) { return 2 * ((pr & 3) | (((pr >> 2) & 1) << 3)); }

// The limbs of pair pr into the planes.
__device__ __forceinline__ void put_limbs(unsigned char *planes, int plane_stride, int pr, long long e0, long long e1)
{
    constexpr unsigned long long bias =
        512ull * (1ull + (1ull << 10) + (1ull << 20) + (1ull << 30) + (1ull << 40) + (1ull << 50));
    const unsigned long long b0 = (unsigned long long)e0 + bias, b1 = (unsigned long long)e1 + bias;
    unsigned char *dst = planes + 4 * pr;
#pragma unroll
    for (int k = 0; k < kLimbs; ++k) {
        const int col = k < 3 ? k : k + 1;
        unsigned v0, v1;
        half2 off;
        if (k < kLimbs - 1) {
            v0 = (unsigned)(b0 >> (10 * k)) & 1023u;
            v1 = (unsigned)(b1 >> (10 * k)) & 1023u;
            off = __half2half2(__ushort_as_half(0x6600));   // 1024 + 512
        } else {
            v0 = (unsigned)((long long)b0 >> 60) + 8u;
            v1 = (unsigned)((long long)b1 >> 60) + 8u;
            off = __half2half2(__ushort_as_half(0x6408));   // 1024 + 8
        }
        // 0x6400 | v is the FP16 value 1024 + v
        const unsigned w = 0x64006400u | v0 | (v1 << 16);
        *reinterpret_cast<half2 *>(dst + (size_t)col * plane_stride) = __hsub2(*reinterpret_cast<const half2 *>(&w), off);
    }
}

// 16 genotypes of a code word as FP16 pairs, pair K in the order above.  `table`
// holds the high byte of the FP16 value of each 2-bit code.
constexpr unsigned kGenoTable = 0x003C0040u;   // codes 0: 2.0, 1 (missing): 0, 2: 1.0, 3: 0
constexpr unsigned kMissTable = 0x00003C00u;   // code 1: 1.0
template <int K>
__device__ __forceinline__ unsigned geno_pair(unsigned w, unsigned table)
{
    const unsigned s = K == 0 ? w << 4 : K == 1 ? w << 2 : K == 2 ? w : w >> (K == 3 ? 2 : 4 + 2 * K);
    return __byte_perm(table, 0u, (s & 0x3030u) | 0x0404u);
}

__device__ __forceinline__ void mma_f16(float (&c)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0,
                                        unsigned b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                 "{%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// One 64-individual chunk of a 16-marker tile: code words w0 (this lane's marker
// row) and w1 (that + 8) against the chunk's limbs x, y.
__device__ __forceinline__ void mma_chunk(float (&c)[4], unsigned w0, unsigned w1, unsigned table, uint4 x, uint4 y)
{
    mma_f16(c, geno_pair<0>(w0, table), geno_pair<0>(w1, table), geno_pair<1>(w0, table), geno_pair<1>(w1, table), x.x,
            x.y);
    mma_f16(c, geno_pair<2>(w0, table), geno_pair<2>(w1, table), geno_pair<3>(w0, table), geno_pair<3>(w1, table), x.z,
            x.w);
    mma_f16(c, geno_pair<4>(w0, table), geno_pair<4>(w1, table), geno_pair<5>(w0, table), geno_pair<5>(w1, table), y.x,
            y.y);
    mma_f16(c, geno_pair<6>(w0, table), geno_pair<6>(w1, table), geno_pair<7>(w0, table), geno_pair<7>(w1, table), y.z,
            y.w);
}

// A tile's sums for marker row m: the warps of the tile left them in `part` as rows of
// eight columns, `n` parts `stride` float4 apart; word 0 is the low part of the sum
// (limbs 0-2), word 1 the high part, the sum being high 2^30 + low.
__device__ __forceinline__ long long limb_sum(const float *part, int m, int word, int n, int stride)
{
    const float4 *src = reinterpret_cast<const float4 *>(part + (size_t)m * 8) + word;
    // integers below 2^24 in any order of addition
    float4 f = src[0];
    for (int k = 1; k < n; ++k) {
        const float4 g = src[(size_t)k * stride];
        f.x += g.x; f.y += g.y; f.z += g.z; f.w += g.w;
    }
    return (long long)(int)f.x + ((long long)(int)f.y << 10) + ((long long)(int)f.z << 20) + ((long long)(int)f.w << 30);
}

}  // namespace brr
