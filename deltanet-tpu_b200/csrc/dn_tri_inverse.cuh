// (I + A)^-1 of a strictly lower triangular 128 x 128 fp32 matrix in shared memory, in place, and the
// two products that consume it (W = T X, U = T Y): the tail shared by the forward prepass kernels.
//
// Storage: only the 36 blocks of 16 x 16 on and below the diagonal are kept, block (bi, bj) at
// (bi (bi + 1) / 2 + bj), rows of 20 floats (rows r and r + 8 of a block then fall into different banks,
// and so do eight consecutive rows read 16 bytes at a time): 45 KB instead of the 66 KB of a padded square, which is
// what lets two CTAs share an SM.
//
// Method: substitution on the diagonal blocks, then block merges T21 = -T22 (A21 T11) at 16, 32, 64 rows; blocks that
// are zero by triangularity are skipped and a warp owns one 16 x 16 block of a merge's result.  On the CUDA cores the
// merges are bound by shared memory: a 16-byte load moves 512 bytes into registers whether or not lanes share
// addresses, 96 cycles per block product against 32 of multiply-adds.  As warp-level tensor products on
// operands split in two (fp32 accuracy) a block product loads each element once per warp, 16 cycles.
#pragma once
#include "dn_chunkprep.cuh"
#include "dn_umma.cuh"

namespace dn {
namespace tri {

constexpr int BP = 20;                  // floats per row of a block
constexpr int BS = 16 * BP;             // floats per block
constexpr int BLOCKS = 36;
constexpr int BYTES = BLOCKS * BS * 4;
constexpr int TMP_BYTES = 16 * BS * 4;  // products of the widest merge

__device__ __forceinline__ float* blk(float* t, int bi, int bj) { return t + (bi * (bi + 1) / 2 + bj) * BS; }

// One m16n8k8 product on the warp-level tensor path, tf32 operands, fp32 accumulation.
__device__ __forceinline__ void mma_tf32(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// x = hi + lo with hi the 11 leading bits and lo the next ones (the subtraction is exact; the tensor path reads
// the 11 leading bits of lo, so 22 bits of x take part)
__device__ __forceinline__ void split(float x, uint32_t& hi, uint32_t& lo) {
  hi = __float_as_uint(x) & 0xffffe000u;
  lo = __float_as_uint(x - __uint_as_float(hi));
}

// A product's rows, columns and contraction index may be dealt to the fragments in any order.  With row slot gr holding row pi(gr) (three bits
// reversed), contraction slots tc and tc + 4 the indices 2 tc and 2 tc + 1, and column slot c of tile n column 2 c + n, a lane's
// operands are pairs of neighbours, its results are four neighbouring columns of a row, and a block's 20-float rows keep the
// quarter-warps of all of these accesses apart in the banks: a block product takes 8 shared-memory loads instead of 16 and 16 passes
// of the data stage instead of about 24, and a block is stored by 2 stores instead of 4.
__device__ __forceinline__ int row_slot(int gr) { return ((gr & 1) << 2) | (gr & 2) | (gr >> 2); }

// acc (two 16 x 8 column tiles) += A B of two 16 x 16 fp32 blocks, each factor split in two:
// hi hi + hi lo + lo hi, so the result keeps fp32 accuracy (what is dropped is 2^-22 of a term).  The two column tiles take
// turns: a product waits 21 cycles for one that it adds to and 8 for the unit.  r: row_slot(lane >> 2)
__device__ __forceinline__ void block_mac(const float* A, const float* B, int gr, int r, int tc, float (&acc)[2][4]) {
  A += r * BP + 2 * tc;
  B += 2 * tc * BP + 2 * gr;
#pragma unroll
  for (int k = 0; k < 16; k += 8) {
    const float2 a0 = *reinterpret_cast<const float2*>(A + k), a1 = *reinterpret_cast<const float2*>(A + 8 * BP + k);
    const float2 b0 = *reinterpret_cast<const float2*>(B + k * BP), b1 = *reinterpret_cast<const float2*>(B + (k + 1) * BP);
    uint32_t ah[4], al[4], bh[2][2], bl[2][2];
    split(a0.x, ah[0], al[0]);
    split(a1.x, ah[1], al[1]);
    split(a0.y, ah[2], al[2]);
    split(a1.y, ah[3], al[3]);
    split(b0.x, bh[0][0], bl[0][0]);
    split(b1.x, bh[0][1], bl[0][1]);
    split(b0.y, bh[1][0], bl[1][0]);
    split(b1.y, bh[1][1], bl[1][1]);
    mma_tf32(acc[0], al, bh[0]);
    mma_tf32(acc[1], al, bh[1]);
    mma_tf32(acc[0], ah, bh[0]);
    mma_tf32(acc[1], ah, bh[1]);
    mma_tf32(acc[0], ah, bl[0]);
    mma_tf32(acc[1], ah, bl[1]);
  }
}
__device__ __forceinline__ void block_store(float* p, int r, int tc, const float (&acc)[2][4], float sign) {
  p += r * BP + 4 * tc;
  *reinterpret_cast<float4*>(p) = make_float4(sign * acc[0][0], sign * acc[1][0], sign * acc[0][1], sign * acc[1][1]);
  *reinterpret_cast<float4*>(p + 8 * BP) = make_float4(sign * acc[0][2], sign * acc[1][2], sign * acc[0][3], sign * acc[1][3]);
}

__device__ __forceinline__ void bar_sync(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

// One merge level: NB blocks per side, 4 / NB pairs, a warp per block of the results.  SYNC: the barrier among the warps that take part.
template <int NB, class SYNC>
__device__ __forceinline__ void merge(float* t, float* tmp, int warp, int lane, SYNC sync) {
  const int gr = lane >> 2, tc = lane & 3, r = row_slot(gr);
  const int pair = warp / (NB * NB), ib = (warp / NB) % NB, jb = (warp + warp / NB) % NB;   // (jb rotated: the skipped work spreads over the SM's quarters)
  const int J0 = pair * 2 * NB, I0 = J0 + NB;
  {
    float acc[2][4] = {};
#pragma unroll 1
    for (int mb = jb; mb < NB; ++mb) block_mac(blk(t, I0 + ib, J0 + mb), blk(t, J0 + mb, J0 + jb), gr, r, tc, acc);
    block_store(tmp + ((pair * NB + ib) * NB + jb) * BS, r, tc, acc, 1.f);
  }
  sync();
  {
    float acc[2][4] = {};
#pragma unroll 1
    for (int mb = 0; mb <= ib; ++mb) block_mac(blk(t, I0 + ib, I0 + mb), tmp + ((pair * NB + mb) * NB + jb) * BS, gr, r, tc, acc);
    block_store(blk(t, I0 + ib, J0 + jb), r, tc, acc, -1.f);
  }
}

// t: A on entry (diagonal blocks strictly lower, upper part zero), T on return.  512 threads, t visible to all.
// Work comes in fours: warp p's lanes are the columns of the diagonal blocks 2 p and 2 p + 1, which are also all that the first merge
// of warp p reads; the second merge has 8 blocks, the last one 16.  So warps 4 to 7 join at the second merge and 8 to 15 at the
// last, by barriers of their own, and run `others` before (about 2000 cycles for the latter).
template <class OTHERS>
__device__ __forceinline__ void invert(float* t, float* tmp, OTHERS others) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid < 128) {                       // thread = (diagonal block, column)
    const int b = tid >> 4, jl = tid & 15;
    float* d = blk(t, b, b);
    float col[16];
#pragma unroll
    for (int m = 0; m < 16; ++m) col[m] = m == jl ? 1.f : 0.f;
#pragma unroll
    for (int i = 1; i < 16; ++i) {
      float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int u = 0; u < (i + 3) / 4; ++u) {
        const float4 a4 = *reinterpret_cast<const float4*>(d + i * BP + 4 * u);
        const float av[4] = {a4.x, a4.y, a4.z, a4.w};
#pragma unroll
        for (int m = 0; m < 4; ++m)
          if (4 * u + m < i) s[m] = fmaf(av[m], col[4 * u + m], s[m]);
      }
      if (i > jl) col[i] = -((s[0] + s[1]) + (s[2] + s[3]));
    }
    __syncwarp();                        // a block's 16 columns sit in one warp: all of A has been read
#pragma unroll
    for (int i = 0; i < 16; ++i) d[i * BP + jl] = col[i];
    __syncwarp();
    merge<1>(t, tmp, warp, lane, [] { __syncwarp(); });
  } else {
    others();
  }
  if (warp < 8) {
    bar_sync(2, 256);
    merge<2>(t, tmp, warp, lane, [] { bar_sync(2, 256); });
  }
  __syncthreads();
  merge<4>(t, tmp, warp, lane, [] { __syncthreads(); });
  __syncthreads();
}

// bf16 K-major operand image of T ([col / 8][row][8])
__device__ __forceinline__ void image(float* t, uint4* TI) {
#pragma unroll
  for (int it = 0; it < 4; ++it) {
    const int e = it * 512 + threadIdx.x, p = e >> 7, x = e & 127;
    uint4 v = make_uint4(0, 0, 0, 0);
    if ((p >> 1) <= (x >> 4)) v = umma::ld8_f32(blk(t, x >> 4, p >> 1) + (x & 15) * BP + (p & 1) * 8);
    TI[e] = v;
  }
}

}  // namespace tri
}  // namespace dn
