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
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// x = hi + lo with hi the 11 leading bits and lo the next ones (the subtraction is exact; the tensor path reads
// the 11 leading bits of lo, so 22 bits of x take part)
__device__ __forceinline__ void split(float x, uint32_t& hi, uint32_t& lo) {
  hi = __float_as_uint(x) & 0xffffe000u;
  lo = __float_as_uint(x - __uint_as_float(hi));
}

// acc (two 16 x 8 column tiles) += A B of two 16 x 16 fp32 blocks, each factor split in two:
// hi hi + hi lo + lo hi, so the result keeps fp32 accuracy (what is dropped is 2^-22 of a term)
__device__ __forceinline__ void block_mac(const float* A, const float* B, int gr, int tc, float (&acc)[2][4]) {
#pragma unroll
  for (int k = 0; k < 16; k += 8) {
    uint32_t ah[4], al[4];
    split(A[gr * BP + k + tc], ah[0], al[0]);
    split(A[(gr + 8) * BP + k + tc], ah[1], al[1]);
    split(A[gr * BP + k + tc + 4], ah[2], al[2]);
    split(A[(gr + 8) * BP + k + tc + 4], ah[3], al[3]);
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      uint32_t bh[2], bl[2];
      split(B[(k + tc) * BP + 8 * n + gr], bh[0], bl[0]);
      split(B[(k + tc + 4) * BP + 8 * n + gr], bh[1], bl[1]);
      mma_tf32(acc[n], al, bh);
      mma_tf32(acc[n], ah, bl);
      mma_tf32(acc[n], ah, bh);
    }
  }
}
__device__ __forceinline__ void block_store(float* p, int gr, int tc, const float (&acc)[2][4], float sign) {
#pragma unroll
  for (int n = 0; n < 2; ++n) {
    *reinterpret_cast<float2*>(p + gr * BP + 8 * n + 2 * tc) = make_float2(sign * acc[n][0], sign * acc[n][1]);
    *reinterpret_cast<float2*>(p + (gr + 8) * BP + 8 * n + 2 * tc) = make_float2(sign * acc[n][2], sign * acc[n][3]);
  }
}

// One merge level: NB blocks per side, 4 / NB pairs.  16 warps; ends with a __syncthreads().
template <int NB>
__device__ __forceinline__ void merge(float* t, float* tmp, int warp, int lane) {
  const int gr = lane >> 2, tc = lane & 3;
  const int pair = warp / (NB * NB), ib = (warp / NB) % NB, jb = (warp + warp / NB) % NB;   // (jb rotated: the skipped work spreads over the SM's quarters)
  const int J0 = pair * 2 * NB, I0 = J0 + NB;
  const bool on = warp < 4 * NB;
  if (on) {
    float acc[2][4] = {};
#pragma unroll 1
    for (int mb = jb; mb < NB; ++mb) block_mac(blk(t, I0 + ib, J0 + mb), blk(t, J0 + mb, J0 + jb), gr, tc, acc);
    block_store(tmp + ((pair * NB + ib) * NB + jb) * BS, gr, tc, acc, 1.f);
  }
  __syncthreads();
  if (on) {
    float acc[2][4] = {};
#pragma unroll 1
    for (int mb = 0; mb <= ib; ++mb) block_mac(blk(t, I0 + ib, I0 + mb), tmp + ((pair * NB + mb) * NB + jb) * BS, gr, tc, acc);
    block_store(blk(t, I0 + ib, J0 + jb), gr, tc, acc, -1.f);
  }
  __syncthreads();
}

// t: A on entry (diagonal blocks strictly lower, upper part zero), T on return.  512 threads, t visible to all.
// The substitution keeps 128 threads busy; the others run `others` meanwhile.
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
      float s0 = 0.f, s1 = 0.f;
#pragma unroll
      for (int u = 0; u < (i + 3) / 4; ++u) {
        const float4 a4 = *reinterpret_cast<const float4*>(d + i * BP + 4 * u);
        const float av[4] = {a4.x, a4.y, a4.z, a4.w};
#pragma unroll
        for (int m = 0; m < 4; ++m)
          if (4 * u + m < i) { if (m & 1) s1 = fmaf(av[m], col[4 * u + m], s1); else s0 = fmaf(av[m], col[4 * u + m], s0); }
      }
      if (i > jl) col[i] = -(s0 + s1);
    }
    __syncwarp();                        // a block's 16 columns sit in one warp: all of A has been read
#pragma unroll
    for (int i = 0; i < 16; ++i) d[i * BP + jl] = col[i];
  } else {
    others();
  }
  __syncthreads();
  merge<1>(t, tmp, warp, lane);
  merge<2>(t, tmp, warp, lane);
  merge<4>(t, tmp, warp, lane);
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
