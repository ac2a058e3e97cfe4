// The steps either side of the recurrence in a Gated DeltaNet layer, as the reference's layer example
// wires them (examples/qwen3_5_layer_parity.py:144-159 of the reference project):
//
//   producer   mixed (B,L,D), D = 2*Hk*K + Hv*V  --depthwise causal conv (width W <= 4) + SiLU-->  q | k | v
//              a, b (B,L,Hv)  -->  g = -exp(A_log) * softplus(a + dt_bias),  beta = sigmoid(b)
//   consumer   y = weight * rmsnorm(o) * silu(z) per (token, value head), o and z of shape (rows, V)
//
// All of it is element-wise or a short stencil over tokens, i.e. bound by HBM bytes: every kernel
// below reads each input once with 16-byte accesses (a thread owns 8 channels and walks a run of
// tokens with the stencil window in registers, so the halo is 3 rows per run) and writes each output
// once.  Parameter gradients (conv weight, bias, A_log, dt_bias, norm weight) are reduced in a fixed
// order through per-tile partial sums, so results are bit-reproducible.
#include <cooperative_groups.h>

#include <type_traits>

#include "dn_kernels.cuh"
#include "dn_umma.cuh"

namespace dn {
namespace {

constexpr int CG = 8;            // channels per thread (one 16-byte bf16 vector)
constexpr int PT = 128;          // threads per CTA of the producer kernels (= 1024 channels)
constexpr int TT_FWD = 64;       // longest run of tokens of a thread, forward
constexpr int TT_BWD = 256;      // the same, backward (a run is also a tile of the weight-gradient partials)
constexpr int MAXW = 4;

__device__ __forceinline__ float silu(float x) { return x * __frcp_rn(1.f + __expf(-x)); }
// d silu(x) / dx = s + x s (1 - s), s = sigmoid(x)
__device__ __forceinline__ float dsilu(float x) {
  const float s = __frcp_rn(1.f + __expf(-x));
  return s * (1.f + x * (1.f - s));
}

struct ProducerArgs {
  const void* mixed;             // (B,L,D)
  const float* w;                // (D,W) depthwise taps; tap W-1 multiplies the current token
  const float* bias;             // (D) or null
  const int32_t* seg;            // (B,L) or null: taps from another document read as zero
  int B, L, D, W, dt;
  int qk_dim, Hk_K;              // Hk*K: channels [0,HkK) -> q, [HkK, 2HkK) -> k, rest -> v
  int run;                       // tokens per thread run, a multiple of 4
  void *q, *k, *v;               // forward outputs / backward: their cotangents
  void* d_mixed;                 // backward
  float* part;                   // backward: (tiles, D, W+1) partial sums of d w | d bias
};

// sigmoid by one MUFU op (tanh.approx, relative error ~2^-11): used where the result is rounded to bf16 anyway
__device__ __forceinline__ float sigmoid_fast(float x) {
  float t;
  asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(0.5f * x));
  return fmaf(0.5f, t, 0.5f);
}
template <bool FAST> __device__ __forceinline__ float silu_t(float x) {
  if (FAST) return x * sigmoid_fast(x);
  return silu(x);
}

// A lane's 4 or 2 channels of one row as they were loaded (conversion to fp32 happens when the row is used, so a
// batch of loads can be issued back to back without holding CG floats per row).
template <bool BF16, int CG_> struct Raw;
template <> struct Raw<true, 4> {
  uint2 r;
  __device__ __forceinline__ void load(const void* base, size_t off) {
    r = __ldg(reinterpret_cast<const uint2*>(reinterpret_cast<const __nv_bfloat16*>(base) + off));
  }
  __device__ __forceinline__ void get(float (&x)[4]) const {
    x[0] = __uint_as_float(r.x << 16); x[1] = __uint_as_float(r.x & 0xffff0000u);
    x[2] = __uint_as_float(r.y << 16); x[3] = __uint_as_float(r.y & 0xffff0000u);
  }
};
template <> struct Raw<false, 4> {
  float4 a;
  __device__ __forceinline__ void load(const void* base, size_t off) {
    a = __ldg(reinterpret_cast<const float4*>(reinterpret_cast<const float*>(base) + off));
  }
  __device__ __forceinline__ void get(float (&x)[4]) const { x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; }
};
template <> struct Raw<true, 2> {
  uint32_t r;
  __device__ __forceinline__ void load(const void* base, size_t off) {
    r = __ldg(reinterpret_cast<const uint32_t*>(reinterpret_cast<const __nv_bfloat16*>(base) + off));
  }
  __device__ __forceinline__ void get(float (&x)[2]) const { x[0] = __uint_as_float(r << 16); x[1] = __uint_as_float(r & 0xffff0000u); }
};
template <> struct Raw<false, 2> {
  float2 a;
  __device__ __forceinline__ void load(const void* base, size_t off) {
    a = __ldg(reinterpret_cast<const float2*>(reinterpret_cast<const float*>(base) + off));
  }
  __device__ __forceinline__ void get(float (&x)[2]) const { x[0] = a.x; x[1] = a.y; }
};

// The token loops below keep a ring of NS batches of NB rows in shared memory, filled by asynchronous
// copies (cp.async) that cost no registers: while batch i is walked with the stencil window in registers,
// the rows of batches i+1 .. i+NS-1 are on their way (12 rows of 16 or 32 bytes per thread).  A thread
// reads back only the slots it filled itself, so the ring needs no block-wide synchronisation.
template <int BYTES> __device__ __forceinline__ void cp_async_row(void* dst, const void* src);
template <> __device__ __forceinline__ void cp_async_row<16>(void* dst, const void* src) { umma::cp_async16(dst, src); }
template <> __device__ __forceinline__ void cp_async_row<8>(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(umma::smem_u32(dst)), "l"(src) : "memory");
}
// Two neighbouring channels, for the packed fp32 instructions (one issue slot for two results; each rounds as its scalar form)
using F2 = unsigned long long;
__device__ __forceinline__ F2 f2(float lo, float hi) {
  F2 d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ void split2(F2 x, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(x)); }
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
  F2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
  F2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ F2 bf16x2_f2(uint32_t r) { return f2(__uint_as_float(r << 16), __uint_as_float(r & 0xffff0000u)); }
__device__ __forceinline__ uint32_t f2_bf16x2(F2 x) {
  float lo, hi;
  split2(x, lo, hi);
  return umma::pack2(lo, hi);
}
__device__ __forceinline__ float tanh_fast(float x) {
  float t;
  asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(x));
  return t;
}
// With h = x / 2 and t = tanh h:  silu(x) = h + h t,  d silu(x) / dx = s (1 + h (1 - t)),  s = (1 + t) / 2
template <bool FAST> __device__ __forceinline__ F2 silu2(F2 x) {
  float lo, hi;
  if (FAST) {
    const F2 h = mul2(x, f2(0.5f, 0.5f));
    split2(h, lo, hi);
    return fma2(h, f2(tanh_fast(lo), tanh_fast(hi)), h);
  }
  split2(x, lo, hi);
  return f2(silu(lo), silu(hi));
}
template <bool FAST> __device__ __forceinline__ F2 dsilu2(F2 x) {
  float lo, hi;
  if (FAST) {
    const F2 half = f2(0.5f, 0.5f), one = f2(1.f, 1.f), h = mul2(x, half);
    split2(h, lo, hi);
    const F2 t = f2(tanh_fast(lo), tanh_fast(hi));
    return mul2(fma2(t, half, half), fma2(h, fma2(t, f2(-1.f, -1.f), one), one));
  }
  split2(x, lo, hi);
  return f2(dsilu(lo), dsilu(hi));
}
// N pairs of channels of one row, from the ring (pieces of 16 bytes lie PT * 16 bytes apart) or from memory, and to memory
template <bool BF16, int N> __device__ __forceinline__ void get_row(const uint8_t* p, F2 (&x)[N], int piece) {
  if (BF16 && N == 4) {
    const uint4 r = *reinterpret_cast<const uint4*>(p);
    x[0] = bf16x2_f2(r.x); x[1] = bf16x2_f2(r.y); x[2 % N] = bf16x2_f2(r.z); x[3 % N] = bf16x2_f2(r.w);
  } else if (BF16) {
    const uint2 r = *reinterpret_cast<const uint2*>(p);
    x[0] = bf16x2_f2(r.x); x[1] = bf16x2_f2(r.y);
  } else {
#pragma unroll
    for (int i = 0; i < N; i += 2) {
      const float4 r = *reinterpret_cast<const float4*>(p + (i / 2) * piece);
      x[i] = f2(r.x, r.y); x[i + 1] = f2(r.z, r.w);
    }
  }
}
template <bool BF16, int N> __device__ __forceinline__ void put_row(char* p, const F2 (&x)[N]) {
  if (BF16 && N == 4) {
    *reinterpret_cast<uint4*>(p) = make_uint4(f2_bf16x2(x[0]), f2_bf16x2(x[1]), f2_bf16x2(x[2 % N]), f2_bf16x2(x[3 % N]));
  } else if (BF16) {
    *reinterpret_cast<uint2*>(p) = make_uint2(f2_bf16x2(x[0]), f2_bf16x2(x[1]));
  } else {
#pragma unroll
    for (int i = 0; i < N; i += 2) {
      float4 r;
      split2(x[i], r.x, r.y);
      split2(x[i + 1], r.z, r.w);
      reinterpret_cast<float4*>(p)[i / 2] = r;
    }
  }
}
// Whether the window of every row of batch `bi` lies in one document; ids[0] belongs to the row W - 1 before the run
template <int W, int NB> __device__ __forceinline__ bool one_document(const int* ids, int bi) {
  bool same = true;
#pragma unroll
  for (int i = 1; i < NB + W - 1; ++i) same &= ids[bi * NB + i] == ids[bi * NB];
  return same;
}

// Forward.  A batch of NB rows whose windows lie in one document, within the run, takes an instance of the body without tests
// of ids and ends (nearly every batch does); both instances add in the same order.  Measured at 2 x 4001 tokens of 8192
// channels, bf16, W = 4: 62.2 us with a test per tap and scalar arithmetic, 58.2 without the tests, 54.5 with packed arithmetic
// besides (4.8 TB/s); 4 x 4096 tokens 109.8, 103.6, 96.8.
template <int W, bool BF16, bool LONG>
__global__ void __launch_bounds__(PT, 4) producer_fwd_kernel(ProducerArgs a) {
  const int run = LONG ? TT_FWD : a.run;
  constexpr int NB = 4, NS = BF16 ? 4 : 2;           // rows per batch, batches in the ring (32 KB either way)
  constexpr int ES = BF16 ? 2 : 4, NP = CG * ES / 16;  // element size; 16-byte copies per row and thread
  __shared__ __align__(16) uint8_t ring[NS * NB * NP * PT * 16];
  __shared__ int seg_sm[TT_FWD + MAXW];              // document ids of rows t0-(W-1) .. t_end-1 (-1 before the sequence)
  const int tid = threadIdx.x;
  const bool active = (blockIdx.y * PT + tid) * CG < a.D;
  const int c0 = active ? (blockIdx.y * PT + tid) * CG : 0;
  const int tiles_per_row = (a.L + run - 1) / run;
  const int b = blockIdx.x / tiles_per_row, t0 = (blockIdx.x % tiles_per_row) * run;
  const size_t row0 = (size_t)b * a.L;
  const int t_end = min(t0 + run, a.L);
  const int nbatch = (t_end - t0 + NB - 1) / NB;
  const char* src = reinterpret_cast<const char*>(a.mixed);
  const char* first = src + ((row0 + t0) * a.D + c0) * ES;
  auto fetch = [&](int bi) {                           // rows past the end read the last row and are not stored
    if (bi < nbatch) {
#pragma unroll
      for (int n = 0; n < NB; ++n) {
        const char* g = first + (uint64_t)(uint32_t)min(bi * NB + n, a.L - 1 - t0) * (uint32_t)(a.D * ES);
        uint8_t* d = ring + ((size_t)(((bi % NS) * NB + n) * NP) * PT + tid) * 16;
#pragma unroll
        for (int h = 0; h < NP; ++h) umma::cp_async16(d + h * PT * 16, g + h * 16);
      }
    }
    umma::cp_async_commit();
  };
#pragma unroll
  for (int bi = 0; bi < NS - 1; ++bi) fetch(bi);
  for (int i = tid; i < run + W - 1; i += PT) {
    const int t = t0 - (W - 1) + i;
    seg_sm[i] = t < 0 ? -1 : (a.seg ? __ldg(a.seg + row0 + min(t, a.L - 1)) : 0);
  }
  constexpr int N2 = CG / 2;
  F2 wt[W][N2], bs[N2], xw[W][N2];                   // xw[j] = x[t - (W-1) + j], j = 0..W-1 (tap j)
#pragma unroll
  for (int i = 0; i < N2; ++i) {
#pragma unroll
    for (int j = 0; j < W; ++j) {
      wt[j][i] = f2(__ldg(a.w + (size_t)(c0 + 2 * i) * W + j), __ldg(a.w + (size_t)(c0 + 2 * i + 1) * W + j));
      xw[j][i] = 0;
    }
    bs[i] = a.bias ? f2(__ldg(a.bias + c0 + 2 * i), __ldg(a.bias + c0 + 2 * i + 1)) : 0;
  }
#pragma unroll
  for (int j = 0; j < W - 1; ++j) {                  // halo rows
    const int t = t0 - (W - 1) + j;
    if (t >= 0) get_row<BF16>(reinterpret_cast<const uint8_t*>(src) + ((row0 + t) * a.D + c0) * ES, xw[j], 16);
  }
  const int HkK = a.Hk_K, Dv = a.D - 2 * HkK;
  // where this thread's channels go: q, k or v, each token-major
  char* obase; uint32_t ostride; int ooff;
  if (c0 < HkK) { obase = (char*)a.q; ostride = HkK; ooff = c0; }
  else if (c0 < 2 * HkK) { obase = (char*)a.k; ostride = HkK; ooff = c0 - HkK; }
  else { obase = (char*)a.v; ostride = Dv; ooff = c0 - 2 * HkK; }
  ostride *= ES;
  obase += (row0 + t0) * ostride + (size_t)ooff * ES;
  __syncthreads();
  // PLAIN: every row of the batch is this run's and has its whole window in its own document
  auto rows = [&](auto plain, int bi) {
    constexpr bool PLAIN = decltype(plain)::value;
    const uint8_t* slot = ring + ((size_t)((bi % NS) * NB * NP) * PT + tid) * 16;
    char* dst = obase + (uint64_t)(uint32_t)(bi * NB) * ostride;
#pragma unroll
    for (int n = 0; n < NB; ++n, dst += ostride) {
      const int* ids = seg_sm + bi * NB + n;
      get_row<BF16>(slot + n * NP * PT * 16, xw[W - 1], PT * 16);
      F2 y[N2];
#pragma unroll
      for (int i = 0; i < N2; ++i) y[i] = bs[i];
#pragma unroll
      for (int j = 0; j < W; ++j) {
        if (PLAIN || ids[j] == ids[W - 1]) {
#pragma unroll
          for (int i = 0; i < N2; ++i) y[i] = fma2(wt[j][i], xw[j][i], y[i]);
        }
      }
#pragma unroll
      for (int i = 0; i < N2; ++i) y[i] = silu2<BF16>(y[i]);
      if (active && (PLAIN || t0 + bi * NB + n < t_end)) put_row<BF16>(dst, y);
#pragma unroll
      for (int j = 0; j + 1 < W; ++j)
#pragma unroll
        for (int i = 0; i < N2; ++i) xw[j][i] = xw[j + 1][i];
    }
  };
#pragma unroll 1
  for (int bi = 0; bi < nbatch; ++bi) {
    fetch(bi + NS - 1);
    umma::cp_async_wait<NS - 1>();
    if (t0 + (bi + 1) * NB <= t_end && one_document<W, NB>(seg_sm, bi)) rows(std::true_type{}, bi);
    else rows(std::false_type{}, bi);
  }
  umma::cp_async_wait<0>();
}

// Backward of the producer over one run of tokens: with pre[u] the conv output of token u and
// dpre[u] = dy[u] * silu'(pre[u]),
//   d x[s]    = sum_j w[j] * dpre[s + (W-1-j)]      (taps inside the same document)
//   d w[j]   += dpre[u] * x[u - (W-1) + j],   d bias += dpre[u]    (u inside this run)
// The loop walks u over the run plus W-1 rows of look-ahead and emits d x with a lag of W-1.  A thread
// owns CB = 4 channels here (the windows of x and dpre and the parameter-gradient accumulators are
// 10 CB + registers), so that twice as many threads are resident as with 8.
// Bound by instruction issue (three stencils, SiLU', unpacking) until whole batches lost their tests, as in the forward, and the
// arithmetic was packed by pairs; a pair's results are those of the scalar instructions.  2 x 4001 tokens of 8192 channels, bf16, W = 4:
// 123.4 us with a test per tap and scalar arithmetic, 118.3 without the tests, 94.5 with packed arithmetic besides (4.2 TB/s;
// packed arithmetic under the tests was slower, 137); 4 x 4096 tokens 210.8, 200.0, 157.7.
constexpr int CB = 4;
template <int W, bool BF16, bool LONG>
__global__ void __launch_bounds__(PT, 4) producer_bwd_kernel(ProducerArgs a) {
  const int run = LONG ? TT_BWD : a.run;
  constexpr int NB = 4, NS = BF16 ? 4 : 2;
  constexpr int ES = BF16 ? 2 : 4, RB = CB * ES;     // bytes per row, thread and tensor: 8 or 16
  __shared__ __align__(16) uint8_t ring[NS * NB * 2 * PT * RB];       // x rows | cotangent rows
  __shared__ int seg_sm[TT_BWD + 2 * MAXW];          // document ids of rows t0-(W-1) .. u_end-1 (-1 / -2 outside the sequence)
  const int tid = threadIdx.x;
  const bool active = (blockIdx.y * PT + tid) * CB < a.D;
  const int c0 = active ? (blockIdx.y * PT + tid) * CB : 0;
  const int tiles_per_row = (a.L + run - 1) / run;
  const int b = blockIdx.x / tiles_per_row, t0 = (blockIdx.x % tiles_per_row) * run;
  const size_t row0 = (size_t)b * a.L;
  const int t_end = min(t0 + run, a.L);
  const int u_end = t_end + W - 1;                   // look-ahead rows; rows >= L contribute nothing
  const int nbatch = (u_end - t0 + NB - 1) / NB;
  const int HkK = a.Hk_K, Dv = a.D - 2 * HkK;
  const char* gbase; size_t gstride, goff;           // this thread's channels of the cotangent of q, k or v
  if (c0 < HkK) { gbase = (const char*)a.q; gstride = HkK; goff = c0; }
  else if (c0 < 2 * HkK) { gbase = (const char*)a.k; gstride = HkK; goff = c0 - HkK; }
  else { gbase = (const char*)a.v; gstride = Dv; goff = c0 - 2 * HkK; }
  const char* xsrc = reinterpret_cast<const char*>(a.mixed);
  const char *xfirst = xsrc + ((row0 + t0) * a.D + c0) * ES, *gfirst = gbase + ((row0 + t0) * gstride + goff) * ES;
  auto fetch = [&](int bi) {                         // rows past the end read the last row and count as not live
    if (bi < nbatch) {
#pragma unroll
      for (int n = 0; n < NB; ++n) {
        const uint32_t u = min(bi * NB + n, a.L - 1 - t0);
        uint8_t* d = ring + ((size_t)(((bi % NS) * NB + n) * 2) * PT + tid) * RB;
        cp_async_row<RB>(d, xfirst + (uint64_t)u * (uint32_t)(a.D * ES));
        cp_async_row<RB>(d + PT * RB, gfirst + (uint64_t)u * (uint32_t)(gstride * ES));
      }
    }
    umma::cp_async_commit();
  };
#pragma unroll
  for (int bi = 0; bi < NS - 1; ++bi) fetch(bi);
  for (int i = tid; i < run + 2 * MAXW; i += PT) {
    const int t = t0 - (W - 1) + i;
    seg_sm[i] = t < 0 ? -1 : (t >= a.L ? -2 : (a.seg ? __ldg(a.seg + row0 + t) : 0));
  }
  constexpr int N2 = CB / 2;
  F2 wt[W][N2], bs[N2], dwt[W][N2], dbs[N2];
  F2 xw[W][N2], dp[W][N2];               // xw[j] = x[u-(W-1)+j]; dp[j] = dpre[u-(W-1)+j]
#pragma unroll
  for (int i = 0; i < N2; ++i) {
#pragma unroll
    for (int j = 0; j < W; ++j) {
      wt[j][i] = f2(__ldg(a.w + (size_t)(c0 + 2 * i) * W + j), __ldg(a.w + (size_t)(c0 + 2 * i + 1) * W + j));
      dwt[j][i] = xw[j][i] = dp[j][i] = 0;
    }
    bs[i] = a.bias ? f2(__ldg(a.bias + c0 + 2 * i), __ldg(a.bias + c0 + 2 * i + 1)) : 0;
    dbs[i] = 0;
  }
#pragma unroll
  for (int j = 0; j < W - 1; ++j) {
    const int t = t0 - (W - 1) + j;
    if (t >= 0) get_row<BF16>(reinterpret_cast<const uint8_t*>(xsrc) + ((row0 + t) * a.D + c0) * ES, xw[j], 16);
  }
  const uint32_t xstride = (uint32_t)a.D * ES;
  char* dbase = reinterpret_cast<char*>(a.d_mixed) + ((row0 + t0) * a.D + c0) * ES;
  __syncthreads();
  // PLAIN: this run owns every row of the batch, and they and the W - 1 rows before each lie in one document and in the run
  auto rows = [&](auto plain, int bi) {
    constexpr bool PLAIN = decltype(plain)::value;
    const uint8_t* slot = ring + ((size_t)((bi % NS) * NB * 2) * PT + tid) * RB;
    char* dst = dbase + (int64_t)(bi * NB - (W - 1)) * xstride;
#pragma unroll
    for (int n = 0; n < NB; ++n, dst += xstride) {
      const int u = t0 + bi * NB + n;
      const int* ids = seg_sm + bi * NB + n;         // ids[W - 1] is -2 past the end of the sequence
      F2 dy[N2], pre[N2];
      get_row<BF16>(slot + n * 2 * PT * RB, xw[W - 1], PT * 16);
      get_row<BF16>(slot + (n * 2 + 1) * PT * RB, dy, PT * 16);
#pragma unroll
      for (int i = 0; i < N2; ++i) pre[i] = bs[i];
#pragma unroll
      for (int j = 0; j < W; ++j) {
        if (PLAIN || ids[j] == ids[W - 1]) {
#pragma unroll
          for (int i = 0; i < N2; ++i) pre[i] = fma2(wt[j][i], xw[j][i], pre[i]);
        }
      }
#pragma unroll
      for (int i = 0; i < N2; ++i) dp[W - 1][i] = PLAIN || u < a.L ? mul2(dy[i], dsilu2<BF16>(pre[i])) : 0;
      if (PLAIN || u < t_end) {                      // parameter gradients of the rows this run owns
#pragma unroll
        for (int j = 0; j < W; ++j) {
          if (PLAIN || ids[j] == ids[W - 1]) {
#pragma unroll
            for (int i = 0; i < N2; ++i) dwt[j][i] = fma2(dp[W - 1][i], xw[j][i], dwt[j][i]);
          }
        }
#pragma unroll
        for (int i = 0; i < N2; ++i) dbs[i] = add2(dbs[i], dp[W - 1][i]);
      }
      // d x of token sx = u - (W-1): output token sx + (W-1-j) used it through tap j; that token sits at window slot W-1-j
      const int sx = u - (W - 1);
      if (PLAIN || (sx >= t0 && sx < t_end)) {
        F2 dx[N2];
#pragma unroll
        for (int i = 0; i < N2; ++i) dx[i] = 0;
#pragma unroll
        for (int j = 0; j < W; ++j) {
          if (PLAIN || ids[W - 1 - j] == ids[0]) {
#pragma unroll
            for (int i = 0; i < N2; ++i) dx[i] = fma2(wt[j][i], dp[W - 1 - j][i], dx[i]);
          }
        }
        if (active) put_row<BF16>(dst, dx);
      }
#pragma unroll
      for (int j = 0; j + 1 < W; ++j)
#pragma unroll
        for (int i = 0; i < N2; ++i) { xw[j][i] = xw[j + 1][i]; dp[j][i] = dp[j + 1][i]; }
    }
  };
#pragma unroll 1
  for (int bi = 0; bi < nbatch; ++bi) {
    fetch(bi + NS - 1);
    umma::cp_async_wait<NS - 1>();
    if (bi * NB >= W - 1 && t0 + (bi + 1) * NB <= t_end && one_document<W, NB>(seg_sm, bi)) rows(std::true_type{}, bi);
    else rows(std::false_type{}, bi);
  }
  umma::cp_async_wait<0>();
  if (!active) return;
  float* p = a.part + ((size_t)blockIdx.x * a.D + c0) * (W + 1);
#pragma unroll
  for (int i = 0; i < N2; ++i, p += 2 * (W + 1)) {
#pragma unroll
    for (int j = 0; j < W; ++j) split2(dwt[j][i], p[j], p[W + 1 + j]);
    split2(dbs[i], p[W], p[2 * W + 1]);
  }
}

// out[e] = sum over tiles of part[tile][e] in a fixed order: a CTA takes 32 elements; each of its 8 warps
// adds one eighth of the tiles in ascending order (independent loads, several in flight), and the eight
// partial sums are added in ascending order.
__global__ void __launch_bounds__(256) tile_sum_kernel(const float* part, int tiles, size_t n, float* out_a, float* out_b,
                                                       int W) {
  __shared__ float red[8][32];
  const int lane = threadIdx.x & 31, grp = threadIdx.x >> 5;
  const size_t e = (size_t)blockIdx.x * 32 + lane;
  const int per = (tiles + 7) / 8, tb = grp * per, te = min(tb + per, tiles);
  float s = 0.f;
  if (e < n) {
    int t = tb;
    for (; t + 8 <= te; t += 8) {
      float v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = __ldg(part + (size_t)(t + u) * n + e);
#pragma unroll
      for (int u = 0; u < 8; ++u) s += v[u];
    }
    for (; t < te; ++t) s += __ldg(part + (size_t)t * n + e);
  }
  red[grp][lane] = s;
  __syncthreads();
  if (grp != 0 || e >= n) return;
  s = red[0][lane];
#pragma unroll
  for (int k = 1; k < 8; ++k) s += red[k][lane];
  if (W < 0) { out_a[e] = s; return; }
  const size_t c = e / (W + 1);
  const int j = (int)(e - c * (W + 1));
  if (j < W) out_a[c * W + j] = s;
  else if (out_b) out_b[c] = s;
}

// ---- gates ------------------------------------------------------------------------------------------
__device__ __forceinline__ float softplus(float x) { return x > 20.f ? x : log1pf(expf(x)); }

__global__ void __launch_bounds__(256) gates_fwd_kernel(const void* a_, const void* b_, int dt, const float* A_log,
                                                        const float* dt_bias, size_t n, int Hv, float* g, float* beta) {
  const size_t e = (size_t)blockIdx.x * 256 + threadIdx.x;
  if (e >= n) return;
  const int h = (int)(e % Hv);
  g[e] = -expf(A_log[h]) * softplus(ldf_ro(a_, e, dt) + dt_bias[h]);
  beta[e] = 1.f / (1.f + expf(-ldf_ro(b_, e, dt)));
}

// da, db element-wise; dA_log[h] = sum dg * g, d dt_bias[h] = sum dg * dg/d(a).  A cluster of 8 CTAs takes 4 heads (so that a
// thread's neighbours read next to it) and adds its partial sums in a fixed order through distributed shared memory:
// 52 us -> 17 us at 8002 tokens x 32 heads, where one CTA per head walked the tokens alone.  A thread's tokens are a chain of loads and
// special functions, four tokens in flight: with THREADS = 512 instead of 256 17.6 -> 11.4 us there and 28.2 -> 15.9 at 16384 tokens; 1024
// threads leave 64 registers, which spill with four in flight: 9.7 and 13.7 with two.  Up to 512 tokens the threads of 256 have one token
// each and 512 would only lengthen the sum over threads: both directions together 5.4 us against 5.8 at 128 and 301 tokens, 5.9 and 5.9 at 600.
constexpr int GB_CTAS = 8, GB_HEADS = 4;
inline bool gates_bwd_narrow(size_t tokens) { return tokens <= (size_t)GB_CTAS * (256 / GB_HEADS); }
template <int THREADS>
__global__ void __cluster_dims__(GB_CTAS, 1, 1) __launch_bounds__(THREADS, 1)
    gates_bwd_kernel(const void* a_, const void* b_, int dt, const float* A_log, const float* dt_bias, const float* dg, const float* dbeta,
                     size_t tokens, int Hv, void* da, void* db, float* dA_log, float* d_dt_bias) {
  __shared__ float red[2][THREADS], sums[2][GB_HEADS];
  const int rank = blockIdx.x % GB_CTAS, tid = threadIdx.x, hl = tid % GB_HEADS, h = blockIdx.x / GB_CTAS * GB_HEADS + hl;
  float sA = 0.f, sB = 0.f;
  if (h < Hv) {
    const float Ae = -expf(A_log[h]), bias = dt_bias[h];
#pragma unroll 4
    for (size_t t = rank * (THREADS / GB_HEADS) + tid / GB_HEADS; t < tokens; t += GB_CTAS * (THREADS / GB_HEADS)) {
      const size_t e = t * Hv + h;
      const float x = ldf_ro(a_, e, dt) + bias, braw = ldf_ro(b_, e, dt), d = __ldg(dg + e), dbe = __ldg(dbeta + e);
      const float sp = softplus(x), sg = 1.f / (1.f + expf(-x));
      const float dx = d * Ae * sg;
      stf(da, e, dx, dt);
      const float be = 1.f / (1.f + expf(-braw));
      stf(db, e, dbe * be * (1.f - be), dt);
      sA += d * Ae * sp;
      sB += dx;
    }
  }
  red[0][tid] = sA;
  red[1][tid] = sB;
  __syncthreads();
  for (int o = THREADS / 2; o >= GB_HEADS; o >>= 1) {
    if (tid < o) { red[0][tid] += red[0][tid + o]; red[1][tid] += red[1][tid + o]; }
    __syncthreads();
  }
  if (tid < GB_HEADS) { sums[0][tid] = red[0][tid]; sums[1][tid] = red[1][tid]; }
  auto cluster = cooperative_groups::this_cluster();
  cluster.sync();
  if (rank == 0 && tid < GB_HEADS && h < Hv) {
    float tA = 0.f, tB = 0.f;
    for (int r = 0; r < GB_CTAS; ++r) {
      const float* peer = cluster.map_shared_rank(&sums[0][0], r);
      tA += peer[tid];
      tB += peer[GB_HEADS + tid];
    }
    dA_log[h] = tA;
    d_dt_bias[h] = tB;
  }
  cluster.sync();                                        // the peers' shared memory has been read
}

// ---- gated RMSNorm -----------------------------------------------------------------------------------
// One warp per row of V (64 or 128) elements, EPL = V / 32 per lane.  The normalised value is rounded to
// the input dtype before the weight is applied, as the layer this mirrors does.
template <int EPL>
__device__ __forceinline__ void st_row(void* base, size_t off, int dt, const float (&x)[EPL]) {
  if (dt == DN_BF16) {
    __nv_bfloat16* p = reinterpret_cast<__nv_bfloat16*>(base) + off;
    if (EPL == 4) *reinterpret_cast<uint2*>(p) = make_uint2(umma::pack2(x[0], x[1]), umma::pack2(x[2], x[3]));
    else *reinterpret_cast<uint32_t*>(p) = umma::pack2(x[0], x[1]);
  } else {
    float* p = reinterpret_cast<float*>(base) + off;
    if (EPL == 4) *reinterpret_cast<float4*>(p) = make_float4(x[0], x[1], x[2], x[3]);
    else *reinterpret_cast<float2*>(p) = make_float2(x[0], x[1]);
  }
}

// A warp takes NR rows per batch with two sets of registers: the rows of batch i + 1 are requested
// before batch i is worked on (rows past the end read the last row and are not stored), so 2 NR
// (forward) or 3 NR (backward) loads per lane are always in flight.
template <int EPL, bool BF16>
__global__ void __launch_bounds__(256) gated_rmsnorm_fwd_kernel(const void* o, const void* z, const float* weight,
                                                                size_t rows, float eps, void* y, float* rstd) {
  constexpr int V = EPL * 32, NR = 4, dt = BF16 ? DN_BF16 : DN_F32;
  const int lane = threadIdx.x & 31;
  float w[EPL];
#pragma unroll
  for (int i = 0; i < EPL; ++i) w[i] = __ldg(weight + lane * EPL + i);
  const size_t stride = (size_t)gridDim.x * 8;
  const size_t rbeg = (size_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  Raw<BF16, EPL> rx[2][NR], rz[2][NR];
  auto fetch = [&](size_t r0, int slot) {
#pragma unroll
    for (int u = 0; u < NR; ++u) {
      const size_t r = min(r0 + u * stride, rows - 1);
      rx[slot][u].load(o, r * V + lane * EPL);
      rz[slot][u].load(z, r * V + lane * EPL);
    }
  };
  if (rbeg < rows) fetch(rbeg, 0);
  int slot = 0;
#pragma unroll 2
  for (size_t r0 = rbeg; r0 < rows; r0 += stride * NR, slot ^= 1) {
    if (r0 + stride * NR < rows) fetch(r0 + stride * NR, slot ^ 1);
#pragma unroll
    for (int u = 0; u < NR; ++u) {
      const size_t r = r0 + u * stride;
      float x[EPL], zz[EPL], out[EPL];
      rx[slot][u].get(x);
      rz[slot][u].get(zz);
      float ss = 0.f;
#pragma unroll
      for (int i = 0; i < EPL; ++i) ss = fmaf(x[i], x[i], ss);
      ss = warp_sum(ss);
      const float rs = rsqrtf(ss * (1.f / V) + eps);
#pragma unroll
      for (int i = 0; i < EPL; ++i) {
        float n = x[i] * rs;
        if (BF16) n = bf16r(n);
        out[i] = w[i] * n * silu_t<BF16>(zz[i]);
      }
      if (r < rows) {
        st_row<EPL>(y, r * V + lane * EPL, dt, out);
        if (rstd && lane == 0) rstd[r] = rs;
      }
    }
  }
}

template <int EPL, bool BF16>
__global__ void __launch_bounds__(256) gated_rmsnorm_bwd_kernel(const void* o, const void* z, const float* weight,
                                                                size_t rows, float eps, const void* dy, void* d_o, void* d_z,
                                                                float* part) {
  constexpr int V = EPL * 32, NR = 2, dt = BF16 ? DN_BF16 : DN_F32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float w[EPL], dwp[EPL];
#pragma unroll
  for (int i = 0; i < EPL; ++i) { w[i] = __ldg(weight + lane * EPL + i); dwp[i] = 0.f; }
  const size_t stride = (size_t)gridDim.x * 8;
  const size_t rbeg = (size_t)blockIdx.x * 8 + warp;
  Raw<BF16, EPL> rx[2][NR], rz[2][NR], rg[2][NR];
  auto fetch = [&](size_t r0, int slot) {
#pragma unroll
    for (int u = 0; u < NR; ++u) {
      const size_t r = min(r0 + u * stride, rows - 1);
      rx[slot][u].load(o, r * V + lane * EPL);
      rz[slot][u].load(z, r * V + lane * EPL);
      rg[slot][u].load(dy, r * V + lane * EPL);
    }
  };
  if (rbeg < rows) fetch(rbeg, 0);
  int slot = 0;
#pragma unroll 2
  for (size_t r0 = rbeg; r0 < rows; r0 += stride * NR, slot ^= 1) {
    if (r0 + stride * NR < rows) fetch(r0 + stride * NR, slot ^ 1);
#pragma unroll
    for (int u = 0; u < NR; ++u) {                   // rows in ascending order: the weight gradient's order of addition is fixed
      const size_t r = r0 + u * stride;
      if (r >= rows) break;
      float x[EPL], zz[EPL], g[EPL], dn_[EPL], n[EPL], dzo[EPL], dxo[EPL];
      rx[slot][u].get(x);
      rz[slot][u].get(zz);
      rg[slot][u].get(g);
      float ss = 0.f;
#pragma unroll
      for (int i = 0; i < EPL; ++i) ss = fmaf(x[i], x[i], ss);
      ss = warp_sum(ss);
      const float rs = rsqrtf(ss * (1.f / V) + eps);
      float dot = 0.f;
#pragma unroll
      for (int i = 0; i < EPL; ++i) {
        n[i] = x[i] * rs;
        const float nr = BF16 ? bf16r(n[i]) : n[i];
        const float sg = BF16 ? sigmoid_fast(zz[i]) : __frcp_rn(1.f + __expf(-zz[i]));
        const float sl = zz[i] * sg;
        dzo[i] = g[i] * w[i] * nr * (sg * (1.f + zz[i] * (1.f - sg)));
        dn_[i] = g[i] * w[i] * sl;
        dwp[i] = fmaf(g[i] * nr, sl, dwp[i]);
        dot = fmaf(dn_[i], n[i], dot);
      }
      dot = warp_sum(dot) * (1.f / V);
#pragma unroll
      for (int i = 0; i < EPL; ++i) dxo[i] = rs * (dn_[i] - n[i] * dot);
      st_row<EPL>(d_o, r * V + lane * EPL, dt, dxo);
      st_row<EPL>(d_z, r * V + lane * EPL, dt, dzo);
    }
  }
  __shared__ float red[8][V];
#pragma unroll
  for (int i = 0; i < EPL; ++i) red[warp][lane * EPL + i] = dwp[i];
  __syncthreads();
  for (int c = threadIdx.x; c < V; c += 256) {
    float sacc = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) sacc += red[k][c];
    part[(size_t)blockIdx.x * V + c] = sacc;
  }
}

// CTAs of 8 warps that walk the rows with a grid stride: as many as are resident at once (per_sm per SM,
// from the occupancy of the kernel instance; 8 is the upper bound the scratch is sized for)
int norm_grid(size_t rows, int per_sm = 8) {
  const size_t want = (rows + 7) / 8, cap = (size_t)sm_count() * (per_sm < 1 ? 1 : (per_sm > 8 ? 8 : per_sm));
  return (int)(want < cap ? (want ? want : 1) : cap);
}
template <typename KernelT> int resident_ctas(KernelT kernel) {
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, 256, 0) != cudaSuccess) { cudaGetLastError(); n = 4; }
  return n;
}

}  // namespace
}  // namespace dn

using namespace dn;

// Length of the producer's runs.  A run is walked row by row, so a small call takes as long as one run does: runs are halved
// while all CTAs, at half the length, still fit the chip together: four per SM in the backward (its runs are long); one in the
// forward, where more only add halo rows and the set-up of taps.  Backward, D channels and L tokens: D = 2048, L = 301
// 37.6 -> 9.1 us (runs of 32), D = 3072, L = 1501 37.9 -> 12.5 (32), D = 1024, L = 9001 37.5 -> 20.7 (32).  Forward, at D = 2048, L = 301
// 11.9 -> 6.3 (16); up to four per SM, D = 1024, L = 9001 had gone from 13.8 to 17.9.  The longest run keeps an instance with its length
// known (with the length in a register: 94.7 -> 95.9 us at 2 x 4001 tokens of 8192 channels).  The length is a function of the sizes
// alone (148 SMs): the scratch is sized by it, and the order of the weight gradient's sum must not depend on the device.
static int producer_run(int B, int L, int D, bool bwd) {
  const int per_cta = PT * (bwd ? CB : CG), shortest = bwd ? 32 : 16, room = (bwd ? 4 : 1) * 148;
  const int64_t cols = (D + per_cta - 1) / per_cta;
  int run = bwd ? TT_BWD : TT_FWD;
  while (run > shortest && B * cols * ((L + run / 2 - 1) / (run / 2)) <= room) run /= 2;
  return run;
}

extern "C" {

size_t dn_gdn_producer_scratch_bytes(int32_t B, int32_t L, int32_t D, int32_t W) {
  if (B < 1 || L < 1 || D < 1 || W < 2 || W > 4) return 0;
  const int run = producer_run(B, L, D, true);
  const size_t tiles = (size_t)B * ((L + run - 1) / run);
  return tiles * D * (W + 1) * sizeof(float);
}

static int producer_args(ProducerArgs& a, const void* mixed, const float* conv_w, const float* conv_b, const int32_t* seg,
                         int32_t B, int32_t L, int32_t Hk, int32_t Hv, int32_t K, int32_t V, int32_t W, int32_t dtype) {
  if (!mixed || !conv_w) return DN_ERR_NULL_POINTER;
  if (B < 1 || L < 1 || Hk < 1 || Hv < 1 || (K != 64 && K != 128) || (V != 64 && V != 128) || W < 2 || W > MAXW) return DN_ERR_BAD_SHAPE;
  if (dtype != DN_F32 && dtype != DN_BF16) return DN_ERR_BAD_DTYPE;
  a.mixed = mixed; a.w = conv_w; a.bias = conv_b; a.seg = seg;
  a.B = B; a.L = L; a.D = 2 * Hk * K + Hv * V; a.W = W; a.dt = dtype; a.Hk_K = Hk * K; a.qk_dim = K;
  return DN_OK;
}

int dn_gdn_producer_fwd(const void* mixed, const float* conv_w, const float* conv_b, const int32_t* seg,
                        int32_t B, int32_t L, int32_t Hk, int32_t Hv, int32_t K, int32_t V, int32_t W, int32_t dtype,
                        void* q, void* k, void* v, void* stream) {
  ProducerArgs a{};
  int rc = producer_args(a, mixed, conv_w, conv_b, seg, B, L, Hk, Hv, K, V, W, dtype);
  if (rc) return rc;
  if (!q || !k || !v) return DN_ERR_NULL_POINTER;
  a.q = q; a.k = k; a.v = v;
  a.run = producer_run(B, L, a.D, false);
  dim3 grid(B * ((L + a.run - 1) / a.run), (a.D / CG + PT - 1) / PT);
  cudaStream_t st = (cudaStream_t)stream;
  const bool bf = dtype == DN_BF16;
  auto go = [&](auto width, auto is_long) {
    constexpr int WW = decltype(width)::value;
    constexpr bool LONG = decltype(is_long)::value;
    if (bf) producer_fwd_kernel<WW, true, LONG><<<grid, PT, 0, st>>>(a); else producer_fwd_kernel<WW, false, LONG><<<grid, PT, 0, st>>>(a);
  };
  auto pick = [&](auto width) { if (a.run == TT_FWD) go(width, std::true_type{}); else go(width, std::false_type{}); };
  if (W == 4) pick(std::integral_constant<int, 4>{});
  else if (W == 3) pick(std::integral_constant<int, 3>{});
  else pick(std::integral_constant<int, 2>{});
  return launch_status();
}

int dn_gdn_producer_bwd(const void* mixed, const float* conv_w, const float* conv_b, const int32_t* seg,
                        int32_t B, int32_t L, int32_t Hk, int32_t Hv, int32_t K, int32_t V, int32_t W, int32_t dtype,
                        const void* dq, const void* dk, const void* dv, void* d_mixed, float* d_conv_w, float* d_conv_b,
                        void* scratch, size_t scratch_bytes, void* stream) {
  ProducerArgs a{};
  int rc = producer_args(a, mixed, conv_w, conv_b, seg, B, L, Hk, Hv, K, V, W, dtype);
  if (rc) return rc;
  if (!dq || !dk || !dv || !d_mixed || !d_conv_w || !scratch) return DN_ERR_NULL_POINTER;
  if (scratch_bytes < dn_gdn_producer_scratch_bytes(B, L, a.D, W)) return DN_ERR_SCRATCH_TOO_SMALL;
  a.q = const_cast<void*>(dq); a.k = const_cast<void*>(dk); a.v = const_cast<void*>(dv);
  a.d_mixed = d_mixed; a.part = reinterpret_cast<float*>(scratch);
  a.run = producer_run(B, L, a.D, true);
  const int tiles = B * ((L + a.run - 1) / a.run);
  dim3 grid(tiles, (a.D / CB + PT - 1) / PT);
  cudaStream_t st = (cudaStream_t)stream;
  const bool bf = dtype == DN_BF16;
  auto go = [&](auto width, auto is_long) {
    constexpr int WW = decltype(width)::value;
    constexpr bool LONG = decltype(is_long)::value;
    if (bf) producer_bwd_kernel<WW, true, LONG><<<grid, PT, 0, st>>>(a); else producer_bwd_kernel<WW, false, LONG><<<grid, PT, 0, st>>>(a);
  };
  auto pick = [&](auto width) { if (a.run == TT_BWD) go(width, std::true_type{}); else go(width, std::false_type{}); };
  if (W == 4) pick(std::integral_constant<int, 4>{});
  else if (W == 3) pick(std::integral_constant<int, 3>{});
  else pick(std::integral_constant<int, 2>{});
  if ((rc = launch_status())) return rc;
  const size_t n = (size_t)a.D * (W + 1);
  tile_sum_kernel<<<(unsigned)((n + 31) / 32), 256, 0, st>>>(a.part, tiles, n, d_conv_w, d_conv_b, W);
  return launch_status();
}

int dn_gdn_gates_fwd(const void* a, const void* b, const float* A_log, const float* dt_bias, int32_t B, int32_t L,
                     int32_t Hv, int32_t dtype, float* g, float* beta, void* stream) {
  if (!a || !b || !A_log || !dt_bias || !g || !beta) return DN_ERR_NULL_POINTER;
  if (B < 1 || L < 1 || Hv < 1) return DN_ERR_BAD_SHAPE;
  if (dtype != DN_F32 && dtype != DN_BF16) return DN_ERR_BAD_DTYPE;
  const size_t n = (size_t)B * L * Hv;
  gates_fwd_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(a, b, dtype, A_log, dt_bias, n, Hv, g, beta);
  return launch_status();
}

int dn_gdn_gates_bwd(const void* a, const void* b, const float* A_log, const float* dt_bias, const float* dg,
                     const float* dbeta, int32_t B, int32_t L, int32_t Hv, int32_t dtype, void* da, void* db,
                     float* dA_log, float* d_dt_bias, void* stream) {
  if (!a || !b || !A_log || !dt_bias || !dg || !dbeta || !da || !db || !dA_log || !d_dt_bias) return DN_ERR_NULL_POINTER;
  if (B < 1 || L < 1 || Hv < 1) return DN_ERR_BAD_SHAPE;
  if (dtype != DN_F32 && dtype != DN_BF16) return DN_ERR_BAD_DTYPE;
  const unsigned grid = (Hv + GB_HEADS - 1) / GB_HEADS * GB_CTAS;
  const size_t tokens = (size_t)B * L;
  auto go = [&](auto kernel, int threads) { kernel<<<grid, threads, 0, (cudaStream_t)stream>>>(a, b, dtype, A_log, dt_bias, dg, dbeta, tokens, Hv, da, db, dA_log, d_dt_bias); };
  if (gates_bwd_narrow(tokens)) go(gates_bwd_kernel<256>, 256);
  else go(gates_bwd_kernel<512>, 512);
  return launch_status();
}

size_t dn_gated_rmsnorm_scratch_bytes(int64_t rows, int32_t V) {
  if (rows < 1 || V < 1) return 0;
  return (size_t)norm_grid((size_t)rows) * V * sizeof(float);
}

int dn_gated_rmsnorm_fwd(const void* o, const void* z, const float* weight, int64_t rows, int32_t V, int32_t dtype,
                         float eps, void* y, void* stream) {
  if (!o || !z || !weight || !y) return DN_ERR_NULL_POINTER;
  if (rows < 1 || (V != 64 && V != 128)) return DN_ERR_BAD_SHAPE;
  if (dtype != DN_F32 && dtype != DN_BF16) return DN_ERR_BAD_DTYPE;
  cudaStream_t st = (cudaStream_t)stream;
  auto go = [&](auto kernel) {
    const int grid = norm_grid((size_t)rows, resident_ctas(kernel));
    kernel<<<grid, 256, 0, st>>>(o, z, weight, (size_t)rows, eps, y, nullptr);
  };
  if (dtype == DN_BF16) { if (V == 128) go(gated_rmsnorm_fwd_kernel<4, true>); else go(gated_rmsnorm_fwd_kernel<2, true>); }
  else { if (V == 128) go(gated_rmsnorm_fwd_kernel<4, false>); else go(gated_rmsnorm_fwd_kernel<2, false>); }
  return launch_status();
}

int dn_gated_rmsnorm_bwd(const void* o, const void* z, const float* weight, int64_t rows, int32_t V, int32_t dtype,
                         float eps, const void* dy, void* d_o, void* d_z, float* d_weight, void* scratch,
                         size_t scratch_bytes, void* stream) {
  if (!o || !z || !weight || !dy || !d_o || !d_z || !d_weight || !scratch) return DN_ERR_NULL_POINTER;
  if (rows < 1 || (V != 64 && V != 128)) return DN_ERR_BAD_SHAPE;
  if (dtype != DN_F32 && dtype != DN_BF16) return DN_ERR_BAD_DTYPE;
  if (scratch_bytes < dn_gated_rmsnorm_scratch_bytes(rows, V)) return DN_ERR_SCRATCH_TOO_SMALL;
  cudaStream_t st = (cudaStream_t)stream;
  float* part = reinterpret_cast<float*>(scratch);
  int grid = 0;
  auto go = [&](auto kernel) {
    grid = norm_grid((size_t)rows, resident_ctas(kernel));
    kernel<<<grid, 256, 0, st>>>(o, z, weight, (size_t)rows, eps, dy, d_o, d_z, part);
  };
  if (dtype == DN_BF16) { if (V == 128) go(gated_rmsnorm_bwd_kernel<4, true>); else go(gated_rmsnorm_bwd_kernel<2, true>); }
  else { if (V == 128) go(gated_rmsnorm_bwd_kernel<4, false>); else go(gated_rmsnorm_bwd_kernel<2, false>); }
  int rc = launch_status();
  if (rc) return rc;
  tile_sum_kernel<<<(unsigned)((V + 31) / 32), 256, 0, st>>>(part, grid, (size_t)V, d_weight, nullptr, -1);
  return launch_status();
}

}  // extern "C"
