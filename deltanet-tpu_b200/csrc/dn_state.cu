// Inter-chunk recurrence, fp32 SIMT formulation: the forward chain (with or without the
// output) and the reverse chain of the state cotangent.
//
// The recurrence is independent per value column, so one CTA carries a (K x VS) slice of
// the state of one (batch, exec head) through all chunks; a grid of (Vw/VS, H, B) CTAs
// covers the job.  Forward, per chunk (src/deltanet_tpu/gdn2.py:585-652):
//     S      <- 0 at a document start (or the initial state at chunk 0)
//     V_new   = U - W S
//     O       = qe S + M V_new
//     S      <- [chunk is one document] exp(Lambda_end) * S + ke^T V_new
// Reverse, per chunk (the V-column-independent part of gdn2.py:698-769):
//     dV      = M^T dO + ke dH
//     dH     <- [one document] exp(Lambda_end) * dH + qe^T dO - W^T dV ; 0 at a document start
// The contractions over the value width (dW, dM, dqe, dke, dLambda_end) are left to the
// chunk-parallel backward kernel, which gets dV and the per-chunk dH from here.
#include "dn_kernels.cuh"

namespace dn {

// VS: value columns per CTA, 64, or 16 where 64 would occupy less than half of the chip: 64 x 64 heads, 4 CTAs of 64 columns
// took 122 us over 4 chunks, 16 CTAs of 16 columns 51 to 62.

__device__ __forceinline__ size_t native_state_index(const Geo& g, int b, int h, int k, int jj) {
  const int hv = h * g.G + jj / g.V, cv = jj % g.V;   // exec column jj -> (value head, column)
  return (((size_t)b * g.Hv + hv) * g.K + k) * g.V + cv;
}

template <int VS, bool WITH_OUT>
__global__ void __launch_bounds__(DN_THREADS) state_fwd_kernel(StateArgs a) {
  extern __shared__ __align__(16) float smem[];
  const Geo& g = a.g;
  const int C = g.C, K = g.K, Vw = g.Vw;
  const int h = blockIdx.y, b = blockIdx.z;
  // slices past the value width carry the transition columns (see StateArgs::P_out)
  const bool trans = (int)blockIdx.x * VS >= Vw;
  const int v0 = trans ? 0 : blockIdx.x * VS, p0 = trans ? blockIdx.x * VS - Vw : 0;
  const int tid = threadIdx.x;
  float* S = smem;               // K*VS
  float* Vn = S + K * VS;        // C*VS
  float* tile = Vn + C * VS;
  const bool sbf = g.state_bf16(), ibf = g.bf16_mode();
  const int pre = g.pre_dt;

  for (int c = 0; c < g.NC; ++c) {
    bool is_new, all_same;
    chunk_flags(a.seg, g, b, c, is_new, all_same);
    if (c == 0 || is_new) {
      for (int e = tid; e < K * VS; e += DN_THREADS) {
        float s0 = 0.f;
        if (c == 0 && !is_new && trans) s0 = (e / VS == p0 + e % VS) ? 1.f : 0.f;
        else if (c == 0 && !is_new && a.init_state)
          s0 = a.init_state[native_state_index(g, b, h, e / VS, v0 + e % VS)];
        S[e] = s0;
      }
      __syncthreads();
    }
    const size_t item = ((size_t)b * g.H + h) * g.NC + c;
    if (a.states && !trans)
      for (int e = tid; e < K * VS; e += DN_THREADS)
        a.states[item * K * Vw + (size_t)(e / VS) * Vw + v0 + e % VS] = S[e];

    const size_t bW = item * C * K, bU = item * C * Vw, bM = item * C * C;
    // V_new = U - W S
    cta_gemm<true, true, VS>(C, VS, K,
        [&](int i, int kk) { return ldf(a.res.W, bW + (size_t)i * K + kk, pre); },
        [&](int kk, int j) { float s = S[kk * VS + j]; return sbf ? bf16r(s) : s; },
        [&](int i, int j, float acc) {
          const float u = (a.res.U && !trans) ? ldf(a.res.U, bU + (size_t)i * Vw + v0 + j, pre) : 0.f;   // transition columns: U = 0
          Vn[i * VS + j] = u - acc;
        },
        tile);
    if (WITH_OUT && !trans) {
      // O = [qe | M] [S ; V_new]
      cta_gemm<true, true, VS>(C, VS, K + C,
          [&](int i, int kk) {
            return kk < K ? ldf(a.res.qe, bW + (size_t)i * K + kk, pre)
                          : ldf(a.res.M, bM + (size_t)i * C + kk - K, pre);
          },
          [&](int kk, int j) {
            if (kk < K) { float s = S[kk * VS + j]; return sbf ? bf16r(s) : s; }
            float x = Vn[(kk - K) * VS + j];
            return ibf ? bf16r(x) : x;
          },
          [&](int i, int j, float acc) {
            const int t = c * C + i;
            if (t < g.L) stf(a.out, ((size_t)b * g.L + t) * g.Hv * g.V + (size_t)h * Vw + v0 + j, acc, g.qkv_dt);
          },
          tile);
    }
    // S <- decay * S + ke^T V_new
    cta_gemm<false, true, VS>(K, VS, C,
        [&](int i, int kk) { return ldf(a.res.ke, bW + (size_t)kk * K + i, pre); },
        [&](int kk, int j) { float x = Vn[kk * VS + j]; return sbf ? bf16r(x) : x; },
        [&](int i, int j, float acc) {
          float carried = 0.f;
          if (all_same) carried = S[i * VS + j] * expf(fminf(a.res.lam_end[item * K + i], 0.f));
          S[i * VS + j] = carried + acc;
        },
        tile);
    if (a.until_independent && !all_same) break;       // (uniform over the CTA: the flags depend on the chunk only)
    if (a.until_independent && c + 1 < g.NC) {
      bool nn, na;
      chunk_flags(a.seg, g, b, c + 1, nn, na);
      if (nn) break;
    }
  }
  if (a.until_independent) return;                     // the caller has the final state from the shard's affine summary
  if (trans) {
    for (int e = tid; e < K * VS; e += DN_THREADS)
      if (p0 + e % VS < K) a.P_out[(((size_t)b * g.H + h) * K + e / VS) * K + p0 + e % VS] = S[e];
  } else if (a.final_state)
    for (int e = tid; e < K * VS; e += DN_THREADS)
      a.final_state[native_state_index(g, b, h, e / VS, v0 + e % VS)] = S[e];
}

template <int VS>
__global__ void __launch_bounds__(DN_THREADS) state_bwd_kernel(StateArgs a) {
  extern __shared__ __align__(16) float smem[];
  const Geo& g = a.g;
  const int C = g.C, K = g.K, Vw = g.Vw;
  const int v0 = blockIdx.x * VS, h = blockIdx.y, b = blockIdx.z;
  const int tid = threadIdx.x;
  float* dH = smem;              // K*VS
  float* dOs = dH + K * VS;      // C*VS
  float* dVs = dOs + C * VS;     // C*VS
  float* tile = dVs + C * VS;
  const bool sbf = g.state_bf16(), ibf = g.bf16_mode();
  const int pre = g.pre_dt;

  for (int e = tid; e < K * VS; e += DN_THREADS)
    dH[e] = a.d_final ? a.d_final[native_state_index(g, b, h, e / VS, v0 + e % VS)] : 0.f;
  __syncthreads();

  for (int c = g.NC - 1; c >= 0; --c) {
    bool is_new, all_same;
    chunk_flags(a.seg, g, b, c, is_new, all_same);
    const size_t item = ((size_t)b * g.H + h) * g.NC + c;
    const size_t bW = item * C * K, bM = item * C * C;
    for (int e = tid; e < C * VS; e += DN_THREADS) {
      const int i = e / VS, j = e - i * VS, t = c * C + i;
      dOs[e] = t < g.L ? ldf(a.d_out, ((size_t)b * g.L + t) * g.Hv * g.V + (size_t)h * Vw + v0 + j, g.qkv_dt) : 0.f;
    }
    for (int e = tid; e < K * VS; e += DN_THREADS)
      a.dH[item * K * Vw + (size_t)(e / VS) * Vw + v0 + e % VS] = dH[e];
    __syncthreads();
    // dV = M^T dO + ke dH
    cta_gemm<false, true, VS>(C, VS, C + K,
        [&](int i, int kk) {
          return kk < C ? ldf(a.res.M, bM + (size_t)kk * C + i, pre)
                        : ldf(a.res.ke, bW + (size_t)i * K + kk - C, pre);
        },
        [&](int kk, int j) {
          if (kk < C) { float x = dOs[kk * VS + j]; return ibf ? bf16r(x) : x; }
          float x = dH[(kk - C) * VS + j];
          return sbf ? bf16r(x) : x;
        },
        [&](int i, int j, float acc) {
          dVs[i * VS + j] = acc;
          a.dV[item * C * Vw + (size_t)i * Vw + v0 + j] = acc;
        },
        tile);
    // dH <- decay * dH + qe^T dO - W^T dV, cleared at a document start
    cta_gemm<false, true, VS>(K, VS, 2 * C,
        [&](int i, int kk) {
          return kk < C ? ldf(a.res.qe, bW + (size_t)kk * K + i, pre)
                        : -ldf(a.res.W, bW + (size_t)(kk - C) * K + i, pre);
        },
        [&](int kk, int j) {
          float x = kk < C ? dOs[kk * VS + j] : dVs[(kk - C) * VS + j];
          return sbf ? bf16r(x) : x;
        },
        [&](int i, int j, float acc) {
          float carried = 0.f;
          if (all_same) carried = dH[i * VS + j] * expf(fminf(a.res.lam_end[item * K + i], 0.f));
          dH[i * VS + j] = is_new ? 0.f : carried + acc;
        },
        tile);
    if (a.until_independent && (is_new || !all_same)) break;
  }
  if (a.until_independent) return;                     // the caller has d_init from the shard's affine summary
  if (a.d_init)
    for (int e = tid; e < K * VS; e += DN_THREADS)
      a.d_init[native_state_index(g, b, h, e / VS, v0 + e % VS)] = dH[e];
}

// ---------------------------------------------------------------- fp32 residuals, staged
// The same two chains for fp32 throughout, where a chunk's W, qe, ke and M fit in shared memory: a CTA carries 16 columns, and the
// next chunk's factors travel while this one's are used (two stages where both fit, else one).  Nothing but the recurrence
// itself is then on the critical path: 64 x 64 heads, chunks of 64: 30 us a chunk with the kernels above, 5 with these.  Thread (ty, tx) has rows
// 4 ty .. 4 ty + 3 (and 64 more) of column tx; rows are padded by 16 bytes, so that the two row groups of a warp read
// different banks.
constexpr int ST_VS = 16;

template <int C, int K>
struct Staged {
  static constexpr int PK = K + 4, PC = C + 4;
  static constexpr int W = 0, QE = W + C * PK, KE = QE + C * PK, M = KE + C * PK, STAGE = M + C * PC;   // floats
  static constexpr int REST = (K + 2 * C) * ST_VS + 2 * K;                  // state, two (C x 16) panels, end decays per stage
  static constexpr int STAGES = (2 * STAGE + REST) * 4 <= 227 * 1024 ? 2 : 1;
  static constexpr size_t BYTES = ((size_t)STAGES * STAGE + REST) * 4;
  static_assert(BYTES <= 227 * 1024, "no room");
};

__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
template <int ROWS, int COLS>
__device__ __forceinline__ void stage_rows(float* dst, const float* src) {
  for (int e = threadIdx.x; e < ROWS * COLS / 4; e += DN_THREADS) {
    const int r = e / (COLS / 4), c = e % (COLS / 4) * 4;
    cp_async16(dst + r * (COLS + 4) + c, src + (size_t)r * COLS + c);
  }
}
template <int C, int K>
__device__ __forceinline__ void stage_chunk(const StateArgs& a, size_t item, float* st, float* lend, bool all) {
  using L = Staged<C, K>;
  stage_rows<C, K>(st + L::W, reinterpret_cast<const float*>(a.res.W) + item * C * K);
  stage_rows<C, K>(st + L::KE, reinterpret_cast<const float*>(a.res.ke) + item * C * K);
  if (all) {
    stage_rows<C, K>(st + L::QE, reinterpret_cast<const float*>(a.res.qe) + item * C * K);
    stage_rows<C, C>(st + L::M, reinterpret_cast<const float*>(a.res.M) + item * C * C);
  }
  if (threadIdx.x < K / 4) cp_async16(lend + threadIdx.x * 4, a.res.lam_end + item * K + threadIdx.x * 4);
  asm volatile("cp.async.commit_group;" ::: "memory");
}
__device__ __forceinline__ void stage_wait() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

__device__ __forceinline__ int st_row(int r) { return (r & 3) + 4 * ((int)threadIdx.x >> 4) + 64 * (r >> 2); }

// acc[r] += sign * sum_k A[row(r)][k] * B[k][column]
template <int NR, int KC>
__device__ __forceinline__ void rows_times(float (&acc)[NR], const float* A, int pitch, const float* B, float sign) {
  const int tx = threadIdx.x & 15;
#pragma unroll 4
  for (int k = 0; k < KC; k += 4) {
    float b[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) b[u] = sign * B[(k + u) * ST_VS + tx];
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      const float4 x = *reinterpret_cast<const float4*>(A + st_row(r) * pitch + k);
      acc[r] = fmaf(x.w, b[3], fmaf(x.z, b[2], fmaf(x.y, b[1], fmaf(x.x, b[0], acc[r]))));
    }
  }
}
// acc[r] += sign * sum_i A[i][row(r)] * B[i][column]
template <int NR, int KC>
__device__ __forceinline__ void columns_times(float (&acc)[NR], const float* A, int pitch, const float* B, float sign) {
  const int tx = threadIdx.x & 15;
#pragma unroll 8
  for (int i = 0; i < KC; ++i) {
    const float b = sign * B[i * ST_VS + tx];
#pragma unroll
    for (int q = 0; q < NR / 4; ++q) {
      const float4 x = *reinterpret_cast<const float4*>(A + i * pitch + st_row(4 * q));
      acc[4 * q] = fmaf(x.x, b, acc[4 * q]);
      acc[4 * q + 1] = fmaf(x.y, b, acc[4 * q + 1]);
      acc[4 * q + 2] = fmaf(x.z, b, acc[4 * q + 2]);
      acc[4 * q + 3] = fmaf(x.w, b, acc[4 * q + 3]);
    }
  }
}

template <int C, int K>
__global__ void __launch_bounds__(DN_THREADS, 1) state_fwd_staged_kernel(StateArgs a) {
  using L = Staged<C, K>;
  constexpr int NC = C / 16, NK = K / 16;
  extern __shared__ __align__(16) float smem[];
  const Geo& g = a.g;
  const int Vw = g.Vw, h = blockIdx.y, b = blockIdx.z, tid = threadIdx.x, tx = tid & 15;
  const bool trans = (int)blockIdx.x * ST_VS >= Vw;             // the slices past the value width: see state_fwd_kernel
  const int v0 = trans ? 0 : blockIdx.x * ST_VS, p0 = trans ? blockIdx.x * ST_VS - Vw : 0;
  float* S = smem + L::STAGES * L::STAGE;
  float* Vn = S + K * ST_VS;
  float* lend = Vn + 2 * C * ST_VS;
  const bool with_out = a.out && !trans;
  const size_t item0 = ((size_t)b * g.H + h) * g.NC;
  stage_chunk<C, K>(a, item0, smem, lend, with_out);

  for (int c = 0; c < g.NC; ++c) {
    const int sl = L::STAGES == 2 ? c & 1 : 0;
    const float* st = smem + sl * L::STAGE;
    const size_t item = item0 + c;
    bool is_new, all_same;
    chunk_flags(a.seg, g, b, c, is_new, all_same);
    float u[NC];
#pragma unroll
    for (int r = 0; r < NC; ++r)
      u[r] = a.res.U && !trans ? reinterpret_cast<const float*>(a.res.U)[(item * C + st_row(r)) * Vw + v0 + tx] : 0.f;
    if (c == 0 || is_new)
      for (int e = tid; e < K * ST_VS; e += DN_THREADS) {
        float s0 = 0.f;
        if (c == 0 && !is_new && trans) s0 = (e / ST_VS == p0 + e % ST_VS) ? 1.f : 0.f;
        else if (c == 0 && !is_new && a.init_state) s0 = a.init_state[native_state_index(g, b, h, e / ST_VS, v0 + e % ST_VS)];
        S[e] = s0;
      }
    stage_wait();
    __syncthreads();
    if (L::STAGES == 2 && c + 1 < g.NC)
      stage_chunk<C, K>(a, item + 1, smem + (sl ^ 1) * L::STAGE, lend + (sl ^ 1) * K, with_out);
    if (a.states && !trans)
      for (int e = tid; e < K * ST_VS; e += DN_THREADS)
        a.states[item * K * Vw + (size_t)(e / ST_VS) * Vw + v0 + e % ST_VS] = S[e];

    rows_times<NC, K>(u, st + L::W, L::PK, S, -1.f);            // V_new = U - W S
#pragma unroll
    for (int r = 0; r < NC; ++r) Vn[st_row(r) * ST_VS + tx] = u[r];
    __syncthreads();
    if (with_out) {                                            // O = qe S + M V_new
      float o[NC] = {};
      rows_times<NC, K>(o, st + L::QE, L::PK, S, 1.f);
      rows_times<NC, C>(o, st + L::M, L::PC, Vn, 1.f);
#pragma unroll
      for (int r = 0; r < NC; ++r) {
        const int t = c * C + st_row(r);
        if (t < g.L) stf(a.out, ((size_t)b * g.L + t) * g.Hv * g.V + (size_t)h * Vw + v0 + tx, o[r], g.qkv_dt);
      }
    }
    float s[NK];                                               // S <- decay * S + ke^T V_new
#pragma unroll
    for (int r = 0; r < NK; ++r)
      s[r] = all_same ? S[st_row(r) * ST_VS + tx] * expf(fminf(lend[sl * K + st_row(r)], 0.f)) : 0.f;
    columns_times<NK, C>(s, st + L::KE, L::PK, Vn, 1.f);
    __syncthreads();
#pragma unroll
    for (int r = 0; r < NK; ++r) S[st_row(r) * ST_VS + tx] = s[r];
    if (L::STAGES == 1 && c + 1 < g.NC) stage_chunk<C, K>(a, item + 1, smem, lend, with_out);
    __syncthreads();
    if (a.until_independent) {                                 // (uniform over the CTA)
      bool nn = !all_same, na;
      if (!nn && c + 1 < g.NC) chunk_flags(a.seg, g, b, c + 1, nn, na);
      if (nn) break;
    }
  }
  stage_wait();
  if (a.until_independent) return;                             // the caller has the final state from the shard's affine summary
  if (trans) {
    for (int e = tid; e < K * ST_VS; e += DN_THREADS)
      if (p0 + e % ST_VS < K) a.P_out[(((size_t)b * g.H + h) * K + e / ST_VS) * K + p0 + e % ST_VS] = S[e];
  } else if (a.final_state) {
    for (int e = tid; e < K * ST_VS; e += DN_THREADS)
      a.final_state[native_state_index(g, b, h, e / ST_VS, v0 + e % ST_VS)] = S[e];
  }
}

template <int C, int K>
__global__ void __launch_bounds__(DN_THREADS, 1) state_bwd_staged_kernel(StateArgs a) {
  using L = Staged<C, K>;
  constexpr int NC = C / 16, NK = K / 16;
  extern __shared__ __align__(16) float smem[];
  const Geo& g = a.g;
  const int Vw = g.Vw, h = blockIdx.y, b = blockIdx.z, v0 = blockIdx.x * ST_VS, tid = threadIdx.x, tx = tid & 15;
  float* dH = smem + L::STAGES * L::STAGE;
  float* dOs = dH + K * ST_VS;
  float* dVs = dOs + C * ST_VS;
  float* lend = dVs + C * ST_VS;
  const size_t item0 = ((size_t)b * g.H + h) * g.NC;
  stage_chunk<C, K>(a, item0 + g.NC - 1, smem, lend, true);
  float next[NC];                                              // the chunk's dO, fetched one chunk ahead
  auto fetch = [&](int c) {
#pragma unroll
    for (int r = 0; r < NC; ++r) {
      const int t = c * C + st_row(r);
      next[r] = t < g.L ? ldf(a.d_out, ((size_t)b * g.L + t) * g.Hv * g.V + (size_t)h * Vw + v0 + tx, g.qkv_dt) : 0.f;
    }
  };
  fetch(g.NC - 1);
  for (int e = tid; e < K * ST_VS; e += DN_THREADS)
    dH[e] = a.d_final ? a.d_final[native_state_index(g, b, h, e / ST_VS, v0 + e % ST_VS)] : 0.f;

  for (int c = g.NC - 1, n = 0; c >= 0; --c, ++n) {
    const int sl = L::STAGES == 2 ? n & 1 : 0;
    const float* st = smem + sl * L::STAGE;
    const size_t item = item0 + c;
    bool is_new, all_same;
    chunk_flags(a.seg, g, b, c, is_new, all_same);
#pragma unroll
    for (int r = 0; r < NC; ++r) dOs[st_row(r) * ST_VS + tx] = next[r];
    stage_wait();
    __syncthreads();
    if (L::STAGES == 2 && c > 0) stage_chunk<C, K>(a, item - 1, smem + (sl ^ 1) * L::STAGE, lend + (sl ^ 1) * K, true);
    if (c > 0) fetch(c - 1);
    for (int e = tid; e < K * ST_VS; e += DN_THREADS)
      a.dH[item * K * Vw + (size_t)(e / ST_VS) * Vw + v0 + e % ST_VS] = dH[e];
    float dv[NC] = {};                                         // dV = M^T dO + ke dH
    columns_times<NC, C>(dv, st + L::M, L::PC, dOs, 1.f);
    rows_times<NC, K>(dv, st + L::KE, L::PK, dH, 1.f);
#pragma unroll
    for (int r = 0; r < NC; ++r) {
      dVs[st_row(r) * ST_VS + tx] = dv[r];
      a.dV[(item * C + st_row(r)) * Vw + v0 + tx] = dv[r];
    }
    __syncthreads();
    float d[NK];                                               // dH <- decay * dH + qe^T dO - W^T dV, cleared at a document start
#pragma unroll
    for (int r = 0; r < NK; ++r)
      d[r] = all_same ? dH[st_row(r) * ST_VS + tx] * expf(fminf(lend[sl * K + st_row(r)], 0.f)) : 0.f;
    columns_times<NK, C>(d, st + L::QE, L::PK, dOs, 1.f);
    columns_times<NK, C>(d, st + L::W, L::PK, dVs, -1.f);
    __syncthreads();
#pragma unroll
    for (int r = 0; r < NK; ++r) dH[st_row(r) * ST_VS + tx] = is_new ? 0.f : d[r];
    if (L::STAGES == 1 && c > 0) stage_chunk<C, K>(a, item - 1, smem, lend, true);
    if (a.until_independent && (is_new || !all_same)) break;
  }
  stage_wait();
  if (a.until_independent) return;                             // the caller has d_init from the shard's affine summary
  __syncthreads();
  if (a.d_init)
    for (int e = tid; e < K * ST_VS; e += DN_THREADS)
      a.d_init[native_state_index(g, b, h, e / ST_VS, v0 + e % ST_VS)] = dH[e];
}

template <int VS>
static size_t state_smem(const Geo& g, bool bwd) {
  size_t fl = (size_t)g.K * VS + (size_t)g.C * VS * (bwd ? 2 : 1) + GEMM_SMEM_FLOATS;
  return fl * sizeof(float);
}
static bool narrow(const Geo& g) { return g.Vw / 64 * g.H * g.B * 2 <= sm_count(); }

template <int VS>
static int launch_fwd(const StateArgs& a, cudaStream_t st) {
  const Geo& g = a.g;
  const dim3 grid(g.Vw / VS + (a.P_out ? (g.K + VS - 1) / VS : 0), g.H, g.B);
  const size_t smem = state_smem<VS>(g, false);
  // (the attribute is per device: set on every launch, like the tensor-core launchers do)
  if (a.out) {
    cudaFuncSetAttribute(state_fwd_kernel<VS, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    state_fwd_kernel<VS, true><<<grid, DN_THREADS, smem, st>>>(a);
  } else {
    cudaFuncSetAttribute(state_fwd_kernel<VS, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    state_fwd_kernel<VS, false><<<grid, DN_THREADS, smem, st>>>(a);
  }
  return launch_status();
}
template <int VS>
static int launch_bwd(const StateArgs& a, cudaStream_t st) {
  const Geo& g = a.g;
  const size_t smem = state_smem<VS>(g, true);
  cudaFuncSetAttribute(state_bwd_kernel<VS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  state_bwd_kernel<VS><<<dim3(g.Vw / VS, g.H, g.B), DN_THREADS, smem, st>>>(a);
  return launch_status();
}

// fp32 residuals and products, and factors that 16-byte copies can fetch.
static bool staged(const StateArgs& a) {
  const Geo& g = a.g;
  uintptr_t bits = 0;
  for (const void* p : {(const void*)a.res.W, (const void*)a.res.qe, (const void*)a.res.ke, (const void*)a.res.M, (const void*)a.res.lam_end})
    bits |= reinterpret_cast<uintptr_t>(p);
  return g.pre_dt == DN_F32 && !g.state_bf16() && !g.bf16_mode() && (bits & 15) == 0;
}
template <int C, int K>
static int launch_staged(const StateArgs& a, bool bwd, cudaStream_t st) {
  const Geo& g = a.g;
  auto kernel = bwd ? state_bwd_staged_kernel<C, K> : state_fwd_staged_kernel<C, K>;
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Staged<C, K>::BYTES);
  kernel<<<dim3((g.Vw + (!bwd && a.P_out ? g.K : 0)) / ST_VS, g.H, g.B), DN_THREADS, Staged<C, K>::BYTES, st>>>(a);
  return launch_status();
}
static int launch_staged(const StateArgs& a, bool bwd, cudaStream_t st) {
  return a.g.K == 128 ? launch_staged<64, 128>(a, bwd, st) : launch_staged<64, 64>(a, bwd, st);
}

int launch_state_fwd(const StateArgs& a, cudaStream_t st) {
  if (state_tc_eligible(a.g) && !force_simt()) return launch_state_fwd_tc(a, st);
  if (staged(a)) return launch_staged(a, false, st);
  return narrow(a.g) ? launch_fwd<16>(a, st) : launch_fwd<64>(a, st);
}

int launch_state_bwd(const StateArgs& a, cudaStream_t st) {
  if (state_tc_eligible(a.g) && !force_simt()) return launch_state_bwd_tc(a, st);
  if (staged(a)) return launch_staged(a, true, st);
  return narrow(a.g) ? launch_bwd<16>(a, st) : launch_bwd<64>(a, st);
}

}  // namespace dn
