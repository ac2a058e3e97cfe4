// Inter-chunk recurrence on the tcgen05 tensor cores (bf16 precision, 128-row tiles).
//
// Same math as the fp32 formulation in dn_state.cu (reference: src/deltanet_tpu/gdn2.py:585-769): one CTA carries a
// (128 x VS) column slice of the state of one (batch, exec head) through all chunks.  A chunk step is two dependent
// products with a drain of tensor memory behind each,
//     forward:  P = W S;  V = U - P;   S' = dec S + ke^T V          (off the chain: O = qe S + M V)
//     reverse:  dV = M^T dO + ke dH;   dH' = dec dH + qe^T dO - W^T dV
// and nothing else belongs on the serial path.  So the CTA is specialised by warp:
//   * state warps (row of the state per lane, 32 columns per warp) hold the fp32 master in registers, turn
//     accumulators into bf16 operands in shared memory and touch global memory only before and after the walk;
//   * one thread issues every product, in an order that puts the products off the chain into the time in
//     which the state warps drain;
//   * one thread streams the chunk's tiles (W, qe, ke, M: operand images of 32 KB) through a ring of slots in the
//     order of use, one brings the rows (U or the entry state, and Lambda_end), one stores what the
//     state warps staged (entry states; dH, dV and the partial sums of dLambda_end), all by bulk copies;
//   * four warps write the outputs from a second accumulator, or stage dO ahead (reverse).
// Every hand-over is an mbarrier with one phase per use of the buffer it guards, so that no barrier can run two
// phases ahead of a slow waiter.  Every wait is bounded; after one that gave up a thread skips the rest of its waits,
// raises the library's error word and runs to its end.
//
// With narrow heads (K = 64 or value width 64) rows and columns past the end are zeros.
#include "dn_kernels.cuh"
#include "dn_umma.cuh"

namespace dn {

namespace {

constexpr uint32_t TILE_B = 32768;                    // a 128 x 128 bf16 operand image
constexpr int C = 128, KT = 128;

template <int VS, bool BWD>
struct Plan {
  static constexpr int NG = VS / 32;                  // state warps: 4 NG
  static constexpr int ST = 128 * NG;                 // state threads; then 128 threads for O / dO; then four single-thread roles
  static constexpr int NT = ST + 128 + 128;
  static constexpr uint32_t SL = VS * 256;            // bytes of a (128 x VS) operand
  static constexpr int DO_BUF = 2;                    // reverse: copies of dO
  static constexpr int ROWS = BWD ? 2 : 3;            // buffers of the row loader
  // forward: S, V (U arrives in V's place); reverse: dO, dH, dV, S rows
  static constexpr int OPS = BWD ? DO_BUF + 2 + ROWS : 1 + ROWS;
  static constexpr int SLOTS = VS == 32 ? (BWD ? 5 : 6) : (BWD ? 4 : 5);
  static constexpr uint32_t SMEM = SLOTS * TILE_B + OPS * SL + ROWS * 512 + (BWD ? NG * 512 : 0);
  static constexpr uint32_t TMEM = 4 * VS;
  static_assert(SMEM + 512 <= 227 * 1024, "shared memory, with the static arrays");
};

__device__ __forceinline__ void arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(umma::smem_u32(bar)) : "memory");
}
// one arrival per warp, behind the shared-memory and tensor-memory accesses of all its lanes
__device__ __forceinline__ void warp_arrive(uint64_t* bar) {
  umma::fence_async_smem();
  umma::tc_fence_before();
  __syncwarp();
  if ((threadIdx.x & 31) == 0) arrive(bar);
}
struct Waiter {
  int* err;
  bool dead;
  __device__ __forceinline__ void operator()(uint64_t* bar, uint32_t parity) {
    if (dead) return;
    if (!umma::mbar_wait(bar, parity)) { dead = true; umma::report_timeout(err); }
  }
};
// D[128 x N] (+)= A B over a contraction of 128, by a converged warp; operands are images of 128-row panels
template <bool MN>
__device__ __forceinline__ uint64_t operand(const void* p) {
  return umma::smem_desc(umma::smem_u32(p), MN ? 128u : 2048u, MN ? 2048u : 128u);
}
template <int N, bool A_MN, bool B_MN>
__device__ __forceinline__ void product(uint32_t d, uint64_t ad, uint64_t bd, bool accumulate) {
  constexpr uint32_t idesc = umma::instr_desc(N, A_MN ? 1 : 0, B_MN ? 1 : 0);
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    umma::mma_bf16_warp(d, ad, bd, idesc, (accumulate || k > 0) ? 1u : 0u);
    ad += (A_MN ? 256u : 4096u) >> 4;
    bd += (B_MN ? 256u : 4096u) >> 4;
  }
}
// Position in a ring of N buffers: index and the parity of the current use
template <int N>
struct Ring {
  uint32_t at = 0, parity = 0;
  __device__ __forceinline__ void next() {
    if (++at == N) { at = 0; parity ^= 1u; }
  }
};
__device__ __forceinline__ void ld32(bool dead, uint32_t addr, float (&v)[32]) {
  if (!dead) {
    umma::tmem_ld32_nowait(addr, v);
    umma::tmem_wait_ld();
  } else {
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = 0.f;
  }
}
__device__ __forceinline__ void image32(uint4* img, int row, const float (&v)[32]) {
#pragma unroll
  for (int p = 0; p < 4; ++p) img[p * 128 + row] = umma::pack8p(v + 8 * p);
}

// Document flags of the chunks a chain walks, 32 at a time as bit masks a warp keeps in registers: bit i is chunk
// top + dir * i.  (is_new: the chunk starts a document; all_same: the chunk is one document.)
struct Flags {
  uint32_t is_new, all_same;
  __device__ __forceinline__ void fill(const int32_t* seg, const Geo& g, int b, int top, int dir, int lo, int hi) {
    const int c = top + dir * (int)(threadIdx.x & 31);
    bool n = false, s = false;
    if (c >= lo && c < hi) chunk_flags(seg, g, b, c, n, s);
    is_new = __ballot_sync(0xffffffffu, n);
    all_same = __ballot_sync(0xffffffffu, s);
  }
  __device__ __forceinline__ void next() { is_new >>= 1; all_same >>= 1; }
};
// 32 columns of one row of a native (B, Hv, K, V) state: offset, or none where the row or the columns do not exist
__device__ __forceinline__ bool native_row(const Geo& g, int b, int h, int k, int col, size_t& off) {
  off = (((size_t)b * g.Hv + h * g.G + col / g.V) * g.K + k) * g.V + col % g.V;
  return k < g.K && col < g.G * g.V;
}
__device__ __forceinline__ void load32(const float* p, float (&v)[32]) {
  if ((reinterpret_cast<uintptr_t>(p) & 15) == 0) {
#pragma unroll
    for (int j = 0; j < 32; j += 4) {
      const float4 t = *reinterpret_cast<const float4*>(p + j);
      v[j] = t.x; v[j + 1] = t.y; v[j + 2] = t.z; v[j + 3] = t.w;
    }
  } else {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = p[j];
  }
}
__device__ __forceinline__ void store32(float* p, const float (&v)[32]) {
  if ((reinterpret_cast<uintptr_t>(p) & 15) == 0) {
#pragma unroll
    for (int j = 0; j < 32; j += 4) *reinterpret_cast<float4*>(p + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
  } else {
#pragma unroll
    for (int j = 0; j < 32; ++j) p[j] = v[j];
  }
}

// A document boundary cuts the chain: what a chunk that holds one, or starts with one, hands on does not depend on what it is
// handed.  So the range [c_begin, c_end) is dealt out in `parts` equal parts.  The CTA of the first part starts where the
// range does, that of any other at the first cut inside its part, and each ends where the next one starts; a part without a
// cut has no walk and its CTA leaves.  Where the boundary lies inside a chunk, the new walk takes this chunk from zeros, for
// what it hands on alone (`warm` = 1: it stores nothing of it).  Results are those of a single walk, bit for bit.
// `found`: two words of shared memory.  Every thread calls; false: no walk.
template <bool REVERSE, int NT>
__device__ __forceinline__ bool find_walk(const StateArgs& a, int b, int part, int* found, int& lo, int& hi, int& warm) {
  const int begin = a.c_begin, end = a.c_end, len = (end - begin + a.parts - 1) / a.parts, tid = threadIdx.x;
  // the part, in the order of the walk: s0 its first chunk, s1 the first of the next part
  const int s0 = REVERSE ? end - 1 - part * len : begin + part * len;
  const int s1 = REVERSE ? max(begin - 1, s0 - len) : min(end, s0 + len);
  constexpr int dir = REVERSE ? -1 : 1, none = REVERSE ? -1 : 0x7fffffff;
  if (tid < 2) found[tid] = none;
  __syncthreads();
  auto search = [&](int from, int to, int* f) {
    for (int c = from + dir * tid; dir * c < dir * to; c += dir * NT) {
      bool n, s;
      chunk_flags(a.seg, a.g, b, c, n, s);
      // (a cut behind which nothing is left to walk is none)
      if (REVERSE ? (n || !s) && c > begin : n || (!s && c + 1 < end)) {
        const int v = 2 * c + (n ? 0 : 1);
        if (REVERSE) atomicMax(f, v); else atomicMin(f, v);
        break;
      }
    }
  };
  if (part > 0) search(s0, s1, &found[0]);
  search(s1, REVERSE ? begin - 1 : end, &found[1]);
  __syncthreads();
  const int f0 = found[0], f1 = found[1];
  if (part > 0 && f0 == none) return false;
  warm = part > 0 ? f0 & 1 : 0;
  if (REVERSE) {
    hi = part > 0 ? (f0 >> 1) + warm : end;
    lo = f1 == none ? begin : f1 >> 1;
  } else {
    lo = part > 0 ? f0 >> 1 : begin;
    hi = f1 == none ? end : (f1 >> 1) + (f1 & 1);
  }
  return true;
}

// CUT: the range may be cut into several walks (find_walk).  An instance of its own, since bounds that are the launch's
// parameters leave the uncut chain faster (by 17 us of 331 at 256 CTAs and 64 chunks).
template <int VS, bool CUT>
__global__ void __launch_bounds__(Plan<VS, false>::NT, 1) state_fwd_tc_kernel(const __grid_constant__ StateArgs a) {
  using PL = Plan<VS, false>;
  constexpr int ST = PL::ST, NG = PL::NG, SLOTS = PL::SLOTS;
  extern __shared__ __align__(128) uint8_t sm[];
  constexpr int ROWS = PL::ROWS;
  __shared__ uint64_t full[SLOTS], empty[SLOTS], row_full[ROWS], row_empty[ROWS];
  __shared__ uint64_t s_ready, v_ready, p_done, s_done, o_done[2], o_free[2], s_free, all_done;
  __shared__ uint32_t tmem_base;
  __shared__ int stop_s;
  const Geo& g = a.g;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;      // (warp: uniform for the compiler)
  const int Vw = g.Vw, vr = g.G * g.V, h = blockIdx.y, b = CUT ? blockIdx.z % g.B : blockIdx.z;
  // slices past the value width carry the transition columns (see StateArgs::P_out)
  const bool trans = (int)blockIdx.x * VS >= Vw;
  const int v0 = trans ? 0 : blockIdx.x * VS, p0 = trans ? blockIdx.x * VS - Vw : 0;
  uint8_t* tiles = sm;
  uint8_t* sS = sm + SLOTS * TILE_B;
  uint8_t* sV = sS + PL::SL;                            // ROWS buffers
  float* lam_s = reinterpret_cast<float*>(sV + ROWS * PL::SL);
  int cb = a.c_begin, ce = a.c_end, warm = 0;
  __shared__ int found_s[2];
  if (CUT && !find_walk<false, PL::NT>(a, b, blockIdx.z / g.B, found_s, cb, ce, warm)) return;
  const bool first_walk = !CUT || cb == a.c_begin, last_walk = !CUT || ce == a.c_end;
  if (tid == 0) {
    for (int i = 0; i < SLOTS; ++i) { umma::mbar_init(&full[i], 1); umma::mbar_init(&empty[i], 1); }
    for (int i = 0; i < ROWS; ++i) { umma::mbar_init(&row_full[i], 1); umma::mbar_init(&row_empty[i], 1); }
    for (int i = 0; i < 2; ++i) { umma::mbar_init(&o_done[i], 1); umma::mbar_init(&o_free[i], 4); }
    umma::mbar_init(&s_ready, 4 * NG); umma::mbar_init(&v_ready, 4 * NG);
    umma::mbar_init(&p_done, 1); umma::mbar_init(&s_done, 1); umma::mbar_init(&s_free, 1); umma::mbar_init(&all_done, 1);
    umma::fence_mbar_init();
    stop_s = ce;
  }
  if (warp == 0) umma::tmem_alloc(&tmem_base, PL::TMEM);
  umma::tc_fence_before();
  __syncthreads();
  // the first chunk behind which nothing depends on the state that this launch starts from
  if (a.until_independent || a.skip_provisional) {
    for (int c = cb + tid; c < ce; c += PL::NT) {
      bool n, s, n2 = false, s2;
      chunk_flags(a.seg, g, b, c, n, s);
      if (c + 1 < ce) chunk_flags(a.seg, g, b, c + 1, n2, s2);
      if (!s || n2) { atomicMin(&stop_s, c); break; }
    }
    __syncthreads();
  }
  umma::tc_fence_after();
  const int stop = stop_s;
  if (a.until_independent && stop + 1 < ce) ce = stop + 1;
  const int n = ce - cb;
  // index of the first chunk whose outputs are wanted
  const int o_from = (!a.out || trans) ? n : (a.skip_provisional ? (stop + 1 < ce ? stop + 1 - cb : n) : warm);
  const uint32_t tm = tmem_base;
  constexpr uint32_t colP = 0, colS = VS, colO = 2 * VS;
  const size_t item0 = ((size_t)b * g.H + h) * g.NC + cb;
  const bool keep_states = a.states && !trans;
  const bool has_u = a.res.U && !trans;
  Waiter wait{a.err, false};

  if (tid < ST) {
    // ------------------------------------------------------------------------------------------ state warps
    const int row = (warp & 3) * 32 + lane, ng = warp >> 2, col = v0 + 32 * ng;
    const uint32_t tb = tm + ((uint32_t)((warp & 3) * 32) << 16) + 32 * ng;
    uint4* S_img = reinterpret_cast<uint4*>(sS) + ng * 512;
    float* carry = a.carry ? a.carry + (((size_t)b * g.H + h) * KT + row) * Vw + col : nullptr;
    size_t noff;
    const bool native = native_row(g, b, h, row, col, noff);
    float S[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) S[j] = 0.f;
    if (cb > 0 && first_walk) load32(carry, S);
    Flags fl;
    fl.fill(a.seg, g, b, cb, 1, cb, ce);
    if (cb == 0 && !(fl.is_new & 1u)) {
      if (trans) {
#pragma unroll
        for (int j = 0; j < 32; ++j) S[j] = row == p0 + 32 * ng + j ? 1.f : 0.f;
      } else if (a.init_state && native) {
        load32(a.init_state + noff, S);
      }
    }
    if (fl.is_new & 1u) {
#pragma unroll
      for (int j = 0; j < 32; ++j) S[j] = 0.f;
    }
    Ring<ROWS> rows;
    Ring<SLOTS> ring;                                   // follows the tiles the products take
#pragma unroll 1
    for (int i = 0; i < n; ++i) {
      const bool outs = i >= o_from;
      if (keep_states && i > 0) wait(&s_free, (i - 1) & 1);
      image32(S_img, row, S);
      warp_arrive(&s_ready);
      // V = U - W S, over U
      wait(&row_full[rows.at], rows.parity);
      uint4* V_img = reinterpret_cast<uint4*>(sV + rows.at * PL::SL) + ng * 512;
      uint4 u[4];
#pragma unroll
      for (int p = 0; p < 4; ++p) u[p] = has_u ? V_img[p * 128 + row] : make_uint4(0, 0, 0, 0);
      float dec = fl.all_same & 1u ? expf(fminf(lam_s[rows.at * 128 + row], 0.f)) : 0.f;
      const uint32_t row_at = rows.at;
      rows.next();
      fl.next();
      if ((i & 31) == 31) fl.fill(a.seg, g, b, cb + i + 1, 1, cb, ce);
      // the next chunk starts a document: nothing of this one is handed on
      const bool drop = fl.is_new & 1u;
      float x[32];
      wait(&p_done, i & 1);
      umma::tc_fence_after();
      ld32(wait.dead, tb + colP, x);
      // (released by the threads that see a product complete: a commit of its own costs the issuing warp 67 cycles)
      if (tid == 0) arrive(&empty[ring.at]);            // W
      ring.next();
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        float t[8];
        umma::unpack8(u[p], t);
#pragma unroll
        for (int k = 0; k < 8; ++k) t[k] -= x[8 * p + k];
        V_img[p * 128 + row] = umma::pack8(t);
      }
      warp_arrive(&v_ready);
      wait(&s_done, i & 1);
      umma::tc_fence_after();
      ld32(wait.dead, tb + colS, x);
      if (outs) {
        if (tid == 32) arrive(&empty[ring.at]);         // qe
        ring.next();
      }
      if (tid == 64) arrive(&empty[ring.at]);           // ke
      ring.next();
      if (outs) ring.next();                            // M: released by the output warps, with V
      else if (tid == 96) arrive(&row_empty[row_at]);
#pragma unroll
      for (int j = 0; j < 32; ++j) S[j] = fmaf(dec, S[j], x[j]);
      if (drop) {
#pragma unroll
        for (int j = 0; j < 32; ++j) S[j] = 0.f;
      }
    }
    umma::tc_fence_before();
    if (a.until_independent) {
      // nothing to hand on: the caller has the final state from the shard's affine summary
    } else if (trans) {
      if (row < g.K) store32(a.P_out + (((size_t)b * g.H + h) * g.K + row) * g.K + p0 + 32 * ng, S);
    } else if (!last_walk) {
      // the next walk does not need it
    } else if (ce < g.NC) {
      store32(carry, S);
    } else if (a.final_state && native) {
      store32(a.final_state + noff, S);
    }
  } else if (tid < ST + 128) {
    // ------------------------------------------------------------------------------------------ outputs, a row per lane
    const int q = warp & 3, row = q * 32 + lane;
    Ring<ROWS> rows;
    rows.at = o_from % ROWS;
    uint32_t m_at = (2 * o_from + 3) % SLOTS;           // M's slot (two tiles per chunk without outputs, four with)
#pragma unroll 1
    for (int i = o_from; i < n; ++i) {
      const int oi = i - o_from;
      wait(&o_done[oi & 1], (oi >> 1) & 1);
      umma::tc_fence_after();
      if (q == 0 && lane == 0) arrive(&empty[m_at]);
      if (q == 1 && lane == 0) arrive(&row_empty[rows.at]);
      rows.next();
      m_at = (m_at + 4) % SLOTS;
      const int t = (cb + i) * C + row;
      const size_t off = ((size_t)b * g.L + t) * g.Hv * g.V + (size_t)h * vr + v0;
#pragma unroll 1
      for (int ng = 0; ng < NG; ++ng) {
        float o[32];
        ld32(wait.dead, tm + ((uint32_t)(q * 32) << 16) + colO + (oi & 1) * VS + 32 * ng, o);
        if (ng == NG - 1) {
          umma::tc_fence_before();
          __syncwarp();
          if (lane == 0) arrive(&o_free[oi & 1]);
        }
        if (t < g.L && v0 + 32 * ng < vr) {
          if (g.qkv_dt == DN_BF16) {
            uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(a.out) + off + 32 * ng);
#pragma unroll
            for (int p = 0; p < 4; ++p) dst[p] = umma::pack8p(o + 8 * p);
          } else {
            float4* dst = reinterpret_cast<float4*>(reinterpret_cast<float*>(a.out) + off + 32 * ng);
#pragma unroll
            for (int j = 0; j < 8; ++j) dst[j] = make_float4(o[4 * j], o[4 * j + 1], o[4 * j + 2], o[4 * j + 3]);
          }
        }
      }
    }
  } else {
    const int role = warp - (ST + 128) / 32;
    if (role == 0) {
      // ---------------------------------------------------------------------------------------- products
      Ring<SLOTS> ring;
      Ring<ROWS> rows;
      Ring<2> ob;
      const uint64_t tk = operand<false>(tiles), tt = operand<true>(tiles), bS = operand<true>(sS), bV = operand<true>(sV);
#pragma unroll 1
      for (int i = 0; i < n; ++i) {
        const bool outs = i >= o_from;
        const uint32_t colOi = tm + colO + ob.at * VS;
        const uint64_t bVi = bV + rows.at * (PL::SL >> 4);
        wait(&full[ring.at], ring.parity);
        wait(&s_ready, i & 1);
        umma::tc_fence_after();
        product<VS, false, true>(tm + colP, tk + ring.at * (TILE_B >> 4), bS, false);            // P = W S
        umma::mma_commit_warp(&p_done);
        ring.next();
        if (outs) {
          wait(&full[ring.at], ring.parity);
          if (i - o_from >= 2) { wait(&o_free[ob.at], ob.parity ^ 1u); umma::tc_fence_after(); }
          product<VS, false, true>(colOi, tk + ring.at * (TILE_B >> 4), bS, false);              // O  = qe S
          ring.next();
        }
        wait(&full[ring.at], ring.parity);
        wait(&v_ready, i & 1);
        umma::tc_fence_after();
        product<VS, true, true>(tm + colS, tt + ring.at * (TILE_B >> 4), bVi, false);            // ke^T V
        umma::mma_commit_warp(&s_done);
        ring.next();
        if (outs) {
          wait(&full[ring.at], ring.parity);
          product<VS, false, true>(colOi, tk + ring.at * (TILE_B >> 4), bVi, true);              //    + M V
          umma::mma_commit_warp(&o_done[ob.at]);
          ring.next();
          ob.next();
        }
        rows.next();
      }
      umma::mma_commit_warp(&all_done);                 // every arrival above has happened before the CTA leaves
      wait(&all_done, 0);
    } else if (role == 1 && lane == 0) {
      // ---------------------------------------------------------------------------------------- tiles, in the order of use
      Ring<SLOTS> ring;
      bool again = false;                               // the slot has been used before
      auto load = [&](const void* base, size_t item) {
        if (again) wait(&empty[ring.at], ring.parity ^ 1u);
        umma::mbar_expect_tx(&full[ring.at], TILE_B);
        umma::bulk_load(tiles + ring.at * TILE_B, reinterpret_cast<const uint8_t*>(base) + item * TILE_B, TILE_B, &full[ring.at]);
        ring.next();
        again |= ring.at == 0;
      };
#pragma unroll 1
      for (int i = 0; i < n && !wait.dead; ++i) {
        const bool outs = i >= o_from;
        load(a.res.W, item0 + i);
        if (outs) load(a.res.qe, item0 + i);
        load(a.res.ke, item0 + i);
        if (outs) load(a.res.M, item0 + i);
      }
    } else if (role == 2 && lane == 0) {
      // ---------------------------------------------------------------------------------------- rows: U, Lambda_end
      Ring<ROWS> ring;
#pragma unroll 1
      for (int i = 0; i < n && !wait.dead; ++i, ring.next()) {
        const uint32_t s = ring.at;
        if (i >= ROWS) wait(&row_empty[s], ring.parity ^ 1u);
        umma::mbar_expect_tx(&row_full[s], 512 + (has_u ? PL::SL : 0));
        umma::bulk_load(lam_s + s * 128, a.res.lam_end + (item0 + i) * KT, 512, &row_full[s]);
        if (has_u)
          umma::bulk_load(sV + s * PL::SL, reinterpret_cast<const uint8_t*>(a.res.U) + ((item0 + i) * Vw + v0) * 256, PL::SL, &row_full[s]);
      }
    } else if (role == 3 && lane == 0 && keep_states) {
      // ---------------------------------------------------------------------------------------- chunk-entry states
      uint8_t* dst = reinterpret_cast<uint8_t*>(a.states);
      for (int i = 0; i < n && !wait.dead; ++i) {
        wait(&s_ready, i & 1);
        if (!CUT || i >= warm) umma::bulk_store(dst + ((item0 + i) * Vw + v0) * 256, sS, PL::SL);
        umma::bulk_commit();
        umma::bulk_wait_read<0>();
        arrive(&s_free);
      }
      asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
  }
  __syncthreads();
  if (warp == 0) umma::tmem_dealloc(tmem_base, PL::TMEM);
}

template <int VS, bool CUT>
__global__ void __launch_bounds__(Plan<VS, true>::NT, 1) state_bwd_tc_kernel(const __grid_constant__ StateArgs a) {
  using PL = Plan<VS, true>;
  constexpr int ST = PL::ST, NG = PL::NG, SLOTS = PL::SLOTS, DB = PL::DO_BUF, ROWS = PL::ROWS;
  extern __shared__ __align__(128) uint8_t sm[];
  __shared__ uint64_t full[SLOTS], empty[SLOTS], row_full[ROWS], row_empty[ROWS], do_ready[DB], do_free[DB];
  __shared__ uint64_t h_ready, v_ready, v_done, h_done, h_free, v_free, all_done;
  __shared__ uint32_t tmem_base;
  __shared__ int stop_s;
  const Geo& g = a.g;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;      // (warp: uniform for the compiler)
  const int Vw = g.Vw, vr = g.G * g.V, v0 = blockIdx.x * VS, h = blockIdx.y, b = CUT ? blockIdx.z % g.B : blockIdx.z;
  uint8_t* tiles = sm;
  uint8_t* sdO = sm + SLOTS * TILE_B;                   // DB buffers
  uint8_t* sdH = sdO + DB * PL::SL;
  uint8_t* sdV = sdH + PL::SL;
  uint8_t* sR = sdV + PL::SL;                           // rows of S, ROWS buffers
  float* lam_s = reinterpret_cast<float*>(sR + ROWS * PL::SL);
  float* part_s = lam_s + ROWS * 128;                   // partial sums of dLambda_end: NG x 128
  int cb = a.c_begin, ce = a.c_end, warm = 0;
  __shared__ int found_s[2];
  if (CUT && !find_walk<true, PL::NT>(a, b, blockIdx.z / g.B, found_s, cb, ce, warm)) return;
  const bool first_walk = !CUT || ce == a.c_end, last_walk = !CUT || cb == a.c_begin;
  if (tid == 0) {
    for (int i = 0; i < SLOTS; ++i) { umma::mbar_init(&full[i], 1); umma::mbar_init(&empty[i], 1); }
    for (int i = 0; i < ROWS; ++i) { umma::mbar_init(&row_full[i], 1); umma::mbar_init(&row_empty[i], 1); }
    for (int i = 0; i < DB; ++i) { umma::mbar_init(&do_ready[i], 4); umma::mbar_init(&do_free[i], 1); }
    umma::mbar_init(&h_ready, 4 * NG); umma::mbar_init(&v_ready, 4 * NG);
    umma::mbar_init(&v_done, 1); umma::mbar_init(&h_done, 1);
    umma::mbar_init(&h_free, 1); umma::mbar_init(&v_free, 1); umma::mbar_init(&all_done, 1);
    umma::fence_mbar_init();
    stop_s = cb;
  }
  if (warp == 0) umma::tmem_alloc(&tmem_base, PL::TMEM);
  umma::tc_fence_before();
  __syncthreads();
  if (a.until_independent) {                            // the last chunk whose results depend on the incoming cotangent
    for (int c = ce - 1 - tid; c >= cb; c -= PL::NT) {
      bool n, s;
      chunk_flags(a.seg, g, b, c, n, s);
      if (n || !s) { atomicMax(&stop_s, c); break; }
    }
    __syncthreads();
  }
  umma::tc_fence_after();
  cb = stop_s;
  const int n = ce - cb;
  const uint32_t tm = tmem_base;
  constexpr uint32_t colV = 0, colQ = VS, colW = 2 * VS;
  const size_t last = ((size_t)b * g.H + h) * g.NC + ce - 1;      // item of step i: last - i
  Waiter wait{a.err, false};

  if (tid < ST) {
    // ------------------------------------------------------------------------------------------ state warps
    const int row = (warp & 3) * 32 + lane, ng = warp >> 2, col = v0 + 32 * ng;
    const uint32_t tb = tm + ((uint32_t)((warp & 3) * 32) << 16) + 32 * ng;
    uint4* H_img = reinterpret_cast<uint4*>(sdH) + ng * 512;
    uint4* V_img = reinterpret_cast<uint4*>(sdV) + ng * 512;
    float* carry = a.carry ? a.carry + (((size_t)b * g.H + h) * KT + row) * Vw + col : nullptr;
    size_t noff;
    const bool native = native_row(g, b, h, row, col, noff);
    float dH[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) dH[j] = 0.f;
    if (!first_walk) { /* zeros */ }
    else if (ce < g.NC) load32(carry, dH);
    else if (a.d_final && native) load32(a.d_final + noff, dH);
    Flags fl;
    fl.fill(a.seg, g, b, ce - 1, -1, cb, ce);
    Ring<ROWS> rows;
    Ring<SLOTS> ring;                                   // follows the tiles the products take
#pragma unroll 1
    for (int i = 0; i < n; ++i) {
      if (i > 0) wait(&h_free, (i - 1) & 1);
      image32(H_img, row, dH);
      warp_arrive(&h_ready);
      // off the chain: this slice's share of dLambda_end = sum_v dH S, in fp32
      wait(&row_full[rows.at], rows.parity);
      const uint4* R_img = reinterpret_cast<const uint4*>(sR + rows.at * PL::SL) + ng * 512;
      float part = 0.f;
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        float s8[8];
        umma::unpack8(R_img[p * 128 + row], s8);
#pragma unroll
        for (int k = 0; k < 8; ++k) part = fmaf(dH[8 * p + k], s8[k], part);
      }
      if (i > 0) wait(&v_free, (i - 1) & 1);            // dV and the sums of the step before have been read
      part_s[ng * 128 + row] = part;
      const float dec = fl.all_same & 1u ? expf(fminf(lam_s[rows.at * 128 + row], 0.f)) : 0.f;
      const bool is_new = fl.is_new & 1u;
      const uint32_t row_at = rows.at;
      rows.next();
      fl.next();
      if ((i & 31) == 31) fl.fill(a.seg, g, b, ce - 2 - i, -1, cb, ce);
      float x[32];
      wait(&v_done, i & 1);
      umma::tc_fence_after();
      ld32(wait.dead, tb + colV, x);
      // (released by the threads that see a product complete: a commit of its own costs the issuing warp 67 cycles)
      if (tid == 0) arrive(&empty[ring.at]);            // M
      ring.next();
      if (tid == 32) arrive(&empty[ring.at]);           // ke
      ring.next();
      image32(V_img, row, x);
      warp_arrive(&v_ready);
      wait(&h_done, i & 1);
      umma::tc_fence_after();
      if (tid == 0) arrive(&empty[ring.at]);            // qe
      ring.next();
      if (tid == 32) arrive(&empty[ring.at]);           // W
      ring.next();
      if (tid == 64) arrive(&do_free[i & 1]);
      if (tid == 96) arrive(&row_empty[row_at]);
      if (is_new) {
#pragma unroll
        for (int j = 0; j < 32; ++j) dH[j] = 0.f;
      } else if (wait.dead) {
        // nothing to add
      } else {
        float w[32];
        umma::tmem_ld32_nowait(tb + colQ, x);
        umma::tmem_ld32_nowait(tb + colW, w);
        umma::tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 32; ++j) dH[j] = fmaf(dec, dH[j], x[j] - w[j]);
      }
    }
    umma::tc_fence_before();
    if (a.until_independent) {
      // nothing to hand on: the caller has d_init from the shard's affine summary
    } else if (!last_walk) {
      // the next walk does not need it
    } else if (cb > 0) {
      store32(carry, dH);
    } else if (a.d_init && native) {
      store32(a.d_init + noff, dH);
    }
  } else if (tid < ST + 128) {
    // ------------------------------------------------------------------------------------------ dO, rounded to bf16 (gdn2.py:731)
    const int row = (warp & 3) * 32 + lane;
    for (int i = 0; i < n; ++i) {
      const int t = (ce - 1 - i) * C + row;
      const size_t off = ((size_t)b * g.L + (t < g.L ? t : 0)) * g.Hv * g.V + (size_t)h * vr + v0;
      uint4 raw[4 * NG];
#pragma unroll
      for (int p = 0; p < 4 * NG; ++p) {
        const bool on = t < g.L && v0 + 8 * p < vr;
        if (g.qkv_dt == DN_BF16) raw[p] = on ? __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(a.d_out) + off) + p) : make_uint4(0, 0, 0, 0);
        else raw[p] = on ? umma::ld8_f32_ro(reinterpret_cast<const float*>(a.d_out) + off + 8 * p) : make_uint4(0, 0, 0, 0);
      }
      if (i >= DB) wait(&do_free[i % DB], (i / DB - 1) & 1);
      uint4* img = reinterpret_cast<uint4*>(sdO + (i % DB) * PL::SL);
#pragma unroll
      for (int p = 0; p < 4 * NG; ++p) img[p * 128 + row] = raw[p];
      warp_arrive(&do_ready[i % DB]);
    }
  } else {
    const int role = warp - (ST + 128) / 32;
    if (role == 0) {
      // ---------------------------------------------------------------------------------------- products
      Ring<SLOTS> ring;
      Ring<DB> dos;
      const uint64_t tk = operand<false>(tiles), tt = operand<true>(tiles), bO = operand<true>(sdO), bH = operand<true>(sdH), bV = operand<true>(sdV);
#pragma unroll 1
      for (int i = 0; i < n; ++i) {
        const uint64_t bOi = bO + dos.at * (PL::SL >> 4);
        wait(&full[ring.at], ring.parity);
        wait(&do_ready[dos.at], dos.parity);
        umma::tc_fence_after();
        product<VS, true, true>(tm + colV, tt + ring.at * (TILE_B >> 4), bOi, false);            // dV  = M^T dO
        ring.next();
        wait(&full[ring.at], ring.parity);
        wait(&h_ready, i & 1);
        umma::tc_fence_after();
        product<VS, false, true>(tm + colV, tk + ring.at * (TILE_B >> 4), bH, true);             //     + ke dH
        umma::mma_commit_warp(&v_done);
        ring.next();
        wait(&full[ring.at], ring.parity);
        product<VS, true, true>(tm + colQ, tt + ring.at * (TILE_B >> 4), bOi, false);            // qe^T dO
        ring.next();
        dos.next();
        wait(&full[ring.at], ring.parity);
        wait(&v_ready, i & 1);
        umma::tc_fence_after();
        product<VS, true, true>(tm + colW, tt + ring.at * (TILE_B >> 4), bV, false);             // W^T dV
        umma::mma_commit_warp(&h_done);
        ring.next();
      }
      umma::mma_commit_warp(&all_done);
      wait(&all_done, 0);
    } else if (role == 1 && lane == 0) {
      // ---------------------------------------------------------------------------------------- tiles, in the order of use
      Ring<SLOTS> ring;
      bool again = false;                               // the slot has been used before
      auto load = [&](const void* base, size_t item) {
        if (again) wait(&empty[ring.at], ring.parity ^ 1u);
        umma::mbar_expect_tx(&full[ring.at], TILE_B);
        umma::bulk_load(tiles + ring.at * TILE_B, reinterpret_cast<const uint8_t*>(base) + item * TILE_B, TILE_B, &full[ring.at]);
        ring.next();
        again |= ring.at == 0;
      };
#pragma unroll 1
      for (int i = 0; i < n && !wait.dead; ++i) {
        load(a.res.M, last - i);
        load(a.res.ke, last - i);
        load(a.res.qe, last - i);
        load(a.res.W, last - i);
      }
    } else if (role == 2 && lane == 0) {
      // ---------------------------------------------------------------------------------------- rows: entry state, Lambda_end
      Ring<ROWS> ring;
#pragma unroll 1
      for (int i = 0; i < n && !wait.dead; ++i, ring.next()) {
        const uint32_t s = ring.at;
        if (i >= ROWS) wait(&row_empty[s], ring.parity ^ 1u);
        umma::mbar_expect_tx(&row_full[s], 512 + PL::SL);
        umma::bulk_load(lam_s + s * 128, a.res.lam_end + (last - i) * KT, 512, &row_full[s]);
        umma::bulk_load(sR + s * PL::SL, reinterpret_cast<const uint8_t*>(a.res.states) + ((last - i) * Vw + v0) * 256, PL::SL, &row_full[s]);
      }
    } else if (role == 3 && lane == 0) {
      // ---------------------------------------------------------------------------------------- dH, dV, partial sums
      float* parts = dlend_part(g, a.dV);
      for (int i = 0; i < n && !wait.dead; ++i) {
        wait(&h_ready, i & 1);
        if (!CUT || i >= warm) umma::bulk_store(reinterpret_cast<uint8_t*>(a.dH) + ((last - i) * Vw + v0) * 256, sdH, PL::SL);
        umma::bulk_commit();
        umma::bulk_wait_read<0>();
        arrive(&h_free);
        wait(&v_ready, i & 1);
        if (!CUT || i >= warm) {
          umma::bulk_store(reinterpret_cast<uint8_t*>(a.dV) + ((last - i) * Vw + v0) * 256, sdV, PL::SL);
          umma::bulk_store(parts + ((last - i) * (Vw / 32) + v0 / 32) * KT, part_s, NG * 512);
        }
        umma::bulk_commit();
        umma::bulk_wait_read<0>();
        arrive(&v_free);
      }
      asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
  }
  __syncthreads();
  if (warp == 0) umma::tmem_dealloc(tmem_base, PL::TMEM);
}

// Parts to cut the range into (find_walk): four times as many walks as SMs, where documents are given and one walk per column
// slice leaves half of the chip idle.  A part is 4 chunks at least and the range 24, because a walk costs about two steps more than
// its chunks.  32 heads, 1024 chunks in 8 documents: forward 2361 us -> 1185, with entry states 1587 -> 1185, reverse 2243 -> 1725;
// 24 heads, 47 chunks in documents of 8 on average: forward 117 -> 75, reverse 105 -> 82; over 12 chunks it loses (51 -> 56).
// (Twice the SMs: 73 and 81, but 2194 for the reverse above: documents that share a part are one walk.)
int pick_parts(const StateArgs& a) {
  const int ctas = a.g.B * a.g.H * (a.g.Vw / 64), chunks = a.c_end - a.c_begin;
  if (!a.seg || a.P_out || a.until_independent || a.skip_provisional || ctas * 2 > sm_count() || chunks < 24) return 1;
  const int want = 4 * sm_count() / ctas, most = chunks / 4;
  return want < most ? want : most;
}

// Columns of the value width per CTA, 32 or 64.  What bounds a chunk step is shared memory: the products read their
// operands at its full width (46 cycles per 128 x 32 x 16 MMA, 48 at 64 columns, 64 at 128: the tile, 4 KB of each, dominates),
// the four tiles are written to it, and loads and stores of the threads wait their turn.  64 columns read the tiles half as
// often and leave the step 2.0 us as against 1.9 (forward, storing entry states), 2.2 as against 3.2 (reverse); at 128 it was 4.4.
// So: 64, except for uncut forward passes that store entry states and fit the SMs at 32 (fused prologue L=6001, 96 CTAs:
// 117 us against 139; the KDA pass over 131072 tokens with one launch of each kind: 3.92 ms against 4.18).
int pick_vs_fwd(const StateArgs& a) {
  if (a.P_out) return 64;                               // Vw + K columns of 32 heads in few enough CTAs for one wave
  return a.states && a.g.B * a.g.H * (a.g.Vw / 32) <= sm_count() ? 32 : 64;
}


template <int VS, bool CUT>
int launch_fwd(const StateArgs& a, cudaStream_t st) {
  using PL = Plan<VS, false>;
  const dim3 grid((a.g.Vw + (a.P_out ? a.g.K : 0)) / VS, a.g.H, a.g.B * a.parts);
  cudaFuncSetAttribute(state_fwd_tc_kernel<VS, CUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PL::SMEM);
  state_fwd_tc_kernel<VS, CUT><<<grid, PL::NT, PL::SMEM, st>>>(a);
  return launch_status();
}
template <int VS, bool CUT>
int launch_bwd(const StateArgs& a, cudaStream_t st) {
  using PL = Plan<VS, true>;
  const dim3 grid(a.g.Vw / VS, a.g.H, a.g.B * a.parts);
  cudaFuncSetAttribute(state_bwd_tc_kernel<VS, CUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PL::SMEM);
  state_bwd_tc_kernel<VS, CUT><<<grid, PL::NT, PL::SMEM, st>>>(a);
  return launch_status();
}

StateArgs with_range(const StateArgs& in) {
  StateArgs a = in;
  if (a.c_end <= 0) { a.c_begin = 0; a.c_end = a.g.NC; }
  a.err = device_error_ptr();
  a.parts = pick_parts(a);
  return a;
}

}  // namespace

bool state_tc_eligible(const Geo& g) { return g.img; }

int launch_state_fwd_tc(const StateArgs& in, cudaStream_t st) {
  const StateArgs a = with_range(in);
  if (a.parts > 1) return launch_fwd<64, true>(a, st);
  return pick_vs_fwd(a) == 64 ? launch_fwd<64, false>(a, st) : launch_fwd<32, false>(a, st);
}

int launch_state_bwd_tc(const StateArgs& in, cudaStream_t st) {
  const StateArgs a = with_range(in);
  return a.parts > 1 ? launch_bwd<64, true>(a, st) : launch_bwd<64, false>(a, st);
}

}  // namespace dn
