// Flash-style attention forward and backward on tcgen05 tensor cores (causal or full, MHA and
// GQA, head_dim 64 or 128), with Q/K/V/dO tiles staged by TMA (128-byte swizzle) and every
// matrix product accumulated in tensor memory.
//
// Forward (attn_fwd3_kernel), per item of 256 query rows of one (head, batch), looping over blocks of 64 keys:
//   S = Q K^T in TMEM -> softmax warps read one row per thread (no shuffles needed), keep the
//   running max / sum, write P (bf16) back over S in TMEM -> O += P V in TMEM, rescaled in place when
//   the maximum has grown by much. attn_fwd_kernel is the older form: one CTA per 128 query rows, P
//   through shared memory, O folded into registers.
// Backward, per item of 128 key rows of one (kv head, batch), looping over the query blocks (and,
// for GQA, over the query heads of the group):
//   S^T = K Q^T and dP^T = V dO^T (TMEM) -> threads rebuild P^T = exp(S^T*scale - lse) and
//   dS^T = P^T o (dP^T - delta) and write both back to tensor memory -> dV += P^T dO, dK += dS^T Q
//   (TMEM, accumulated over the whole loop), dQ^T = K^T dS^T (TMEM, then a TMA reduce-add into the
//   fp32 accumulator in global memory).
// The tiles loaded once by TMA serve both as K-major and as MN-major operands: a 128-row tile
// whose rows are 128 swizzled bytes is the canonical layout of either, read with a different
// descriptor.
//
// The reference attention is a forward-only scalar loop that builds one score row at a time
// (legacy/src/momijo/learn/nn/attention.mojo:122-161); softmax is the default normaliser here.
#include "common.cuh"

#include <cstdlib>

namespace mmj {

constexpr int kAttnThreads = 192;     // forward: TMA warp, MMA warp, 4 softmax warps
constexpr int kPanelBytes = 128 * 128;  // 128 rows x 64 bf16

struct AttnParams {
  int B, T, Hq, Hkv;
  int q_col0, k_col0, v_col0;  // column of head 0 inside the Q / K / V tensor maps
  float scale;                 // softmax scale (1/sqrt(D))
  int causal;
  // forward outputs
  __nv_bfloat16* O;
  long long ldo;
  float* lse;  // [B, Hq, T]
  // backward
  const float* delta;  // [B, Hq, T]
  float scale_log2;    // scale * log2(e); a factor too small to reach a sum where scale is 0
  uint32_t dead_score; // bits of the infinity that scale_log2 turns into -inf
  float* dQ;           // fp32 accumulator [B*T, ld_dq]
  long long ld_dq;
  __nv_bfloat16* dK;
  __nv_bfloat16* dV;
  long long ld_dk, ld_dv;
  int dk_col0, dv_col0, dq_col0, o_col0;
  int* status;
  long long* trace;  // nullable; kTraceSlots stamps per CTA
};

// K-major operand descriptor for k-step `k` (16 elements each) of a tile made of 64-column panels.
__device__ __forceinline__ uint64_t desc_kmajor(uint32_t tile_addr, int k) {
  return make_smem_desc(tile_addr + (uint32_t)(k >> 2) * kPanelBytes + (uint32_t)(k & 3) * 32, 16,
                        1024);
}
// MN-major operand descriptor: rows are the contraction index, 16 rows per k-step.
__device__ __forceinline__ uint64_t desc_mnmajor(uint32_t tile_addr, int k) {
  return make_smem_desc(tile_addr + (uint32_t)k * 2048, kPanelBytes, 1024);
}

// Write 32 consecutive columns [col0, col0+32) of row r into a 128 x 128 bf16 tile stored as
// two 64-column panels with the 128-byte swizzle (16-byte chunk index ^= row & 7).
__device__ __forceinline__ void store_chunk_sw128(uint8_t* tile, int r, int col0,
                                                  const float (&v)[32]) {
  uint8_t* rowp = tile + (col0 >> 6) * kPanelBytes + r * 128;
  const int cbase = (col0 & 63) >> 3;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint4 q;
    q.x = pack_bf16x2(v[8 * i + 0], v[8 * i + 1]);
    q.y = pack_bf16x2(v[8 * i + 2], v[8 * i + 3]);
    q.z = pack_bf16x2(v[8 * i + 4], v[8 * i + 5]);
    q.w = pack_bf16x2(v[8 * i + 6], v[8 * i + 7]);
    const int phys = (cbase + i) ^ (r & 7);
    *reinterpret_cast<uint4*>(rowp + phys * 16) = q;
  }
}

// TMA reduce-add of a shared-memory box into a global tensor (element type from the map).
// The x coordinate times the element size must be a multiple of 16 bytes; coordinates are
// never negative here.
__device__ __forceinline__ void tma_reduce_add_3d(const void* tmap, const void* smem_src, int c0,
                                                  int c1, int c2) {
  asm volatile(
      "cp.reduce.async.bulk.tensor.3d.global.shared::cta.add.bulk_group [%0, {%2, %3, %4}], [%1];"
      :
      : "l"(reinterpret_cast<uint64_t>(tmap)), "r"(smem_u32(smem_src)), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
__device__ __forceinline__ void bulk_commit_group() {
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
__device__ __forceinline__ void bulk_wait_group_read0() {
  asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}
__device__ __forceinline__ void bulk_wait_group0() {
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

// Optional kernel timeline: when a trace buffer is installed, one softmax (or compute) thread and the
// MMA thread of every CTA store clock64() stamps at their stage boundaries (64 slots per CTA).
constexpr int kTraceSlots = 64;
__device__ __forceinline__ void trace_stamp(long long* trace, int cta, int slot) {
  if (trace != nullptr && slot < kTraceSlots) trace[(long long)cta * kTraceSlots + slot] = clock64();
}

// =============================================================================================
// Forward
// =============================================================================================
template <int D>
__global__ void __launch_bounds__(kAttnThreads, (D == 64) ? 2 : 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                const __grid_constant__ CUtensorMap tmV, const AttnParams p) {
  constexpr int NP = D / 64;             // 64-column panels per tile
  constexpr int kTile = NP * kPanelBytes;
  constexpr uint32_t kTmemCols = 256;
  constexpr uint32_t kColS = 0, kColO = 128;
  // head_dim 64 keeps a single V stage so that two CTAs fit in one SM's shared memory (the
  // second CTA's softmax then overlaps this CTA's MMAs); head_dim 128 runs one CTA per SM.
  constexpr int VS = (D == 64) ? 1 : 2;

  extern __shared__ uint8_t smem_raw[];
  // (offset arithmetic on the __shared__ symbol, not an integer round trip, so that the compiler
  // keeps the shared address space and emits shared rather than generic loads and stores)
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t* sQ = smem;
  uint8_t* sK = sQ + kTile;      // 2 stages
  uint8_t* sV = sK + 2 * kTile;  // VS stages
  // head_dim 128 (one CTA per SM) has room for two P tiles, so the softmax of block j+1 need not
  // wait for P(j) V(j); head_dim 64 keeps one (its second CTA on the SM fills the gap)
  constexpr int PB = (D == 64) ? 1 : 2;
  constexpr int kPTile = 2 * kPanelBytes;
  uint8_t* sP = sV + VS * kTile;  // PB tiles of 128 x 128 bf16

  __shared__ __align__(8) uint64_t q_full, s_full, p_full, o_full;
  __shared__ __align__(8) uint64_t k_full[2], k_empty[2], v_full[2], v_empty[2], p_free[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int num_qb = (p.T + 127) / 128;
  const int qb = num_qb - 1 - (int)blockIdx.x;  // heaviest (latest) query blocks first
  const int h = blockIdx.y, b = blockIdx.z;
  const int hkv = h / (p.Hq / p.Hkv);
  const int q0 = qb * 128;
  int kv_end = p.causal ? min(p.T, q0 + 128) : p.T;
  const int nkv = (kv_end + 127) / 128;
  const int cta_lin = (blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
  const bool tracer = (threadIdx.x == 64);
  if (tracer) {
    trace_stamp(p.trace, cta_lin, 0);
    if (p.trace) {
      uint32_t smid;
      asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
      p.trace[(long long)cta_lin * kTraceSlots + 1] = smid;
      p.trace[(long long)cta_lin * kTraceSlots + 7] = nkv;
    }
  }

  if (threadIdx.x == 0) {
    mbar_init(&q_full, 1);
    mbar_init(&s_full, 1);
    mbar_init(&p_full, 4);
    mbar_init(&o_full, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&k_empty[s], 1);
      mbar_init(&v_full[s], 1);
      mbar_init(&v_empty[s], 1);
      mbar_init(&p_free[s], 1);
    }
    abort_flag = 0;
    mbar_fence_init();
    prefetch_tmap(&tmQ);
    prefetch_tmap(&tmK);
    prefetch_tmap(&tmV);
  }
  if (warp == 1) {
    tmem_alloc(&tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;
  pdl_wait();  // the set-up above read no tensor of the step
  pdl_trigger();
  if (tracer) trace_stamp(p.trace, cta_lin, 2);

  if (warp == 0) {
    if (lane == 0) {
      mbar_expect_tx(&q_full, kTile);
#pragma unroll
      for (int pn = 0; pn < NP; ++pn)
        tma_load_3d(sQ + pn * kPanelBytes, &tmQ, &q_full, p.q_col0 + h * D + pn * 64, q0, b);
      for (int j = 0; j < nkv; ++j) {
        const int s = j & 1;
        const uint32_t ph = (j >> 1) & 1;
        if (!mbar_wait(&k_empty[s], ph ^ 1, &abort_flag, p.status, kTimeoutEmpty, j)) break;
        mbar_expect_tx(&k_full[s], kTile);
#pragma unroll
        for (int pn = 0; pn < NP; ++pn)
          tma_load_3d(sK + s * kTile + pn * kPanelBytes, &tmK, &k_full[s],
                      p.k_col0 + hkv * D + pn * 64, j * 128, b);
        const int sv = j % VS;
        const uint32_t phv = (j / VS) & 1;
        if (!mbar_wait(&v_empty[sv], phv ^ 1, &abort_flag, p.status, kTimeoutEmpty, 100 + j)) break;
        mbar_expect_tx(&v_full[sv], kTile);
#pragma unroll
        for (int pn = 0; pn < NP; ++pn)
          tma_load_3d(sV + sv * kTile + pn * kPanelBytes, &tmV, &v_full[sv],
                      p.v_col0 + hkv * D + pn * 64, j * 128, b);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc_s = make_idesc_bf16(128, 128, 0, 0);
      const uint32_t idesc_o = make_idesc_bf16(128, D, 0, 1);
      const uint32_t aQ = smem_u32(sQ), aP = smem_u32(sP);
      bool ok = mbar_wait(&q_full, 0, &abort_flag, p.status, kTimeoutFull, -1);
      auto issue_s = [&](int j) -> bool {
        const int s = j & 1;
        const uint32_t ph = (j >> 1) & 1;
        if (!mbar_wait(&k_full[s], ph, &abort_flag, p.status, kTimeoutFull, j)) return false;
        tc_fence_after();
        const uint32_t aK = smem_u32(sK + s * kTile);
#pragma unroll
        for (int k = 0; k < D / 16; ++k)
          umma_bf16_ss(tmem_base + kColS, desc_kmajor(aQ, k), desc_kmajor(aK, k), idesc_s,
                       k > 0 ? 1u : 0u);
        umma_commit(&k_empty[s]);
        umma_commit(&s_full);
        return true;
      };
      if (ok) ok = issue_s(0);
      for (int j = 0; j < nkv && ok; ++j) {
        const int sv = j % VS;
        const uint32_t phv = (j / VS) & 1;
        if (!mbar_wait(&p_full, j & 1, &abort_flag, p.status, kTimeoutFlag, j)) break;
        trace_stamp(p.trace, cta_lin, 8 + j * 6 + 3);
        // P(j) written means S(j) has been consumed: the next score tile goes first, so that
        // the softmax of block j+1 can start while P(j) V(j) is still running
        if (j + 1 < nkv) ok = issue_s(j + 1);
        if (!ok) break;
        if (!mbar_wait(&v_full[sv], phv, &abort_flag, p.status, kTimeoutFull, 100 + j)) break;
        tc_fence_after();
        const uint32_t aV = smem_u32(sV + sv * kTile);
#pragma unroll
        for (int k = 0; k < 8; ++k)
          umma_bf16_ss(tmem_base + kColO, desc_kmajor(aP + (uint32_t)((j % PB) * kPTile), k), desc_mnmajor(aV, k), idesc_o,
                       (j > 0 || k > 0) ? 1u : 0u);
        umma_commit(&v_empty[sv]);
        umma_commit(&p_free[j % PB]);  // this P tile may be overwritten
        umma_commit(&o_full);
      }
    }
  } else {
    // ---------------- softmax / output warps: one query row per thread ----------------
    const int quad = warp & 3;
    const int row = quad * 32 + lane;
    const int q_idx = q0 + row;
    const uint32_t t_lane = tmem_base + ((uint32_t)(quad * 32) << 16);
    const float c = p.scale * 1.4426950408889634f;
    // The output accumulator stays in tensor memory (P V accumulates into it); it is rescaled
    // in place only when the running row maximum grows by more than kTau (in the exp2 domain),
    // so most iterations neither read nor write it. Probabilities are then bounded by 2^kTau,
    // which bf16 / fp32 hold comfortably, and the final 1/l normalisation makes the result exact.
    constexpr float kTau = 8.0f;
    float m_used = -1.0e30f, l = 0.f;
    bool ok = true;
    for (int j = 0; j < nkv; ++j) {
      if (!mbar_wait_warp(&s_full, j & 1, &abort_flag, p.status, kTimeoutTmemFull, j)) { ok = false; break; }
      tc_fence_after();
      if (tracer) trace_stamp(p.trace, cta_lin, 8 + j * 6 + 0);
      const int kv0 = j * 128;
      const bool need_mask = (p.causal && (kv0 + 127 > q0)) || (kv0 + 128 > p.T);
      uint32_t s[128];
      tmem_ld_32x32(t_lane + kColS + 0, *reinterpret_cast<uint32_t(*)[32]>(&s[0]));
      tmem_ld_32x32(t_lane + kColS + 32, *reinterpret_cast<uint32_t(*)[32]>(&s[32]));
      tmem_ld_32x32(t_lane + kColS + 64, *reinterpret_cast<uint32_t(*)[32]>(&s[64]));
      tmem_ld_32x32(t_lane + kColS + 96, *reinterpret_cast<uint32_t(*)[32]>(&s[96]));
      tmem_ld_wait();
      if (tracer) trace_stamp(p.trace, cta_lin, 8 + j * 6 + 1);
      if (need_mask) {
#pragma unroll
        for (int i = 0; i < 128; ++i) {
          const int kv = kv0 + i;
          if (kv >= p.T || (p.causal && kv > q_idx)) s[i] = 0xff800000u;  // -inf
        }
      }
      float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY;
#pragma unroll
      for (int i = 0; i < 128; i += 4) {
        mx0 = fmaxf(mx0, __uint_as_float(s[i + 0]));
        mx1 = fmaxf(mx1, __uint_as_float(s[i + 1]));
        mx2 = fmaxf(mx2, __uint_as_float(s[i + 2]));
        mx3 = fmaxf(mx3, __uint_as_float(s[i + 3]));
      }
      const float mx = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3));
      const bool grow = (mx - m_used) * c > kTau;  // false for fully masked rows (mx = -inf)
      if (__any_sync(0xffffffffu, grow ? 1 : 0)) {
        float alpha = 1.0f;
        if (grow) {
          alpha = exp2f((m_used - mx) * c);
          l *= alpha;
          m_used = mx;
        }
        if (j > 0) {
          // P(j-1) V(j-1) must have landed before the accumulator is rescaled
          if (!mbar_wait_warp(&o_full, (j - 1) & 1, &abort_flag, p.status, kTimeoutTmemFull, 100 + j)) { ok = false; break; }
          tc_fence_after();
#pragma unroll
          for (int cc = 0; cc < D / 32; ++cc) {
            uint32_t r[32];
            tmem_ld_32x32(t_lane + kColO + cc * 32, r);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * alpha);
            tmem_st_32x32(t_lane + kColO + cc * 32, r);
          }
          tmem_st_wait();
        }
      }
      // P(j-1) V(j-1) reads the P tile that is about to be overwritten: it must have finished. (It
      // was issued after S(j) and takes a fraction of the time spent above, so this wait is normally
      // already satisfied; without it the order would only be a matter of timing.)
      // (one barrier per P tile: each sees one completion per use of its tile, so a wait for the
      // previous use can never be overtaken by a later phase)
      if (j >= PB) {
        if (!mbar_wait_warp(&p_free[j % PB], ((j / PB) - 1) & 1, &abort_flag, p.status, kTimeoutTmemFull, 200 + j)) { ok = false; break; }
      }
      const float mc = m_used * c;
      float sum0 = 0.f, sum1 = 0.f, sum2 = 0.f, sum3 = 0.f;
#pragma unroll
      for (int cc = 0; cc < 4; ++cc) {
        float(&pv)[32] = *reinterpret_cast<float(*)[32]>(&s[cc * 32]);  // exponentiate in place
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
          pv[i + 0] = exp2f(fmaf(pv[i + 0], c, -mc));
          pv[i + 1] = exp2f(fmaf(pv[i + 1], c, -mc));
          pv[i + 2] = exp2f(fmaf(pv[i + 2], c, -mc));
          pv[i + 3] = exp2f(fmaf(pv[i + 3], c, -mc));
          sum0 += pv[i + 0]; sum1 += pv[i + 1]; sum2 += pv[i + 2]; sum3 += pv[i + 3];
        }
        store_chunk_sw128(sP + (j % PB) * kPTile, row, cc * 32, pv);
      }
      l += (sum0 + sum1) + (sum2 + sum3);
      fence_proxy_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full);
      if (tracer) trace_stamp(p.trace, cta_lin, 8 + j * 6 + 2);
    }
    if (tracer) trace_stamp(p.trace, cta_lin, 4);
    // final: wait for the last P V, normalise and store
    if (ok && nkv > 0)
      ok = mbar_wait_warp(&o_full, (nkv - 1) & 1, &abort_flag, p.status, kTimeoutTmemFull, 999);
    if (ok) {
      tc_fence_after();
      const float inv = (l > 0.f) ? 1.0f / l : 0.f;
      __nv_bfloat16* dst = p.O + ((long long)b * p.T + q_idx) * p.ldo + p.o_col0 + h * D;
#pragma unroll
      for (int cc = 0; cc < D / 32; ++cc) {
        uint32_t r[32];
        tmem_ld_32x32(t_lane + kColO + cc * 32, r);
        tmem_ld_wait();
        if (q_idx < p.T) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            uint4 q;
            q.x = pack_bf16x2(__uint_as_float(r[8 * i + 0]) * inv, __uint_as_float(r[8 * i + 1]) * inv);
            q.y = pack_bf16x2(__uint_as_float(r[8 * i + 2]) * inv, __uint_as_float(r[8 * i + 3]) * inv);
            q.z = pack_bf16x2(__uint_as_float(r[8 * i + 4]) * inv, __uint_as_float(r[8 * i + 5]) * inv);
            q.w = pack_bf16x2(__uint_as_float(r[8 * i + 6]) * inv, __uint_as_float(r[8 * i + 7]) * inv);
            reinterpret_cast<uint4*>(dst + cc * 32)[i] = q;
          }
        }
      }
      if (q_idx < p.T && p.lse != nullptr)
        p.lse[((long long)b * p.Hq + h) * p.T + q_idx] =
            (l > 0.f) ? (m_used * p.scale + __logf(l)) : -INFINITY;
    }
  }

  if (tracer) trace_stamp(p.trace, cta_lin, 5);
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tmem_dealloc(tmem_base, kTmemCols);
  }
  if (tracer) trace_stamp(p.trace, cta_lin, 6);
}

// =============================================================================================
// Forward, two query tiles per CTA, 64-key blocks, double-buffered score tiles (the default)
// =============================================================================================
// One persistent CTA per SM walks a list of work items, heaviest first; an item is 256 query rows (two
// 128-row tiles) of one (batch, head). Three warpgroups: warps 0..3 = TMA producer (warp 0), one MMA issuer
// per query tile (warps 1 and 2; warp 1 owns the TMEM allocation) and an idle warp; warps 4..7 = softmax
// group of tile 0; warps 8..11 = softmax group of tile 1 (one query row per thread). A softmax group reads
// its score tile from tensor memory, writes the probabilities back over the first columns of the same tile
// as packed bf16 pairs, and the P V product takes them from there as its tensor-memory A operand: P never
// touches shared memory. Three things keep the groups' dependency chain short:
//   * each query tile has its own MMA-issuing thread (warps 1 and 2);
//   * a key block is 64 keys and every query tile owns TWO score buffers in tensor memory
//     (S_t[0], S_t[1], 64 columns each): the MMA thread issues S_t(j+1) before the group has finished
//     block j, so a group that has stored P_t(j) finds S_t(j+1) waiting and starts on it at once;
//     per key block the MMA thread does  [wait P_t(j)]  P_t(j) V_j -> O_t,  Q_t K_(j+2)^T -> S_t[j & 1];
//   * three-operand maxima, paired multiply-adds and sums and the paired conversion shorten the softmax's own chain
//     (B6 T1777 H16 D128 full 196 -> 183 us).
// No unit bounds it: counters of that call read issue slots 34 %, exponentials' unit 46 % (64 exponentials and 32
// conversions a row and block), tensor pipe 45 %, L2 21 %; at head_dim 64 (B16 T1024 H12 causal) 34, 41, 20 and 15 %.
// 0.46 warps are ready a cycle and scheduler, out of three: fixed-latency waits (2.3 of 8.8 cycles an instruction), TMEM
// loads (1.4 and 1.8) and the stores' queue (1.0 and 0.5) are the chain of one row per thread, one warp a scheduler and tile.
// Tensor memory: S0[0] S0[1] S1[0] S1[1] | O0 | O1 = 256 + 2 D columns; P_t(j) overwrites the first 32
// columns of S_t[j & 1] (64 probabilities as bf16 pairs). Every P_t(j) V_j commits to o_done[t][j & 1];
// a group waits on it only before it rescales O_t (rare: the running maximum must have grown by more
// than 2^8) and before the final normalisation.
template <int D>
__global__ void __launch_bounds__(384, 1)
attn_fwd3_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                 const __grid_constant__ CUtensorMap tmV, const AttnParams p) {
  constexpr int NP = D / 64;
  constexpr int kQTile = NP * kPanelBytes;         // 128 query rows
  constexpr int kKVPanel = 64 * 128;               // 64 key rows x 64 bf16
  constexpr int kKVTile = NP * kKVPanel;           // 64 key rows x D
  constexpr int KS = (D == 64) ? 6 : 4;            // K and V stages
  constexpr uint32_t kTmemCols = 512;
  constexpr uint32_t kColO = 256;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t* sQ = smem;                   // 2 tiles
  uint8_t* sK = sQ + 2 * kQTile;        // KS stages
  uint8_t* sV = sK + KS * kKVTile;      // KS stages

  __shared__ __align__(8) uint64_t q_full[2], q_empty[2], o_free[2];
  __shared__ __align__(8) uint64_t s_full[2][2], p_full[2][2], o_done[2][2];
  __shared__ __align__(8) uint64_t k_full[KS], k_empty[KS], v_full[KS], v_empty[KS];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nqp = (p.T + 255) / 256;
  const int nbh = p.B * p.Hq;
  const int n_items = nqp * nbh;
  const int group = p.Hq / p.Hkv;

  if (threadIdx.x == 0) {
    for (int t = 0; t < 2; ++t) {
      mbar_init(&q_full[t], 1);
      mbar_init(&q_empty[t], 1);
      mbar_init(&o_free[t], 4);
      for (int b = 0; b < 2; ++b) {
        mbar_init(&s_full[t][b], 1);
        mbar_init(&p_full[t][b], 4);
        mbar_init(&o_done[t][b], 1);
      }
    }
    for (int s = 0; s < KS; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&k_empty[s], 2);   // one arrival per query tile (its MMA thread)
      mbar_init(&v_full[s], 1);
      mbar_init(&v_empty[s], 2);
    }
    abort_flag = 0;
    mbar_fence_init();
    prefetch_tmap(&tmQ);
    prefetch_tmap(&tmK);
    prefetch_tmap(&tmV);
  }
  if (warp == 1) {
    tmem_alloc(&tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  constexpr uint32_t tmem_base = 0;   // an allocation of all 512 columns starts at column 0
  pdl_wait();  // the set-up above touched no global memory
  pdl_trigger();

  auto decode = [&](int w, int& qp, int& h, int& b) {
    qp = nqp - 1 - w / nbh;  // later (longer) query pairs first
    const int bh = w % nbh;
    h = bh % p.Hq;
    b = bh / p.Hq;
  };
  // 64-key blocks of tile t of query pair qp (0 when the tile lies beyond T)
  auto blocks_of = [&](int qp, int t) -> int {
    const int q0 = qp * 256 + t * 128;
    if (q0 >= p.T) return 0;
    const int kv_end = p.causal ? min(p.T, q0 + 128) : p.T;
    return (kv_end + 63) / 64;
  };

  if (warp == 0) {
    // ======================= TMA producer =======================
    if (lane == 0) {
      uint32_t qn[2] = {0, 0};
      uint32_t kc = 0;  // ring position of this item's block 0 (K and V rings advance together per item)
      bool ok = true;
      for (int w = blockIdx.x; w < n_items && ok; w += gridDim.x) {
        int qp, h, b;
        decode(w, qp, h, b);
        const int hkv = h / group;
        const int nb[2] = {blocks_of(qp, 0), blocks_of(qp, 1)};
        const int n1 = max(nb[0], nb[1]);
        for (int t = 0; t < 2 && ok; ++t) {
          if (nb[t] == 0) continue;
          if (!mbar_wait(&q_empty[t], (qn[t] & 1) ^ 1, &abort_flag, p.status, kTimeoutEmpty, 300 + t)) { ok = false; break; }
          ++qn[t];
          mbar_expect_tx(&q_full[t], kQTile);
#pragma unroll
          for (int pn = 0; pn < NP; ++pn)
            tma_load_3d(sQ + t * kQTile + pn * kPanelBytes, &tmQ, &q_full[t], p.q_col0 + h * D + pn * 64,
                        qp * 256 + t * 128, b);
        }
        auto load_k = [&](int j) -> bool {
          const uint32_t c = kc + (uint32_t)j;
          const int s = c % KS;
          if (!mbar_wait(&k_empty[s], ((c / KS) & 1) ^ 1, &abort_flag, p.status, kTimeoutEmpty, j)) return false;
          mbar_expect_tx(&k_full[s], kKVTile);
#pragma unroll
          for (int pn = 0; pn < NP; ++pn)
            tma_load_3d(sK + s * kKVTile + pn * kKVPanel, &tmK, &k_full[s], p.k_col0 + hkv * D + pn * 64, j * 64, b);
          return true;
        };
        auto load_v = [&](int j) -> bool {
          const uint32_t c = kc + (uint32_t)j;
          const int s = c % KS;
          if (!mbar_wait(&v_empty[s], ((c / KS) & 1) ^ 1, &abort_flag, p.status, kTimeoutEmpty, 100 + j)) return false;
          mbar_expect_tx(&v_full[s], kKVTile);
#pragma unroll
          for (int pn = 0; pn < NP; ++pn)
            tma_load_3d(sV + s * kKVTile + pn * kKVPanel, &tmV, &v_full[s], p.v_col0 + hkv * D + pn * 64, j * 64, b);
          return true;
        };
        // the order the MMA thread consumes them in: K0 K1 V0 K2 V1 K3 ...
        for (int j = 0; j < n1 && ok; ++j) {
          ok = load_k(j);
          if (ok && j >= 1) ok = load_v(j - 1);
        }
        if (ok && n1 > 0) ok = load_v(n1 - 1);
        kc += (uint32_t)n1;
      }
    }
  } else if (warp == 1 || warp == 2) {
    // ======================= MMA issuers: warp 1 drives query tile 0, warp 2 tile 1 =======================
    // (the warps stay converged and elect a lane to issue; one issuer for both tiles queued their chains behind each
    // other)
    {
      const int t = warp - 1;
      const uint32_t idesc_s = make_idesc_bf16(128, 64, 0, 0);
      const uint32_t idesc_o = make_idesc_bf16(128, D, 0, 1);
      const uint32_t lo_q = smem_desc_lo(smem_u32(sQ) + t * kQTile, 16), lo_k = smem_desc_lo(smem_u32(sK), 16);
      const uint32_t lo_v = smem_desc_lo(smem_u32(sV), kKVPanel);
      uint32_t qn = 0;
      uint32_t pc[2] = {0, 0};  // P tiles consumed so far, per buffer
      uint32_t on = 0;
      uint32_t kc = 0;
      bool ok = true;
      for (int w = blockIdx.x; w < n_items && ok; w += gridDim.x) {
        int qp, h, b;
        decode(w, qp, h, b);
        const int nbt = blocks_of(qp, t);
        const int n1 = max(blocks_of(qp, 0), blocks_of(qp, 1));
        // S_t(j) = Q_t K_j^T into buffer j & 1
        auto issue_s = [&](int j) -> bool {
          const uint32_t c = kc + (uint32_t)j;
          const int s = c % KS;
          if (!mbar_wait_warp(&k_full[s], (c / KS) & 1, &abort_flag, p.status, kTimeoutFull, j)) return false;
          tc_fence_after();
          if (elect_one()) {
            const uint32_t d = (uint32_t)(t * 128 + (j & 1) * 64), bk = lo_k + s * (kKVTile >> 4);
#pragma unroll
            for (int k = 0; k < D / 16; ++k)
              // K tile: 64 rows, 64-column panels of 8 KiB
              umma_bf16_ss(d, smem_desc(lo_q + ((k >> 2) * kPanelBytes + (k & 3) * 32) / 16),
                           smem_desc(bk + ((k >> 2) * kKVPanel + (k & 3) * 32) / 16), idesc_s, k > 0 ? 1u : 0u);
            umma_commit(&s_full[t][j & 1]);
            umma_commit(&k_empty[s]);   // this tile's share of the K block's release
            if (j + 1 == nbt) umma_commit(&q_empty[t]);
          }
          __syncwarp();
          return true;
        };
        if (nbt > 0) {
          if (!mbar_wait_warp(&q_full[t], qn & 1, &abort_flag, p.status, kTimeoutFull, 400 + t)) { ok = false; break; }
          ++qn;
          ok = issue_s(0);
          if (ok && nbt > 1) ok = issue_s(1);
        }
        for (int j = 0; j < n1 && ok; ++j) {
          const uint32_t c = kc + (uint32_t)j;
          const int sv = c % KS;
          if (j >= nbt) {
            // a key block only the other tile reads: hand in this tile's share of its release, but only
            // once the block has been loaded (an earlier arrival would count for the stage's previous block)
            if (!mbar_wait_warp(&k_full[sv], (c / KS) & 1, &abort_flag, p.status, kTimeoutFull, 800 + j)) { ok = false; break; }
            if (lane == 0) mbar_arrive(&k_empty[sv]);
            if (!mbar_wait_warp(&v_full[sv], (c / KS) & 1, &abort_flag, p.status, kTimeoutFull, 900 + j)) { ok = false; break; }
            if (lane == 0) mbar_arrive(&v_empty[sv]);
            continue;
          }
          const int bf = j & 1;
          if (!mbar_wait_warp(&v_full[sv], (c / KS) & 1, &abort_flag, p.status, kTimeoutFull, 100 + j)) { ok = false; break; }
          if (j == 0 && on > 0) {
            if (!mbar_wait_warp(&o_free[t], (on - 1) & 1, &abort_flag, p.status, kTimeoutTmemEmpty, 600 + t)) { ok = false; break; }
          }
          if (!mbar_wait_warp(&p_full[t][bf], pc[bf] & 1, &abort_flag, p.status, kTimeoutFlag, 500 + j)) { ok = false; break; }
          ++pc[bf];
          tc_fence_after();
          if (elect_one()) {
            const uint32_t bv = lo_v + sv * (kKVTile >> 4), aP = (uint32_t)(t * 128 + bf * 64);
#pragma unroll
            for (int k = 0; k < 4; ++k)
              // V tile as an MN-major B operand: 16 key rows per step, 64-wide panels 8 KiB apart
              umma_bf16_ts(kColO + t * D, aP + k * 8, smem_desc(bv + k * 128), idesc_o, (j > 0 || k > 0) ? 1u : 0u);
            umma_commit(&o_done[t][bf]);   // P_t(j) V_j has landed in O_t
            umma_commit(&v_empty[sv]);
          }
          __syncwarp();
          if (j + 1 == nbt) ++on;
          if (j + 2 < nbt) ok = issue_s(j + 2);
        }
        kc += (uint32_t)n1;
      }
    }
  } else if (warp >= 4) {
    // ======================= softmax groups: one query row per thread =======================
    const int t = (warp - 4) >> 2;
    const int quad = warp & 3;
    const int row = quad * 32 + lane;
    const uint32_t t_lane = tmem_base + ((uint32_t)(quad * 32) << 16);
    const uint32_t colO = kColO + t * D;
    const float c = p.scale * 1.4426950408889634f;
    constexpr float kTau = 8.0f;
    uint32_t sn[2] = {0, 0};   // score tiles consumed so far, per buffer
    uint32_t pn[2] = {0, 0};   // P tiles produced so far, per buffer (= P V products expected)
    bool ok = true;
    const bool tracer = (p.trace != nullptr) && (lane == 0) && (quad == 0) && (t == 0);
    for (int w = blockIdx.x; w < n_items && ok; w += gridDim.x) {
      int qp, h, b;
      decode(w, qp, h, b);
      const int nkv = blocks_of(qp, t);
      if (nkv == 0) continue;
      const int q0 = qp * 256 + t * 128;
      const int q_idx = q0 + row;
      const bool tr = tracer && (w == (int)blockIdx.x);
      if (tr && t == 0) {
        p.trace[(long long)blockIdx.x * kTraceSlots + 7] = nkv;
        trace_stamp(p.trace, blockIdx.x, 0);
      }
      float m_used = -1.0e30f, l = 0.f;
      for (int j = 0; j < nkv; ++j) {
        const int bf = j & 1;
        const uint32_t colS = (uint32_t)(t * 128 + bf * 64);
        if (!mbar_wait_warp(&s_full[t][bf], sn[bf] & 1, &abort_flag, p.status, kTimeoutTmemFull, j)) { ok = false; break; }
        ++sn[bf];
        tc_fence_after();
        if (tr && j < 6) trace_stamp(p.trace, blockIdx.x, 8 + 24 * t + 4 * j + 0);
        const int kv0 = j * 64;
        const bool need_mask = (p.causal && (kv0 + 63 > q0)) || (kv0 + 64 > p.T);
        uint32_t s[64];
        tmem_ld_32x32(t_lane + colS + 0, *reinterpret_cast<uint32_t(*)[32]>(&s[0]));
        tmem_ld_32x32(t_lane + colS + 32, *reinterpret_cast<uint32_t(*)[32]>(&s[32]));
        tmem_ld_wait();
        if (tr && j < 6) trace_stamp(p.trace, blockIdx.x, 8 + 24 * t + 4 * j + 1);
        if (need_mask) {
          // keys behind the query (causal) and past the end: one bit per column
          const int n = min(p.T, p.causal ? q_idx + 1 : p.T) - kv0;   // live columns
          const uint32_t m0 = n >= 32 ? 0xffffffffu : n <= 0 ? 0u : (1u << n) - 1u;
          const uint32_t m1 = n >= 64 ? 0xffffffffu : n <= 32 ? 0u : (1u << (n - 32)) - 1u;
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            s[i] = (m0 & (1u << i)) ? s[i] : 0xff800000u;  // -inf
            s[i + 32] = (m1 & (1u << i)) ? s[i + 32] : 0xff800000u;
          }
        }
        float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY;
#pragma unroll
        for (int i = 0; i < 64; i += 8) {
          mx0 = fmax3(mx0, __uint_as_float(s[i + 0]), __uint_as_float(s[i + 1]));
          mx1 = fmax3(mx1, __uint_as_float(s[i + 2]), __uint_as_float(s[i + 3]));
          mx2 = fmax3(mx2, __uint_as_float(s[i + 4]), __uint_as_float(s[i + 5]));
          mx3 = fmax3(mx3, __uint_as_float(s[i + 6]), __uint_as_float(s[i + 7]));
        }
        const float mx = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3));
        if (tr && j < 6) trace_stamp(p.trace, blockIdx.x, 8 + 24 * t + 4 * j + 2);
        const bool grow = (mx - m_used) * c > kTau;  // false for fully masked rows (mx = -inf)
        if (__any_sync(0xffffffffu, grow ? 1 : 0)) {
          float alpha = 1.0f;
          if (grow) {
            alpha = exp2f((m_used - mx) * c);
            l *= alpha;
            m_used = mx;
          }
          if (j > 0) {
            // O_t holds the blocks up to j - 1 once P_t(j-1) V has landed (its commit is the newest on
            // the other buffer's barrier; never more than one completion away, so the parity is safe)
            const int ob = bf ^ 1;
            if (!mbar_wait_warp(&o_done[t][ob], (pn[ob] - 1) & 1, &abort_flag, p.status, kTimeoutTmemFull, 700 + j)) { ok = false; break; }
            tc_fence_after();
#pragma unroll
            for (int cc = 0; cc < D / 32; ++cc) {
              uint32_t r[32];
              tmem_ld_32x32(t_lane + colO + cc * 32, r);
              tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * alpha);
              tmem_st_32x32(t_lane + colO + cc * 32, r);
            }
          }
        }
        const f32x2 c2 = f2_pack(c, c), mc2 = f2_pack(-m_used * c, -m_used * c);
        f32x2 sum0 = 0ull, sum1 = 0ull;   // two zeros each
        // 64 probabilities as bf16 pairs, packed in place: pair m lands in s[m], which the loop has
        // already consumed (it reads s[2m ...], never behind its writes)
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          float e0, e1, e2, e3;
          f2_unpack(f2_fma(f2_pack(__uint_as_float(s[2 * i + 0]), __uint_as_float(s[2 * i + 1])), c2, mc2), e0, e1);
          f2_unpack(f2_fma(f2_pack(__uint_as_float(s[2 * i + 2]), __uint_as_float(s[2 * i + 3])), c2, mc2), e2, e3);
          e0 = exp2f(e0); e1 = exp2f(e1); e2 = exp2f(e2); e3 = exp2f(e3);
          sum0 = f2_add(sum0, f2_pack(e0, e1));
          sum1 = f2_add(sum1, f2_pack(e2, e3));
          s[i + 0] = pack_bf16x2(e0, e1);
          s[i + 1] = pack_bf16x2(e2, e3);
        }
        tmem_st_32x32(t_lane + colS, *reinterpret_cast<uint32_t(*)[32]>(&s[0]));
        float l0, l1;
        f2_unpack(f2_add(sum0, sum1), l0, l1);
        l += l0 + l1;
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[t][bf]);
        ++pn[bf];
        if (tr && j < 6) trace_stamp(p.trace, blockIdx.x, 8 + 24 * t + 4 * j + 3);
      }
      if (!ok) break;
      if (tr) trace_stamp(p.trace, blockIdx.x, 2 + 2 * t);
      // final: wait for the last P V of this tile, normalise and store
      {
        const int lb = (nkv - 1) & 1;
        if (!mbar_wait_warp(&o_done[t][lb], (pn[lb] - 1) & 1, &abort_flag, p.status, kTimeoutTmemFull, 999)) { ok = false; break; }
      }
      tc_fence_after();
      const float inv = (l > 0.f) ? 1.0f / l : 0.f;
      __nv_bfloat16* dst = p.O + ((long long)b * p.T + q_idx) * p.ldo + p.o_col0 + h * D;
#pragma unroll
      for (int cc = 0; cc < D / 32; ++cc) {
        uint32_t r[32];
        tmem_ld_32x32(t_lane + colO + cc * 32, r);
        tmem_ld_wait();
        if (cc == D / 32 - 1) {
          // the accumulator is in registers: the next item may overwrite O_t
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&o_free[t]);
        }
        if (q_idx < p.T) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            uint4 q;
            q.x = pack_bf16x2(__uint_as_float(r[8 * i + 0]) * inv, __uint_as_float(r[8 * i + 1]) * inv);
            q.y = pack_bf16x2(__uint_as_float(r[8 * i + 2]) * inv, __uint_as_float(r[8 * i + 3]) * inv);
            q.z = pack_bf16x2(__uint_as_float(r[8 * i + 4]) * inv, __uint_as_float(r[8 * i + 5]) * inv);
            q.w = pack_bf16x2(__uint_as_float(r[8 * i + 6]) * inv, __uint_as_float(r[8 * i + 7]) * inv);
            reinterpret_cast<uint4*>(dst + cc * 32)[i] = q;
          }
        }
      }
      if (q_idx < p.T && p.lse != nullptr)
        p.lse[((long long)b * p.Hq + h) * p.T + q_idx] = (l > 0.f) ? (m_used * p.scale + __logf(l)) : -INFINITY;
      if (tr) trace_stamp(p.trace, blockIdx.x, 3 + 2 * t);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// =============================================================================================
// Backward
// =============================================================================================
// delta[b, h, t] = sum_d dO[b, t, h, d] * O[b, t, h, d]; D/8 lanes per (row, head), 16 bytes per
// lane and tensor, so a warp covers 4 (head_dim 64) or 2 (head_dim 128) heads of a row at once.
// The same lanes clear the fp32 dQ accumulator (8 values each) that the backward kernel adds into.
__global__ void attn_delta_kernel(const __nv_bfloat16* __restrict__ O, long long ldo, int o_col0,
                                  const __nv_bfloat16* __restrict__ dO, long long lddo, int do_col0,
                                  float* __restrict__ delta, float* __restrict__ dq_zero, long long ld_dq,
                                  int dq_col0, int B, int T, int H, int D) {
  pdl_wait();
  pdl_trigger();
  const int lp = D >> 3;  // lanes per item: 8 or 16
  const long long gt = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long item = gt / lp;
  const int sub = (int)(gt - item * lp);
  const long long total = (long long)B * T * H;
  const bool live = item < total;
  float s = 0.f;
  int h = 0;
  long long bt = 0;
  if (live) {
    h = (int)(item % H);
    bt = item / H;
    const uint4 a = *reinterpret_cast<const uint4*>(O + bt * ldo + o_col0 + h * D + sub * 8);
    const uint4 c = *reinterpret_cast<const uint4*>(dO + bt * lddo + do_col0 + h * D + sub * 8);
    if (dq_zero != nullptr) {
      float4* z = reinterpret_cast<float4*>(dq_zero + bt * ld_dq + dq_col0 + h * D + sub * 8);
      z[0] = make_float4(0.f, 0.f, 0.f, 0.f);
      z[1] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const uint32_t av[4] = {a.x, a.y, a.z, a.w}, cv[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 x = unpack_bf16x2(av[i]), y = unpack_bf16x2(cv[i]);
      s = fmaf(x.x, y.x, fmaf(x.y, y.y, s));
    }
  }
  for (int o = lp >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (live && sub == 0) {
    const long long b = bt / T, t = bt - b * T;
    delta[(b * H + h) * T + t] = s;
  }
}

// Backward kernel: one persistent CTA per SM walks (key block, kv head, batch) items; inside an item it visits
// 64-query blocks of every query head of the group. Warps: 0 = TMA producer, 1 = issuer of the score products and owner
// of TMEM, 2 = issuer of the gradient products, 3 = idle, then one (head_dim 128) or two (64) compute groups of eight
// warps, then four dQ drain warps.
//
// What bounds it: a block's chain, by the clock stamps at head_dim 64 (B16 T1024 H12): 240 cycles to read the scores, 1320
// for the exponentials and the stores, 140 to the gradient issuer, 1980 until dQ^T is complete behind the products queued
// before it. It is several times the tensor core's own time (about 55 cycles for each of 24 or 32 products, which read 2 to 4
// KB of A and B from shared memory each), so blocks have to overlap: one every 1790 cycles, at 52 % of the issue slots, 35 %
// of the tensor pipe and 39 % of the shared-memory pipe. At head_dim 128 (B2 T4096 H32:8: 190, 1120, 150, 790, one every 2390) the L2's
// rate of fp32 reductions costs another sixth (785 -> 655 us without them).
//   * 64 queries to a block, because two 128-query blocks do not fit (at head_dim 128 one block of 128 left a single
//     Q / dO stage, and every block waited out a TMA round trip). Three blocks are in flight at head_dim 64, where two
//     compute groups take them in turn (two blocks and one group: 160 us against 151; sixteen warps on one block: 170);
//     tensor memory holds two at head_dim 128, where a second group only lengthens the chain (883 us against 765).
//   * P^T and dS^T are written back over their scores in tensor memory and are the A operands of dV and dK from there;
//     dS^T goes to shared memory as well, as the B operand of dQ^T.
//   * dQ is computed transposed (dQ^T = K^T dS^T, 128 lanes = head_dim, 64 columns = queries) into the columns of the
//     dP^T it came from. At head_dim 64 the upper 64 lanes read the V tile that lies behind K and are ignored. A drain
//     warp owns 32 of head_dim and writes rows of 32 contiguous values, conflict free, for a TMA reduce-add (one
//     red.global per value instead: 2.5 times slower).
//   * items are dealt in a snake over CTAs, longest first; at head_dim 64 K and V are double-buffered, so that the
//     next item's scores run under the last block of this one.
// Measured with the delta kernel, 128-query blocks before -> now, us: B16 T1024 H12 D64 causal 221 -> 151, B4 T4096 H16
// D64 causal 733 -> 545, B2 T4096 H32:8 D128 causal 1224 -> 765, B6 T1777 H16 D128 full 788 -> 538, B2 T777 H8:2 D128
// causal 147 -> 73.
// TMEM columns: buffer b at 128 b: S^T / (P^T, dS^T) 64 | dP^T / dQ^T 64; dV and dK behind the last buffer.
template <int kWarps>
struct BwdCtl {
  float neg_lse[kWarps][32], neg_delta[kWarps][32];   // one row per compute warp: the 32 query columns it works on
  uint64_t kv_full[2], kv_empty[2], qdo_full[4], qdo_empty[4];
  uint64_t s_full[3], pds_full[3], dq_full[3], dq_read[3], ds_free[3], acc_full, acc_empty;
  uint32_t tmem_slot;
  int abort_flag;
};

__device__ __forceinline__ void bulk_wait_group_read1() {
  asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
}
// 16 consecutive 32-bit columns of this thread's lane
__device__ __forceinline__ void tmem_st_cols(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      :
      : "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}

__device__ __forceinline__ void tmem_st_cols(uint32_t taddr, const uint32_t (&r)[32]) { tmem_st_32x32(taddr, r); }
__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t (&r)[32]) { tmem_ld_32x32(taddr, r); }

template <int D>
struct BwdCfg {
  static constexpr int kBufs = (D == 64) ? 3 : 2;     // S^T / dP^T buffers (128 TMEM columns each) and dS^T tiles
  static constexpr int kGroups = (D == 64) ? 2 : 1;   // compute groups of 8 warps; they take the blocks in turn
  static constexpr int kCols = (D == 64) ? 16 : 32;   // query columns a thread holds at a time (80 / 128 registers)
  static constexpr int kThreads = (8 + 8 * kGroups) * 32;
};

// kPlain: the scale is positive and no timeline is recorded, as nearly always; what the other form needs costs registers
// that head_dim 64 does not have to spare. Its timeline: slot 0 start, 1 SM, 2 set up, 3 K / V landed (score issuer),
// 4 first dK / dV complete, 5 first compute warp done, 6 end, 7 blocks of the first item; block g of the CTA's sequence,
// g < 9: 8 + 6 g + 0 scores seen, 1 read from TMEM, 2 P^T and dS^T stored (first warp of the block's
// compute group), 3 dQ^T seen, 4 its reduce-add issued (drain warp), 5 P^T and dS^T seen by the gradient issuer.
template <int D, bool kPlain>
__global__ void __launch_bounds__(BwdCfg<D>::kThreads, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                const __grid_constant__ CUtensorMap tmdQ, const AttnParams p) {
  constexpr int NP = D / 64;
  constexpr int kTile = NP * kPanelBytes;      // 128 key rows
  constexpr int kQPanel = 64 * 128;            // 64 query rows x 64 bf16
  constexpr int kQTile = NP * kQPanel;         // 64 query rows
  constexpr int kStages = (D == 64) ? 4 : 3;   // Q / dO blocks in flight
  constexpr int kKV = (D == 64) ? 2 : 1;       // K / V tiles
  constexpr int kDrain = D / 32;               // active drain warps
  constexpr int kDsBytes = 128 * 128;          // 128 keys x 64 queries
  constexpr int kDqBytes = 32 * 32 * 4;        // 32 queries x 32 of head_dim
  constexpr int kBufs = BwdCfg<D>::kBufs, kGroups = BwdCfg<D>::kGroups, kCols = BwdCfg<D>::kCols;
  constexpr uint32_t kTmemCols = 512, kColV = 128 * kBufs, kColK = kColV + D;

  extern __shared__ uint8_t smem_raw[];
  // (offset arithmetic on the __shared__ symbol, not an integer round trip, so that the compiler
  // keeps the shared address space and emits shared rather than generic loads and stores)
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t* sKV = smem;                          // kKV x (K | V)
  uint8_t* sQO = sKV + kKV * 2 * kTile;         // kStages x (Q | dO)
  uint8_t* sdS = sQO + kStages * 2 * kQTile;    // kBufs x dS^T
  uint8_t* sDQ = sdS + kBufs * kDsBytes;            // 4 warps x 2
  typedef BwdCtl<8 * kGroups> Ctl;
  Ctl& ctl = *reinterpret_cast<Ctl*>(sDQ + 8 * kDqBytes);
  {
    uint32_t dyn_bytes;
    asm volatile("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn_bytes));
    const uint32_t need = (uint32_t)(reinterpret_cast<uint8_t*>(&ctl) - smem_raw) + sizeof(Ctl);
    if (need > dyn_bytes) {  // uniform over the CTA: nothing allocated yet, just leave
      if (threadIdx.x == 0) report(p.status, kBadArgument, (int)need);
      return;
    }
  }
  int& abort_flag = ctl.abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_heads_b = p.Hkv * p.B;
  const int group = p.Hq / p.Hkv;
  const int num_qb = (p.T + 63) / 64;
  const int n_items = ((p.T + 127) / 128) * n_heads_b;
  const int G = (int)gridDim.x, cta = (int)blockIdx.x;
  const int rounds = (n_items + G - 1) / G;
  // item of round k, or -1 (only in the last round). Items are ordered by work: with a causal mask key block 0 meets
  // every query block and the last key block only its own.
  auto item_at = [&](int k) -> int {
    const int w = k * G + ((k & 1) ? G - 1 - cta : cta);
    return (k < rounds && w < n_items) ? w : -1;
  };
  auto first_block = [&](int w) -> int { return p.causal ? 2 * (w / n_heads_b) : 0; };

  // slots past the last recorded block fall off the end of the CTA's row
  auto stamp = [&](int slot) {
    if constexpr (!kPlain) trace_stamp(p.trace, cta, slot);
  };
  auto stamp_block = [&](uint32_t g, int what) {
    if constexpr (!kPlain) trace_stamp(p.trace, cta, g < 9u ? 8 + 6 * (int)g + what : kTraceSlots);
  };
  if (threadIdx.x == 0) {
    stamp(0);
    if (!kPlain && p.trace != nullptr) {
      uint32_t smid;
      asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
      p.trace[(long long)cta * kTraceSlots + 1] = smid;
      p.trace[(long long)cta * kTraceSlots + 7] = (num_qb - first_block(item_at(0))) * group;
    }
    mbar_init(&ctl.acc_full, 1);
    mbar_init(&ctl.acc_empty, kBufs == 3 ? 4 : 8 * kGroups);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&ctl.kv_full[s], 1);
      mbar_init(&ctl.kv_empty[s], 1);
    }
    for (int s = 0; s < 3; ++s) {
      mbar_init(&ctl.s_full[s], 1);
      mbar_init(&ctl.pds_full[s], 8);
      mbar_init(&ctl.dq_full[s], 1);
      mbar_init(&ctl.dq_read[s], kDrain);
      mbar_init(&ctl.ds_free[s], 1);
    }
    for (int s = 0; s < 4; ++s) {
      mbar_init(&ctl.qdo_full[s], 1);
      mbar_init(&ctl.qdo_empty[s], 1);
    }
    abort_flag = 0;
    mbar_fence_init();
    prefetch_tmap(&tmQ);
    prefetch_tmap(&tmK);
    prefetch_tmap(&tmV);
    prefetch_tmap(&tmdO);
    prefetch_tmap(&tmdQ);
  }
  if (warp == 1) {
    tmem_alloc(&ctl.tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  constexpr uint32_t tmem_base = 0;   // an allocation of all 512 columns starts at column 0
  pdl_wait();  // the set-up above read no tensor of the step
  pdl_trigger();
  if (threadIdx.x == 0) stamp(2);

  // dV / dK of item n: 32 key rows (one per lane), 32-column chunks [c0, c1) of head_dim. With one accumulator the
  // compute warps do this; with two the drain warps do, while the compute warps are already at the next item.
  // `st`: 2 KB of the calling warp's own, through which rows leave four lanes to 64 bytes; nullptr: a lane stores its
  // own row.
  auto store_grads = [&](int quad, int c0, int c1, uint32_t n, int jb, int hkv, int b, uint8_t* st) -> bool {
    if (!mbar_wait_warp(&ctl.acc_full, n & 1, &abort_flag, p.status, kTimeoutTmemFull, 700)) return false;
    tc_fence_after();
    if (n == 0 && quad == 0 && c0 == 0 && lane == 0) stamp(4);
    const int row0 = jb * 128 + quad * 32;
    const uint32_t colV = ((uint32_t)(quad * 32) << 16) + kColV;
    __nv_bfloat16* dk = p.dK + ((long long)b * p.T + row0) * p.ld_dk + p.dk_col0 + hkv * D;
    __nv_bfloat16* dv = p.dV + ((long long)b * p.T + row0) * p.ld_dv + p.dv_col0 + hkv * D;
#pragma unroll 1
    for (int cc = 2 * c0; cc < 2 * c1; ++cc) {   // dV chunk, dK chunk, ...
      const bool is_k = cc & 1;
      const int c = (cc >> 1) * 32;
      uint32_t r[32];
      tmem_ld_32x32(colV + (is_k ? D : 0) + c, r);
      tmem_ld_wait();
      if (cc + 1 == 2 * c1) {   // in registers: the accumulator may be overwritten
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&ctl.acc_empty);
      }
      const float f = is_k ? p.scale : 1.f;
      __nv_bfloat16* dst = (is_k ? dk : dv) + c;
      const long long ld = is_k ? p.ld_dk : p.ld_dv;
      uint4 q[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        q[i].x = pack_bf16x2(__uint_as_float(r[8 * i + 0]) * f, __uint_as_float(r[8 * i + 1]) * f);
        q[i].y = pack_bf16x2(__uint_as_float(r[8 * i + 2]) * f, __uint_as_float(r[8 * i + 3]) * f);
        q[i].z = pack_bf16x2(__uint_as_float(r[8 * i + 4]) * f, __uint_as_float(r[8 * i + 5]) * f);
        q[i].w = pack_bf16x2(__uint_as_float(r[8 * i + 6]) * f, __uint_as_float(r[8 * i + 7]) * f);
      }
      if (st != nullptr) {
        // 16-byte pieces of a 64-byte row are XORed with bits 1-2 of the row: conflict free both ways
#pragma unroll
        for (int i = 0; i < 4; ++i) *reinterpret_cast<uint4*>(st + lane * 64 + ((i ^ ((lane >> 1) & 3)) << 4)) = q[i];
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int rr = 8 * i + (lane >> 2);
          const uint4 v = *reinterpret_cast<const uint4*>(st + rr * 64 + (((lane & 3) ^ ((rr >> 1) & 3)) << 4));
          if (row0 + rr < p.T) reinterpret_cast<uint4*>(dst + rr * ld)[lane & 3] = v;
        }
        __syncwarp();
      } else if (row0 + lane < p.T) {
#pragma unroll
        for (int i = 0; i < 4; ++i) reinterpret_cast<uint4*>(dst + lane * ld)[i] = q[i];
      }
    }
    return true;
  };

  if (warp == 0) {
    // ======================= TMA producer =======================
    if (lane == 0) {
      uint32_t g = 0, n = 0;
      bool ok = true;
      for (int k = 0; k < rounds && ok; ++k) {
        const int w = item_at(k);
        if (w < 0) break;
        const int jb = w / n_heads_b, hb = w - jb * n_heads_b;
        const int hkv = hb % p.Hkv, b = hb / p.Hkv;
        const int i0 = first_block(w);
        bool kv_loaded = false;
        for (int hq = hkv * group; hq < (hkv + 1) * group && ok; ++hq) {
          for (int qi = i0; qi < num_qb; ++qi, ++g) {
            const uint32_t s = g % kStages;
            if (!mbar_wait(&ctl.qdo_empty[s], ((g / kStages) & 1) ^ 1, &abort_flag, p.status, kTimeoutEmpty, (int)g)) { ok = false; break; }
            mbar_expect_tx(&ctl.qdo_full[s], 2 * kQTile);
            uint8_t* st = sQO + s * 2 * kQTile;
#pragma unroll
            for (int pn = 0; pn < NP; ++pn) {
              tma_load_3d(st + pn * kQPanel, &tmQ, &ctl.qdo_full[s], p.q_col0 + hq * D + pn * 64, qi * 64, b);
              tma_load_3d(st + kQTile + pn * kQPanel, &tmdO, &ctl.qdo_full[s], p.o_col0 + hq * D + pn * 64, qi * 64, b);
            }
            if (!kv_loaded) {   // behind the item's first block: its stage is free before the K / V tile is
              const uint32_t kb = n % kKV;
              if (!mbar_wait(&ctl.kv_empty[kb], ((n / kKV) & 1) ^ 1, &abort_flag, p.status, kTimeoutEmpty, 1000)) { ok = false; break; }
              mbar_expect_tx(&ctl.kv_full[kb], 2 * kTile);
              uint8_t* kv = sKV + kb * 2 * kTile;
#pragma unroll
              for (int pn = 0; pn < NP; ++pn) {
                tma_load_3d(kv + pn * kPanelBytes, &tmK, &ctl.kv_full[kb], p.k_col0 + hkv * D + pn * 64, jb * 128, b);
                tma_load_3d(kv + kTile + pn * kPanelBytes, &tmV, &ctl.kv_full[kb], p.v_col0 + hkv * D + pn * 64, jb * 128, b);
              }
              kv_loaded = true;
            }
          }
        }
        ++n;
      }
    }
  } else if (warp == 1) {
    // ======================= scores: S^T = K Q^T and dP^T = V dO^T =======================
    // (both issuing warps stay converged and elect a lane; see the GEMM kernels)
    const uint32_t idesc_st = make_idesc_bf16(128, 64, 0, 0);   // K / V (K-major) x Q / dO (K-major)
    const uint32_t lo_k = smem_desc_lo(smem_u32(sKV), 16), lo_q = smem_desc_lo(smem_u32(sQO), 16);
    uint32_t g = 0, n = 0, s = 0, ph = 0, bf = 0, bph = 0;
    bool ok = true;
    for (int k = 0; k < rounds && ok; ++k) {
      const int w = item_at(k);
      if (w < 0) break;
      const uint32_t kb = n % kKV;
      const int n_iter = (num_qb - first_block(w)) * group;
      if (!mbar_wait_warp(&ctl.kv_full[kb], (n / kKV) & 1, &abort_flag, p.status, kTimeoutFull, 1001)) break;
      if (n == 0 && lane == 0) stamp(3);
      ++n;
      const uint32_t ak = lo_k + kb * (2 * kTile >> 4);
      for (int it = 0; it < n_iter; ++it, ++g) {
        if (!mbar_wait_warp(&ctl.qdo_full[s], ph, &abort_flag, p.status, kTimeoutFull, (int)g)) { ok = false; break; }
        // the buffer's columns were last P^T and dQ^T of kBufs blocks ago: dQ^T is drained and the products are done
        if (!mbar_wait_warp(&ctl.dq_read[bf], bph ^ 1, &abort_flag, p.status, kTimeoutFlag, 200) ||
            !mbar_wait_warp(&ctl.ds_free[bf], bph ^ 1, &abort_flag, p.status, kTimeoutFlag, 201)) { ok = false; break; }
        tc_fence_after();
        const uint32_t bq = lo_q + s * (2 * kQTile >> 4), d = bf * 128;
        if (elect_one()) {
#pragma unroll
          for (int j = 0; j < D / 16; ++j)
            umma_bf16_ss(d, smem_desc(ak + ((j >> 2) * kPanelBytes + (j & 3) * 32) / 16),
                         smem_desc(bq + ((j >> 2) * kQPanel + (j & 3) * 32) / 16), idesc_st, j > 0 ? 1u : 0u);
#pragma unroll
          for (int j = 0; j < D / 16; ++j)
            umma_bf16_ss(d + 64, smem_desc(ak + (kTile + (j >> 2) * kPanelBytes + (j & 3) * 32) / 16),
                         smem_desc(bq + (kQTile + (j >> 2) * kQPanel + (j & 3) * 32) / 16), idesc_st, j > 0 ? 1u : 0u);
          umma_commit(&ctl.s_full[bf]);
        }
        __syncwarp();
        if (++s == kStages) { s = 0; ph ^= 1; }
        if (++bf == kBufs) { bf = 0; bph ^= 1; }
      }
    }
  } else if (warp == 2) {
    // ======================= gradients: dV += P^T dO, dK += dS^T Q, dQ^T = K^T dS^T =======================
    const uint32_t idesc_dkv = make_idesc_bf16(128, D, 0, 1);   // P^T (TMEM) / dS^T (K-major) x dO / Q (MN)
    const uint32_t idesc_dq = make_idesc_bf16(128, 64, 1, 1);   // K as MN-major A x dS^T (MN)
    const uint32_t lo_kmn = smem_desc_lo(smem_u32(sKV), kPanelBytes), lo_qmn = smem_desc_lo(smem_u32(sQO), kQPanel);
    const uint32_t lo_dsmn = smem_desc_lo(smem_u32(sdS), kDsBytes);
    uint32_t g = 0, n = 0, s = 0, ph = 0, bf = 0, bph = 0;
    bool ok = true;
    for (int k = 0; k < rounds && ok; ++k) {
      const int w = item_at(k);
      if (w < 0) break;
      const uint32_t kb = n % kKV;
      const int n_iter = (num_qb - first_block(w)) * group;
      if (!mbar_wait_warp(&ctl.kv_full[kb], (n / kKV) & 1, &abort_flag, p.status, kTimeoutFull, 1002)) break;
      if (!mbar_wait_warp(&ctl.acc_empty, (n & 1) ^ 1, &abort_flag, p.status, kTimeoutTmemEmpty, 1003)) break;
      ++n;
      const uint32_t ak = lo_kmn + kb * (2 * kTile >> 4);
      for (int it = 0; it < n_iter; ++it, ++g) {
        if (!mbar_wait_warp(&ctl.qdo_full[s], ph, &abort_flag, p.status, kTimeoutFull, (int)g) ||
            !mbar_wait_warp(&ctl.pds_full[bf], bph, &abort_flag, p.status, kTimeoutFlag, (int)g)) { ok = false; break; }
        tc_fence_after();
        if (lane == 0) stamp_block(g, 5);
        const uint32_t bq = lo_qmn + s * (2 * kQTile >> 4);
        const uint32_t bds = lo_dsmn + bf * (kDsBytes >> 4);
        const uint32_t acc = it > 0 ? 1u : 0u;
        // kCols columns of TMEM hold P^T and dS^T of kCols queries, half of them each, as bf16 pairs
        auto pcol = [](int j) -> uint32_t { return (uint32_t)(kCols == 16 ? j * 16 : (j >> 1) * 32 + (j & 1) * 8); };
        if (elect_one()) {
          // dQ^T first: its drain is what the scores of two blocks on wait for. Contraction over the 128 key rows.
#pragma unroll
          for (int j = 0; j < 8; ++j)
            umma_bf16_ss(bf * 128 + 64, smem_desc(ak + j * 128), smem_desc(bds + j * 128), idesc_dq, j > 0 ? 1u : 0u);
          umma_commit(&ctl.dq_full[bf]);
          // contraction over the 64 query rows
#pragma unroll
          for (int j = 0; j < 4; ++j)
            umma_bf16_ts(kColV, bf * 128 + pcol(j), smem_desc(bq + (kQTile + j * 2048) / 16),
                         idesc_dkv, j > 0 ? 1u : acc);
#pragma unroll
          for (int j = 0; j < 4; ++j)
            umma_bf16_ts(kColK, bf * 128 + pcol(j) + kCols / 2, smem_desc(bq + j * 128), idesc_dkv,
                         j > 0 ? 1u : acc);
          umma_commit(&ctl.qdo_empty[s]);
          umma_commit(&ctl.ds_free[bf]);   // P^T and dS^T of this buffer have been read
          if (it + 1 == n_iter) {
            umma_commit(&ctl.kv_empty[kb]);
            umma_commit(&ctl.acc_full);
          }
        }
        __syncwarp();
        if (++s == kStages) { s = 0; ph ^= 1; }
        if (++bf == kBufs) { bf = 0; bph ^= 1; }
      }
    }
  } else if (warp >= 4 && warp < 4 + 8 * kGroups) {
    // ---------------- compute warps: group 0 takes the even blocks, group 1 the odd ones --------
    // (a block's chain of waits, TMEM reads and stores takes a group about 1900 cycles with two thirds of its issue
    // slots empty: sixteen warps on one block gained nothing, two groups on two blocks overlap)
    const int grp = (warp - 4) >> 3;
    const int quad = warp & 3, chalf = ((warp - 4) >> 2) & 1;
    const int row = quad * 32 + lane;
    const uint32_t t_lane = (uint32_t)(quad * 32) << 16;
    const float l2e = 1.4426950408889634f;
    const f32x2 c2 = kPlain ? f2_pack(p.scale * l2e, p.scale * l2e) : f2_pack(p.scale_log2, p.scale_log2);
    float* my_lse = ctl.neg_lse[warp - 4];
    float* my_delta = ctl.neg_delta[warp - 4];
    // position in the CTA's sequence of blocks
    struct Pos {
      int k, w, b, hkv, hq, qi, i0;
    };
    auto enter = [&](Pos& q, int k) {
      q.k = k;
      q.w = item_at(k);
      if (q.w >= 0) {
        const int hb = q.w % n_heads_b;
        q.hkv = hb % p.Hkv;
        q.b = hb / p.Hkv;
        q.hq = q.hkv * group;
        q.i0 = q.qi = first_block(q.w);
      }
    };
    auto advance = [&](Pos& q) {
      if (q.w < 0) return;
      if (++q.qi < num_qb) return;
      q.qi = q.i0;
      if (++q.hq < (q.hkv + 1) * group) return;
      enter(q, q.k + 1);
    };
    // lse / delta of the warp's 32 columns, one (own) block ahead; queries past the end get lse = +inf, i.e. P = 0
    // (raw values: arithmetic on them would wait for the loads here, a block early)
    float st_l = 0.f, st_d = 0.f;
    auto stat_load = [&](const Pos& z) {
      st_l = INFINITY;
      st_d = 0.f;
      const int q = z.qi * 64 + chalf * 32 + lane;
      if (z.w >= 0 && q < p.T) {
        const long long off = ((long long)z.b * p.Hq + z.hq) * p.T + q;
        st_l = p.lse[off];
        st_d = p.delta[off];
      }
    };
    Pos cur, ahead;
    enter(cur, 0);
    if (grp == 1) advance(cur);
    ahead = cur;
    stat_load(ahead);
    uint32_t bf = grp, bph = 0;   // the block's buffer and its phase
    int stored = 0;   // items whose dV / dK this warp has stored (head_dim 128)
    const bool tracer = !kPlain && ((warp - 4) & 7) == 0 && lane == 0;
    uint32_t blk = grp;   // position in the CTA's sequence (timeline)
    bool ok = true;
    while (true) {
      if (kBufs == 2) {
        // items that lie behind: all MMAs into dV / dK have completed once acc_full fires
        while (ok && item_at(stored) >= 0 && stored < cur.k) {
          const int w = item_at(stored), hb = w % n_heads_b;
          ok = store_grads(quad, chalf * (D / 64), (chalf + 1) * (D / 64), (uint32_t)stored, w / n_heads_b, hb % p.Hkv, hb / p.Hkv, nullptr);
          ++stored;
        }
      }
      if (!ok || cur.w < 0) break;
      const int kv_idx = cur.w / n_heads_b * 128 + row;
      __syncwarp();   // every lane has read the previous block's values
      my_lse[lane] = -st_l * l2e;
      my_delta[lane] = -st_d;
      __syncwarp();
#pragma unroll
      for (int i = 0; i < kGroups; ++i) advance(ahead);
      stat_load(ahead);
      if (!mbar_wait_warp(&ctl.s_full[bf], bph, &abort_flag, p.status, kTimeoutTmemFull, (int)bf)) break;
      tc_fence_after();
      if (tracer) stamp_block(blk, 0);
      // (the scores waited for the products that last read this buffer, its dS^T tile among them)
      uint8_t* rowp = sdS + bf * kDsBytes + row * 128;
#pragma unroll
      for (int sub = 0; sub < 32 / kCols; ++sub) {
        const uint32_t col = bf * 128 + chalf * 32 + sub * kCols;
        uint32_t rs[kCols], rp[kCols];
        tmem_ld_cols(t_lane + col, rs);
        tmem_ld_cols(t_lane + col + 64, rp);
        tmem_ld_wait();
        if (tracer && sub == 0) stamp_block(blk, 1);
        // Queries below the key row (causal) and key rows past the end have P = 0: their scaled scores become -inf. (A
        // second, masked copy of the block below ran twice an item, each time from a cold instruction cache, and took
        // 2000 cycles longer than the plain one.)
        const int lim = p.causal ? kv_idx - (cur.qi * 64 + chalf * 32 + sub * kCols) : 0;   // columns below it are dead
        const bool past = kv_idx >= p.T;
        if (__any_sync(0xffffffffu, (lim > 0) | past)) {
          const uint32_t live = (past || lim >= kCols) ? 0u : lim <= 0 ? 0xffffffffu : 0xffffffffu << lim;
#pragma unroll
          for (int i = 0; i < kCols; ++i) rs[i] = (live & (1u << i)) ? rs[i] : kPlain ? 0xff800000u : p.dead_score;
        }
        uint32_t pw[kCols];   // P^T as bf16 pairs, then dS^T
#pragma unroll
        for (int i4 = 0; i4 < kCols / 4; ++i4) {
          const ulonglong2 l4 = *reinterpret_cast<const ulonglong2*>(&my_lse[sub * kCols + 4 * i4]);
          const ulonglong2 d4 = *reinterpret_cast<const ulonglong2*>(&my_delta[sub * kCols + 4 * i4]);
          float e[4], ds[4];
#pragma unroll
          for (int v = 0; v < 2; ++v) {
            const int i = 4 * i4 + 2 * v;
            f2_unpack(f2_fma(f2_pack(__uint_as_float(rs[i]), __uint_as_float(rs[i + 1])), c2, v ? l4.y : l4.x), e[2 * v],
                      e[2 * v + 1]);
            e[2 * v] = exp2f(e[2 * v]);
            e[2 * v + 1] = exp2f(e[2 * v + 1]);
            const f32x2 t = f2_add(f2_pack(__uint_as_float(rp[i]), __uint_as_float(rp[i + 1])), v ? d4.y : d4.x);
            f2_unpack(f2_mul(f2_pack(e[2 * v], e[2 * v + 1]), t), ds[2 * v], ds[2 * v + 1]);
          }
          pw[2 * i4] = pack_bf16x2(e[0], e[1]);
          pw[2 * i4 + 1] = pack_bf16x2(e[2], e[3]);
          pw[kCols / 2 + 2 * i4] = pack_bf16x2(ds[0], ds[1]);
          pw[kCols / 2 + 2 * i4 + 1] = pack_bf16x2(ds[2], ds[3]);
          if (i4 & 1)   // eight columns of dS^T
            *reinterpret_cast<uint4*>(rowp + (((chalf * 4 + sub * (kCols / 8) + (i4 >> 1)) ^ (row & 7)) << 4)) =
                make_uint4(pw[kCols / 2 + 2 * i4 - 2], pw[kCols / 2 + 2 * i4 - 1], pw[kCols / 2 + 2 * i4],
                           pw[kCols / 2 + 2 * i4 + 1]);
        }
        tmem_st_cols(t_lane + col, pw);
      }
      fence_proxy_async_smem();
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl.pds_full[bf]);
      if (tracer) stamp_block(blk, 2);
      blk += kGroups;
#pragma unroll
      for (int i = 0; i < kGroups; ++i) {
        advance(cur);
        if (++bf == kBufs) { bf = 0; bph ^= 1; }
      }
    }
    if (tracer && grp == 0) stamp(5);
  } else if (warp >= 4 + 8 * kGroups) {
    // ---------------- dQ drain warps: 32 values of head_dim (one per lane), 64 queries --------
    const int quad = warp & 3;
    const uint32_t t_lane = tmem_base + ((uint32_t)(quad * 32) << 16);
    float* stg = reinterpret_cast<float*>(sDQ + quad * 2 * kDqBytes);
    uint32_t n = 0, bf = 0, bph = 0, blk = 0;
    bool ok = true;
    for (int k = 0; k < rounds && ok; ++k) {
      const int w = item_at(k);
      if (w < 0) break;
      const int jb = w / n_heads_b, hb = w - jb * n_heads_b;
      const int hkv = hb % p.Hkv, b = hb / p.Hkv;
      const int i0 = first_block(w);
      for (int hq = hkv * group; quad < kDrain && hq < (hkv + 1) * group && ok; ++hq) {
        for (int qi = i0; qi < num_qb; ++qi) {
          if (!mbar_wait_warp(&ctl.dq_full[bf], bph, &abort_flag, p.status, kTimeoutTmemFull, 100)) { ok = false; break; }
          tc_fence_after();
          if (quad == 0 && lane == 0) stamp_block(blk, 3);
          // 64 queries at once where registers allow it, so that the columns are handed back early
          constexpr int kAtOnce = (kGroups == 1) ? 2 : 1;
          uint32_t r[kAtOnce][32];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if (h % kAtOnce == 0) {
#pragma unroll
              for (int i = 0; i < kAtOnce; ++i) tmem_ld_32x32(t_lane + bf * 128 + 64 + (h + i) * 32, r[i]);
              tmem_ld_wait();
              if (h + kAtOnce == 2) {   // dQ^T is in registers: its columns are free
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&ctl.dq_read[bf]);
              }
            }
            if (lane == 0) bulk_wait_group_read1();   // at most the other half's reduction still reads its tile
            __syncwarp();
            float* t = stg + h * (kDqBytes / 4);
#pragma unroll
            for (int q = 0; q < 32; ++q) t[q * 32 + lane] = __uint_as_float(r[h % kAtOnce][q]) * p.scale;
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              // queries past T are clipped by the tensor map (3-D: columns, rows of one batch, batch)
              if (qi * 64 + h * 32 < p.T)
                tma_reduce_add_3d(&tmdQ, t, p.dq_col0 + hq * D + quad * 32, qi * 64 + h * 32, b);
              bulk_commit_group();
            }
          }
          if (quad == 0 && lane == 0) stamp_block(blk, 4);
          ++blk;
          if (++bf == kBufs) { bf = 0; bph ^= 1; }
        }
      }
      if (kBufs == 3 && ok) {
        if (lane == 0) bulk_wait_group_read0();   // the staging tiles are free
        __syncwarp();
        ok = store_grads(quad, 0, D / 32, n++, jb, hkv, b, sDQ + quad * 2 * kDqBytes);
      }
    }
    if (lane == 0) bulk_wait_group0();  // reductions in flight finish before the CTA retires
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tmem_dealloc(tmem_base, kTmemCols);
  }
  if (threadIdx.x == 0) stamp(6);
}

static long long* g_attn_trace = nullptr;
static long long g_attn_trace_ctas = 0;

// ---------------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

void ensure_context();  // gemm_sm100.cu

static EncodeTiledFn attn_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (fn == nullptr) {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &qres) ==
            cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(f);
  }
  return fn;
}

// [B, T, cols] bf16 view with row stride ld: dims {cols, T, B}, box {64, 128, 1}.
static int make_tmap_btc(CUtensorMap* out, const void* base, int B, int T, long long cols,
                         long long ld, int box_rows = 128) {
  EncodeTiledFn fn = attn_encode_fn();
  if (fn == nullptr) return -1;
  ensure_context();
  if (ld % 8 || ((uintptr_t)base & 15)) return -2;
  cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)T, (cuuint64_t)B};
  cuuint64_t strides[2] = {(cuuint64_t)ld * 2, (cuuint64_t)ld * 2 * (cuuint64_t)T};
  cuuint32_t box[3] = {64, (cuuint32_t)box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides,
                  box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return (r == CUDA_SUCCESS) ? 0 : (int)r;
}

// fp32 accumulator [B*T, ld] viewed as [B][T][ld]; boxes of 32 columns x 32 rows
static int make_tmap_f32_btc(CUtensorMap* out, const void* base, int B, int T, long long ld) {
  EncodeTiledFn fn = attn_encode_fn();
  if (fn == nullptr) return -1;
  ensure_context();
  if (ld % 4 || ((uintptr_t)base & 15)) return -2;
  cuuint64_t dims[3] = {(cuuint64_t)ld, (cuuint64_t)T, (cuuint64_t)B};
  cuuint64_t strides[2] = {(cuuint64_t)ld * 4, (cuuint64_t)ld * 4 * (cuuint64_t)T};
  cuuint32_t box[3] = {32, 32, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<void*>(base), dims, strides,
                  box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return (r == CUDA_SUCCESS) ? 0 : (int)r;
}

}  // namespace mmj

using namespace mmj;

// q/k/v: [B*T, ld*] bf16 matrices in which head h of Q starts at column q_col0 + h*D (same for
// K/V with Hkv heads). O: [B*T, ldo] with head h at o_col0 + h*D. lse: [B, Hq, T] fp32.
MMJ_API int mmj_attn_fwd(const void* q, long long ldq, int q_col0, const void* k, long long ldk,
                         int k_col0, const void* v, long long ldv, int v_col0, void* O,
                         long long ldo, int o_col0, float* lse, int B, int T, int Hq, int Hkv,
                         int D, float scale, int causal, int* status, void* stream) {
  if (D != 64 && D != 128) return -10;
  if (Hkv <= 0 || Hq % Hkv) return -11;
  if (ldo % 8 || o_col0 % 8) return -12;
  CUtensorMap tq, tk, tv;
  int rc;
  if ((rc = make_tmap_btc(&tq, q, B, T, ldq, ldq))) return rc;
  if ((rc = make_tmap_btc(&tk, k, B, T, ldk, ldk))) return rc;
  if ((rc = make_tmap_btc(&tv, v, B, T, ldv, ldv))) return rc;
  AttnParams p = {};
  p.B = B; p.T = T; p.Hq = Hq; p.Hkv = Hkv;
  p.q_col0 = q_col0; p.k_col0 = k_col0; p.v_col0 = v_col0;
  p.scale = scale; p.causal = causal;
  p.O = (__nv_bfloat16*)O; p.ldo = ldo; p.o_col0 = o_col0;
  p.lse = lse;
  p.status = status;
  // Default (3): persistent kernel, two query tiles per CTA, 64-key blocks with double-buffered score
  // tiles. MOMIJO_ATTN_FWD=1 selects the older one-tile-per-CTA kernel (kept for comparison).
  static int fwd_mode = -1;
  if (fwd_mode < 0) {
    const char* e = getenv("MOMIJO_ATTN_FWD");
    fwd_mode = e ? atoi(e) : 3;
  }
  if (fwd_mode == 3) {
    static bool b64 = false, b128 = false;
    static int sms3 = 0;
    if (sms3 == 0) {
      int dev = 0;
      cudaGetDevice(&dev);
      cudaDeviceGetAttribute(&sms3, cudaDevAttrMultiProcessorCount, dev);
    }
    CUtensorMap tk64, tv64;
    if ((rc = make_tmap_btc(&tk64, k, B, T, ldk, ldk, 64))) return rc;
    if ((rc = make_tmap_btc(&tv64, v, B, T, ldv, ldv, 64))) return rc;
    const long long n_items = (long long)((T + 255) / 256) * Hq * B;
    const unsigned g = (unsigned)(n_items < sms3 ? n_items : sms3);
    p.trace = (g_attn_trace && (long long)g <= g_attn_trace_ctas) ? g_attn_trace : nullptr;
    if (D == 64) {
      const int smem = 2 * kPanelBytes + 2 * 6 * 8192 + 1024;
      if (!b64) {
        cudaFuncSetAttribute(attn_fwd3_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        b64 = true;
      }
      launch_pdl(attn_fwd3_kernel<64>, dim3(g), dim3(384), (size_t)smem, (cudaStream_t)stream, tq, tk64, tv64,
                 p);
    } else {
      const int smem = 2 * 2 * kPanelBytes + 2 * 4 * 16384 + 1024;
      if (!b128) {
        cudaFuncSetAttribute(attn_fwd3_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        b128 = true;
      }
      launch_pdl(attn_fwd3_kernel<128>, dim3(g), dim3(384), (size_t)smem, (cudaStream_t)stream, tq, tk64, tv64,
                 p);
    }
    return (int)cudaGetLastError();
  }
  dim3 grid((T + 127) / 128, Hq, B);
  p.trace = (g_attn_trace && (long long)grid.x * grid.y * grid.z <= g_attn_trace_ctas) ? g_attn_trace : nullptr;
  static bool attr64 = false, attr128 = false;
  if (D == 64) {
    const int smem = 4 * kPanelBytes + 2 * kPanelBytes + 1024;  // Q + 2 K + 1 V + P
    if (!attr64) {
      cudaFuncSetAttribute(attn_fwd_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
      attr64 = true;
    }
    attn_fwd_kernel<64><<<grid, kAttnThreads, smem, (cudaStream_t)stream>>>(tq, tk, tv, p);
  } else {
    const int smem = 5 * 2 * kPanelBytes + 2 * 2 * kPanelBytes + 1024;  // Q + 2 K + 2 V + 2 P
    if (!attr128) {
      cudaFuncSetAttribute(attn_fwd_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
      attr128 = true;
    }
    attn_fwd_kernel<128><<<grid, kAttnThreads, smem, (cudaStream_t)stream>>>(tq, tk, tv, p);
  }
  return (int)cudaGetLastError();
}

// Install (or clear, with nullptr) the timeline buffer of the attention kernels: int64
// [ctas * 64], written by whichever of them is launched next. Launches whose grid has more CTAs than `ctas` leave it untouched.
MMJ_API int mmj_attn_set_trace(void* buf, long long ctas) {
  g_attn_trace = reinterpret_cast<long long*>(buf);
  g_attn_trace_ctas = buf ? ctas : 0;
  return 0;
}

// dQ_accum: fp32 [B*T, ld_dq]; its Hq*D columns from dq_col0 are cleared by the delta kernel, then the
// backward kernel adds into them.
// delta: fp32 scratch [B, Hq, T] (filled here). dK/dV: bf16 outputs.
MMJ_API int mmj_attn_bwd(const void* q, long long ldq, int q_col0, const void* k, long long ldk,
                         int k_col0, const void* v, long long ldv, int v_col0, const void* O,
                         long long ldo, int o_col0, const void* dO, long long lddo, int do_col0,
                         const float* lse, float* delta, float* dQ_accum, long long ld_dq,
                         int dq_col0, void* dK, long long ld_dk, int dk_col0, void* dV,
                         long long ld_dv, int dv_col0, int B, int T, int Hq, int Hkv, int D,
                         float scale, int causal, int* status, void* stream) {
  if (D != 64 && D != 128) return -10;
  if (Hkv <= 0 || Hq % Hkv) return -11;
  if (ld_dk % 8 || ld_dv % 8 || dk_col0 % 8 || dv_col0 % 8 || ld_dq % 4 || dq_col0 % 4) return -12;
  CUtensorMap tq, tk, tv, tdo;
  int rc;
  if ((rc = make_tmap_btc(&tq, q, B, T, ldq, ldq, 64))) return rc;
  if ((rc = make_tmap_btc(&tk, k, B, T, ldk, ldk))) return rc;
  if ((rc = make_tmap_btc(&tv, v, B, T, ldv, ldv))) return rc;
  if ((rc = make_tmap_btc(&tdo, dO, B, T, lddo, lddo, 64))) return rc;
  CUtensorMap tdq;
  if (dq_col0 % 4) return -13;
  if ((rc = make_tmap_f32_btc(&tdq, dQ_accum, B, T, ld_dq))) return rc;
  {
    if (((uintptr_t)O & 15) || (ldo & 7) || (o_col0 & 7) || (do_col0 & 7)) return -1;
    const long long lanes = (long long)B * T * Hq * (D / 8);
    const int threads = 256;
    const long long blocks = (lanes + threads - 1) / threads;
    launch_pdl(attn_delta_kernel, dim3((unsigned)blocks), dim3(threads), 0, (cudaStream_t)stream,
               (const __nv_bfloat16*)O, ldo, o_col0, (const __nv_bfloat16*)dO, lddo, do_col0, delta,
               (((uintptr_t)dQ_accum & 15) == 0) ? dQ_accum : (float*)nullptr, ld_dq, dq_col0, B, T, Hq, D);
  }
  AttnParams p = {};
  p.B = B; p.T = T; p.Hq = Hq; p.Hkv = Hkv;
  p.q_col0 = q_col0; p.k_col0 = k_col0; p.v_col0 = v_col0;
  p.o_col0 = do_col0;  // the dO map is addressed with o_col0 inside the kernel
  p.scale = scale; p.causal = causal;
  p.scale_log2 = scale == 0.f ? 1e-30f : scale * 1.4426950408889634f;
  p.dead_score = scale < 0.f ? 0x7f800000u : 0xff800000u;
  p.lse = const_cast<float*>(lse);
  p.delta = delta;
  p.dQ = dQ_accum; p.ld_dq = ld_dq; p.dq_col0 = dq_col0;
  p.dK = (__nv_bfloat16*)dK; p.ld_dk = ld_dk; p.dk_col0 = dk_col0;
  p.dV = (__nv_bfloat16*)dV; p.ld_dv = ld_dv; p.dv_col0 = dv_col0;
  p.status = status;
  const long long n_items = (long long)((T + 127) / 128) * Hkv * B;
  static int sms = 0;
  if (sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  }
  const dim3 grid((unsigned)(n_items < sms ? n_items : sms));
  // head_dim 128: 224 KB of tiles, the control block and the alignment padding take what is left of the 227 KB a CTA
  // may have (the kernel checks that they fit); head_dim 64 needs 208 KB of tiles
  const int smem = 232448;
  p.trace = (g_attn_trace && (long long)grid.x <= g_attn_trace_ctas) ? g_attn_trace : nullptr;
  static bool attr_set[4] = {};
  const bool plain = scale > 0.f && p.trace == nullptr;
  auto* kernel = (D == 64) ? (plain ? &attn_bwd_kernel<64, true> : &attn_bwd_kernel<64, false>)
                           : (plain ? &attn_bwd_kernel<128, true> : &attn_bwd_kernel<128, false>);
  bool& attr = attr_set[(D == 64 ? 0 : 2) + (plain ? 1 : 0)];
  if (!attr) {
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    attr = true;
  }
  launch_pdl(kernel, grid, dim3(D == 64 ? BwdCfg<64>::kThreads : BwdCfg<128>::kThreads), (size_t)smem, (cudaStream_t)stream, tq, tk, tv, tdo, tdq, p);
  return (int)cudaGetLastError();
}
