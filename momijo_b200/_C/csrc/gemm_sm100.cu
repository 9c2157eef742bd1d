// bf16 GEMM on the 5th-generation tensor cores: D[M,N] = op(A) * op(B)^T-style products with
// fp32 accumulation in tensor memory (TMEM), operands staged in shared memory by TMA with a
// 128-byte swizzle, issued by one thread per CTA (tcgen05.mma), persistent over output tiles.
//
// Warp roles inside a 320-thread CTA:
//   warp 0      TMA producer (one lane)
//   warp 1      TMEM allocator + MMA issuer (one lane)
//   warps 2..9  epilogue: tcgen05.ld the accumulator (one output row per thread, two warps per
//               TMEM lane quadrant taking alternate 32-column chunks), apply the fused epilogue
//               (bias / GELU / GELU' / residual / SiLU / scale / accumulate), store bf16 or fp32
// Two accumulators (2 x 256 TMEM columns) let the epilogue of tile i overlap the main loop
// of tile i+1. Tiles are 128 rows tall, or 256 (two MMAs per B stage) for long contractions.
//
// The same kernel also carries the fused communication paths:
//   * gathered operand: extra CTAs pull peer shards over NVLink into local memory and publish
//     per-tile flags that the TMA producer waits on (all-gather -> GEMM);
//   * scattered result: the epilogue stores each row block straight into the memory of the
//     rank that owns it (GEMM -> reduce-scatter, summed by the owner afterwards);
//   * grouped mode for MoE experts (per-tile group table, tile count read from the device).
//
// This replaces the reference's scalar one-thread-per-output kernels
// (legacy/src/momijo/tensor/gpu/runtime.mojo:52-119) and its CPU matmul loops
// (legacy/src/momijo/tensor/broadcast.mojo:1612, legacy/src/momijo/tensor/indexing.mojo:2702).
#include "common.cuh"
#include "gemm_sm100.cuh"

#include <mutex>

namespace mmj {

constexpr int kEpiWarps = 8;
constexpr int kThreads = (2 + kEpiWarps) * 32;  // TMA producer warp, MMA warp, epilogue warps
constexpr int kAStageBytes = kGemmBM * kGemmBK * 2;  // 16 KiB
constexpr int kTmemCols = 512;
constexpr int kAccCols = 256;

__device__ __forceinline__ int ld_acquire_gpu(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_gpu(int* p, int v) {
  asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ int ld_acquire_sys(const int* p) {
  int v;
  asm volatile("ld.acquire.sys.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Bounded wait until *flag >= want. Returns false on timeout / abort.
__device__ __forceinline__ bool wait_flag_ge(const int* flag, int want, bool sys_scope,
                                             volatile int* abort_flag, int* status, int detail) {
  int v = sys_scope ? ld_acquire_sys(flag) : ld_acquire_gpu(flag);
  if (v >= want) return true;
  uint64_t t0 = 0;  // %globaltimer is slow to read: start the clock only after many polls
  uint32_t it = 0;
  while (true) {
    v = sys_scope ? ld_acquire_sys(flag) : ld_acquire_gpu(flag);
    if (v >= want) return true;
    __nanosleep(32);
    if (((++it) & 0xff) == 0) {
      if (*abort_flag) return false;
      if (status_failed(status)) {
        *abort_flag = 1;
        return false;
      }
      if (t0 == 0) {
        t0 = globaltimer_ns();
        continue;
      }
      if (globaltimer_ns() - t0 > MMJ_WAIT_BUDGET_NS) {
        *abort_flag = 1;
        report(status, kTimeoutFlag, detail);
        return false;
      }
    }
  }
}

struct TileCoord {
  int m_tile, n_tile;
};

// Contraction range of a tile. Plain GEMMs contract over [0, K); in grouped-K mode (expert
// weight gradients) tile t belongs to group g = t / tiles_per_group and contracts over the rows
// [group_k[2g], group_k[2g+1]) of both MN-major operands.
struct KRange {
  int g, tt, k_begin, nk;
};
__device__ __forceinline__ KRange krange_of(int t, int per_group, int num_k, const GemmParams& p) {
  KRange r;
  if (p.groups_k <= 0) {
    r.g = 0; r.tt = t; r.k_begin = 0; r.nk = num_k;
    return r;
  }
  r.g = t / per_group;
  r.tt = t - r.g * per_group;
  r.k_begin = p.group_k[2 * r.g];
  const int k_end = p.group_k[2 * r.g + 1];
  r.nk = (k_end > r.k_begin) ? (k_end - r.k_begin + kGemmBK - 1) / kGemmBK : 0;
  return r;
}

__device__ __forceinline__ TileCoord tile_of(int t, int num_m, int num_n, const GemmParams& p) {
  // n fastest by default: concurrently running CTAs share A rows and sweep B (weights stay in
  // L2). With a gathered B operand the order is m fastest, so that the first waves only need
  // the B tiles that are already local.
  int m_lin, n_lin;
  if (p.flag_mode == 2) {
    n_lin = t / num_m;
    m_lin = t - n_lin * num_m;
  } else if (p.flag_mode == 1 || num_n <= 12) {
    m_lin = t / num_n;
    n_lin = t - m_lin * num_n;
  } else {
    // wide outputs: walk groups of 16 row tiles with n outer / m inner, so that one wave of
    // CTAs covers a roughly square block of tiles and re-reads fewer operand panels from DRAM
    constexpr int kGroupM = 16;
    const int per_group = kGroupM * num_n;
    const int g = t / per_group;
    const int first_m = g * kGroupM;
    const int rows_in_group = min(kGroupM, num_m - first_m);
    const int r = t - g * per_group;
    n_lin = r / rows_in_group;
    m_lin = first_m + (r - n_lin * rows_in_group);
  }
  TileCoord c;
  c.m_tile = m_lin + p.m_tile_rot;
  if (c.m_tile >= num_m) c.m_tile -= num_m;
  c.n_tile = n_lin + p.n_tile_rot;
  if (c.n_tile >= num_n) c.n_tile -= num_n;
  return c;
}

// Byte offset of 16-byte piece `c` (0..3) of row `row` (0..31) in a per-warp staging area of 32 rows x
// 64 bytes. The piece index is XORed with bits 1-2 of the row: the eight lanes of a quarter warp then hit
// eight different 16-byte bank groups both when every lane writes piece c of its own row and when four
// neighbouring lanes read the four pieces of one row (a padded pitch of 80 bytes left the reads of two
// adjacent rows sharing a bank group).
__device__ __forceinline__ int stage_off(int row, int c) {
  return row * 64 + ((c ^ ((row >> 1) & 3)) << 4);
}

// Stores a 32-row x 32-column bf16 chunk (lane = row, v = its 32 columns) through a per-warp
// staging area so that four neighbouring lanes write 64 contiguous bytes of one row: full 32-byte
// sectors per request instead of 32 half-sector pieces. `tile` points at (first row, first column).
__device__ __forceinline__ void staged_store_bf16(uint8_t* st, int lane, const float (&v)[32],
                                                  __nv_bfloat16* tile, long long ld) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint4 q;
    q.x = pack_bf16x2(v[8 * i + 0], v[8 * i + 1]);
    q.y = pack_bf16x2(v[8 * i + 2], v[8 * i + 3]);
    q.z = pack_bf16x2(v[8 * i + 4], v[8 * i + 5]);
    q.w = pack_bf16x2(v[8 * i + 6], v[8 * i + 7]);
    *reinterpret_cast<uint4*>(st + stage_off(lane, i)) = q;
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int rr = 8 * i + (lane >> 2);
    const uint4 q = *reinterpret_cast<const uint4*>(st + stage_off(rr, lane & 3));
    *reinterpret_cast<uint4*>(tile + rr * ld + (lane & 3) * 8) = q;
  }
  __syncwarp();
}

template <bool kOutF32>
__device__ __forceinline__ void epilogue_store_chunk(const GemmParams& p, const uint32_t (&acc)[32],
                                                     int row, int col0, uint8_t* st = nullptr,
                                                     int lane = 0, const uint4* auxq = nullptr) {
  // One thread owns 32 consecutive columns [col0, col0+32) of output row `row`. With `st` set the
  // whole warp is here (32 valid rows, lane = row offset) and full chunks leave through it. `auxq`:
  // the chunk's 32 aux values, already loaded by the caller (full chunks only).
  const int epi = p.epi;
  float v[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(acc[i]);

  const bool full = p.vec_ok && (col0 + 32 <= p.N);
  if (epi & kEpiBias) {
    const __nv_bfloat16* b = reinterpret_cast<const __nv_bfloat16*>(p.bias) + col0;
    if (full) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        uint4 q = __ldg(reinterpret_cast<const uint4*>(b) + i);
        float2 f0 = unpack_bf16x2(q.x), f1 = unpack_bf16x2(q.y), f2 = unpack_bf16x2(q.z),
               f3 = unpack_bf16x2(q.w);
        v[8 * i + 0] += f0.x; v[8 * i + 1] += f0.y; v[8 * i + 2] += f1.x; v[8 * i + 3] += f1.y;
        v[8 * i + 4] += f2.x; v[8 * i + 5] += f2.y; v[8 * i + 6] += f3.x; v[8 * i + 7] += f3.y;
      }
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i)
        if (col0 + i < p.N) v[i] += __bfloat162float(b[i]);
    }
  }
  if (epi & kEpiGelu) {
    __nv_bfloat16* d2 = reinterpret_cast<__nv_bfloat16*>(p.D2) + (long long)row * p.ldd2 + col0;
    if (full && st != nullptr) {
      staged_store_bf16(st, lane, v, d2 - (long long)lane * p.ldd2, p.ldd2);
    } else if (full) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        uint4 q;
        q.x = pack_bf16x2(v[8 * i + 0], v[8 * i + 1]);
        q.y = pack_bf16x2(v[8 * i + 2], v[8 * i + 3]);
        q.z = pack_bf16x2(v[8 * i + 4], v[8 * i + 5]);
        q.w = pack_bf16x2(v[8 * i + 6], v[8 * i + 7]);
        reinterpret_cast<uint4*>(d2)[i] = q;
      }
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i)
        if (col0 + i < p.N) d2[i] = __float2bfloat16(v[i]);
    }
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = gelu_tanh(v[i]);
  }
  if (epi & kEpiSilu) {
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = v[i] / (1.0f + __expf(-v[i]));
  }
  if (epi & (kEpiDGelu | kEpiAddAux | kEpiMulAux)) {
    const __nv_bfloat16* a =
        reinterpret_cast<const __nv_bfloat16*>(p.aux) + (long long)row * p.ldaux + col0;
    float x[32];
    if (full) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        uint4 q = (auxq != nullptr) ? auxq[i] : reinterpret_cast<const uint4*>(a)[i];
        float2 f0 = unpack_bf16x2(q.x), f1 = unpack_bf16x2(q.y), f2 = unpack_bf16x2(q.z),
               f3 = unpack_bf16x2(q.w);
        x[8 * i + 0] = f0.x; x[8 * i + 1] = f0.y; x[8 * i + 2] = f1.x; x[8 * i + 3] = f1.y;
        x[8 * i + 4] = f2.x; x[8 * i + 5] = f2.y; x[8 * i + 6] = f3.x; x[8 * i + 7] = f3.y;
      }
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i) x[i] = (col0 + i < p.N) ? __bfloat162float(a[i]) : 0.f;
    }
    if (epi & kEpiDGelu) {
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] *= gelu_tanh_grad(x[i]);
    } else if (epi & kEpiMulAux) {
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] *= x[i];
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] += x[i];
    }
  }
  if (epi & kEpiRowScale) {
    const float s = p.row_scale[row];
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] *= s;
  }

  // Destination row: local, or the owner's staging slot for the reduce-scatter epilogue.
  long long off;
  void* base = p.D;
  if (epi & kEpiScatterPeers) {
    int owner = row / p.rows_per_rank;
    int lrow = row - owner * p.rows_per_rank;
    base = p.peer_D[owner];
    off = (long long)p.rank * p.slot_stride + (long long)lrow * p.ldd + col0;
  } else {
    off = (long long)row * p.ldd + col0;
  }

  if (kOutF32) {
    float* d = reinterpret_cast<float*>(base) + off;
    if (full) {
      if (epi & kEpiAccumulate) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          float4 o = reinterpret_cast<float4*>(d)[i];
          v[4 * i + 0] += o.x; v[4 * i + 1] += o.y; v[4 * i + 2] += o.z; v[4 * i + 3] += o.w;
        }
      }
#pragma unroll
      for (int i = 0; i < 8; ++i)
        reinterpret_cast<float4*>(d)[i] =
            make_float4(v[4 * i + 0], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i)
        if (col0 + i < p.N) d[i] = (epi & kEpiAccumulate) ? d[i] + v[i] : v[i];
    }
  } else {
    __nv_bfloat16* d = reinterpret_cast<__nv_bfloat16*>(base) + off;
    if (full && st != nullptr && !(epi & (kEpiAccumulate | kEpiScatterPeers))) {
      staged_store_bf16(st, lane, v, d - (long long)lane * p.ldd, p.ldd);
    } else if (full) {
      if (epi & kEpiAccumulate) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          uint4 q = reinterpret_cast<uint4*>(d)[i];
          float2 f0 = unpack_bf16x2(q.x), f1 = unpack_bf16x2(q.y), f2 = unpack_bf16x2(q.z),
                 f3 = unpack_bf16x2(q.w);
          v[8 * i + 0] += f0.x; v[8 * i + 1] += f0.y; v[8 * i + 2] += f1.x; v[8 * i + 3] += f1.y;
          v[8 * i + 4] += f2.x; v[8 * i + 5] += f2.y; v[8 * i + 6] += f3.x; v[8 * i + 7] += f3.y;
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        uint4 q;
        q.x = pack_bf16x2(v[8 * i + 0], v[8 * i + 1]);
        q.y = pack_bf16x2(v[8 * i + 2], v[8 * i + 3]);
        q.z = pack_bf16x2(v[8 * i + 4], v[8 * i + 5]);
        q.w = pack_bf16x2(v[8 * i + 6], v[8 * i + 7]);
        reinterpret_cast<uint4*>(d)[i] = q;
      }
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i)
        if (col0 + i < p.N) {
          float o = (epi & kEpiAccumulate) ? __bfloat162float(d[i]) : 0.f;
          d[i] = __float2bfloat16(v[i] + o);
        }
    }
  }
}

__global__ void __launch_bounds__(kThreads, 1)
gemm_bf16_tcgen05_kernel(const __grid_constant__ CUtensorMap tmA,
                         const __grid_constant__ CUtensorMap tmB, const GemmParams p) {
  extern __shared__ uint8_t smem_raw[];
  // 128-byte swizzled tiles need 1024-byte aligned bases.
  // (offset arithmetic on the __shared__ symbol, not an integer round trip, so that the compiler
  // keeps the shared address space and emits shared rather than generic loads and stores)
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  __shared__ __align__(8) uint64_t full_bar[kGemmMaxStages];
  __shared__ __align__(8) uint64_t empty_bar[kGemmMaxStages];
  __shared__ __align__(8) uint64_t tfull_bar[2];
  __shared__ __align__(8) uint64_t tempty_bar[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  // per-warp staging for the transposing stores: 32 rows x 64 bytes, pieces swizzled (stage_off)
  __shared__ __align__(16) uint8_t epi_stage[kEpiWarps][32 * 64];

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int gemm_ctas = (p.gemm_ctas > 0) ? p.gemm_ctas : (int)gridDim.x;

  // ---------------- communication CTAs: pull peer shards, publish per-tile flags ----------
  // One thread per CTA drives bulk asynchronous copies (peer memory -> shared memory ->
  // local memory) through a ring of 32 KiB buffers, so that ~190 KiB per CTA stay in flight
  // over NVLink without occupying the other threads. No multicast is involved.
  if ((int)blockIdx.x >= gemm_ctas) {
    constexpr int kNBuf = 6;
    constexpr int kBufBytes = 32 * 1024;
    if (threadIdx.x == 0) {
      abort_flag = 0;
      for (int b = 0; b < kNBuf; ++b) mbar_init(&full_bar[b], 1);
      mbar_fence_init();
      const int n_comm = (int)gridDim.x - gemm_ctas;
      const int cid = (int)blockIdx.x - gemm_ctas;
      const int ntiles = (int)((p.gather_total_bytes + p.tile_bytes - 1) / p.tile_bytes);
      const int rot = p.comm_rot;
      uint32_t issued = 0, drained = 0;  // chunk counters over the ring
      bool ok = true;
      for (int i = cid; i < ntiles && ok; i += n_comm) {
        int t = i + rot;  // same visiting order as the GEMM CTAs consume tiles
        if (t >= ntiles) t -= ntiles;
        long long lo = (long long)t * p.tile_bytes;
        long long hi = lo + p.tile_bytes;
        if (hi > p.gather_total_bytes) hi = p.gather_total_bytes;
        // a tile may straddle shard boundaries: copy it owner by owner
        while (lo < hi && ok) {
          const long long abs_off = p.gather_flat_off + lo;
          const int owner = (int)(abs_off / p.shard_bytes);
          long long seg_hi = (long long)(owner + 1) * p.shard_bytes - p.gather_flat_off;
          if (seg_hi > hi) seg_hi = hi;
          if ((owner != p.rank || p.src_compact) && owner < p.world) {
            if (p.peer_ready != nullptr && owner != p.rank)
              ok = wait_flag_ge(p.peer_ready + owner, p.ready_epoch, true, &abort_flag, p.status,
                                100 + owner);
            if (!ok) break;
            const long long nbytes = seg_hi - lo;
            const uint8_t* src = reinterpret_cast<const uint8_t*>(p.peer_src[owner]) +
                                 (p.src_compact ? (abs_off - (long long)owner * p.shard_bytes) : lo);
            uint8_t* dst = reinterpret_cast<uint8_t*>(p.gather_dst) + lo;
            const int nchunks = (int)((nbytes + kBufBytes - 1) / kBufBytes);
            int next_load = 0;
            for (int c = 0; c < nchunks && ok; ++c) {
              // keep up to kNBuf loads in flight
              while (next_load < nchunks && issued - drained < (uint32_t)kNBuf) {
                const int b = issued % kNBuf;
                const long long co = (long long)next_load * kBufBytes;
                const uint32_t sz =
                    (uint32_t)((nbytes - co < kBufBytes) ? (nbytes - co) : kBufBytes);
                mbar_expect_tx(&full_bar[b], sz);
                asm volatile(
                    "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                    ::"r"(smem_u32(smem + (size_t)b * kBufBytes)), "l"(src + co), "r"(sz),
                    "r"(smem_u32(&full_bar[b]))
                    : "memory");
                ++issued;
                ++next_load;
              }
              const int b = drained % kNBuf;
              const uint32_t par = (drained / kNBuf) & 1u;
              if (!mbar_wait(&full_bar[b], par, &abort_flag, p.status, kTimeoutFull, 1000 + c)) {
                ok = false;
                break;
              }
              const long long co = (long long)c * kBufBytes;
              const uint32_t sz = (uint32_t)((nbytes - co < kBufBytes) ? (nbytes - co) : kBufBytes);
              asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst + co),
                           "r"(smem_u32(smem + (size_t)b * kBufBytes)), "r"(sz)
                           : "memory");
              asm volatile("cp.async.bulk.commit_group;" ::: "memory");
              // the buffer may be refilled once the store has read it
              asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
              ++drained;
            }
            // all bytes of this piece written before the tile's flag is published
            asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
          }
          lo = seg_hi;
        }
        if (!ok) break;
        asm volatile("fence.proxy.async;" ::: "memory");
        __threadfence();
        st_release_gpu(p.flags_rw + t, p.ready_epoch);
      }
      // never leave with loads in flight into this CTA's shared memory
      while (drained < issued) {
        const int b = drained % kNBuf;
        const uint32_t par = (drained / kNBuf) & 1u;
        int local_abort = 0;
        if (!mbar_wait(&full_bar[b], par, &local_abort, p.status, kTimeoutFull, 2000)) break;
        ++drained;
      }
    }
    return;
  }

  // ---------------- GEMM CTAs --------------------------------------------------------------
  const int bn = p.bn;
  const int stages = p.stages;
  const int b_stage_bytes = bn * kGemmBK * 2;
  // Tall tiles (bm2): 256 rows per tile as two 128-row sub-tiles that share each B stage, which
  // halves the B bytes pulled from L2 per FLOP. With bn = 256 the two accumulators take all 512
  // TMEM columns, so the epilogue of a tile no longer overlaps the next tile's main loop.
  const int subs = p.bm2 ? 2 : 1;
  const int bm = kGemmBM * subs;
  const int a_bytes = kAStageBytes * subs;
  const int stage_bytes = a_bytes + b_stage_bytes;
  const int n_acc = (subs * bn > kAccCols) ? 1 : 2;

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tfull_bar[a], 1);
      mbar_init(&tempty_bar[a], kEpiWarps);
    }
    abort_flag = 0;
    mbar_fence_init();
    prefetch_tmap(&tmA);
    prefetch_tmap(&tmB);
  }
  if (warp == 1) {
    tmem_alloc(&tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;
  // everything above touched no global memory: it may run under the previous kernel's tail
  pdl_wait();
  pdl_trigger();

  const int num_m = (p.num_m_tiles_dev != nullptr) ? *p.num_m_tiles_dev
                                                   : (p.M + bm - 1) / bm;
  const int num_n = (p.N + bn - 1) / bn;
  const int num_k = (p.K + kGemmBK - 1) / kGemmBK;
  const int per_group = num_m * num_n;
  const int num_tiles = (p.groups_k > 0) ? p.groups_k * per_group : per_group;

  if (num_k > 0 || p.groups_k > 0) {
    if (warp == 0) {
      // ======================= TMA producer =======================
      if (lane == 0) {
        int s = 0;
        uint32_t ph = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < num_tiles && ok; t += gemm_ctas) {
          const KRange kr = krange_of(t, per_group, num_k, p);
          const TileCoord tc = tile_of(kr.tt, num_m, num_n, p);
          const int m0 = tc.m_tile * bm;
          const int n0 = tc.n_tile * bn;
          const int g = (p.tile_group != nullptr) ? p.tile_group[tc.m_tile] : 0;
          const int b_row_base = g * p.b_group_rows;
          if (p.flag_mode == 1) {
            // flags are per 128-row granule of the gathered operand: a tall tile needs two
            const int n_gran = (p.M + kGemmBM - 1) / kGemmBM;
            for (int sub = 0; sub < subs && ok; ++sub) {
              const int gt = tc.m_tile * subs + sub;
              if (gt < n_gran)
                ok = wait_flag_ge(p.ready_flags + gt, p.ready_epoch, false, &abort_flag, p.status, gt);
            }
            asm volatile("fence.proxy.async;" ::: "memory");
          } else if (p.flag_mode == 2) {
            ok = wait_flag_ge(p.ready_flags + tc.n_tile, p.ready_epoch, false, &abort_flag,
                              p.status, tc.n_tile);
            asm volatile("fence.proxy.async;" ::: "memory");
          }
          if (!ok) break;
          for (int kb = 0; kb < kr.nk; ++kb) {
            if (!mbar_wait(&empty_bar[s], ph ^ 1, &abort_flag, p.status, kTimeoutEmpty, kb)) {
              ok = false;
              break;
            }
            uint8_t* sA = smem + (size_t)s * stage_bytes;
            uint8_t* sB = sA + a_bytes;
            mbar_expect_tx(&full_bar[s], (uint32_t)stage_bytes);
            const int k0 = kr.k_begin + kb * kGemmBK;
            for (int sub = 0; sub < subs; ++sub) {
              uint8_t* sAs = sA + sub * kAStageBytes;
              const int ms = m0 + sub * kGemmBM;
              if (!p.a_mn) {
                tma_load_2d(sAs, &tmA, &full_bar[s], k0, ms);
              } else {
                tma_load_2d(sAs, &tmA, &full_bar[s], ms, k0);
                tma_load_2d(sAs + 8192, &tmA, &full_bar[s], ms + 64, k0);
              }
            }
            if (!p.b_mn) {
              tma_load_2d(sB, &tmB, &full_bar[s], k0, b_row_base + n0);
            } else {
              for (int j = 0; j < bn / 64; ++j)
                tma_load_2d(sB + j * 8192, &tmB, &full_bar[s], n0 + 64 * j, b_row_base + k0);
            }
            if (++s == stages) { s = 0; ph ^= 1; }
          }
        }
      }
    } else if (warp == 1) {
      // ======================= MMA issuer =======================
      if (lane == 0) {
        const uint32_t idesc = make_idesc_bf16(kGemmBM, bn, p.a_mn, p.b_mn);
        const uint32_t a_lbo = p.a_mn ? 8192u : 16u;
        const uint32_t b_lbo = p.b_mn ? 8192u : 16u;
        const uint32_t a_kstep = p.a_mn ? 2048u : 32u;
        const uint32_t b_kstep = p.b_mn ? 2048u : 32u;
        int s = 0;
        uint32_t ph = 0;
        int acc = 0;
        uint32_t acc_ph = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < num_tiles && ok; t += gemm_ctas) {
          const KRange kr = krange_of(t, per_group, num_k, p);
          if (kr.nk == 0) continue;  // empty contraction: the epilogue writes zeros on its own
          if (!mbar_wait(&tempty_bar[acc], acc_ph ^ 1, &abort_flag, p.status, kTimeoutTmemEmpty,
                         t)) {
            break;
          }
          tc_fence_after();
          const uint32_t d_tmem = tmem_base + (uint32_t)(acc * kAccCols);
          const uint32_t d_tmem1 = d_tmem + (uint32_t)bn;  // second sub-tile of a tall tile
          for (int kb = 0; kb < kr.nk; ++kb) {
            if (!mbar_wait(&full_bar[s], ph, &abort_flag, p.status, kTimeoutFull, kb)) {
              ok = false;
              break;
            }
            tc_fence_after();
            const uint32_t a_base = smem_u32(smem + (size_t)s * stage_bytes);
            const uint32_t b_base = a_base + (uint32_t)a_bytes;
#pragma unroll
            for (int k = 0; k < kGemmBK / 16; ++k) {
              const uint64_t da = make_smem_desc(a_base + k * a_kstep, a_lbo, 1024);
              const uint64_t db = make_smem_desc(b_base + k * b_kstep, b_lbo, 1024);
              umma_bf16_ss(d_tmem, da, db, idesc, (kb > 0 || k > 0) ? 1u : 0u);
              if (subs == 2) {
                const uint64_t da1 = make_smem_desc(a_base + kAStageBytes + k * a_kstep, a_lbo, 1024);
                umma_bf16_ss(d_tmem1, da1, db, idesc, (kb > 0 || k > 0) ? 1u : 0u);
              }
            }
            umma_commit(&empty_bar[s]);  // frees the smem stage once these MMAs retire
            if (++s == stages) { s = 0; ph ^= 1; }
          }
          if (!ok) break;
          umma_commit(&tfull_bar[acc]);  // accumulator complete
          if (++acc == n_acc) { acc = 0; acc_ph ^= 1; }
        }
      }
    } else {
      // ======================= epilogue warps =======================
      // Eight epilogue warps: two per TMEM lane quadrant (a warp reaches the 32 lanes of quadrant
      // warp % 4 only), taking alternate 32-column chunks. With four warps the fused GELU / GELU'
      // epilogues of the K = 768 products took longer than the next tile's main loop.
      const int quad = warp & 3;
      const int chalf = (warp - 2) >> 2;
      int acc = 0;
      uint32_t acc_ph = 0;
      for (int t = blockIdx.x; t < num_tiles; t += gemm_ctas) {
        const KRange kr = krange_of(t, per_group, num_k, p);
        const TileCoord tc = tile_of(kr.tt, num_m, num_n, p);
        const int m0 = tc.m_tile * bm;
        const int n0 = tc.n_tile * bn;
        const int out_row0 = kr.g * p.M;  // grouped-K: group g writes rows [g*M, (g+1)*M)
        if (kr.nk == 0) {
          // nothing to contract (an expert without tokens): the result is zero
          for (int sub = 0; sub < subs; ++sub) {
          const int zrow = m0 + sub * kGemmBM + quad * 32 + lane;
          if (zrow < p.M) {
            uint32_t z[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) z[i] = 0u;
            for (int c = chalf; c < bn / 32; c += 2) {
              const int col0 = n0 + c * 32;
              if (col0 < p.N) {
                if (p.epi & kEpiOutF32)
                  epilogue_store_chunk<true>(p, z, zrow + out_row0, col0);
                else
                  epilogue_store_chunk<false>(p, z, zrow + out_row0, col0);
              }
            }
          }
          }
          continue;
        }
        if (!mbar_wait_warp(&tfull_bar[acc], acc_ph, &abort_flag, p.status, kTimeoutTmemFull, t)) break;
        tc_fence_after();
        for (int sub = 0; sub < subs; ++sub) {
          const int row = m0 + sub * kGemmBM + quad * 32 + lane;
          const uint32_t t_row = tmem_base + ((uint32_t)(quad * 32) << 16) +
                                 (uint32_t)(acc * kAccCols + sub * bn);
          for (int c = chalf; c < bn / 32; c += 2) {
            uint32_t r[32];
            tmem_ld_32x32(t_row + (uint32_t)(c * 32), r);
            tmem_ld_wait();
            const int col0 = n0 + c * 32;
            if ((p.epi & kEpiScatterPeers) && p.vec_ok && col0 + 32 <= p.N) {
              // Stores into a peer's memory travel over NVLink: transpose the chunk through shared
              // memory so that four neighbouring lanes write 64 contiguous bytes of one row (one
              // thread per row would send 16-byte pieces).
              uint8_t* st = epi_stage[warp - 2];
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                uint4 q;
                q.x = pack_bf16x2(__uint_as_float(r[8 * i + 0]), __uint_as_float(r[8 * i + 1]));
                q.y = pack_bf16x2(__uint_as_float(r[8 * i + 2]), __uint_as_float(r[8 * i + 3]));
                q.z = pack_bf16x2(__uint_as_float(r[8 * i + 4]), __uint_as_float(r[8 * i + 5]));
                q.w = pack_bf16x2(__uint_as_float(r[8 * i + 6]), __uint_as_float(r[8 * i + 7]));
                *reinterpret_cast<uint4*>(st + stage_off(lane, i)) = q;
              }
              __syncwarp();
              const int row_base = m0 + sub * kGemmBM + quad * 32;
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const int rr = 8 * i + (lane >> 2);
                const uint4 q = *reinterpret_cast<const uint4*>(st + stage_off(rr, lane & 3));
                const int grow = row_base + rr;
                if (grow < p.M) {
                  const int owner = grow / p.rows_per_rank;
                  const int lrow = grow - owner * p.rows_per_rank;
                  __nv_bfloat16* d = reinterpret_cast<__nv_bfloat16*>(p.peer_D[owner]) +
                                     (long long)p.rank * p.slot_stride + (long long)lrow * p.ldd + col0 +
                                     (lane & 3) * 8;
                  *reinterpret_cast<uint4*>(d) = q;
                }
              }
              __syncwarp();
            } else if (row < p.M && col0 < p.N) {
              if (p.epi & kEpiOutF32)
                epilogue_store_chunk<true>(p, r, row + out_row0, col0);
              else
                epilogue_store_chunk<false>(
                    p, r, row + out_row0, col0,
                    (m0 + sub * kGemmBM + quad * 32 + 32 <= p.M) ? epi_stage[warp - 2] : nullptr, lane);
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tempty_bar[acc]);
        if (++acc == n_acc) { acc = 0; acc_ph ^= 1; }
      }
    }
  }

  // ---------------- teardown ----------------
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// ---------------------------------------------------------------------------------------------
// CTA-pair variant (cta_group::2) for plain products: two CTAs of a cluster own one 256 x 256 tile.
// Each CTA stages its own 128 rows of A and its own 128-column half of B (32 KiB per 64-deep K
// block instead of 48 KiB for a 128 x 256 tile on one CTA: a third less traffic from L2 into shared
// memory per FLOP), keeps 128 x 256 of the accumulator in its own TMEM (two accumulators, so the
// epilogue still overlaps the next main loop) and stores its own rows. The rank-0 CTA issues the
// MMAs for the pair; both CTAs' loads are credited to rank 0's "full" barrier, the MMA's commits
// release the stage in both CTAs, and both CTAs' epilogue warps arrive on rank 0's "accumulator
// free" barrier. No load uses multicast.
// ---------------------------------------------------------------------------------------------
constexpr int kPairBN = 256;
constexpr int kPairStageBytes = kAStageBytes + (kPairBN / 2) * kGemmBK * 2;  // 32 KiB

// The fused GELU / GELU' epilogues lengthen the chain of a tile's 32-column chunks; no unit bounds them. Counters at
// 16384 x 3072 x 768, bias only / GELU / GELU': tensor pipe 72 / 52 / 50 %, issue slots 19 / 25 / 27 %, exponentials' unit 1 /
// 18 / 17 %, 6 / 11 / 13 instructions an element, 2.5 warps a scheduler that mostly wait for TMEM and shared memory.
// the two bf16 halves of a word, widened (their bits are the upper halves of the fp32 values)
__device__ __forceinline__ f32x2 f2_from_bf16(uint32_t u) {
  return f2_pack(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u));
}
__device__ __forceinline__ uint32_t f2_to_bf16(f32x2 v) {
  float a, b;
  f2_unpack(v, a, b);
  return pack_bf16x2(a, b);
}
constexpr float kGeluK0 = 0.7978845608028654f, kGeluK1 = 0.7978845608028654f * 0.044715f;
__device__ __forceinline__ f32x2 f2_tanh(f32x2 u) {
  float a, b;
  f2_unpack(u, a, b);
  return f2_pack(tanh_fast(a), tanh_fast(b));
}
__device__ __forceinline__ f32x2 f2_gelu(f32x2 x) {
  const f32x2 x2 = f2_mul(x, x);
  const f32x2 t = f2_tanh(f2_mul(x, f2_fma(x2, f2_pack(kGeluK1, kGeluK1), f2_pack(kGeluK0, kGeluK0))));
  const f32x2 h = f2_mul(x, f2_pack(0.5f, 0.5f));
  return f2_fma(h, t, h);
}
__device__ __forceinline__ f32x2 f2_gelu_grad(f32x2 x) {
  const f32x2 x2 = f2_mul(x, x), half = f2_pack(0.5f, 0.5f), one = f2_pack(1.f, 1.f);
  const f32x2 k0 = f2_pack(kGeluK0, kGeluK0);
  const f32x2 t = f2_tanh(f2_mul(x, f2_fma(x2, f2_pack(kGeluK1, kGeluK1), k0)));
  const f32x2 du = f2_fma(x2, f2_pack(3.f * kGeluK1, 3.f * kGeluK1), k0);
  const f32x2 sech2 = f2_fma(f2_mul(t, f2_pack(-1.f, -1.f)), t, one);
  return f2_fma(f2_mul(f2_mul(x, half), sech2), du, f2_fma(t, half, half));
}

// Stores 32 rows x 32 bf16 columns (lane = row, 16 packed words) through the warp's staging area.
__device__ __forceinline__ void staged_store_words(uint8_t* st, int lane, const uint32_t (&w)[16],
                                                   __nv_bfloat16* tile, long long ld) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
    *reinterpret_cast<uint4*>(st + stage_off(lane, i)) = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int rr = 8 * i + (lane >> 2);
    const uint4 q = *reinterpret_cast<const uint4*>(st + stage_off(rr, lane & 3));
    *reinterpret_cast<uint4*>(tile + rr * ld + (lane & 3) * 8) = q;
  }
  __syncwarp();
}

// Epilogue of a full 32-row, 32-column chunk (16384 x 3072 x 768: GELU 86 -> 75 us, GELU' 99 -> 78 us, of which 13 us
// came from fetching aux four lanes to a row instead of a row per lane; sixteen epilogue warps instead of eight measured
// 78 and 81) with the options fixed at compile time. kMode: 1 = bf16 result with an
// optional bias, 2 = bias, pre-activation kept, GELU, 3 = times GELU'(aux), 4 = fp32 result. `bias` / `auxq` hold the chunk's 16 words.
template <int kMode>
__device__ __forceinline__ void epilogue_chunk_fixed(const GemmParams& p, const uint32_t (&acc)[32], bool has_bias,
                                                     const uint4 (&extra)[4], long long row0, int col0, uint8_t* st,
                                                     int lane) {
  const uint32_t* ew = reinterpret_cast<const uint32_t*>(extra);
  uint32_t w[16];
  if (kMode == 4) {   // fp32, 16 columns (64 bytes of a row) at a time
    float* d = reinterpret_cast<float*>(p.D) + row0 * p.ldd + col0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        *reinterpret_cast<uint4*>(st + stage_off(lane, i)) =
            make_uint4(acc[16 * h + 4 * i], acc[16 * h + 4 * i + 1], acc[16 * h + 4 * i + 2], acc[16 * h + 4 * i + 3]);
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int rr = 8 * i + (lane >> 2);
        *reinterpret_cast<uint4*>(d + rr * p.ldd + 16 * h + (lane & 3) * 4) =
            *reinterpret_cast<const uint4*>(st + stage_off(rr, lane & 3));
      }
      __syncwarp();
    }
    return;
  }
  if (kMode == 2) {
    uint32_t act[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      f32x2 v = f2_pack(__uint_as_float(acc[2 * i]), __uint_as_float(acc[2 * i + 1]));
      if (has_bias) v = f2_add(v, f2_from_bf16(ew[i]));
      w[i] = f2_to_bf16(v);
      act[i] = f2_to_bf16(f2_gelu(v));
    }
    staged_store_words(st, lane, w, reinterpret_cast<__nv_bfloat16*>(p.D2) + row0 * p.ldd2 + col0, p.ldd2);
    staged_store_words(st, lane, act, reinterpret_cast<__nv_bfloat16*>(p.D) + row0 * p.ldd + col0, p.ldd);
    return;
  }
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    f32x2 v = f2_pack(__uint_as_float(acc[2 * i]), __uint_as_float(acc[2 * i + 1]));
    if (kMode == 1) {
      if (has_bias) v = f2_add(v, f2_from_bf16(ew[i]));
    } else {
      v = f2_mul(v, f2_gelu_grad(f2_from_bf16(ew[i])));
    }
    w[i] = f2_to_bf16(v);
  }
  staged_store_words(st, lane, w, reinterpret_cast<__nv_bfloat16*>(p.D) + row0 * p.ldd + col0, p.ldd);
}

// kMode 0: every combination of epilogue options; 1 to 4: the fixed ones of epilogue_chunk_fixed; 5: as 4, and the column
// sums of A (an MN-major dy: the bias gradient of the layer whose weight gradient this is) into p.bias_part. The epilogue
// warps are idle during a split product's one main loop: those of the CTAs with the first column tile add up their A
// stages once the products have read them, and every CTA's stages return through its epilogue warps. The four column
// sums of a GPT-2 layer (19 + 15 + 8 + 8 us and a 3 us fold each) re-read the same dy from HBM.
template <int kMode>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
gemm_bf16_pair_kernel(const __grid_constant__ CUtensorMap tmA,
                      const __grid_constant__ CUtensorMap tmB, const GemmParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  __shared__ __align__(8) uint64_t full_bar[kGemmMaxStages];
  __shared__ __align__(8) uint64_t empty_bar[kGemmMaxStages];
  __shared__ __align__(8) uint64_t done_bar[kGemmMaxStages];   // kMode 5: the stage's products have read it
  __shared__ __align__(8) uint64_t sums_bar[2];                // kMode 5: the warps' sums are written / have been read
  __shared__ __align__(8) uint64_t tfull_bar[2];
  __shared__ __align__(8) uint64_t tempty_bar[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  __shared__ __align__(16) uint8_t epi_stage[kEpiWarps][32 * 64];

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;
  const int pair = (int)blockIdx.x >> 1;
  const int num_pairs = (int)gridDim.x >> 1;
  const int stages = p.stages;

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], kMode == 5 ? kEpiWarps : 1);
      if (kMode == 5) mbar_init(&done_bar[s], 1);
    }
    if (kMode == 5) {
      mbar_init(&sums_bar[0], kEpiWarps);
      mbar_init(&sums_bar[1], kEpiWarps / 2);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tfull_bar[a], 1);
      mbar_init(&tempty_bar[a], 2 * kEpiWarps);  // epilogue warps of both CTAs (used on rank 0)
    }
    abort_flag = 0;
    mbar_fence_init();
    prefetch_tmap(&tmA);
    prefetch_tmap(&tmB);
  }
  if (warp == 1) {
    tmem_alloc_pair(&tmem_slot, kTmemCols);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the peer's barriers are initialised before anything arrives on them
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;
  pdl_wait();  // nothing above touched global memory
  pdl_trigger();

  const int num_m = (p.M + 2 * kGemmBM - 1) / (2 * kGemmBM);
  const int num_n = (p.N + kPairBN - 1) / kPairBN;
  const int num_k = (p.K + kGemmBK - 1) / kGemmBK;
  const int per_group = num_m * num_n;
  const int num_tiles = (p.groups_k > 0) ? p.groups_k * per_group : per_group;

  if (num_k > 0 || p.groups_k > 0) {
    if (warp == 0) {
      // ======================= TMA producer (both CTAs) =======================
      const uint32_t full0 = mapa_shared(smem_u32(&full_bar[0]), 0);  // rank 0's barriers
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int t = pair; t < num_tiles && ok; t += num_pairs) {
        const KRange kr = krange_of(t, per_group, num_k, p);
        const TileCoord tc = tile_of(kr.tt, num_m, num_n, p);
        const int m0 = tc.m_tile * 2 * kGemmBM + (int)rank * kGemmBM;
        const int n0 = tc.n_tile * kPairBN + (int)rank * (kPairBN / 2);
        for (int kb = 0; kb < kr.nk; ++kb) {
          if (!mbar_wait_warp(&empty_bar[s], ph ^ 1, &abort_flag, p.status, kTimeoutEmpty, kb)) {
            ok = false;
            break;
          }
          if (elect_one()) {
            uint8_t* sA = smem + (size_t)s * kPairStageBytes;
            uint8_t* sB = sA + kAStageBytes;
            if (leader) mbar_expect_tx(&full_bar[s], 2u * (uint32_t)kPairStageBytes);
            const uint32_t fb = full0 + (uint32_t)(s * sizeof(uint64_t));
            const int k0 = kr.k_begin + kb * kGemmBK;
            if (!p.a_mn) {
              tma_load_2d_pair(sA, &tmA, fb, k0, m0);
            } else if (p.a_panels) {
              tma_load_3d_pair(sA, &tmA, fb, 0, k0, m0 >> 6);
            } else {
              tma_load_2d_pair(sA, &tmA, fb, m0, k0);
              tma_load_2d_pair(sA + 8192, &tmA, fb, m0 + 64, k0);
            }
            if (!p.b_mn) {
              tma_load_2d_pair(sB, &tmB, fb, k0, n0);
            } else if (p.b_panels) {
              tma_load_3d_pair(sB, &tmB, fb, 0, k0, n0 >> 6);
            } else {
              tma_load_2d_pair(sB, &tmB, fb, n0, k0);
              tma_load_2d_pair(sB + 8192, &tmB, fb, n0 + 64, k0);
            }
          }
          __syncwarp();
          if (++s == stages) { s = 0; ph ^= 1; }
        }
      }
    } else if (warp == 1) {
      // ======================= MMA issuer (rank 0 only) =======================
      // The whole warp walks the loop and an elected lane issues; stage descriptors are one addition and both CTAs'
      // barriers take one multicast commit. With lane 0 alone in a divergent loop and two commits, a 64-deep K block
      // cost about 900 cycles of issue against 512 of tensor time: 16384 x 2304 x 768 51.0 -> 47.2 us,
      // x 768 x 3072 64.0 -> 57.9, x 50304 x 768 1058 -> 991 (cuBLAS 47.5, 58.0, 1072 beside it). The one-SM kernel
      // keeps lane 0: its 256-row tiles have twice the tensor time per block, and measured 349 -> 376 us this way.
      if (leader) {
        const uint32_t idesc = make_idesc_bf16(2 * kGemmBM, kPairBN, p.a_mn, p.b_mn);
        const uint32_t a_lbo = p.a_mn ? 8192u : 16u;
        const uint32_t b_lbo = p.b_mn ? 8192u : 16u;
        const uint32_t a_kstep = (p.a_mn ? 2048u : 32u) >> 4;
        const uint32_t b_kstep = (p.b_mn ? 2048u : 32u) >> 4;
        const uint32_t a_lo0 = smem_desc_lo(smem_u32(smem), a_lbo);
        const uint32_t b_lo0 = smem_desc_lo(smem_u32(smem) + (uint32_t)kAStageBytes, b_lbo);
        int s = 0;
        uint32_t ph = 0;
        int acc = 0;
        uint32_t acc_ph = 0;
        bool ok = true;
        for (int t = pair; t < num_tiles && ok; t += num_pairs) {
          const KRange kr = krange_of(t, per_group, num_k, p);
          if (kr.nk == 0) continue;  // empty contraction: the epilogues write zeros on their own
          if (!mbar_wait_warp(&tempty_bar[acc], acc_ph ^ 1, &abort_flag, p.status, kTimeoutTmemEmpty, t)) break;
          tc_fence_after();
          const uint32_t d_tmem = tmem_base + (uint32_t)(acc * kAccCols);
          for (int kb = 0; kb < kr.nk; ++kb) {
            if (!mbar_wait_warp(&full_bar[s], ph, &abort_flag, p.status, kTimeoutFull, kb)) {
              ok = false;
              break;
            }
            tc_fence_after();
            if (elect_one()) {
              const uint32_t a_lo = a_lo0 + (uint32_t)(s * (kPairStageBytes >> 4));
              const uint32_t b_lo = b_lo0 + (uint32_t)(s * (kPairStageBytes >> 4));
#pragma unroll
              for (int k = 0; k < kGemmBK / 16; ++k)
                umma_bf16_ss_pair(d_tmem, smem_desc(a_lo + k * a_kstep), smem_desc(b_lo + k * b_kstep), idesc,
                                  (kb > 0 || k > 0) ? 1u : 0u);
              // the stage is free in both CTAs once these MMAs retire
              umma_commit_pair_both(kMode == 5 ? &done_bar[s] : &empty_bar[s]);
              if (kb + 1 == kr.nk) umma_commit_pair_both(&tfull_bar[acc]);
            }
            __syncwarp();
            if (++s == stages) { s = 0; ph ^= 1; }
          }
          if (++acc == 2) { acc = 0; acc_ph ^= 1; }
        }
      }
    } else {
      // ======================= epilogue warps (both CTAs) =======================
      const int quad = warp & 3;
      const int chalf = (warp - 2) >> 2;
      const uint32_t tempty0 = mapa_shared(smem_u32(&tempty_bar[0]), 0);
      int acc = 0;
      uint32_t acc_ph = 0;
      int cs = 0;          // kMode 5: the stage whose columns come next
      uint32_t cph = 0, sph = 0;
      for (int t = pair; t < num_tiles; t += num_pairs) {
        const KRange kr = krange_of(t, per_group, num_k, p);
        const TileCoord tc = tile_of(kr.tt, num_m, num_n, p);
        const int m0 = tc.m_tile * 2 * kGemmBM + (int)rank * kGemmBM;
        const int n0 = tc.n_tile * kPairBN;
        const int out_row0 = kr.g * p.M;  // grouped-K: group g writes rows [g*M, (g+1)*M)
        if (kMode == 5) {
          // warp: one 64-column panel of A, 16 of the stage's 64 rows; lane: two columns
          const int panel = (warp - 2) & 1, r0 = ((warp - 2) >> 1) * 16;
          f32x2 total = 0ull, part = 0ull;   // short chains: eight stages, then into the total
          bool ok = true;
          for (int kb = 0; kb < kr.nk; ++kb) {
            if (!mbar_wait_warp(&done_bar[cs], cph, &abort_flag, p.status, kTimeoutFull, kb)) { ok = false; break; }
            if (tc.n_tile == 0) {
              const uint8_t* base = smem + (size_t)cs * kPairStageBytes + panel * 8192;
#pragma unroll
              for (int i = 0; i < 16; ++i) {
                const int rr = r0 + i;   // 128-byte rows, 16-byte pieces XORed with the row's low bits
                part = f2_add(part, f2_from_bf16(*reinterpret_cast<const uint32_t*>(
                                        base + rr * 128 + (((lane >> 2) ^ (rr & 7)) << 4) + (lane & 3) * 4)));
              }
              if ((kb & 7) == 7) {
                total = f2_add(total, part);
                part = 0ull;
              }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty_bar[cs]);
            if (++cs == stages) { cs = 0; cph ^= 1; }
          }
          if (!ok) break;
          if (tc.n_tile == 0) {
            // The warps meet on mbarriers: a warp that gives up leaves this loop alone, on any tile, and the others then
            // run out of time as well, where a named barrier would wait for it for good.
            total = f2_add(total, part);
            float* mine = reinterpret_cast<float*>(epi_stage[warp - 2]);
            f2_unpack(total, mine[2 * lane], mine[2 * lane + 1]);
            __syncwarp();
            if (lane == 0) mbar_arrive(&sums_bar[0]);
            const int c = (int)threadIdx.x - 64;
            if (c < 128) {   // four of the eight warps
              if (!mbar_wait_warp(&sums_bar[0], sph, &abort_flag, p.status, kTimeoutFlag, t)) break;
              if (m0 + c < p.M) {
                float v = 0.f;
#pragma unroll
                for (int q = 0; q < kEpiWarps / 2; ++q)
                  v += reinterpret_cast<const float*>(epi_stage[(c >> 6) + 2 * q])[c & 63];
                p.bias_part[(long long)kr.g * p.M + m0 + c] = v;
              }
              __syncwarp();
              if (lane == 0) mbar_arrive(&sums_bar[1]);
            }
            // the staging areas are free again
            if (!mbar_wait_warp(&sums_bar[1], sph, &abort_flag, p.status, kTimeoutFlag, t)) break;
            sph ^= 1;
          }
        }
        if (kr.nk == 0) {
          const int zrow = m0 + quad * 32 + lane;
          if (zrow < p.M) {
            uint32_t z[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) z[i] = 0u;
            for (int c = chalf; c < kPairBN / 32; c += kEpiWarps / 4) {
              const int col0 = n0 + c * 32;
              if (col0 < p.N) {
                if (p.epi & kEpiOutF32)
                  epilogue_store_chunk<true>(p, z, zrow + out_row0, col0);
                else
                  epilogue_store_chunk<false>(p, z, zrow + out_row0, col0);
              }
            }
          }
          continue;
        }
        if (!mbar_wait_warp(&tfull_bar[acc], acc_ph, &abort_flag, p.status, kTimeoutTmemFull, t)) break;
        tc_fence_after();
        const int row = m0 + quad * 32 + lane;
        const uint32_t t_row = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(acc * kAccCols);
        uint8_t* st = (m0 + quad * 32 + 32 <= p.M) ? epi_stage[warp - 2] : nullptr;
        if (kMode != 0 && st != nullptr && n0 + kPairBN <= p.N) {
          // full tile: the next chunk's accumulator and operand are requested before this chunk is worked on
          const bool has_bias = kMode <= 2 && (p.epi & kEpiBias) != 0;
          const uint4* ext = kMode == 3
              ? reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(p.aux) +
                                               (long long)(m0 + quad * 32 + (lane >> 2)) * p.ldaux + n0) + (lane & 3)
              : reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(p.bias) + n0);
          const long long row0 = m0 + quad * 32 + out_row0;
          constexpr int kStep = kEpiWarps / 4, kChunks = kPairBN / 32 / kStep;
          uint32_t r[2][32];
          uint4 e[2][4];
#pragma unroll
          for (int i = 0; i < 4; ++i) e[0][i] = e[1][i] = make_uint4(0u, 0u, 0u, 0u);
          // a bias chunk is the same for every lane; four lanes fetch the 64 bytes of an aux row, eight rows at a time
          auto fetch = [&](int c, uint4 (&q)[4]) {
            if (kMode == 3) {
#pragma unroll
              for (int i = 0; i < 4; ++i)
                q[i] = __ldg(ext + (long long)(8 * i) * (p.ldaux >> 3) + c * 4);
            } else if (has_bias) {
#pragma unroll
              for (int i = 0; i < 4; ++i) q[i] = __ldg(ext + c * 4 + i);
            }
          };
          tmem_ld_32x32(t_row + (uint32_t)(chalf * 32), r[0]);
          fetch(chalf, e[0]);
#pragma unroll
          for (int j = 0; j < kChunks; ++j) {
            const int c = chalf + kStep * j;
            uint4(&q)[4] = e[j & 1];
            if (kMode == 3) {   // to one row per lane
#pragma unroll
              for (int i = 0; i < 4; ++i)
                *reinterpret_cast<uint4*>(st + stage_off(8 * i + (lane >> 2), lane & 3)) = q[i];
              __syncwarp();
#pragma unroll
              for (int i = 0; i < 4; ++i) q[i] = *reinterpret_cast<const uint4*>(st + stage_off(lane, i));
              __syncwarp();
            }
            tmem_ld_wait();
            if (j + 1 < kChunks) {
              tmem_ld_32x32(t_row + (uint32_t)((c + kStep) * 32), r[(j + 1) & 1]);
              fetch(c + kStep, e[(j + 1) & 1]);
            } else {
              // every column is in registers: the accumulator can be overwritten while they are worked on
              tc_fence_before();
              __syncwarp();
              if (lane == 0) mbar_arrive_cluster(tempty0 + (uint32_t)(acc * sizeof(uint64_t)));
            }
            epilogue_chunk_fixed<kMode == 5 ? 4 : kMode>(p, r[j & 1], has_bias, q, row0, n0 + c * 32, st, lane);
          }
          if (++acc == 2) { acc = 0; acc_ph ^= 1; }
          continue;
        }
        // The aux operand of the GELU' / add / multiply epilogues is requested one chunk ahead, so that
        // its latency hides behind the previous chunk instead of following every TMEM read.
        const bool has_aux = (p.epi & (kEpiDGelu | kEpiAddAux | kEpiMulAux)) != 0 && p.vec_ok && row < p.M;
        const __nv_bfloat16* aux_row =
            reinterpret_cast<const __nv_bfloat16*>(p.aux) + (long long)(row + out_row0) * p.ldaux;
        uint4 aq[4], aq_next[4];
        bool aq_ok = false, aq_next_ok = false;
#pragma unroll
        for (int i = 0; i < 4; ++i) aq_next[i] = make_uint4(0u, 0u, 0u, 0u);
        if (has_aux && n0 + chalf * 32 + 32 <= p.N) {
#pragma unroll
          for (int i = 0; i < 4; ++i)
            aq_next[i] = reinterpret_cast<const uint4*>(aux_row + n0 + chalf * 32)[i];
          aq_next_ok = true;
        }
        for (int c = chalf; c < kPairBN / 32; c += kEpiWarps / 4) {
          uint32_t r[32];
          tmem_ld_32x32(t_row + (uint32_t)(c * 32), r);
#pragma unroll
          for (int i = 0; i < 4; ++i) aq[i] = aq_next[i];
          aq_ok = aq_next_ok;
          aq_next_ok = false;
          const int ncol0 = n0 + (c + kEpiWarps / 4) * 32;
          if (has_aux && c + kEpiWarps / 4 < kPairBN / 32 && ncol0 + 32 <= p.N) {
#pragma unroll
            for (int i = 0; i < 4; ++i) aq_next[i] = reinterpret_cast<const uint4*>(aux_row + ncol0)[i];
            aq_next_ok = true;
          }
          tmem_ld_wait();
          const int col0 = n0 + c * 32;
          if (row < p.M && col0 < p.N) {
            if (p.epi & kEpiOutF32)
              epilogue_store_chunk<true>(p, r, row + out_row0, col0, nullptr, 0, aq_ok ? aq : nullptr);
            else
              epilogue_store_chunk<false>(p, r, row + out_row0, col0, st, lane, aq_ok ? aq : nullptr);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(tempty0 + (uint32_t)(acc * sizeof(uint64_t)));
        if (++acc == 2) { acc = 0; acc_ph ^= 1; }
      }
    }
  }

  // ---------------- teardown: neither CTA leaves (or frees TMEM) while its peer may still signal it
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  if (warp == 1) {
    __syncwarp();
    tmem_dealloc_pair(tmem_base, kTmemCols);
  }
}

// ---------------------------------------------------------------------------------------------
// Split kernel: 128 x 64 tiles whose contraction is cut over a cluster of S CTAs
// ---------------------------------------------------------------------------------------------
// For products with few output tiles (a handful of rows through a projection, short prompts). There the time is one
// CTA's walk along K, about 900 cycles for each 64-deep block (one SM's share of the L2 plus latency), while most SMs
// idle: 16 x 2304 x 768 takes 9.4 us on 18 CTAs, 113 x 768 x 3072 26.0 us on 6. Narrow tiles (500 cycles a block) and up
// to eight ranges of K put the operands' bytes on as many SMs as there are; the partial tiles meet in distributed shared
// memory, where CTA r of a cluster adds columns [64 r / S, 64 (r + 1) / S) over the ranks in order (the result does not
// depend on timing) and runs the epilogue on them: 7.3 us and 10.3 us (2 and 4 ranges of K; the rule that picks them, with
// every count's time, is the front end's).
constexpr int kSplitBN = 64, kSplitStages = 4, kSplitThreads = 192;
constexpr int kSplitStageBytes = kAStageBytes + kSplitBN * kGemmBK * 2;   // 24 KiB
constexpr int kSplitPitch = 68;                                          // floats; rows 16-byte aligned, conflict free

// Epilogue of eight consecutive columns of one row.
__device__ __forceinline__ void epilogue_cols8(const GemmParams& p, float (&v)[8], int row, int col0) {
  const int epi = p.epi;
  const bool full = p.vec_ok && col0 + 8 <= p.N;
  auto load8 = [&](const __nv_bfloat16* src, float (&x)[8]) {
    if (full) {
      const uint4 q = *reinterpret_cast<const uint4*>(src);
      const float2 f0 = unpack_bf16x2(q.x), f1 = unpack_bf16x2(q.y), f2 = unpack_bf16x2(q.z), f3 = unpack_bf16x2(q.w);
      x[0] = f0.x; x[1] = f0.y; x[2] = f1.x; x[3] = f1.y; x[4] = f2.x; x[5] = f2.y; x[6] = f3.x; x[7] = f3.y;
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) x[i] = (col0 + i < p.N) ? __bfloat162float(src[i]) : 0.f;
    }
  };
  auto store8 = [&](__nv_bfloat16* dst, const float (&x)[8]) {
    if (full) {
      *reinterpret_cast<uint4*>(dst) = make_uint4(pack_bf16x2(x[0], x[1]), pack_bf16x2(x[2], x[3]),
                                                  pack_bf16x2(x[4], x[5]), pack_bf16x2(x[6], x[7]));
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (col0 + i < p.N) dst[i] = __float2bfloat16(x[i]);
    }
  };
  float x[8];
  if (epi & kEpiBias) {
    load8(reinterpret_cast<const __nv_bfloat16*>(p.bias) + col0, x);
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] += x[i];
  }
  if (epi & kEpiGelu) {
    store8(reinterpret_cast<__nv_bfloat16*>(p.D2) + (long long)row * p.ldd2 + col0, v);
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = gelu_tanh(v[i]);
  }
  if (epi & kEpiSilu) {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = v[i] / (1.0f + __expf(-v[i]));
  }
  if (epi & (kEpiDGelu | kEpiAddAux | kEpiMulAux)) {
    load8(reinterpret_cast<const __nv_bfloat16*>(p.aux) + (long long)row * p.ldaux + col0, x);
#pragma unroll
    for (int i = 0; i < 8; ++i)
      v[i] = (epi & kEpiDGelu) ? v[i] * gelu_tanh_grad(x[i]) : (epi & kEpiMulAux) ? v[i] * x[i] : v[i] + x[i];
  }
  if (epi & kEpiRowScale) {
    const float sc = p.row_scale[row];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] *= sc;
  }
  if (epi & kEpiOutF32) {
    float* d = reinterpret_cast<float*>(p.D) + (long long)row * p.ldd + col0;
    if (full) {
      float4* d4 = reinterpret_cast<float4*>(d);
      if (epi & kEpiAccumulate) {
        const float4 a = d4[0], b = d4[1];
        v[0] += a.x; v[1] += a.y; v[2] += a.z; v[3] += a.w;
        v[4] += b.x; v[5] += b.y; v[6] += b.z; v[7] += b.w;
      }
      d4[0] = make_float4(v[0], v[1], v[2], v[3]);
      d4[1] = make_float4(v[4], v[5], v[6], v[7]);
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (col0 + i < p.N) d[i] = (epi & kEpiAccumulate) ? d[i] + v[i] : v[i];
    }
  } else {
    __nv_bfloat16* d = reinterpret_cast<__nv_bfloat16*>(p.D) + (long long)row * p.ldd + col0;
    if (epi & kEpiAccumulate) {
      load8(d, x);
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] += x[i];
    }
    store8(d, v);
  }
}

template <int S>
__global__ void __launch_bounds__(kSplitThreads)
gemm_bf16_split_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                       const GemmParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  __shared__ __align__(8) uint64_t full_bar[kSplitStages], empty_bar[kSplitStages], tfull_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = S > 1 ? (int)cluster_ctarank() : 0;
  const int num_m = (p.M + kGemmBM - 1) / kGemmBM;
  const int num_k = (p.K + kGemmBK - 1) / kGemmBK;
  const int tile = (int)blockIdx.x / S;
  const int n_tile = tile / num_m;
  const int m0 = (tile - n_tile * num_m) * kGemmBM, n0 = n_tile * kSplitBN;
  const int kb0 = rank * num_k / S, kb1 = (rank + 1) * num_k / S;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kSplitStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(&tfull_bar, 1);
    abort_flag = 0;
    mbar_fence_init();
    prefetch_tmap(&tmA);
    prefetch_tmap(&tmB);
  }
  if (warp == 1) {
    tmem_alloc(&tmem_slot, kSplitBN);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;
  pdl_wait();  // nothing above touched global memory
  pdl_trigger();

  uint32_t acc[kSplitBN];
  bool ok = true;
  if (warp == 0) {
    if (lane == 0) {
      for (int kb = kb0, i = 0; kb < kb1; ++kb, ++i) {
        const int s = i % kSplitStages;
        if (!mbar_wait(&empty_bar[s], ((i / kSplitStages) & 1) ^ 1, &abort_flag, p.status, kTimeoutEmpty, kb)) break;
        uint8_t* sA = smem + s * kSplitStageBytes;
        mbar_expect_tx(&full_bar[s], kSplitStageBytes);
        tma_load_2d(sA, &tmA, &full_bar[s], kb * kGemmBK, m0);
        if (!p.b_mn) tma_load_2d(sA + kAStageBytes, &tmB, &full_bar[s], kb * kGemmBK, n0);
        else tma_load_2d(sA + kAStageBytes, &tmB, &full_bar[s], n0, kb * kGemmBK);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    const uint32_t idesc = make_idesc_bf16(kGemmBM, kSplitBN, 0, p.b_mn);
    const uint32_t b_kstep = (p.b_mn ? 2048u : 32u) >> 4;
    const uint32_t a_lo0 = smem_desc_lo(smem_u32(smem), 16);
    const uint32_t b_lo0 = smem_desc_lo(smem_u32(smem) + (uint32_t)kAStageBytes, p.b_mn ? 8192u : 16u);
    for (int kb = kb0, i = 0; kb < kb1; ++kb, ++i) {
      const int s = i % kSplitStages;
      if (!mbar_wait_warp(&full_bar[s], (i / kSplitStages) & 1, &abort_flag, p.status, kTimeoutFull, kb)) break;
      tc_fence_after();
      if (elect_one()) {
        const uint32_t a_lo = a_lo0 + s * (kSplitStageBytes >> 4), b_lo = b_lo0 + s * (kSplitStageBytes >> 4);
#pragma unroll
        for (int k = 0; k < kGemmBK / 16; ++k)
          umma_bf16_ss(tmem_base, smem_desc(a_lo + k * 2), smem_desc(b_lo + k * b_kstep), idesc,
                       (i > 0 || k > 0) ? 1u : 0u);
        umma_commit(&empty_bar[s]);
        if (kb + 1 == kb1) umma_commit(&tfull_bar);
      }
      __syncwarp();
    }
  } else {
    const int quad = warp & 3;
    const int row = quad * 32 + lane;
    ok = mbar_wait_warp(&tfull_bar, 0, &abort_flag, p.status, kTimeoutTmemFull, tile);
    if (ok) {
      tc_fence_after();
      const uint32_t t_row = tmem_base + ((uint32_t)(quad * 32) << 16);
      tmem_ld_32x32(t_row, *reinterpret_cast<uint32_t(*)[32]>(&acc[0]));
      tmem_ld_32x32(t_row + 32, *reinterpret_cast<uint32_t(*)[32]>(&acc[32]));
      tmem_ld_wait();
      if (S == 1) {
        if (m0 + row < p.M) {
#pragma unroll
          for (int c = 0; c < kSplitBN; c += 8) {
            float v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(acc[c + i]);
            if (n0 + c < p.N) epilogue_cols8(p, v, m0 + row, n0 + c);
          }
        }
      } else {
        // every product of this CTA has completed: its stages are free for the partial tile
        float* red = reinterpret_cast<float*>(smem) + row * kSplitPitch;
#pragma unroll
        for (int c = 0; c < kSplitBN; c += 4)
          *reinterpret_cast<float4*>(red + c) = make_float4(__uint_as_float(acc[c]), __uint_as_float(acc[c + 1]),
                                                             __uint_as_float(acc[c + 2]), __uint_as_float(acc[c + 3]));
      }
    }
  }
  if (S > 1) {
    cluster_sync_all();
    if (warp >= 2) {
      constexpr int kCols = kSplitBN / S;
      const int row = (warp & 3) * 32 + lane;
      const int c0 = rank * kCols;
      float v[kCols];
#pragma unroll
      for (int i = 0; i < kCols; ++i) v[i] = 0.f;
      const uint32_t mine = smem_u32(smem) + (uint32_t)(row * kSplitPitch + c0) * 4u;
#pragma unroll
      for (int r = 0; r < S; ++r) {
        const uint32_t peer = mapa_shared(mine, (uint32_t)r);
#pragma unroll
        for (int i = 0; i < kCols; i += 4) {
          float4 q;
          asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                       : "=f"(q.x), "=f"(q.y), "=f"(q.z), "=f"(q.w)
                       : "r"(peer + i * 4u)
                       : "memory");
          v[i] += q.x; v[i + 1] += q.y; v[i + 2] += q.z; v[i + 3] += q.w;
        }
      }
      if (ok && m0 + row < p.M) {
#pragma unroll
        for (int c = 0; c < kCols; c += 8) {
          float u[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) u[i] = v[c + i];
          if (n0 + c0 + c < p.N) epilogue_cols8(p, u, m0 + row, n0 + c0 + c);
        }
      }
    }
    cluster_sync_all();  // no CTA leaves while a peer may still read its partial tile
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tmem_dealloc(tmem_base, kSplitBN);
  }
}

// ---------------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &qres) ==
            cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(f);
  });
  return fn;
}

// The driver call below needs the primary context to be current on the calling thread; threads
// that have only been handed a device ordinal (e.g. autograd workers) bind it on first use.
void ensure_context() {
  static thread_local bool ready = false;
  if (!ready) {
    cudaFree(0);
    ready = true;
  }
}

// 2-D bf16 tensor map: `inner` contiguous elements, `outer` rows `row_stride_elems` apart.
// A descriptor is a pure function of (address, extents, stride, box), and a training step asks for the
// same few hundred of them every iteration, so encoded maps are kept in a small per-thread
// direct-mapped cache instead of calling into the driver twice per GEMM launch.
struct TmapKey {
  const void* base;
  uint64_t inner, outer, stride;
  uint32_t box_inner, box_outer;
  bool operator==(const TmapKey& o) const {
    return base == o.base && inner == o.inner && outer == o.outer && stride == o.stride &&
           box_inner == o.box_inner && box_outer == o.box_outer;
  }
};
struct TmapSlot {
  TmapKey key;
  CUtensorMap map;
  bool used;
};
constexpr int kTmapCacheSlots = 1024;
constexpr uint32_t kPanelBox = 0xffffffffu;   // box_outer of a panel map: {64 columns, rows, panels}, box {64, 64, 2}

int make_tmap_bf16_2d(CUtensorMap* out, const void* base, uint64_t inner, uint64_t outer,
                      uint64_t row_stride_elems, uint32_t box_inner, uint32_t box_outer) {
  static thread_local TmapSlot* cache = nullptr;
  if (cache == nullptr) cache = new TmapSlot[kTmapCacheSlots]();
  const TmapKey key{base, inner, outer, row_stride_elems, box_inner, box_outer};
  uint64_t h = (uint64_t)(uintptr_t)base * 0x9E3779B97F4A7C15ull;
  h ^= (inner * 0xC2B2AE3D27D4EB4Full) ^ (outer * 0x165667B19E3779F9ull) ^ (row_stride_elems << 17) ^
       ((uint64_t)box_inner << 40) ^ ((uint64_t)box_outer << 48);
  TmapSlot& slot = cache[(h >> 20) & (kTmapCacheSlots - 1)];
  if (slot.used && slot.key == key) {
    *out = slot.map;
    return 0;
  }
  EncodeTiledFn fn = get_encode_fn();
  if (fn == nullptr) return -1;
  ensure_context();
  const bool panels = box_outer == kPanelBox;
  cuuint64_t dims[3] = {panels ? 64 : inner, outer, panels ? inner / 64 : 1};
  cuuint64_t strides[2] = {row_stride_elems * 2, 128};
  cuuint32_t box[3] = {box_inner, panels ? 64u : box_outer, 2};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, panels ? 3 : 2, const_cast<void*>(base), dims, strides,
                  box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return (int)r;
  slot.key = key;
  slot.map = *out;
  slot.used = true;
  return 0;
}

static int make_tmap_bf16_panels(CUtensorMap* out, const void* base, uint64_t inner, uint64_t outer,
                                 uint64_t row_stride_elems) {
  return make_tmap_bf16_2d(out, base, inner, outer, row_stride_elems, 64, kPanelBox);
}

static int g_sm_count = 0;
static int sm_count() {
  if (g_sm_count == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_sm_count, cudaDevAttrMultiProcessorCount, dev);
    if (g_sm_count <= 0) g_sm_count = 148;
  }
  return g_sm_count;
}

static bool g_attr_set = false;
static int g_max_dyn_smem = 0;

int launch_gemm(GemmParams& p, const void* A, long long lda, long long a_rows, const void* B,
                long long ldb, long long b_rows, int comm_ctas, cudaStream_t stream) {
  if (p.M <= 0 || p.N <= 0) return 0;
  if ((lda % 8) != 0 || (ldb % 8) != 0) return -2;
  {
    // 16-byte vector accesses in the epilogue need aligned bases and leading dimensions.
    const int out_elems = (p.epi & kEpiOutF32) ? 4 : 8;
    bool ok = (p.ldd % out_elems == 0) && (((uintptr_t)p.D & 15) == 0);
    if (p.epi & kEpiScatterPeers)
      for (int r = 0; r < p.world; ++r) ok = ok && (((uintptr_t)p.peer_D[r] & 15) == 0);
    if (p.epi & kEpiScatterPeers) ok = ok && (p.slot_stride % out_elems == 0);
    if (p.epi & kEpiBias) ok = ok && (((uintptr_t)p.bias & 15) == 0);
    if (p.epi & kEpiGelu) ok = ok && (p.ldd2 % 8 == 0) && (((uintptr_t)p.D2 & 15) == 0);
    if (p.epi & (kEpiDGelu | kEpiAddAux | kEpiMulAux))
      ok = ok && (p.ldaux % 8 == 0) && (((uintptr_t)p.aux & 15) == 0);
    p.vec_ok = ok ? 1 : 0;
  }
  if (((uintptr_t)A & 15) || ((uintptr_t)B & 15)) return -3;
  if (p.bn != 64 && p.bn != 128 && p.bn != 256) return -4;
  CUtensorMap tmA, tmB;
  int rc;
  // A: K-major [a_rows(M), K] or MN-major [a_rows(K), M]
  if (!p.a_mn)
    rc = make_tmap_bf16_2d(&tmA, A, (uint64_t)p.K, (uint64_t)a_rows, (uint64_t)lda, 64, 128);
  else
    rc = make_tmap_bf16_2d(&tmA, A, (uint64_t)p.M, (uint64_t)a_rows, (uint64_t)lda, 64, 64);
  if (rc) return rc;
  if (!p.b_mn)
    rc = make_tmap_bf16_2d(&tmB, B, (uint64_t)p.K, (uint64_t)b_rows, (uint64_t)ldb, 64,
                           (uint32_t)p.bn);
  else
    rc = make_tmap_bf16_2d(&tmB, B, (uint64_t)p.N, (uint64_t)b_rows, (uint64_t)ldb, 64, 64);
  if (rc) return rc;

  if (p.bm2 && p.tile_group != nullptr) return -5;
  const int stage_bytes = kAStageBytes * (p.bm2 ? 2 : 1) + p.bn * kGemmBK * 2;
  int stages = (200 * 1024) / stage_bytes;
  if (stages > kGemmMaxStages) stages = kGemmMaxStages;
  p.stages = stages;
  const int smem_bytes = stages * stage_bytes + 1024;
  if (!g_attr_set) {
    // static shared memory (barriers, the scatter staging) counts against the same 227 KB
    cudaFuncAttributes fa;
    cudaError_t e = cudaFuncGetAttributes(&fa, gemm_bf16_tcgen05_kernel);
    if (e != cudaSuccess) return (int)e;
    g_max_dyn_smem = 232448 - (int)fa.sharedSizeBytes;
    e = cudaFuncSetAttribute(gemm_bf16_tcgen05_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             g_max_dyn_smem);
    if (e != cudaSuccess) return (int)e;
    g_attr_set = true;
  }
  if (smem_bytes > g_max_dyn_smem) return -6;
  const int bm = kGemmBM * (p.bm2 ? 2 : 1);
  const int num_m = (p.M + bm - 1) / bm;
  const int num_n = (p.N + p.bn - 1) / p.bn;
  long long tiles = (long long)num_m * num_n;
  if (p.groups_k > 0) tiles *= p.groups_k;
  int gemm_ctas = sm_count() - comm_ctas;
  if (gemm_ctas < 1) gemm_ctas = 1;
  if (tiles < gemm_ctas) gemm_ctas = (int)tiles;
  p.gemm_ctas = gemm_ctas;
  if (comm_ctas == 0 && p.flag_mode == 0) {
    // plain product: set-up may overlap the previous kernel's tail
    cudaError_t e = launch_pdl(gemm_bf16_tcgen05_kernel, dim3(gemm_ctas), dim3(kThreads), (size_t)smem_bytes,
                               stream, tmA, tmB, p);
    return (int)(e != cudaSuccess ? e : cudaGetLastError());
  }
  // products fused with a collective wait on other ranks: ordinary stream order
  gemm_bf16_tcgen05_kernel<<<gemm_ctas + comm_ctas, kThreads, smem_bytes, stream>>>(tmA, tmB, p);
  return (int)cudaGetLastError();
}

// 16-byte vector accesses in the epilogue need aligned bases and leading dimensions.
static int epilogue_vec_ok(const GemmParams& p) {
  const int out_elems = (p.epi & kEpiOutF32) ? 4 : 8;
  bool ok = (p.ldd % out_elems == 0) && (((uintptr_t)p.D & 15) == 0);
  if (p.epi & kEpiBias) ok = ok && (((uintptr_t)p.bias & 15) == 0);
  if (p.epi & kEpiGelu) ok = ok && (p.ldd2 % 8 == 0) && (((uintptr_t)p.D2 & 15) == 0);
  if (p.epi & (kEpiDGelu | kEpiAddAux | kEpiMulAux)) ok = ok && (p.ldaux % 8 == 0) && (((uintptr_t)p.aux & 15) == 0);
  return ok ? 1 : 0;
}

// Split kernel launcher: plain products with K-major A. `splits`: 1, 2, 4 or 8 ranges of K, none of them empty (a CTA
// without a K block would commit no accumulator, and its peers would add a partial tile that was never written).
int launch_gemm_split(GemmParams& p, const void* A, long long lda, long long a_rows, const void* B, long long ldb,
                      long long b_rows, int splits, cudaStream_t stream) {
  if (p.M <= 0 || p.N <= 0) return 0;
  if ((lda % 8) != 0 || (ldb % 8) != 0) return -2;
  if (((uintptr_t)A & 15) || ((uintptr_t)B & 15)) return -3;
  if (p.a_mn || (p.epi & kEpiScatterPeers) || p.K <= 0) return -7;
  if (splits < 1 || splits > 8 || (splits & (splits - 1)) || splits > (p.K + kGemmBK - 1) / kGemmBK) return -4;
  p.vec_ok = epilogue_vec_ok(p);
  CUtensorMap tmA, tmB;
  int rc = make_tmap_bf16_2d(&tmA, A, (uint64_t)p.K, (uint64_t)a_rows, (uint64_t)lda, 64, 128);
  if (rc) return rc;
  if (!p.b_mn)
    rc = make_tmap_bf16_2d(&tmB, B, (uint64_t)p.K, (uint64_t)b_rows, (uint64_t)ldb, 64, kSplitBN);
  else
    rc = make_tmap_bf16_2d(&tmB, B, (uint64_t)p.N, (uint64_t)b_rows, (uint64_t)ldb, 64, 64);
  if (rc) return rc;
  const int smem_bytes = kSplitStages * kSplitStageBytes + 1024;
  typedef void (*SplitKernel)(CUtensorMap, CUtensorMap, GemmParams);
  SplitKernel kernel = splits == 1   ? &gemm_bf16_split_kernel<1>
                       : splits == 2 ? &gemm_bf16_split_kernel<2>
                       : splits == 4 ? &gemm_bf16_split_kernel<4>
                                     : &gemm_bf16_split_kernel<8>;
  static bool attr_set = false;
  if (!attr_set) {
    for (SplitKernel k : {&gemm_bf16_split_kernel<1>, &gemm_bf16_split_kernel<2>, &gemm_bf16_split_kernel<4>,
                          &gemm_bf16_split_kernel<8>}) {
      const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes);
      if (e != cudaSuccess) return (int)e;
    }
    attr_set = true;
  }
  const long long tiles = (long long)((p.M + kGemmBM - 1) / kGemmBM) * ((p.N + kSplitBN - 1) / kSplitBN);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(tiles * splits));
  cfg.blockDim = dim3(kSplitThreads);
  cfg.dynamicSmemBytes = (size_t)smem_bytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)splits;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, tmA, tmB, p);
  return (int)(e != cudaSuccess ? e : cudaGetLastError());
}

// Pair kernel launcher: plain products only (no flags, groups, gathered or scattered operands).
static int g_pair_max_dyn = 0;
static int g_pair_clusters = 0;

int launch_gemm_pair(GemmParams& p, const void* A, long long lda, long long a_rows, const void* B,
                     long long ldb, long long b_rows, cudaStream_t stream) {
  if (p.M <= 0 || p.N <= 0) return 0;
  if ((lda % 8) != 0 || (ldb % 8) != 0) return -2;
  if (p.epi & kEpiScatterPeers) return -7;
  p.vec_ok = epilogue_vec_ok(p);
  if (((uintptr_t)A & 15) || ((uintptr_t)B & 15)) return -3;
  p.bn = kPairBN;
  CUtensorMap tmA, tmB;
  int rc;
  // An MN-major operand whose width is a multiple of 64 is described as panels of 64 columns, so that one load brings
  // the two panels of a stage; other widths take a load for each (a panel map would run past the last row's end).
  p.a_panels = p.a_mn && p.M % 64 == 0;
  p.b_panels = p.b_mn && p.N % 64 == 0;
  if (!p.a_mn)
    rc = make_tmap_bf16_2d(&tmA, A, (uint64_t)p.K, (uint64_t)a_rows, (uint64_t)lda, 64, 128);
  else if (p.a_panels)
    rc = make_tmap_bf16_panels(&tmA, A, (uint64_t)p.M, (uint64_t)a_rows, (uint64_t)lda);
  else
    rc = make_tmap_bf16_2d(&tmA, A, (uint64_t)p.M, (uint64_t)a_rows, (uint64_t)lda, 64, 64);
  if (rc) return rc;
  if (!p.b_mn)
    rc = make_tmap_bf16_2d(&tmB, B, (uint64_t)p.K, (uint64_t)b_rows, (uint64_t)ldb, 64, kPairBN / 2);
  else if (p.b_panels)
    rc = make_tmap_bf16_panels(&tmB, B, (uint64_t)p.N, (uint64_t)b_rows, (uint64_t)ldb);
  else
    rc = make_tmap_bf16_2d(&tmB, B, (uint64_t)p.N, (uint64_t)b_rows, (uint64_t)ldb, 64, 64);
  if (rc) return rc;

  int stages = (200 * 1024) / kPairStageBytes;
  if (stages > kGemmMaxStages) stages = kGemmMaxStages;
  p.stages = stages;
  const int smem_bytes = stages * kPairStageBytes + 1024;
  if (g_pair_max_dyn == 0) {
    cudaFuncAttributes fa;
    typedef void (*PairKernel)(CUtensorMap, CUtensorMap, GemmParams);
    cudaError_t e = cudaFuncGetAttributes(&fa, gemm_bf16_pair_kernel<5>);
    if (e != cudaSuccess) return (int)e;
    const int max_dyn = 232448 - (int)fa.sharedSizeBytes;
    for (PairKernel k : {&gemm_bf16_pair_kernel<0>, &gemm_bf16_pair_kernel<1>, &gemm_bf16_pair_kernel<2>,
                         &gemm_bf16_pair_kernel<3>, &gemm_bf16_pair_kernel<4>, &gemm_bf16_pair_kernel<5>}) {
      e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, max_dyn);
      if (e != cudaSuccess) return (int)e;
    }
    // how many pairs the device holds at once (a persistent grid must not exceed it)
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * sm_count());
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = (size_t)smem_bytes;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = 2; at.val.clusterDim.y = 1; at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    int n = 0;
    e = cudaOccupancyMaxActiveClusters(&n, gemm_bf16_pair_kernel<0>, &cfg);
    if (e != cudaSuccess || n <= 0) { cudaGetLastError(); n = sm_count() / 2; }
    g_pair_clusters = n;
    g_pair_max_dyn = max_dyn;
  }
  if (smem_bytes > g_pair_max_dyn) return -6;
  const int num_m = (p.M + 2 * kGemmBM - 1) / (2 * kGemmBM);
  const int num_n = (p.N + kPairBN - 1) / kPairBN;
  long long tiles = (long long)num_m * num_n;
  if (p.groups_k > 0) tiles *= p.groups_k;
  int pairs = g_pair_clusters;
  if (tiles < pairs) pairs = (int)tiles;
  p.gemm_ctas = 2 * pairs;
  {
    // the epilogues of the main path are compiled on their own (vector access throughout, ordinary output)
    auto* kernel = &gemm_bf16_pair_kernel<0>;
    if (p.vec_ok && p.groups_k == 0) {
      if ((p.epi & ~kEpiBias) == 0) kernel = &gemm_bf16_pair_kernel<1>;
      else if ((p.epi & ~kEpiBias) == kEpiGelu) kernel = &gemm_bf16_pair_kernel<2>;
      else if (p.epi == kEpiDGelu) kernel = &gemm_bf16_pair_kernel<3>;
    }
    // the slabs of a split weight gradient: one tile to a CTA, so that nothing hides its epilogue
    if (p.vec_ok && p.epi == kEpiOutF32) kernel = &gemm_bf16_pair_kernel<4>;
    if (p.bias_part != nullptr) {
      if (!p.vec_ok || !p.a_panels || p.epi != kEpiOutF32) return -8;
      kernel = &gemm_bf16_pair_kernel<5>;
    }
    cudaError_t e = launch_pdl(kernel, dim3(2 * pairs), dim3(kThreads), (size_t)smem_bytes, stream, tmA, tmB, p);
    if (e != cudaSuccess) return (int)e;
  }
  return (int)cudaGetLastError();
}

}  // namespace mmj

using namespace mmj;

// Number of CTA pairs the device holds at once for the pair kernel (0 before its first launch).
MMJ_API int mmj_gemm_pair_clusters() { return g_pair_clusters; }

// Plain / fused-epilogue GEMM.
//   a_mn = 0: A is [M, K] row-major (lda);  a_mn = 1: A is [K, M] row-major (lda)
//   b_mn = 0: B is [N, K] row-major (ldb);  b_mn = 1: B is [K, N] row-major (ldb)
//   D[M, N] (ldd) = A_op * B_op^T-style contraction over K, then the epilogue flags in `epi`.
MMJ_API int mmj_gemm_bf16(const void* A, long long lda, int a_mn, const void* B, long long ldb,
                          int b_mn, void* D, long long ldd, int M, int N, int K, int epi,
                          const void* bias, const void* aux, long long ldaux, void* D2,
                          long long ldd2, const float* row_scale, int bn, int* status,
                          void* stream) {
  GemmParams p = {};
  p.M = M; p.N = N; p.K = K;
  p.a_mn = a_mn; p.b_mn = b_mn;
  p.bn = bn & 0xfff;          // bit 12 of `bn` asks for 256-row tiles
  p.bm2 = (bn >> 12) & 1;
  p.epi = epi;
  p.D = D; p.ldd = ldd;
  p.D2 = D2; p.ldd2 = ldd2;
  p.bias = bias; p.aux = aux; p.ldaux = ldaux;
  p.row_scale = row_scale;
  p.status = status;
  if ((bn >> 14) & 1)  // bit 14 of `bn`: 128 x 64 tiles, K cut into (bn >> 16) ranges over a cluster
    return launch_gemm_split(p, A, lda, a_mn ? K : M, B, ldb, b_mn ? K : N, bn >> 16, (cudaStream_t)stream);
  if ((bn >> 13) & 1)  // bit 13 of `bn`: CTA-pair kernel, 256 x 256 tiles
    return launch_gemm_pair(p, A, lda, a_mn ? K : M, B, ldb, b_mn ? K : N, (cudaStream_t)stream);
  return launch_gemm(p, A, lda, a_mn ? K : M, B, ldb, b_mn ? K : N, 0, (cudaStream_t)stream);
}

// Grouped GEMM for MoE experts: rows of A are sorted by expert and every expert's segment
// starts on a 128-row boundary. tile_group[m_tile] names the expert of each row tile;
// num_m_tiles_dev (device int) is the number of row tiles in use. B holds `groups` weight
// matrices stacked along its row dimension, b_group_rows rows each.
MMJ_API int mmj_gemm_bf16_grouped(const void* A, long long lda, const void* B, long long ldb,
                                  int b_mn, int groups, int b_group_rows, void* D, long long ldd,
                                  int M_cap, int N, int K, int epi, const void* aux,
                                  long long ldaux, const float* row_scale, const int* tile_group,
                                  const int* num_m_tiles_dev, int bn, int* status, void* stream) {
  GemmParams p = {};
  p.M = M_cap; p.N = N; p.K = K;
  p.a_mn = 0; p.b_mn = b_mn;
  p.bn = bn;
  p.epi = epi;
  p.D = D; p.ldd = ldd;
  p.aux = aux; p.ldaux = ldaux;
  p.row_scale = row_scale;
  p.status = status;
  p.tile_group = tile_group;
  p.b_group_rows = b_group_rows;
  p.num_m_tiles_dev = num_m_tiles_dev;
  return launch_gemm(p, A, lda, M_cap, B, ldb, (long long)groups * b_group_rows, 0,
                     (cudaStream_t)stream);
}

// All-gather fused into the GEMM. One operand (A when gather_a != 0, else B) is the
// concatenation along rows of `world` equal shards that live on different GPUs.
// `gathered` is the local full-size buffer (the GEMM reads it through TMA); comm CTAs copy
// each peer shard from peer_src[r] into it in `granule_rows`-row pieces (128 for A, bn for B)
// and publish flags[piece] = epoch, which the TMA producer waits on (bounded). peer_ready
// (may be null) is the local signal pad where rank r stores `epoch` once its shard is final.
MMJ_API int mmj_gemm_bf16_allgather(const void* const* peer_src, void* gathered, int gather_a,
                                    const void* other, long long ld_gathered, long long ld_other,
                                    int other_mn, void* D, long long ldd, int M, int N, int K,
                                    int epi, const void* bias, const void* aux, long long ldaux,
                                    void* D2, long long ldd2, int bn, int world, int rank,
                                    long long shard_bytes, long long flat_off_bytes,
                                    int* flags, const int* peer_ready, int epoch, int comm_ctas,
                                    int* status, void* stream) {
  if (world < 1 || world > kMaxPeers) return -5;
  GemmParams p = {};
  p.src_compact = (gather_a >> 1) & 1;   // bit 1 of gather_a: peers keep compact shards
  gather_a &= 1;
  p.M = M; p.N = N; p.K = K;
  p.bn = bn & 0xfff;          // bit 12 of `bn` asks for 256-row tiles
  p.bm2 = (bn >> 12) & 1;
  bn = p.bn;
  p.epi = epi;
  p.D = D; p.ldd = ldd;
  p.D2 = D2; p.ldd2 = ldd2;
  p.bias = bias; p.aux = aux; p.ldaux = ldaux;
  p.status = status;
  p.world = world; p.rank = rank;
  p.ready_flags = flags; p.flags_rw = flags;
  p.peer_ready = peer_ready;
  p.ready_epoch = epoch;
  p.gather_dst = gathered;
  for (int r = 0; r < world; ++r) p.peer_src[r] = peer_src[r];
  const long long rows = gather_a ? M : N;
  const int granule = gather_a ? kGemmBM : bn;
  p.tile_bytes = (long long)granule * ld_gathered * 2;
  p.gather_total_bytes = rows * ld_gathered * 2;
  p.gather_flat_off = flat_off_bytes;
  p.shard_bytes = shard_bytes;
  if (shard_bytes <= 0 || (shard_bytes & 15) || (flat_off_bytes & 15)) return -6;
  // first tile that holds local data (if any) is visited first
  long long first_local = (long long)rank * shard_bytes - flat_off_bytes;
  if (first_local < 0) first_local = 0;
  int rot_tile = 0;
  if (first_local < p.gather_total_bytes) rot_tile = (int)((first_local + p.tile_bytes - 1) / p.tile_bytes);
  const int ntiles_g = (int)((p.gather_total_bytes + p.tile_bytes - 1) / p.tile_bytes);
  if (rot_tile >= ntiles_g) rot_tile = 0;
  if (gather_a) {
    p.flag_mode = 1;
    p.a_mn = 0; p.b_mn = other_mn;
    p.comm_rot = rot_tile;
    p.m_tile_rot = p.bm2 ? rot_tile / 2 : rot_tile;
    return launch_gemm(p, gathered, ld_gathered, M, other, ld_other, other_mn ? K : N, comm_ctas,
                       (cudaStream_t)stream);
  } else {
    p.flag_mode = 2;
    p.a_mn = other_mn; p.b_mn = 0;
    p.comm_rot = rot_tile;
    p.n_tile_rot = rot_tile;
    return launch_gemm(p, other, ld_other, other_mn ? K : M, gathered, ld_gathered, N, comm_ctas,
                       (cudaStream_t)stream);
  }
}

// GEMM whose result is reduce-scattered over rows: rank `rank` computes a partial D[M, N];
// rows [r*M/world, (r+1)*M/world) are stored into rank r's staging buffer peer_stage[r] at
// slot `rank` (slot_stride elements apart). Each owner later sums its `world` slots
// (mmj_reduce_slots_bf16). Rows are visited starting after the local block so that ranks
// write to different owners at the same time.
MMJ_API int mmj_gemm_bf16_reduce_scatter(const void* A, long long lda, const void* B,
                                         long long ldb, int b_mn, void* const* peer_stage,
                                         long long ldd, long long slot_stride, int M, int N, int K,
                                         int bn, int world, int rank, int* status, void* stream) {
  if (world < 1 || world > kMaxPeers) return -5;
  if (M % world) return -6;
  GemmParams p = {};
  p.M = M; p.N = N; p.K = K;
  p.a_mn = 0; p.b_mn = b_mn;
  p.bn = bn & 0xfff;          // bit 12 of `bn` asks for 256-row tiles
  p.bm2 = (bn >> 12) & 1;
  p.epi = kEpiScatterPeers;
  p.ldd = ldd;
  p.status = status;
  p.world = world; p.rank = rank;
  p.rows_per_rank = M / world;
  p.slot_stride = slot_stride;
  for (int r = 0; r < world; ++r) p.peer_D[r] = peer_stage[r];
  p.D = peer_stage[rank];
  const int bm = kGemmBM * (p.bm2 ? 2 : 1);
  const int num_m = (M + bm - 1) / bm;
  p.m_tile_rot = (int)(((long long)(rank + 1) % world) * p.rows_per_rank / bm) % num_m;
  return launch_gemm(p, A, lda, M, B, ldb, b_mn ? K : N, 0, (cudaStream_t)stream);
}

// Grouped-K GEMM for expert weight gradients: for every group g,
//   D[g][M, N] = sum over rows k in [group_k[2g], group_k[2g+1]) of A[k, :M]^T B[k, :N]
// with A: [rows, M] and B: [rows, N] row-major (both MN-major operands; rows outside every range
// are never read, rows inside a range that hold no token must be zero). D is [groups, M, N].
// Weight gradient cut into `splits` ranges of the contraction, on CTA pairs: fp32 slabs [splits, M, N] of dy^T x and the
// column sums of dy [splits, M]. dy: [rows, M] (M % 64 == 0), x: [rows, N]; mmj_wgrad_fold adds both up.
MMJ_API int mmj_wgrad_bias(const void* dy, long long lddy, const void* x, long long ldx, float* slabs, float* bias_part,
                           int rows, int M, int N, int splits, const int* ranges_dev, int* status, void* stream) {
  GemmParams p = {};
  p.M = M; p.N = N; p.K = rows;
  p.a_mn = 1; p.b_mn = 1;
  p.epi = kEpiOutF32;
  p.D = slabs; p.ldd = N;
  p.bias_part = bias_part;
  p.status = status;
  p.groups_k = splits;
  p.group_k = ranges_dev;
  return launch_gemm_pair(p, dy, lddy, rows, x, ldx, rows, (cudaStream_t)stream);
}

MMJ_API int mmj_gemm_bf16_grouped_k(const void* A, long long lda, const void* B, long long ldb,
                                    void* D, long long ldd, int rows, int M, int N, int groups,
                                    const int* group_k_dev, int out_f32, int accumulate, int bn,
                                    int* status, void* stream) {
  GemmParams p = {};
  p.M = M; p.N = N; p.K = rows;
  p.a_mn = 1; p.b_mn = 1;
  p.bn = bn & 0xfff;          // bit 12 of `bn` asks for 256-row tiles
  p.bm2 = (bn >> 12) & 1;
  p.epi = (out_f32 ? kEpiOutF32 : 0) | (accumulate ? kEpiAccumulate : 0);
  p.D = D; p.ldd = ldd;
  p.status = status;
  p.groups_k = groups;
  p.group_k = group_k_dev;
  if ((bn >> 13) & 1)  // CTA-pair kernel
    return launch_gemm_pair(p, A, lda, rows, B, ldb, rows, (cudaStream_t)stream);
  return launch_gemm(p, A, lda, rows, B, ldb, rows, 0, (cudaStream_t)stream);
}
