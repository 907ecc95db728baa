// Flash attention for sm_100a on the 5th-generation tensor cores.
//
// S = Q K^T and O += P V are tcgen05.mma instructions issued by one thread; S and O live in tensor memory, Q/K/V tiles are
// brought into 128-byte-swizzled shared memory by TMA. The running maximum is only refreshed when it grew by more than 2^8, so
// the O accumulator is rescaled rarely. Forward of more than 128 query rows: flash_fwd2_kernel, two query tiles a CTA, P in tensor
// memory. Up to 128 rows: flash_fwd_kernel, one tile a CTA, two S buffers, P through shared memory as the A operand of the second
// product; warp 0 TMA producer, warp 1 MMA issuer + TMEM owner, warps 2-9 softmax (two threads per query row, each reading half of it
// from TMEM with tcgen05.ld).
//
// Inputs are packed variable-length batches (`cu_seqlens`), grouped-query heads, causal and
// sliding-window masks; K/V come either from dense [T, Hkv, D] tensors (training) or from the paged
// cache [num_blocks, Hkv, 16, D] through a block table (prefill with a cached prefix).
//
// Replaces F.scaled_dot_product_attention / FlexAttention in the reference
// (rollouts/inference/attention/flex_backend.py:144-185) and the Hopper-only varlen flash kernel of
// dev/speedrun/single-file.py:932-943.
//
// Every wait is bounded; on a timeout the kernel records a status code, drains its copies, frees
// tensor memory and returns.
#include "common.cuh"
#include "tma_host.h"

#include <math.h>
#include <stdlib.h>

namespace rb {

constexpr int FA_BM = 128;        // query rows per CTA
constexpr int FA_BN = 128;        // keys per iteration
constexpr int FA_THREADS = 320;   // 10 warps: TMA, MMA, two softmax warpgroups
constexpr int FA_KV_SLOTS = 3;    // ring of K/V tiles in consumption order: K0 K1 V0 K2 V1 K3 V2 ...
constexpr int FA_TMEM_COLS = 512;
constexpr float FA_RESCALE_THRESHOLD = 8.f;   // log2 units

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Wait for the single-thread producer / MMA roles. `mbarrier.try_wait` with a suspend-time hint parks the thread in
// hardware until the phase completes or the hint runs out: the waiter takes no issue slots from the softmax warps
// on its scheduler (what a plain poll loop did) and wakes as soon as the barrier flips (what a poll + nanosleep
// loop did not: at short sequences every hand-off on the critical path paid a sleep quantum).
__device__ __forceinline__ bool mbar_try_wait_hint(uint32_t bar, uint32_t parity, uint32_t hint_ns) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred P;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, P;\n\t}"
      : "=r"(done)
      : "r"(bar), "r"(parity), "r"(hint_ns)
      : "memory");
  return done != 0;
}
__device__ __forceinline__ bool mbar_wait_backoff(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* status,
                                                  int code) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = globaltimer_ns();
  uint32_t spins = 0;
  while (true) {
    if (mbar_try_wait_hint(bar, parity, 2000u)) return true;
    if ((++spins & 0x3f) == 0) {
      if (*abort_flag != 0) return false;
      if (globaltimer_ns() - t0 > RB_WAIT_BUDGET_NS) {
        *abort_flag = 1;
        set_status(status, code);
        return false;
      }
    }
  }
}

struct FlashFwdParams {
  CUtensorMap q_map;   // [Tq, Hq*D], box 64 x 128
  CUtensorMap k_map;   // dense: [Tk, Hkv*D], box 64 x 128; paged: [num_blocks*Hkv*16, D], box 64 x 16
  CUtensorMap v_map;
  __nv_bfloat16* out;  // [Tq, Hq, D]
  float* lse;          // [Hq, Tq] natural-log sum-exp of the scaled scores
  const int* cu_q;     // [B+1]
  const int* cu_k;     // [B+1] (dense)
  const int* seq_lens; // [B] total keys per sequence (paged)
  const int* block_tables;  // [B, max_blocks] (paged)
  int max_blocks, num_blocks;
  int Hq, Hkv, Tq;
  int causal, window, chunk, paged;     // window: the last so many keys; chunk: keys of the query's own run of so many positions (0: none)
  const float* gate;   // [Tq, ld_gate] or null: a head's output is multiplied by gate_scale * sigmoid(gate)
  long long ld_gate, ldo;
  float gate_scale;
  float scale_log2;
  int* status;
};

// First key the query at position i sees.
__device__ __forceinline__ int flash_first_key(const FlashFwdParams& p, int i) {
  if (p.window > 0) return max(0, i - p.window + 1);
  return p.chunk > 0 ? i - i % p.chunk : 0;
}
__device__ __forceinline__ float flash_gate(const FlashFwdParams& p, long long row, int h) {
  return p.gate != nullptr ? p.gate_scale / (1.f + __expf(-p.gate[row * p.ld_gate + h])) : 1.f;
}

template <int D>
struct FlashCfg {
  static constexpr int kTileBytes = FA_BN * D * 2;          // one K or V tile (and the Q tile)
  static constexpr int kPBytes = FA_BM * FA_BN * 2;
  static constexpr int kSmemBytes = 1024 + kTileBytes + FA_KV_SLOTS * kTileBytes + 2 * kPBytes;
};

template <int D>
__global__ void __launch_bounds__(FA_THREADS, 1) flash_fwd_kernel(const __grid_constant__ FlashFwdParams p) {
  using Cfg = FlashCfg<D>;
  constexpr int DCH = D / 64;                    // 64-column chunks of the head dimension
  constexpr int CHUNK_BYTES = FA_BN * 128;       // 128 rows x 128 B
  extern __shared__ __align__(128) uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t q_full, kv_full[FA_KV_SLOTS], kv_empty[FA_KV_SLOTS];
  __shared__ __align__(8) uint64_t s_full[2], s_empty[2], p_full[2], p_empty[2], o_done, xch_bar[4];
  __shared__ float xch[2][2][FA_BM];
  __shared__ uint32_t tmem_base_smem;
  __shared__ int abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int b = blockIdx.z, h = blockIdx.y;
  const int q_tile = gridDim.x - 1 - blockIdx.x;           // long (late) tiles first
  const int q_begin = p.cu_q[b];
  const int q_len = p.cu_q[b + 1] - q_begin;
  const int q0 = q_tile * FA_BM;
  if (q0 >= q_len) return;                                  // uniform per CTA, before any set-up
  const int kv_len = p.paged ? p.seq_lens[b] : (p.cu_k[b + 1] - p.cu_k[b]);
  const int k_begin = p.paged ? 0 : p.cu_k[b];
  const int off = kv_len - q_len;                           // key position of query 0
  const int kvh = h / (p.Hq / p.Hkv);
  // keys this tile can see
  int hi = p.causal ? min(kv_len, off + q0 + FA_BM) : kv_len;
  const int lo = flash_first_key(p, off + q0);
  const int t_begin = lo / FA_BN;
  const int t_end = (hi + FA_BN - 1) / FA_BN;
  const int n_tiles = max(t_end - t_begin, 0);

  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_al = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t q_s = smem_base;
  const uint32_t kv_s = q_s + Cfg::kTileBytes;
  const uint32_t p_s = kv_s + FA_KV_SLOTS * Cfg::kTileBytes;
  uint8_t* p_ptr = smem_al + Cfg::kTileBytes + FA_KV_SLOTS * Cfg::kTileBytes;

  if (threadIdx.x == 0) {
    abort_flag = 0;
    mbar_init(smem_u32(&q_full), 1);
    for (int i = 0; i < FA_KV_SLOTS; ++i) {
      mbar_init(smem_u32(&kv_full[i]), 1);
      mbar_init(smem_u32(&kv_empty[i]), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&s_full[i]), 1);
      mbar_init(smem_u32(&s_empty[i]), 8);
      mbar_init(smem_u32(&p_full[i]), 8);
      mbar_init(smem_u32(&p_empty[i]), 1);
    }
    for (int i = 0; i < 4; ++i) mbar_init(smem_u32(&xch_bar[i]), 64);
    mbar_init(smem_u32(&o_done), 1);
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&tmem_base_smem), FA_TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_smem;
  const uint32_t tmem_o = tmem_base + 2 * FA_BN;
  volatile int* abortp = &abort_flag;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one_sync()) {
      bool ok = true;
      mbar_expect_tx(smem_u32(&q_full), Cfg::kTileBytes);
#pragma unroll
      for (int c = 0; c < DCH; ++c)
        tma_load_2d(q_s + c * CHUNK_BYTES, &p.q_map, smem_u32(&q_full), h * D + c * 64, q_begin + q0);
      uint32_t it = 0;
      // tiles are loaded in the order the MMA warp consumes them: K0, then (K_{j+1}, V_j) for every j
      auto load_tile = [&](int j, int which) -> bool {   // which 0: K tile, 1: V tile
        const int k0 = (t_begin + j) * FA_BN;
        const int slot = it % FA_KV_SLOTS;
        if (!mbar_wait_backoff(smem_u32(&kv_empty[slot]), ((it / FA_KV_SLOTS) & 1u) ^ 1u, abortp, p.status,
                               ST_TIMEOUT_SMEM_EMPTY))
          return false;
        const uint32_t fb = smem_u32(&kv_full[slot]);
        const uint32_t dst = kv_s + slot * Cfg::kTileBytes;
        const CUtensorMap* map = which == 0 ? &p.k_map : &p.v_map;
        mbar_expect_tx(fb, Cfg::kTileBytes);
        if (!p.paged) {
#pragma unroll
          for (int c = 0; c < DCH; ++c) tma_load_2d(dst + c * CHUNK_BYTES, map, fb, kvh * D + c * 64, k_begin + k0);
        } else {
          const int* bt = p.block_tables + (long long)b * p.max_blocks;
          const int n_blk = (kv_len + 15) >> 4;
#pragma unroll 1
          for (int i = 0; i < FA_BN / 16; ++i) {
            const int bi = (k0 >> 4) + i;
            int blk = p.num_blocks;                         // out of range: the copy fills zeros
            if (bi < n_blk) {
              blk = bt[bi];
              if (blk < 0 || blk >= p.num_blocks) { set_status(p.status, ST_BAD_INDEX); blk = p.num_blocks; }
            }
            const int y = (blk * p.Hkv + kvh) * 16;
#pragma unroll
            for (int c = 0; c < DCH; ++c) tma_load_2d(dst + c * CHUNK_BYTES + i * 2048, map, fb, c * 64, y);
          }
        }
        ++it;
        return true;
      };
      if (n_tiles > 0) ok = load_tile(0, 0);
      for (int j = 0; j < n_tiles && ok; ++j) {
        if (j + 1 < n_tiles) { ok = load_tile(j + 1, 0); if (!ok) break; }
        ok = load_tile(j, 1);
      }
      if (!ok) {   // drain: no bulk copy may land after the CTA has gone
        const uint32_t first = it > (uint32_t)FA_KV_SLOTS ? it - FA_KV_SLOTS : 0;
        for (uint32_t j = first; j < it; ++j) {
          const uint64_t t0 = globaltimer_ns();
          while (!mbar_try_wait(smem_u32(&kv_full[j % FA_KV_SLOTS]), (j / FA_KV_SLOTS) & 1u))
            if (globaltimer_ns() - t0 > 50000000ull) break;
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one_sync()) {
      constexpr uint32_t idesc_s = make_idesc_bf16(FA_BM, FA_BN, 0, 0);   // Q, K both K-major
      constexpr uint32_t idesc_o = make_idesc_bf16(FA_BM, D, 0, 1);       // P K-major, V MN-major
      bool ok = mbar_wait_backoff(smem_u32(&q_full), 0, abortp, p.status, ST_TIMEOUT_SMEM_FULL);
      uint32_t it = 0;   // tiles consumed so far, in the producer's order
      auto issue_s = [&](int j) -> bool {
        const int slot = it % FA_KV_SLOTS;
        if (!mbar_wait_backoff(smem_u32(&kv_full[slot]), (it / FA_KV_SLOTS) & 1u, abortp, p.status, ST_TIMEOUT_SMEM_FULL))
          return false;
        if (!mbar_wait_backoff(smem_u32(&s_empty[j & 1]), ((j >> 1) & 1u) ^ 1u, abortp, p.status, ST_TIMEOUT_TMEM_EMPTY))
          return false;
        tc_fence_after();
        const uint32_t ks = kv_s + slot * Cfg::kTileBytes;
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          const uint64_t adesc = make_smem_desc_sw128(q_s + (k >> 2) * CHUNK_BYTES + (k & 3) * 32, 16, 1024);
          const uint64_t bdesc = make_smem_desc_sw128(ks + (k >> 2) * CHUNK_BYTES + (k & 3) * 32, 16, 1024);
          umma_bf16(tmem_base + (j & 1) * FA_BN, adesc, bdesc, idesc_s, k > 0 ? 1u : 0u);
        }
        umma_commit(smem_u32(&kv_empty[slot]));
        umma_commit(smem_u32(&s_full[j & 1]));
        ++it;
        return true;
      };
      if (ok && n_tiles > 0) ok = issue_s(0);
      for (int j = 0; j < n_tiles && ok; ++j) {
        if (j + 1 < n_tiles) { ok = issue_s(j + 1); if (!ok) break; }
        const int slot = it % FA_KV_SLOTS;
        ok = mbar_wait_backoff(smem_u32(&p_full[j & 1]), (j >> 1) & 1u, abortp, p.status, ST_TIMEOUT_TMEM_FULL);
        if (!ok) break;
        ok = mbar_wait_backoff(smem_u32(&kv_full[slot]), (it / FA_KV_SLOTS) & 1u, abortp, p.status, ST_TIMEOUT_SMEM_FULL);
        if (!ok) break;
        tc_fence_after();
        const uint32_t vs = kv_s + slot * Cfg::kTileBytes;
        const uint32_t ps = p_s + (j & 1) * Cfg::kPBytes;
#pragma unroll
        for (int k = 0; k < FA_BN / 16; ++k) {
          const uint64_t adesc = make_smem_desc_sw128(ps + (k >> 2) * CHUNK_BYTES + (k & 3) * 32, 16, 1024);
          const uint64_t bdesc = make_smem_desc_sw128(vs + k * 2048, CHUNK_BYTES, 1024);
          umma_bf16(tmem_o, adesc, bdesc, idesc_o, (j > 0 || k > 0) ? 1u : 0u);
        }
        umma_commit(smem_u32(&kv_empty[slot]));
        umma_commit(smem_u32(&p_empty[j & 1]));
        umma_commit(smem_u32(&o_done));
        ++it;
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax + epilogue
    // Two warpgroups (warps 2-5 and 6-9) share the 128 rows: `half` owns 64 of the 128 score columns
    // of a row, half of the O columns and one 64-column chunk of P. The two threads of a row swap
    // their partial row maximum (and, at the end, their partial row sum) through shared memory.
    constexpr int HC = FA_BN / 2;                // score columns per thread
    const int qd = warp & 3;                     // TMEM lane quarter of this warp
    const int half = (warp - 2) >> 2;
    const int r = qd * 32 + lane;                // query row inside the tile
    const uint32_t lane_addr = (uint32_t)(qd * 32) << 16;
    const int qpos = off + q0 + r;               // key position of this query
    const int k_first = flash_first_key(p, qpos), last_first = flash_first_key(p, off + q0 + FA_BM - 1);
    float m_used = -INFINITY, l = 0.f;
    bool ok = true;
    uint32_t xph = 0;                            // phase of the pair barrier
    auto swap_with_partner = [&](float mine, float& other) -> bool {
      xch[xph & 1][half][r] = mine;
      mbar_arrive(smem_u32(&xch_bar[qd]));
      bool good = mbar_wait_backoff(smem_u32(&xch_bar[qd]), xph & 1u, abortp, p.status, ST_TIMEOUT_TMEM_FULL);
      other = xch[xph & 1][half ^ 1][r];
      ++xph;
      return __all_sync(0xffffffffu, good);
    };
    for (int j = 0; j < n_tiles; ++j) {
      const int k0 = (t_begin + j) * FA_BN;
      const uint32_t s_addr = tmem_base + (j & 1) * FA_BN + half * HC + lane_addr;
      ok = mbar_wait_backoff(smem_u32(&s_full[j & 1]), (j >> 1) & 1u, abortp, p.status, ST_TIMEOUT_TMEM_FULL);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const bool need_mask = (k0 + FA_BN > kv_len) || (p.causal && k0 + FA_BN - 1 > off + q0) ||
                             k0 < last_first;
      // this thread's 64 score columns go to registers with one wait; then the S buffer is free again
      uint32_t v[HC];
#pragma unroll
      for (int c = 0; c < HC / 32; ++c)
        tmem_ld_32x32(s_addr + c * 32, *reinterpret_cast<uint32_t(*)[32]>(&v[c * 32]));
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&s_empty[j & 1]));
      if (need_mask) {
#pragma unroll
        for (int i = 0; i < HC; ++i) {
          const int kj = k0 + half * HC + i;
          const bool dead = kj >= kv_len || (p.causal && kj > qpos) || kj < k_first;
          if (dead) v[i] = 0xff800000u;   // -inf
        }
      }
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < HC; i += 4) {
        mx[0] = fmaxf(mx[0], __uint_as_float(v[i]));
        mx[1] = fmaxf(mx[1], __uint_as_float(v[i + 1]));
        mx[2] = fmaxf(mx[2], __uint_as_float(v[i + 2]));
        mx[3] = fmaxf(mx[3], __uint_as_float(v[i + 3]));
      }
      const float mine = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
      float other;
      ok = swap_with_partner(mine, other);
      if (!ok) break;
      const float m_new = fmaxf(m_used, fmaxf(mine, other) * p.scale_log2);
      const bool need = m_new > m_used + FA_RESCALE_THRESHOLD || (m_used == -INFINITY && m_new != -INFINITY);
      if (__any_sync(0xffffffffu, need)) {   // same rows, same inputs: both warps of a quarter agree
        if (j > 0) {
          // O holds the products of tiles 0..j-1 once the previous P V has completed
          ok = mbar_wait_backoff(smem_u32(&o_done), (uint32_t)((j - 1) & 1), abortp, p.status, ST_TIMEOUT_TMEM_FULL);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          tc_fence_after();
          const float alpha = need ? fast_exp2((m_used == -INFINITY ? m_new : m_used) - m_new) : 1.f;
#pragma unroll 1
          for (int c = half * (D / 64); c < (half + 1) * (D / 64); ++c) {
            uint32_t o[32];
            tmem_ld_32x32(tmem_o + lane_addr + c * 32, o);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
            tmem_st_32x32(tmem_o + lane_addr + c * 32, o);
          }
          tmem_st_wait();
          l *= alpha;
        }
        if (need) m_used = m_new;
      }
      const float mref = m_used == -INFINITY ? 0.f : m_used;
      // P = exp2(S * scale - m): a masked score is -inf and gives exactly 0
      float ls[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int i = 0; i < HC; i += 4) {
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const float x = fast_exp2(fmaf(__uint_as_float(v[i + t]), p.scale_log2, -mref));
          ls[t] += x;
          v[i + t] = __float_as_uint(x);
        }
      }
      l += (ls[0] + ls[1]) + (ls[2] + ls[3]);
      // bf16 P into shared memory (A operand of P V) once the P V of two tiles ago has read the buffer
      ok = mbar_wait_backoff(smem_u32(&p_empty[j & 1]), ((j >> 1) & 1u) ^ 1u, abortp, p.status, ST_TIMEOUT_SMEM_EMPTY);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      uint8_t* prow = p_ptr + (j & 1) * Cfg::kPBytes + half * CHUNK_BYTES + r * 128;
#pragma unroll
      for (int unit = 0; unit < HC / 8; ++unit) {
        uint4 w;
        w.x = pack_bf16x2(__uint_as_float(v[unit * 8 + 0]), __uint_as_float(v[unit * 8 + 1]));
        w.y = pack_bf16x2(__uint_as_float(v[unit * 8 + 2]), __uint_as_float(v[unit * 8 + 3]));
        w.z = pack_bf16x2(__uint_as_float(v[unit * 8 + 4]), __uint_as_float(v[unit * 8 + 5]));
        w.w = pack_bf16x2(__uint_as_float(v[unit * 8 + 6]), __uint_as_float(v[unit * 8 + 7]));
        *reinterpret_cast<uint4*>(prow + ((unit ^ (r & 7)) << 4)) = w;
      }
      fence_proxy_async_smem();   // P was written with ordinary stores and is read by the tensor core
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&p_full[j & 1]));
    }
    if (ok && n_tiles > 0) {
      float l_other;
      ok = swap_with_partner(l, l_other);   // both halves used the same m_used, so the sums simply add
      l += l_other;
    }
    if (ok && n_tiles > 0) {
      ok = mbar_wait_backoff(smem_u32(&o_done), (uint32_t)((n_tiles - 1) & 1), abortp, p.status, ST_TIMEOUT_TMEM_FULL);
      ok = __all_sync(0xffffffffu, ok);
    }
    if (ok) {
      tc_fence_after();
      const bool row_ok = q0 + r < q_len;
      const float inv = l > 0.f && row_ok ? flash_gate(p, q_begin + q0 + r, h) / l : 0.f;
      __nv_bfloat16* orow = p.out + (long long)(q_begin + q0 + r) * p.ldo + h * D;
#pragma unroll 1
      for (int c = half * (D / 64); c < (half + 1) * (D / 64); ++c) {   // each warpgroup stores half the columns
        uint32_t v[32];
        if (n_tiles > 0) {
          tmem_ld_32x32(tmem_o + lane_addr + c * 32, v);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = 0u;
        }
        if (row_ok) {
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            uint4 w;
            w.x = pack_bf16x2(__uint_as_float(v[u * 8 + 0]) * inv, __uint_as_float(v[u * 8 + 1]) * inv);
            w.y = pack_bf16x2(__uint_as_float(v[u * 8 + 2]) * inv, __uint_as_float(v[u * 8 + 3]) * inv);
            w.z = pack_bf16x2(__uint_as_float(v[u * 8 + 4]) * inv, __uint_as_float(v[u * 8 + 5]) * inv);
            w.w = pack_bf16x2(__uint_as_float(v[u * 8 + 6]) * inv, __uint_as_float(v[u * 8 + 7]) * inv);
            *reinterpret_cast<uint4*>(orow + c * 32 + u * 8) = w;
          }
        }
      }
      if (row_ok && half == 0 && p.lse != nullptr)
        p.lse[(long long)h * p.Tq + q_begin + q0 + r] =
            l > 0.f ? (m_used + log2f(l)) * 0.6931471805599453f : -INFINITY;
      tc_fence_before();
    }
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, FA_TMEM_COLS);
  }
}


// ------------------------------------------------------------------------------------------
// Forward, two query tiles per CTA: 256 query rows of one head, handled as tiles a and b with one softmax warpgroup
// each (a full score row per thread). Both tiles share the K/V tiles in shared memory, and while one warpgroup is in
// its softmax the tensor core works for the other tile.
//
// What bounds it: per 128 x 128 tile the exponentials take 1024 cycles of the SM's special-function unit and the two
// products 1024 (D = 128) or 512 (D = 64) of the tensor core, so everything else has to hide under these:
//  * P goes to tensor memory (packed bf16) and is the A operand from there. From shared memory the two 128 x 128
//    operands of a product alone need the SM's whole shared-memory bandwidth, and P's stores would come on top.
//    D = 128 fills tensor memory with S_a S_b O_a O_b, so P takes the place of its scores and the next scores wait for
//    P V; D = 64 has room for P beside S, and the next scores are computed under the softmax.
//  * P is handed over in halves: P V starts on the first 64 keys while the exponentials of the others run.
//  * Three warpgroups of 168 registers a thread, redistributed to 88 / 208 / 208: the softmax threads keep their 128 scores
//    in registers without spills.
//  * Pairs of fp32 values per instruction (fma / add .f32x2), three-way maxima.
//  * D = 64: both tiles' scores are there at the same time, so both warpgroups would read, search for maxima and exponentiate together, with the
//    special-function unit idle in between. Tile b starts a part of a tile later, and they stay so: 1 x 16384 tokens, 14 / 2 heads 691 -> 633 us,
//    1 x 4096 93 -> 84; 300, 600, 1000, 1500 and 2200 cycles 690, 670, 634, 633, 636. 32 x 300 (three key tiles at most) 51 -> 53, so
//    it takes four. D = 128 issues the scores of the two tiles apart and measures the same with and without.
//  * A CTA stays and takes the next query tile from the launch's own queue (cluster launch control: it cancels a CTA that
//    has not started and does its work), so set-up, the first loads and the epilogue overlap; longest tiles first.
// Measured rates stand beside the dispatch in launch_flash_fwd.
// ------------------------------------------------------------------------------------------
template <int D>
struct Flash2Cfg {
  static constexpr int kTileBytes = FA_BN * D * 2;
  static constexpr int kSlots = D == 128 ? 4 : 6;
  static constexpr int kSmemBytes = 1024 + 2 * kTileBytes + kSlots * kTileBytes;
};
constexpr int FA2_THREADS = 384;
constexpr int FA2_STAGGER_TILES = 4;
constexpr uint32_t FA2_STAGGER_CYCLES = 1000;
constexpr int FA2_REGS_LAUNCH = 168, FA2_REGS_OTHER = 88, FA2_REGS_SOFTMAX = 208;     // 88 + 2 x 208 = 3 x 168

struct FlashItem {       // one query tile pair
  int b, h, q0, q_begin, q_len, kv_len, k_begin, off, kvh, t_begin, n_a, n_b;
  __device__ __forceinline__ bool valid() const { return q0 < q_len; }
  __device__ __forceinline__ int n() const { return max(n_a, n_b); }
};

__device__ __forceinline__ FlashItem flash_item(const FlashFwdParams& p, int x, int y, int z) {
  FlashItem t;
  // blocks start in the order of their index: the late tiles of all heads and sequences, which see the most keys, first
  const int heads = p.Hq, lin = (z * gridDim.y + y) * gridDim.x + x, per = heads * gridDim.z;
  const int q_tile = gridDim.x - 1 - lin / per, rest = lin % per;
  t.b = rest / heads;
  t.h = rest % heads;
  t.q_begin = p.cu_q[t.b];
  t.q_len = p.cu_q[t.b + 1] - t.q_begin;
  t.q0 = q_tile * 2 * FA_BM;
  t.kv_len = p.paged ? p.seq_lens[t.b] : (p.cu_k[t.b + 1] - p.cu_k[t.b]);
  t.k_begin = p.paged ? 0 : p.cu_k[t.b];
  t.off = t.kv_len - t.q_len;
  t.kvh = t.h / (p.Hq / p.Hkv);
  // key tiles: both query tiles start at tile a's first visible tile; each stops at its own last one
  t.t_begin = flash_first_key(p, t.off + t.q0) / FA_BN;
  const int hi_a = p.causal ? min(t.kv_len, t.off + t.q0 + FA_BM) : t.kv_len;
  const int hi_b = p.causal ? min(t.kv_len, t.off + t.q0 + 2 * FA_BM) : t.kv_len;
  t.n_a = max((hi_a + FA_BN - 1) / FA_BN - t.t_begin, 0);
  t.n_b = t.q0 + FA_BM < t.q_len ? max((hi_b + FA_BN - 1) / FA_BN - t.t_begin, 0) : 0;
  return t;
}

// D[tmem] (+)= A[tmem] * B[smem]: A is 128 lanes x 8 columns of packed bf16 pairs.
__device__ __forceinline__ void umma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ uint64_t pair(float lo, float hi) {
  uint64_t v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
  return v;
}
__device__ __forceinline__ void unpair(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// ---- cluster launch control: take over the work of a CTA of this launch that has not started -------------------------
__device__ __forceinline__ void clc_try_cancel(uint32_t response, uint32_t bar) {
  asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(response), "r"(bar) : "memory");
}
__device__ __forceinline__ bool clc_read(uint32_t response, int& x, int& y, int& z) {
  uint32_t got;
  asm volatile(
      "{\n\t.reg .b128 r;\n\t.reg .pred P;\n\t"
      "ld.shared.b128 r, [%4];\n\t"
      "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 P, r;\n\t"
      "selp.u32 %0, 1, 0, P;\n\t"
      "mov.u32 %1, 0;\n\tmov.u32 %2, 0;\n\tmov.u32 %3, 0;\n\t"
      "@P clusterlaunchcontrol.query_cancel.get_first_ctaid.v4.b32.b128 {%1, %2, %3, _}, r;\n\t}"
      : "=r"(got), "=r"(x), "=r"(y), "=r"(z)
      : "r"(response)
      : "memory");
  return got != 0;
}

template <int D>
__global__ void __launch_bounds__(FA2_THREADS, 1) flash_fwd2_kernel(const __grid_constant__ FlashFwdParams p) {
  using Cfg = Flash2Cfg<D>;
  constexpr int DCH = D / 64;
  constexpr int SLOTS = Cfg::kSlots;
  constexpr int CHUNK_BYTES = FA_BN * 128;
  constexpr bool EARLY = D == 64;          // P has columns of its own: the next scores need not wait for P V
  constexpr uint32_t TM_O = 2 * FA_BN, TM_P = EARLY ? 2 * FA_BN + 2 * D : 0, TM_P_STEP = EARLY ? FA_BN / 2 : FA_BN;
  extern __shared__ __align__(128) uint8_t smem_raw[];
  __shared__ __align__(16) uint4 next_item[2];
  __shared__ __align__(8) uint64_t q_full, q_empty, kv_full[SLOTS], kv_empty[SLOTS];
  __shared__ __align__(8) uint64_t s_full[2], s_empty[2], p_full[2][2], o_done[2], item_full[2], item_empty[2];
  __shared__ uint32_t tmem_base_smem;
  __shared__ int abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t q_s = smem_base;                                   // Q_a then Q_b
  const uint32_t kv_s = q_s + 2 * Cfg::kTileBytes;

  if (threadIdx.x == 0) {
    abort_flag = 0;
    mbar_init(smem_u32(&q_full), 1);
    mbar_init(smem_u32(&q_empty), 1);
    for (int i = 0; i < SLOTS; ++i) {
      mbar_init(smem_u32(&kv_full[i]), 1);
      mbar_init(smem_u32(&kv_empty[i]), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&s_full[i]), 1);
      mbar_init(smem_u32(&s_empty[i]), 4);
      mbar_init(smem_u32(&p_full[i][0]), 4);
      mbar_init(smem_u32(&p_full[i][1]), 4);
      mbar_init(smem_u32(&o_done[i]), 1);
      mbar_init(smem_u32(&item_full[i]), 1);
      mbar_init(smem_u32(&item_empty[i]), 10);      // TMA warp, MMA thread, 8 softmax warps
    }
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&tmem_base_smem), FA_TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_smem;
  volatile int* abortp = &abort_flag;

  // The n-th item of this CTA (n > 0), by every role for itself: false when there is none or a wait ran out.
  auto take = [&](int n, FlashItem& t, bool arrive) -> bool {
    const int slot = (n - 1) & 1;
    if (!mbar_wait_backoff(smem_u32(&item_full[slot]), ((n - 1) >> 1) & 1u, abortp, p.status, ST_TIMEOUT_SMEM_FULL)) return false;
    int x, y, z;
    const bool got = clc_read(smem_u32(&next_item[slot]), x, y, z);
    fence_proxy_async_smem();          // read before the next answer is written over it
    if (arrive) mbar_arrive(smem_u32(&item_empty[slot]));
    if (got) t = flash_item(p, x, y, z);
    return got;
  };
  auto take_warp = [&](int n, FlashItem& t) -> bool {      // all lanes read, then one arrives
    const bool got = __all_sync(0xffffffffu, take(n, t, false));
    if (lane == 0 && got) mbar_arrive(smem_u32(&item_empty[(n - 1) & 1]));
    return got;
  };

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(FA2_REGS_OTHER));
    FlashItem t = flash_item(p, blockIdx.x, blockIdx.y, blockIdx.z);
    if (warp == 0) {
      // ------------------------------------------------------------------ TMA producer: the whole warp, a box a lane
      bool ok = true;
      uint32_t it = 0;
      int q_loads = 0;
      auto wait = [&](uint64_t* bar, uint32_t parity) -> bool {
        return __all_sync(0xffffffffu, mbar_wait_backoff(smem_u32(bar), parity, abortp, p.status, ST_TIMEOUT_SMEM_EMPTY));
      };
      auto load_tile = [&](int j, int which) -> bool {          // which 0: K tile, 1: V tile
        const int k0 = (t.t_begin + j) * FA_BN, slot = it % SLOTS;
        if (!wait(&kv_empty[slot], ((it / SLOTS) & 1u) ^ 1u)) return false;
        const uint32_t fb = smem_u32(&kv_full[slot]), dst = kv_s + slot * Cfg::kTileBytes;
        const CUtensorMap* map = which == 0 ? &p.k_map : &p.v_map;
        if (lane == 0) mbar_expect_tx(fb, Cfg::kTileBytes);
        __syncwarp();
        if (!p.paged) {
          if (lane < DCH) tma_load_2d(dst + lane * CHUNK_BYTES, map, fb, t.kvh * D + lane * 64, t.k_begin + k0);
        } else if (lane < 8 * DCH) {
          const int i = lane / DCH, c = lane % DCH, bi = (k0 >> 4) + i;
          int blk = p.num_blocks;                               // out of range: the copy fills zeros
          if (bi < (t.kv_len + 15) >> 4) {
            blk = p.block_tables[(long long)t.b * p.max_blocks + bi];
            if (blk < 0 || blk >= p.num_blocks) { set_status(p.status, ST_BAD_INDEX); blk = p.num_blocks; }
          }
          tma_load_2d(dst + c * CHUNK_BYTES + i * 2048, map, fb, c * 64, (blk * p.Hkv + t.kvh) * 16);
        }
        __syncwarp();
        ++it;
        return true;
      };
      for (int n = 0; ok;) {
        if (t.valid()) {
          const int tiles = t.q0 + FA_BM < t.q_len ? 2 : 1, nt = t.n();
          ok = wait(&q_empty, (q_loads & 1u) ^ 1u);
          if (!ok) break;
          if (lane == 0) mbar_expect_tx(smem_u32(&q_full), tiles * Cfg::kTileBytes);
          __syncwarp();
          if (lane < tiles * DCH) {
            const int x = lane / DCH, c = lane % DCH;
            tma_load_2d(q_s + x * Cfg::kTileBytes + c * CHUNK_BYTES, &p.q_map, smem_u32(&q_full), t.h * D + c * 64, t.q_begin + t.q0 + x * FA_BM);
          }
          __syncwarp();
          ++q_loads;
          // in the order of use
          if (nt > 0) ok = load_tile(0, 0);
          for (int j = 0; j < nt && ok; ++j) {
            if constexpr (EARLY) {
              if (j + 1 < nt) ok = load_tile(j + 1, 0);
              if (ok) ok = load_tile(j, 1);
            } else {
              ok = load_tile(j, 1);
              if (ok && j + 1 < nt) ok = load_tile(j + 1, 0);
            }
          }
          if (!ok) break;
        }
        ++n;
        if (!take_warp(n, t)) break;
      }
      if (!ok && lane == 0) {   // drain: no bulk copy may land after the CTA has gone
        auto drain = [&](uint64_t* bar, uint32_t parity) {
          const uint64_t t0 = globaltimer_ns();
          while (!mbar_try_wait(smem_u32(bar), parity))
            if (globaltimer_ns() - t0 > 50000000ull) break;
        };
        if (q_loads > 0) drain(&q_full, (q_loads - 1) & 1u);
        for (uint32_t j = it > (uint32_t)SLOTS ? it - SLOTS : 0; j < it; ++j) drain(&kv_full[j % SLOTS], (j / SLOTS) & 1u);
      }
    } else if (warp == 1) {
      // ------------------------------------------------------------------ MMA issuer
      if (elect_one_sync()) {
        constexpr uint32_t idesc_s = make_idesc_bf16(FA_BM, FA_BN, 0, 0);   // Q, K both K-major
        constexpr uint32_t idesc_o = make_idesc_bf16(FA_BM, D, 0, 1);       // P in tensor memory, V MN-major
        bool ok = true;
        uint32_t it = 0, s_count[2] = {0, 0}, p_count[2] = {0, 0};
        int q_loads = 0;
        auto wait = [&](uint64_t* bar, uint32_t parity, int code) { return mbar_wait_backoff(smem_u32(bar), parity, abortp, p.status, code); };
        auto wait_kv = [&](uint32_t idx) { return wait(&kv_full[idx % SLOTS], (idx / SLOTS) & 1u, ST_TIMEOUT_SMEM_FULL); };
        auto issue_s = [&](int x, uint32_t idx) -> bool {
          if constexpr (EARLY) {
            if (!wait(&s_empty[x], (s_count[x] & 1u) ^ 1u, ST_TIMEOUT_TMEM_EMPTY)) return false;
          }
          ++s_count[x];
          tc_fence_after();
          const uint32_t ks = kv_s + (idx % SLOTS) * Cfg::kTileBytes, qs = q_s + x * Cfg::kTileBytes;
#pragma unroll
          for (int k = 0; k < D / 16; ++k) {
            const uint64_t adesc = make_smem_desc_sw128(qs + (k >> 2) * CHUNK_BYTES + (k & 3) * 32, 16, 1024);
            const uint64_t bdesc = make_smem_desc_sw128(ks + (k >> 2) * CHUNK_BYTES + (k & 3) * 32, 16, 1024);
            umma_bf16(tmem_base + x * FA_BN, adesc, bdesc, idesc_s, k > 0 ? 1u : 0u);
          }
          umma_commit(smem_u32(&s_full[x]));
          return true;
        };
        auto issue_pv = [&](int x, int j, uint32_t idx) -> bool {
          const uint32_t vs = kv_s + (idx % SLOTS) * Cfg::kTileBytes;
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            if (!wait(&p_full[x][half], p_count[x] & 1u, ST_TIMEOUT_TMEM_FULL)) return false;
            tc_fence_after();
#pragma unroll
            for (int k = half * 4; k < half * 4 + 4; ++k)
              umma_bf16_ts(tmem_base + TM_O + x * D, tmem_base + TM_P + x * TM_P_STEP + k * 8, make_smem_desc_sw128(vs + k * 2048, CHUNK_BYTES, 1024),
                           idesc_o, (j > 0 || k > 0) ? 1u : 0u);
          }
          ++p_count[x];
          umma_commit(smem_u32(&o_done[x]));
          return true;
        };
        auto release = [&](uint32_t idx) { umma_commit(smem_u32(&kv_empty[idx % SLOTS])); };
        for (int n = 0; ok;) {
          if (t.valid()) {
            const int nt = t.n();
            const int n_x[2] = {t.n_a, t.n_b};
            ok = wait(&q_full, q_loads & 1u, ST_TIMEOUT_SMEM_FULL);
            ++q_loads;
            if (!ok) break;
            if (nt > 0) {
              ok = wait_kv(it);
              if (ok && n_x[0] > 0) ok = issue_s(0, it);
              if (ok && n_x[1] > 0) ok = issue_s(1, it);
              if (!ok) break;
              release(it++);
            }
            if (nt <= 1) umma_commit(smem_u32(&q_empty));
            for (int j = 0; j < nt && ok; ++j) {
              const bool more = j + 1 < nt;
              if constexpr (EARLY) {
                if (more) {
                  ok = wait_kv(it);
                  if (ok && j + 1 < n_x[0]) ok = issue_s(0, it);
                  if (ok && j + 1 < n_x[1]) ok = issue_s(1, it);
                  if (!ok) break;
                  release(it++);
                  if (j + 2 == nt) umma_commit(smem_u32(&q_empty));
                }
                ok = wait_kv(it);
                if (ok && j < n_x[0]) ok = issue_pv(0, j, it);
                if (ok && j < n_x[1]) ok = issue_pv(1, j, it);
                if (!ok) break;
                release(it++);
              } else {
                const uint32_t iv = it++, ik = it;
                if (more) ++it;
                ok = wait_kv(iv);
                for (int x = 0; x < 2 && ok; ++x) {
                  if (j < n_x[x]) ok = issue_pv(x, j, iv);
                  if (ok && x == 1) release(iv);
                  if (ok && more && x == 0) ok = wait_kv(ik);
                  if (ok && j + 1 < n_x[x]) ok = issue_s(x, ik);
                }
                if (!ok) break;
                if (more) {
                  release(ik);
                  if (j + 2 == nt) umma_commit(smem_u32(&q_empty));
                }
              }
            }
            if (!ok) break;
          }
          ++n;
          if (!take(n, t, true)) break;
        }
      }
    } else if (warp == 2) {
      // ------------------------------------------------------------------ next items, two answers ahead at most
      if (elect_one_sync()) {
        for (int n = 1;; ++n) {
          const int slot = (n - 1) & 1;
          const uint32_t use = (n - 1) >> 1;
          if (!mbar_wait_backoff(smem_u32(&item_empty[slot]), (use & 1u) ^ 1u, abortp, p.status, ST_TIMEOUT_SMEM_EMPTY)) break;
          mbar_expect_tx(smem_u32(&item_full[slot]), 16);
          clc_try_cancel(smem_u32(&next_item[slot]), smem_u32(&item_full[slot]));
          // the answer is waited for in any case: it must not land after the CTA has gone
          const uint64_t t0 = globaltimer_ns();
          bool there;
          while (!(there = mbar_try_wait_hint(smem_u32(&item_full[slot]), use & 1u, 2000u)))
            if (globaltimer_ns() - t0 > RB_WAIT_BUDGET_NS) break;
          if (!there) {
            *abortp = 1;
            set_status(p.status, ST_TIMEOUT_SMEM_FULL);
            break;
          }
          int x, y, z;
          if (!clc_read(smem_u32(&next_item[slot]), x, y, z)) break;
          fence_proxy_async_smem();
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax + epilogue, one warpgroup per query tile
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(FA2_REGS_SOFTMAX));
    FlashItem t = flash_item(p, blockIdx.x, blockIdx.y, blockIdx.z);
    const int x = (warp >> 2) - 1;               // 0: tile a, 1: tile b
    const int qd = warp & 3;
    const int r = qd * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(qd * 32) << 16;
    const uint32_t tmem_s = tmem_base + x * FA_BN + lane_addr;
    const uint32_t tmem_o = tmem_base + TM_O + x * D + lane_addr;
    const uint32_t tmem_p = tmem_base + TM_P + x * TM_P_STEP + lane_addr;
    const uint64_t scale2 = pair(p.scale_log2, p.scale_log2);
    uint32_t count = 0;                          // key tiles of this query tile so far, all items
    bool ok = true;
    auto wait = [&](uint64_t* bar, uint32_t parity) -> bool {
      return __all_sync(0xffffffffu, mbar_wait_backoff(smem_u32(bar), parity, abortp, p.status, ST_TIMEOUT_TMEM_FULL));
    };
    for (int n = 0; ok;) {
      const int q0x = t.q0 + x * FA_BM;
      if (t.valid() && q0x < t.q_len) {
        const int qpos = t.off + q0x + r;
        const int k_first = flash_first_key(p, qpos), last_first = flash_first_key(p, t.off + q0x + FA_BM - 1);
        const int n_mine = x == 0 ? t.n_a : t.n_b;
        float m_used = -INFINITY, l = 0.f;
        for (int j = 0; j < n_mine; ++j, ++count) {
          const int k0 = (t.t_begin + j) * FA_BN;
          ok = wait(&s_full[x], count & 1u);
          if (!ok) break;
          if (EARLY && x == 1 && j == 0 && n_mine >= FA2_STAGGER_TILES && t.n_a > 0) {
            const uint32_t begun = (uint32_t)clock();
            while ((uint32_t)clock() - begun < FA2_STAGGER_CYCLES) {
            }
            __syncwarp();
          }
          tc_fence_after();
          const bool need_mask = (k0 + FA_BN > t.kv_len) || (p.causal && k0 + FA_BN - 1 > t.off + q0x) || k0 < last_first;
          uint32_t v[FA_BN];
#pragma unroll
          for (int c = 0; c < FA_BN / 32; ++c) tmem_ld_32x32(tmem_s + c * 32, *reinterpret_cast<uint32_t(*)[32]>(&v[c * 32]));
          tmem_ld_wait();
          if constexpr (EARLY) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&s_empty[x]));       // the next scores may take the columns now
          }
          if (need_mask) {
            // keys k_first <= k <= last of this row
            const int last = (p.causal ? min(t.kv_len - 1, qpos) : t.kv_len - 1) - k0, first = k_first - k0;
#pragma unroll
            for (int i = 0; i < FA_BN; ++i)
              if (i > last || i < first) v[i] = 0xff800000u;
          }
          float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
          for (int i = 0; i < FA_BN; i += 8) {
#pragma unroll
            for (int u = 0; u < 4; ++u) mx[u] = max3(mx[u], __uint_as_float(v[i + 2 * u]), __uint_as_float(v[i + 2 * u + 1]));
          }
          const float m_new = fmaxf(m_used, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * p.scale_log2);
          const bool need = m_new > m_used + FA_RESCALE_THRESHOLD || (m_used == -INFINITY && m_new != -INFINITY);
          if (EARLY && j > 0) {      // the previous P V has read P and written O (D = 128: these scores came after it)
            ok = wait(&o_done[x], (count - 1) & 1u);
            if (!ok) break;
            tc_fence_after();
          }
          if (__any_sync(0xffffffffu, need)) {
            if (j > 0) {
              const float alpha = need ? fast_exp2((m_used == -INFINITY ? m_new : m_used) - m_new) : 1.f;
#pragma unroll 1
              for (int c = 0; c < D / 16; ++c) {
                uint32_t o[16];
                tmem_ld_32x16(tmem_o + c * 16, o);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                tmem_st_32x16(tmem_o + c * 16, o);
              }
              l *= alpha;
            }
            if (need) m_used = m_new;
          }
          const float mref = m_used == -INFINITY ? 0.f : m_used;
          const uint64_t neg2 = pair(-mref, -mref);
          uint64_t ls[2] = {0, 0};       // four running sums, keys 4 i + 0 .. 3
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            uint32_t w[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) {
              const int e = half * 64 + 2 * i;
              float a, b;
              unpair(fma2(pair(__uint_as_float(v[e]), __uint_as_float(v[e + 1])), scale2, neg2), a, b);
              a = fast_exp2(a);
              b = fast_exp2(b);
              ls[i & 1] = add2(ls[i & 1], pair(a, b));
              w[i] = pack_bf16x2(a, b);
            }
            tmem_st_32x32(tmem_p + half * 32, w);
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&p_full[x][half]));
          }
          float s0, s1, s2, s3;
          unpair(ls[0], s0, s1);
          unpair(ls[1], s2, s3);
          l += (s0 + s1) + (s2 + s3);
        }
        if (!ok) break;
        if (n_mine > 0) {
          ok = wait(&o_done[x], (count - 1) & 1u);
          if (!ok) break;
        }
        tc_fence_after();
        const bool row_ok = q0x + r < t.q_len;
        const float inv = l > 0.f && row_ok ? flash_gate(p, t.q_begin + q0x + r, t.h) / l : 0.f;
        __nv_bfloat16* orow = p.out + (long long)(t.q_begin + q0x + r) * p.ldo + t.h * D;
#pragma unroll 1
        for (int c = 0; c < D / 32; ++c) {
          uint32_t o[32];
          if (n_mine > 0) {
            tmem_ld_32x32(tmem_o + c * 32, o);
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = 0u;
          }
          if (row_ok) {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              uint4 w;
              w.x = pack_bf16x2(__uint_as_float(o[u * 8 + 0]) * inv, __uint_as_float(o[u * 8 + 1]) * inv);
              w.y = pack_bf16x2(__uint_as_float(o[u * 8 + 2]) * inv, __uint_as_float(o[u * 8 + 3]) * inv);
              w.z = pack_bf16x2(__uint_as_float(o[u * 8 + 4]) * inv, __uint_as_float(o[u * 8 + 5]) * inv);
              w.w = pack_bf16x2(__uint_as_float(o[u * 8 + 6]) * inv, __uint_as_float(o[u * 8 + 7]) * inv);
              *reinterpret_cast<uint4*>(orow + c * 32 + u * 8) = w;
            }
          }
        }
        if (row_ok && p.lse != nullptr)
          p.lse[(long long)t.h * p.Tq + t.q_begin + q0x + r] = l > 0.f ? (m_used + log2f(l)) * 0.6931471805599453f : -INFINITY;
        tc_fence_before();       // O has been read: the next item's first product may overwrite it
      }
      ++n;
      if (!take_warp(n, t)) break;
    }
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, FA_TMEM_COLS);
  }
}

// ------------------------------------------------------------------------------------------
// Forward for latent attention in its expanded form (ops/latent.py): 128 query rows of one head per CTA. A key is the
// head's own part (DN columns of K) followed by 64 rotated columns shared by all heads, so a key tile is loaded from two
// tensors; values have DV columns. Sliding window, causal, dense key rows per sequence. The softmax denominator also holds
// exp(sink[h]), and the output row is scaled by gate[t, h].
// Same roles and pipeline as flash_fwd_kernel; wider keys leave room for two K slots, one V slot and one P buffer.
// ------------------------------------------------------------------------------------------
struct FlashLatentParams {
  CUtensorMap q_map;    // [T, H*(DN+64)]
  CUtensorMap k_map;    // [S, H*DN]
  CUtensorMap r_map;    // [S, 64]
  CUtensorMap v_map;    // [S, H*DV]
  __nv_bfloat16* out;   // [T, H*DV]
  const int* cu_q;
  const int* cu_k;
  const float* sink;    // [H]
  const float* gate;    // [T, H]
  int H, window;
  float scale_log2;
  int* status;
};

template <int DN, int DV>
struct FlashLatentCfg {
  static constexpr int DK = DN + 64;
  static constexpr int kKBytes = FA_BN * DK * 2;            // a K tile, and the Q tile
  static constexpr int kVBytes = FA_BN * DV * 2;
  static constexpr int kPBytes = FA_BM * FA_BN * 2;
  static constexpr int kSmemBytes = 1024 + 3 * kKBytes + kVBytes + kPBytes;
};

template <int DN, int DV>
__global__ void __launch_bounds__(FA_THREADS, 1) flash_latent_kernel(const __grid_constant__ FlashLatentParams p) {
  using Cfg = FlashLatentCfg<DN, DV>;
  constexpr int DK = Cfg::DK;
  constexpr int CHUNK_BYTES = FA_BN * 128;
  extern __shared__ __align__(128) uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t q_full, k_full[2], k_empty[2], v_full, v_empty;
  __shared__ __align__(8) uint64_t s_full[2], s_empty[2], p_full, p_empty, o_done, xch_bar[4];
  __shared__ float xch[2][2][FA_BM];
  __shared__ uint32_t tmem_base_smem;
  __shared__ int abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int b = blockIdx.z, h = blockIdx.y;
  const int q_tile = gridDim.x - 1 - blockIdx.x;
  const int q_begin = p.cu_q[b];
  const int q_len = p.cu_q[b + 1] - q_begin;
  const int q0 = q_tile * FA_BM;
  if (q0 >= q_len) return;                                  // uniform per CTA, before any set-up
  const int k_begin = p.cu_k[b];
  const int kv_len = p.cu_k[b + 1] - k_begin;
  const int off = kv_len - q_len;                           // key index of query 0
  const int hi = min(kv_len, off + q0 + FA_BM);
  const int lo = max(0, off + q0 - p.window + 1);
  const int t_begin = lo / FA_BN;
  const int n_tiles = max((hi + FA_BN - 1) / FA_BN - t_begin, 0);

  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_al = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t q_s = smem_base;
  const uint32_t k_s = q_s + Cfg::kKBytes;
  const uint32_t v_s = k_s + 2 * Cfg::kKBytes;
  const uint32_t p_s = v_s + Cfg::kVBytes;
  uint8_t* p_ptr = smem_al + 3 * Cfg::kKBytes + Cfg::kVBytes;

  if (threadIdx.x == 0) {
    abort_flag = 0;
    mbar_init(smem_u32(&q_full), 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&k_full[i]), 1);
      mbar_init(smem_u32(&k_empty[i]), 1);
      mbar_init(smem_u32(&s_full[i]), 1);
      mbar_init(smem_u32(&s_empty[i]), 8);
    }
    mbar_init(smem_u32(&v_full), 1);
    mbar_init(smem_u32(&v_empty), 1);
    mbar_init(smem_u32(&p_full), 8);
    mbar_init(smem_u32(&p_empty), 1);
    for (int i = 0; i < 4; ++i) mbar_init(smem_u32(&xch_bar[i]), 64);
    mbar_init(smem_u32(&o_done), 1);
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&tmem_base_smem), FA_TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_smem;
  const uint32_t tmem_o = tmem_base + 2 * FA_BN;
  volatile int* abortp = &abort_flag;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one_sync()) {
      bool ok = true;
      mbar_expect_tx(smem_u32(&q_full), Cfg::kKBytes);
#pragma unroll
      for (int c = 0; c < DK / 64; ++c)
        tma_load_2d(q_s + c * CHUNK_BYTES, &p.q_map, smem_u32(&q_full), h * DK + c * 64, q_begin + q0);
      int k_issued = 0, v_issued = 0;
      auto load_k = [&](int j) -> bool {
        const int slot = j & 1, row = k_begin + (t_begin + j) * FA_BN;
        if (!mbar_wait_backoff(smem_u32(&k_empty[slot]), ((j >> 1) & 1u) ^ 1u, abortp, p.status, ST_TIMEOUT_SMEM_EMPTY)) return false;
        const uint32_t fb = smem_u32(&k_full[slot]), dst = k_s + slot * Cfg::kKBytes;
        mbar_expect_tx(fb, Cfg::kKBytes);
#pragma unroll
        for (int c = 0; c < DN / 64; ++c) tma_load_2d(dst + c * CHUNK_BYTES, &p.k_map, fb, h * DN + c * 64, row);
        tma_load_2d(dst + (DN / 64) * CHUNK_BYTES, &p.r_map, fb, 0, row);
        ++k_issued;
        return true;
      };
      auto load_v = [&](int j) -> bool {
        const int row = k_begin + (t_begin + j) * FA_BN;
        if (!mbar_wait_backoff(smem_u32(&v_empty), (j & 1u) ^ 1u, abortp, p.status, ST_TIMEOUT_SMEM_EMPTY)) return false;
        mbar_expect_tx(smem_u32(&v_full), Cfg::kVBytes);
#pragma unroll
        for (int c = 0; c < DV / 64; ++c) tma_load_2d(v_s + c * CHUNK_BYTES, &p.v_map, smem_u32(&v_full), h * DV + c * 64, row);
        ++v_issued;
        return true;
      };
      // order of use: K0, then (K_{j+1}, V_j) for every j
      if (n_tiles > 0) ok = load_k(0);
      for (int j = 0; j < n_tiles && ok; ++j) {
        if (j + 1 < n_tiles) { ok = load_k(j + 1); if (!ok) break; }
        ok = load_v(j);
      }
      if (!ok) {   // drain: no bulk copy may land after the CTA has gone
        auto drain = [&](uint64_t* bar, uint32_t parity) {
          const uint64_t t0 = globaltimer_ns();
          while (!mbar_try_wait(smem_u32(bar), parity))
            if (globaltimer_ns() - t0 > 50000000ull) break;
        };
        drain(&q_full, 0);
        for (int j = max(0, k_issued - 2); j < k_issued; ++j) drain(&k_full[j & 1], (j >> 1) & 1u);
        if (v_issued > 0) drain(&v_full, (v_issued - 1) & 1u);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one_sync()) {
      constexpr uint32_t idesc_s = make_idesc_bf16(FA_BM, FA_BN, 0, 0);    // Q, K both K-major
      constexpr uint32_t idesc_o = make_idesc_bf16(FA_BM, DV, 0, 1);       // P K-major, V MN-major
      bool ok = mbar_wait_backoff(smem_u32(&q_full), 0, abortp, p.status, ST_TIMEOUT_SMEM_FULL);
      auto issue_s = [&](int j) -> bool {
        const int slot = j & 1;
        if (!mbar_wait_backoff(smem_u32(&k_full[slot]), (j >> 1) & 1u, abortp, p.status, ST_TIMEOUT_SMEM_FULL)) return false;
        if (!mbar_wait_backoff(smem_u32(&s_empty[slot]), ((j >> 1) & 1u) ^ 1u, abortp, p.status, ST_TIMEOUT_TMEM_EMPTY)) return false;
        tc_fence_after();
        const uint32_t ks = k_s + slot * Cfg::kKBytes;
#pragma unroll
        for (int k = 0; k < DK / 16; ++k) {
          const uint64_t adesc = make_smem_desc_sw128(q_s + (k >> 2) * CHUNK_BYTES + (k & 3) * 32, 16, 1024);
          const uint64_t bdesc = make_smem_desc_sw128(ks + (k >> 2) * CHUNK_BYTES + (k & 3) * 32, 16, 1024);
          umma_bf16(tmem_base + slot * FA_BN, adesc, bdesc, idesc_s, k > 0 ? 1u : 0u);
        }
        umma_commit(smem_u32(&k_empty[slot]));
        umma_commit(smem_u32(&s_full[slot]));
        return true;
      };
      if (ok && n_tiles > 0) ok = issue_s(0);
      for (int j = 0; j < n_tiles && ok; ++j) {
        if (j + 1 < n_tiles) { ok = issue_s(j + 1); if (!ok) break; }
        ok = mbar_wait_backoff(smem_u32(&p_full), j & 1u, abortp, p.status, ST_TIMEOUT_TMEM_FULL);
        if (!ok) break;
        ok = mbar_wait_backoff(smem_u32(&v_full), j & 1u, abortp, p.status, ST_TIMEOUT_SMEM_FULL);
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int k = 0; k < FA_BN / 16; ++k) {
          const uint64_t adesc = make_smem_desc_sw128(p_s + (k >> 2) * CHUNK_BYTES + (k & 3) * 32, 16, 1024);
          const uint64_t bdesc = make_smem_desc_sw128(v_s + k * 2048, CHUNK_BYTES, 1024);
          umma_bf16(tmem_o, adesc, bdesc, idesc_o, (j > 0 || k > 0) ? 1u : 0u);
        }
        umma_commit(smem_u32(&v_empty));
        umma_commit(smem_u32(&p_empty));
        umma_commit(smem_u32(&o_done));
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax + epilogue
    // two threads per query row, as in flash_fwd_kernel: `half` owns 64 of the 128 score columns and half of O's columns
    constexpr int HC = FA_BN / 2;
    const int qd = warp & 3;
    const int half = (warp - 2) >> 2;
    const int r = qd * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(qd * 32) << 16;
    const int qpos = off + q0 + r;
    float m_used = -INFINITY, l = 0.f;
    bool ok = true;
    uint32_t xph = 0;
    auto swap_with_partner = [&](float mine, float& other) -> bool {
      xch[xph & 1][half][r] = mine;
      mbar_arrive(smem_u32(&xch_bar[qd]));
      bool good = mbar_wait_backoff(smem_u32(&xch_bar[qd]), xph & 1u, abortp, p.status, ST_TIMEOUT_TMEM_FULL);
      other = xch[xph & 1][half ^ 1][r];
      ++xph;
      return __all_sync(0xffffffffu, good);
    };
    for (int j = 0; j < n_tiles; ++j) {
      const int k0 = (t_begin + j) * FA_BN;
      const uint32_t s_addr = tmem_base + (j & 1) * FA_BN + half * HC + lane_addr;
      ok = mbar_wait_backoff(smem_u32(&s_full[j & 1]), (j >> 1) & 1u, abortp, p.status, ST_TIMEOUT_TMEM_FULL);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const bool need_mask = k0 + FA_BN > kv_len || k0 + FA_BN - 1 > off + q0 || k0 <= off + q0 + FA_BM - 1 - p.window;
      uint32_t v[HC];
#pragma unroll
      for (int c = 0; c < HC / 32; ++c)
        tmem_ld_32x32(s_addr + c * 32, *reinterpret_cast<uint32_t(*)[32]>(&v[c * 32]));
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&s_empty[j & 1]));
      if (need_mask) {
#pragma unroll
        for (int i = 0; i < HC; ++i) {
          const int kj = k0 + half * HC + i;
          if (kj >= kv_len || kj > qpos || kj <= qpos - p.window) v[i] = 0xff800000u;   // -inf
        }
      }
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < HC; i += 4) {
        mx[0] = fmaxf(mx[0], __uint_as_float(v[i]));
        mx[1] = fmaxf(mx[1], __uint_as_float(v[i + 1]));
        mx[2] = fmaxf(mx[2], __uint_as_float(v[i + 2]));
        mx[3] = fmaxf(mx[3], __uint_as_float(v[i + 3]));
      }
      const float mine = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
      float other;
      ok = swap_with_partner(mine, other);
      if (!ok) break;
      const float m_new = fmaxf(m_used, fmaxf(mine, other) * p.scale_log2);
      const bool need = m_new > m_used + FA_RESCALE_THRESHOLD || (m_used == -INFINITY && m_new != -INFINITY);
      if (__any_sync(0xffffffffu, need)) {   // same rows, same inputs: both warps of a quarter agree
        if (j > 0) {
          ok = mbar_wait_backoff(smem_u32(&o_done), (uint32_t)((j - 1) & 1), abortp, p.status, ST_TIMEOUT_TMEM_FULL);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          tc_fence_after();
          const float alpha = need ? fast_exp2((m_used == -INFINITY ? m_new : m_used) - m_new) : 1.f;
#pragma unroll 1
          for (int c = half * (DV / 64); c < (half + 1) * (DV / 64); ++c) {
            uint32_t o[32];
            tmem_ld_32x32(tmem_o + lane_addr + c * 32, o);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
            tmem_st_32x32(tmem_o + lane_addr + c * 32, o);
          }
          tmem_st_wait();
          l *= alpha;
        }
        if (need) m_used = m_new;
      }
      const float mref = m_used == -INFINITY ? 0.f : m_used;
      float ls[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int i = 0; i < HC; i += 4) {
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const float x = fast_exp2(fmaf(__uint_as_float(v[i + t]), p.scale_log2, -mref));
          ls[t] += x;
          v[i + t] = __float_as_uint(x);
        }
      }
      l += (ls[0] + ls[1]) + (ls[2] + ls[3]);
      // bf16 P into shared memory once the previous P V has read the buffer
      ok = mbar_wait_backoff(smem_u32(&p_empty), (j & 1u) ^ 1u, abortp, p.status, ST_TIMEOUT_SMEM_EMPTY);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      uint8_t* prow = p_ptr + half * CHUNK_BYTES + r * 128;
#pragma unroll
      for (int unit = 0; unit < HC / 8; ++unit) {
        uint4 w;
        w.x = pack_bf16x2(__uint_as_float(v[unit * 8 + 0]), __uint_as_float(v[unit * 8 + 1]));
        w.y = pack_bf16x2(__uint_as_float(v[unit * 8 + 2]), __uint_as_float(v[unit * 8 + 3]));
        w.z = pack_bf16x2(__uint_as_float(v[unit * 8 + 4]), __uint_as_float(v[unit * 8 + 5]));
        w.w = pack_bf16x2(__uint_as_float(v[unit * 8 + 6]), __uint_as_float(v[unit * 8 + 7]));
        *reinterpret_cast<uint4*>(prow + ((unit ^ (r & 7)) << 4)) = w;
      }
      tc_fence_before();          // a rescale of O above is ordered before the product that reads it
      fence_proxy_async_smem();   // P was written with ordinary stores and is read by the tensor core
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&p_full));
    }
    if (ok && n_tiles > 0) {
      float l_other;
      ok = swap_with_partner(l, l_other);   // both halves used the same m_used, so the sums simply add
      l += l_other;
    }
    if (ok && n_tiles > 0) {
      ok = mbar_wait_backoff(smem_u32(&o_done), (uint32_t)((n_tiles - 1) & 1), abortp, p.status, ST_TIMEOUT_TMEM_FULL);
      ok = __all_sync(0xffffffffu, ok);
    }
    if (ok) {
      tc_fence_after();
      const bool row_ok = q0 + r < q_len;
      const long long t = q_begin + q0 + r;
      float f = 0.f;
      if (row_ok && n_tiles > 0) {
        l += exp2f(p.sink[h] * 1.4426950408889634f - m_used);      // the sink: in the denominator, no value
        f = p.gate[t * p.H + h] / l;
      }
      __nv_bfloat16* orow = p.out + t * p.H * DV + h * DV;
#pragma unroll 1
      for (int c = half * (DV / 64); c < (half + 1) * (DV / 64); ++c) {
        uint32_t v[32];
        if (n_tiles > 0) {
          tmem_ld_32x32(tmem_o + lane_addr + c * 32, v);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = 0u;
        }
        if (row_ok) {
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            uint4 w;
            w.x = pack_bf16x2(__uint_as_float(v[u * 8 + 0]) * f, __uint_as_float(v[u * 8 + 1]) * f);
            w.y = pack_bf16x2(__uint_as_float(v[u * 8 + 2]) * f, __uint_as_float(v[u * 8 + 3]) * f);
            w.z = pack_bf16x2(__uint_as_float(v[u * 8 + 4]) * f, __uint_as_float(v[u * 8 + 5]) * f);
            w.w = pack_bf16x2(__uint_as_float(v[u * 8 + 6]) * f, __uint_as_float(v[u * 8 + 7]) * f);
            *reinterpret_cast<uint4*>(orow + c * 32 + u * 8) = w;
          }
        }
      }
      tc_fence_before();
    }
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, FA_TMEM_COLS);
  }
}

template <int DN, int DV>
static int launch_flash_latent(const FlashLatentParams& p, int max_q, int B, cudaStream_t stream) {
  auto kern = flash_latent_kernel<DN, DV>;
  static bool attr_dev[64] = {};
  int dev_i = 0;
  if (cudaGetDevice(&dev_i) != cudaSuccess || dev_i < 0 || dev_i >= 64) return -10;
  if (!attr_dev[dev_i]) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, FlashLatentCfg<DN, DV>::kSmemBytes) != cudaSuccess) return -10;
    attr_dev[dev_i] = true;
  }
  dim3 grid((max_q + FA_BM - 1) / FA_BM, p.H, B);
  return launch_kernel(kern, grid, dim3(FA_THREADS), FlashLatentCfg<DN, DV>::kSmemBytes, stream, p) == cudaSuccess ? 0 : -11;
}


// ==========================================================================================
// Backward. Three kernels, no atomics, deterministic:
//   prep : -lse (log2 units) and -delta, delta[h,t] = sum_d dO*O, per 128-query tile of every sequence
//   dkdv : one CTA per (128-key tile, kv head); loops over the query heads of the group and their
//          128-query tiles. S^T = K Q^T and dP^T = V dO^T land in tensor memory (keys on the 128 lanes, so a
//          thread owns a key row); P^T and dS^T go back there, packed to bf16, as A operands of
//          dV += P^T dO and dK += dS^T Q, which accumulate in tensor memory over the whole loop.
//   dq   : one CTA per (128-query tile, head); loops over 128-key tiles. S = Q K^T, dP = dO V^T, dS back to
//          tensor memory, dQ += dS K accumulates there.
// The same Q / dO / K / V shared-memory tile serves as a K-major operand of the score products and
// as an MN-major operand of the gradient products: only the descriptor differs.
//
// What bounds it (D = 128, a 128 x 128 tile): 512 cycles of the tensor core for each of the four (dq: three) products and
// 1024 of the special-function unit, while the way from a finished product through the softmax warps to the next one is
// some 800 cycles long. Tensor memory has room for one S and one dP beside the accumulators, so the products are issued in
// an order that always leaves two to run while the softmax warps work (dkdv; dq has one to run):
//     dkdv:  dV(j)  S(j+1)  dK(j)  dP(j+1)      P(j+1) under dK(j), dP(j+1); dS(j) under dV(j), S(j+1)
//     dq:    S(j+1)  dQ(j)  dP(j+1)             P(j+1) under dQ(j), dP(j+1); dS(j) under S(j+1)
// P takes the columns of S and dS those of dP (products run in the order of their issue, so a new score tile never
// overtakes the product that reads the old P). All 16 softmax warps work on one tile, 32 of its columns each. A 64-wide score
// product would read 6 KB of shared memory for 32 cycles of work, one 128 wide 8 KB for 64: just what it delivers; dq
// keeps Q and dO in tensor memory and reads half of that. The row statistics of a query tile arrive with its Q and dO.
// Backward of causal attention, TFLOP/s by 2.5 x the forward's (in brackets with 64-wide tiles, P and dS through shared memory):
// 4 x 8192 tokens, 32 / 8 heads, D 128 772 (443); 8 x 2048 664 (343); 32 x 200 126 (70); 1 x 16384, 14 / 2 heads, D 64 549 (212);
// 16 x 512 163 (74).
// ==========================================================================================
struct FlashBwdParams {
  CUtensorMap q, dout, k, v;             // boxes of 64 columns x 128 rows
  const float* stat;                     // [Hq][stat_tiles][2 (-lse2, -delta)][128]; the tiles of sequence b start at tile cu_q[b] / 128 + b
  int stat_tiles;
  __nv_bfloat16 *dq, *dk, *dv;           // [Tq,Hq,D], [Tk,Hkv,D], [Tk,Hkv,D]
  const int* cu_q;
  const int* cu_k;
  int Hq, Hkv, Tq, Tk;
  int causal, window;
  float scale_log2, scale;
  int* status;
  // dK/dV with one CTA per (key tile, QUERY head) instead of per (key tile, key/value head): the CTAs of a group write
  // fp32 partials [2 (dV, dK)][G][Tk][Hkv][D] here and flash_bwd_reduce_kernel sums them in a fixed order. With few
  // long sequences the per-kv-head form leaves most SMs idle behind its longest CTA (G x the query tiles of the
  // first key tile); null = off.
  float* dkv_part;
};

// One warp per row, four rows in flight; block (tile of 128 queries, sequence, head).
template <int D>
__global__ void __launch_bounds__(256) flash_bwd_prep_kernel(const __nv_bfloat16* __restrict__ dout, const __nv_bfloat16* __restrict__ out,
                                                             const float* __restrict__ lse, float* __restrict__ stat, const int* __restrict__ cu_q,
                                                             int stat_tiles, int Tq, int Hq) {
  const int b = blockIdx.y, h = blockIdx.z, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int q_begin = cu_q[b], q_len = cu_q[b + 1] - q_begin, i0 = blockIdx.x * 128;
  if (i0 >= q_len) return;
  float* dst = stat + ((long long)h * stat_tiles + (q_begin >> 7) + b + blockIdx.x) * 256;
#pragma unroll
  for (int r0 = 0; r0 < 16; r0 += 4) {
    __nv_bfloat162 x[4][D / 64], y[4][D / 64];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = i0 + warp * 16 + r0 + u;
      const long long at = ((long long)(q_begin + min(i, q_len - 1)) * Hq + h) * D;
#pragma unroll
      for (int c = 0; c < D / 64; ++c) {
        x[u][c] = reinterpret_cast<const __nv_bfloat162*>(dout + at)[c * 32 + lane];
        y[u][c] = reinterpret_cast<const __nv_bfloat162*>(out + at)[c * 32 + lane];
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int r = warp * 16 + r0 + u;
      float acc = 0.f;
#pragma unroll
      for (int c = 0; c < D / 64; ++c) {
        const float2 f = __bfloat1622float2(x[u][c]), g = __bfloat1622float2(y[u][c]);
        acc += f.x * g.x + f.y * g.y;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (lane == 0) {
        const bool in = i0 + r < q_len;      // past the end: P is exactly 0
        dst[r] = in ? -(lse[(long long)h * Tq + q_begin + i0 + r] * 1.4426950408889634f) : -INFINITY;
        dst[128 + r] = in ? -acc : 0.f;
      }
    }
  }
}

template <int D>
struct FlashBwdCfg {
  static constexpr int kTile = 128 * D * 2;                 // a 128-row tile
  static constexpr int kStat = 2 * 128 * 4;
  static constexpr int kQdoStages = D == 128 ? 2 : 3;       // dkdv: (Q, dO, statistics) of 128 queries in flight
  static constexpr int kKvStages = D == 128 ? 2 : 4;        // dq: (K, V) tiles in flight
  static constexpr int kSmemDkdv = 1024 + 2 * kTile + kQdoStages * (2 * kTile + kStat);
  static constexpr int kSmemDq = 1024 + 2 * kTile + kKvStages * 2 * kTile;
};

__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
// contiguous copy global -> shared (both 16-byte aligned, whole 16-byte units)
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

// Warps 0 (TMA), 1 (products), 2 and 3 idle, then four softmax warpgroups, each with 32 of a tile's 128 columns.
constexpr int FA_BWD_THREADS = 640;
constexpr int FA_BWD_WARPS = 16;      // softmax warps

// 32 columns of P: exp2(S * scale + statistic); `nl` holds one pair of -lse2 for each pair of columns, `dead` the masked ones
template <typename Neg>
__device__ __forceinline__ void bwd_probabilities(uint32_t (&v)[32], uint64_t scale_l2, Neg neg, uint32_t dead, uint32_t (&packed)[16]) {
#pragma unroll
  for (int c = 0; c < 32; c += 2) {
    float x0, x1;
    unpair(fma2(pair(__uint_as_float(v[c]), __uint_as_float(v[c + 1])), scale_l2, neg(c)), x0, x1);
    x0 = fast_exp2(x0);
    x1 = fast_exp2(x1);
    if (dead != 0) {
      if (dead >> c & 1) x0 = 0.f;
      if (dead >> (c + 1) & 1) x1 = 0.f;
    }
    v[c] = __float_as_uint(x0);
    v[c + 1] = __float_as_uint(x1);
    packed[c >> 1] = pack_bf16x2(x0, x1);
  }
}
// dS = P * (dP - delta) * scale
template <typename Neg>
__device__ __forceinline__ void bwd_scores(const uint32_t (&prob)[32], const uint32_t (&dp)[32], uint64_t scale2, Neg neg, uint32_t (&packed)[16]) {
#pragma unroll
  for (int c = 0; c < 32; c += 2) {
    float y0, y1;
    unpair(mul2(mul2(pair(__uint_as_float(prob[c]), __uint_as_float(prob[c + 1])),
                     add2(pair(__uint_as_float(dp[c]), __uint_as_float(dp[c + 1])), neg(c))), scale2), y0, y1);
    packed[c >> 1] = pack_bf16x2(y0, y1);
  }
}
// bit c: position first + c lies outside [lo, hi]
__device__ __forceinline__ uint32_t outside_mask(int first, int lo, int hi) {
  const int a = lo - first, z = hi - first;          // columns a .. z are inside
  const uint32_t below = a <= 0 ? 0u : a >= 32 ? 0xffffffffu : (1u << a) - 1u;
  const uint32_t upto = z < 0 ? 0u : z >= 31 ? 0xffffffffu : (2u << z) - 1u;
  return below | ~upto;
}
// A operand of the gradient products: 128 columns = 8 k-steps of 8 packed columns, the quarters of a row 32 columns apart
__device__ __forceinline__ uint32_t packed_column(int k) { return (k >> 1) * 32 + (k & 1) * 8; }

template <int D>
__device__ __forceinline__ void flash_bwd_dkdv(const FlashBwdParams& p, const dim3& block, const dim3& grid) {
  using Cfg = FlashBwdCfg<D>;
  constexpr int DCH = D / 64;
  constexpr int ST = Cfg::kQdoStages;
  constexpr int CH = 128 * 128;                    // bytes of one 64-column chunk of a tile
  constexpr uint32_t TM_DP = 128, TM_DV = 256, TM_DK = 256 + D;
  extern __shared__ __align__(128) uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t kv_full, qdo_full[ST], qdo_empty[ST];
  __shared__ __align__(8) uint64_t s_full, p_full, dp_full, ds_full, acc_done;
  __shared__ uint32_t tmem_base_smem;
  __shared__ int abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // Under a causal mask the first key tiles have the longest loops: hand them out first, across all heads (blocks
  // are scheduled in the order of their linear index)
  const int lin = block.x + grid.x * block.y;
  const int b = block.z, hy = lin % grid.y;
  const int G = p.Hq / p.Hkv;
  const bool head_split = p.dkv_part != nullptr;
  const int kvh = head_split ? hy / G : hy, g_base = head_split ? hy % G : 0;
  const int k_begin = p.cu_k[b], kv_len = p.cu_k[b + 1] - k_begin;
  const int k0 = (lin / grid.y) * 128;
  if (k0 >= kv_len) return;
  const int q_begin = p.cu_q[b], q_len = p.cu_q[b + 1] - q_begin;
  const int off = kv_len - q_len;
  // queries that see at least one key of this tile
  const int kmax = min(k0 + 127, kv_len - 1);
  int qi_lo = 0, qi_hi = q_len;
  if (p.causal) qi_lo = max(0, k0 - off);
  if (p.window > 0) qi_hi = min(q_len, kmax + p.window - off);
  const int i_begin = qi_lo / 128;
  const int n_qt = qi_hi > qi_lo ? (qi_hi + 127) / 128 - i_begin : 0;
  const int n_iter = n_qt * (head_split ? 1 : G);

  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint8_t* smem_al = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t k_s = smem_base, v_s = k_s + Cfg::kTile;
  const uint32_t qdo_s = v_s + Cfg::kTile;                       // stage: Q tile then dO tile
  constexpr uint32_t stat_off = 2 * Cfg::kTile + ST * 2 * Cfg::kTile;

  if (threadIdx.x == 0) {
    abort_flag = 0;
    mbar_init(smem_u32(&kv_full), 1);
    for (int i = 0; i < ST; ++i) { mbar_init(smem_u32(&qdo_full[i]), 1); mbar_init(smem_u32(&qdo_empty[i]), 1); }
    mbar_init(smem_u32(&s_full), 1);
    mbar_init(smem_u32(&dp_full), 1);
    mbar_init(smem_u32(&p_full), FA_BWD_WARPS);
    mbar_init(smem_u32(&ds_full), FA_BWD_WARPS);
    mbar_init(smem_u32(&acc_done), 1);
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&tmem_base_smem), FA_TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_smem;
  volatile int* abortp = &abort_flag;

  if (warp == 0) {
    if (elect_one_sync()) {
      bool ok = true;
      mbar_expect_tx(smem_u32(&kv_full), 2 * Cfg::kTile);
#pragma unroll
      for (int c = 0; c < DCH; ++c) {
        tma_load_2d(k_s + c * CH, &p.k, smem_u32(&kv_full), kvh * D + c * 64, k_begin + k0);
        tma_load_2d(v_s + c * CH, &p.v, smem_u32(&kv_full), kvh * D + c * 64, k_begin + k0);
      }
      int it = 0;
      for (; it < n_iter; ++it) {
        const int h = kvh * G + g_base + it / n_qt, i = i_begin + it % n_qt;
        const int stage = it % ST;
        ok = mbar_wait_backoff(smem_u32(&qdo_empty[stage]), ((it / ST) & 1u) ^ 1u, abortp, p.status, ST_TIMEOUT_SMEM_EMPTY);
        if (!ok) break;
        const uint32_t fb = smem_u32(&qdo_full[stage]);
        const uint32_t dst = qdo_s + stage * 2 * Cfg::kTile;
        mbar_expect_tx(fb, 2 * Cfg::kTile + Cfg::kStat);
#pragma unroll
        for (int c = 0; c < DCH; ++c) {
          tma_load_2d(dst + c * CH, &p.q, fb, h * D + c * 64, q_begin + i * 128);
          tma_load_2d(dst + Cfg::kTile + c * CH, &p.dout, fb, h * D + c * 64, q_begin + i * 128);
        }
        bulk_load(smem_base + stat_off + stage * Cfg::kStat, p.stat + ((long long)h * p.stat_tiles + (q_begin >> 7) + b + i) * 256, Cfg::kStat, fb);
      }
      if (!ok) {
        auto drain = [&](uint64_t* bar, uint32_t parity) {
          const uint64_t t0 = globaltimer_ns();
          while (!mbar_try_wait(smem_u32(bar), parity))
            if (globaltimer_ns() - t0 > 50000000ull) break;
        };
        drain(&kv_full, 0);
        for (int j = max(0, it - ST); j < it; ++j) drain(&qdo_full[j % ST], (j / ST) & 1u);
      }
    }
  } else if (warp == 1) {
    if (elect_one_sync()) {
      constexpr uint32_t idesc_st = make_idesc_bf16(128, 128, 0, 0);
      constexpr uint32_t idesc_acc = make_idesc_bf16(128, D, 0, 1);
      auto wait = [&](uint64_t* bar, uint32_t parity, int code) { return mbar_wait_backoff(smem_u32(bar), parity, abortp, p.status, code); };
      bool ok = wait(&kv_full, 0, ST_TIMEOUT_SMEM_FULL);
      // [128 keys x 128 queries] of K Q^T (which 0) or V dO^T (which 1)
      auto issue_scores = [&](int it, int which) {
        const uint32_t a_s = which ? v_s : k_s, b_s = qdo_s + (it % ST) * 2 * Cfg::kTile + which * Cfg::kTile;
#pragma unroll
        for (int k = 0; k < D / 16; ++k)
          umma_bf16(tmem_base + which * TM_DP, make_smem_desc_sw128(a_s + (k >> 2) * CH + (k & 3) * 32, 16, 1024),
                    make_smem_desc_sw128(b_s + (k >> 2) * CH + (k & 3) * 32, 16, 1024), idesc_st, k > 0 ? 1u : 0u);
        umma_commit(smem_u32(which ? &dp_full : &s_full));
      };
      // dV += P^T dO (which 0), dK += dS^T Q (which 1)
      auto issue_grad = [&](int it, int which) {
        const uint32_t b_s = qdo_s + (it % ST) * 2 * Cfg::kTile + (which ? 0 : Cfg::kTile);
#pragma unroll
        for (int k = 0; k < 8; ++k)
          umma_bf16_ts(tmem_base + (which ? TM_DK : TM_DV), tmem_base + which * TM_DP + packed_column(k), make_smem_desc_sw128(b_s + k * 2048, CH, 1024),
                       idesc_acc, (it > 0 || k > 0) ? 1u : 0u);
      };
      if (ok && n_iter > 0) {
        ok = wait(&qdo_full[0], 0, ST_TIMEOUT_SMEM_FULL);
        if (ok) {
          tc_fence_after();
          issue_scores(0, 0);
          issue_scores(0, 1);
        }
      }
      for (int it = 0; it < n_iter && ok; ++it) {
        const bool more = it + 1 < n_iter;
        ok = wait(&p_full, it & 1u, ST_TIMEOUT_TMEM_FULL);
        if (!ok) break;
        tc_fence_after();
        issue_grad(it, 0);
        if (more) {
          ok = wait(&qdo_full[(it + 1) % ST], ((it + 1) / ST) & 1u, ST_TIMEOUT_SMEM_FULL);
          if (!ok) break;
          tc_fence_after();
          issue_scores(it + 1, 0);
        }
        ok = wait(&ds_full, it & 1u, ST_TIMEOUT_TMEM_FULL);
        if (!ok) break;
        tc_fence_after();
        issue_grad(it, 1);
        umma_commit(smem_u32(&qdo_empty[it % ST]));
        if (more) issue_scores(it + 1, 1);
      }
      if (ok) umma_commit(smem_u32(&acc_done));
    }
  } else if (warp >= 4) {
    const int qd = warp & 3;
    const int r = qd * 32 + lane;                  // key row of the tile
    const int kj = k0 + r;
    const uint32_t lane_addr = (uint32_t)(qd * 32) << 16;
    const int wg = (warp >> 2) - 1;                // which 32 of the 128 query columns
    const uint32_t tm_s = tmem_base + wg * 32 + lane_addr, tm_p = tm_s + TM_DP;
    const uint64_t scale_l2 = pair(p.scale_log2, p.scale_log2), scale2 = pair(p.scale, p.scale);
    // this key is seen from the query positions q_lo .. q_hi
    const int q_lo = kj >= kv_len ? 1 << 30 : p.causal ? kj : -(1 << 30), q_hi = p.window > 0 ? kj + min(p.window, 1 << 29) - 1 : 1 << 30;
    bool ok = true;
    auto wait = [&](uint64_t* bar, uint32_t parity) -> bool {
      return __all_sync(0xffffffffu, mbar_wait_backoff(smem_u32(bar), parity, abortp, p.status, ST_TIMEOUT_TMEM_FULL));
    };
    for (int it = 0; it < n_iter; ++it) {
      const int qi0 = (i_begin + it % n_qt) * 128, stage = it % ST;
      const uint64_t* stat = reinterpret_cast<const uint64_t*>(smem_al + stat_off + stage * Cfg::kStat) + wg * 16;
      ok = wait(&qdo_full[stage], (it / ST) & 1u) && wait(&s_full, it & 1u);
      if (!ok) break;
      tc_fence_after();
      uint32_t prob[32], packed[16];
      tmem_ld_32x32(tm_s, prob);
      tmem_ld_wait();
      const bool need_mask = (k0 + 127 >= kv_len) || (p.causal && k0 + 127 > off + qi0) ||
                             (p.window > 0 && k0 <= off + qi0 + 127 - p.window);
      const uint32_t dead = need_mask ? outside_mask(off + qi0 + wg * 32, q_lo, q_hi) : 0u;
      bwd_probabilities(prob, scale_l2, [&](int c) { return stat[c >> 1]; }, dead, packed);
      tmem_st_32x16(tm_s, packed);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&p_full));
      ok = wait(&dp_full, it & 1u);
      if (!ok) break;
      tc_fence_after();
      uint32_t dv[32];
      tmem_ld_32x32(tm_p, dv);
      tmem_ld_wait();
      bwd_scores(prob, dv, scale2, [&](int c) { return stat[64 + (c >> 1)]; }, packed);
      tmem_st_32x16(tm_p, packed);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ds_full));
    }
    if (ok && n_iter > 0) ok = wait(&acc_done, 0);
    if (ok) {
      tc_fence_after();
      const bool row_ok = kj < kv_len;
      const int which = wg >> 1, half = wg & 1;    // warpgroups 0, 1: dV; 2, 3: dK; each half of the columns
      __nv_bfloat16* row = (which == 0 ? p.dv : p.dk) + ((long long)(k_begin + kj) * p.Hkv + kvh) * D;
#pragma unroll 1
      for (int c = half * (D / 64); c < (half + 1) * (D / 64); ++c) {
        uint32_t v[32];
        if (n_iter > 0) {
          tmem_ld_32x32(tmem_base + (which == 0 ? TM_DV : TM_DK) + lane_addr + c * 32, v);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = 0u;
        }
        if (row_ok && head_split) {
          float* dst = p.dkv_part + (((long long)(which * G + g_base) * p.Tk + k_begin + kj) * p.Hkv + kvh) * D + c * 32;
#pragma unroll
          for (int u = 0; u < 8; ++u)
            *reinterpret_cast<float4*>(dst + u * 4) = make_float4(__uint_as_float(v[u * 4]), __uint_as_float(v[u * 4 + 1]),
                                                                  __uint_as_float(v[u * 4 + 2]), __uint_as_float(v[u * 4 + 3]));
        } else if (row_ok) {
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            uint4 w;
            w.x = pack_bf16x2(__uint_as_float(v[u * 8 + 0]), __uint_as_float(v[u * 8 + 1]));
            w.y = pack_bf16x2(__uint_as_float(v[u * 8 + 2]), __uint_as_float(v[u * 8 + 3]));
            w.z = pack_bf16x2(__uint_as_float(v[u * 8 + 4]), __uint_as_float(v[u * 8 + 5]));
            w.w = pack_bf16x2(__uint_as_float(v[u * 8 + 6]), __uint_as_float(v[u * 8 + 7]));
            *reinterpret_cast<uint4*>(row + c * 32 + u * 8) = w;
          }
        }
      }
      tc_fence_before();
    }
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, FA_TMEM_COLS);
  }
}

template <int D>
__device__ __forceinline__ void flash_bwd_dq(const FlashBwdParams& p, const dim3& block, const dim3& grid) {
  using Cfg = FlashBwdCfg<D>;
  constexpr int DCH = D / 64;
  constexpr int ST = Cfg::kKvStages;
  constexpr int CH = 128 * 128;
  constexpr uint32_t TM_DP = 128, TM_DQ = 256, TM_Q = 384, TM_DO = 448;      // Q, dO: packed bf16, D / 2 columns
  extern __shared__ __align__(128) uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t qdo_full, qdo_ready, kv_full[ST], kv_empty[ST];
  __shared__ __align__(8) uint64_t s_full, s_read, dp_full, ds_full, acc_done;
  __shared__ uint32_t tmem_base_smem;
  __shared__ int abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int b = block.z, h = block.y;
  const int q_tile = grid.x - 1 - block.x;
  const int q_begin = p.cu_q[b], q_len = p.cu_q[b + 1] - q_begin;
  const int q0 = q_tile * 128;
  if (q0 >= q_len) return;
  const int k_begin = p.cu_k[b], kv_len = p.cu_k[b + 1] - k_begin;
  const int off = kv_len - q_len;
  const int kvh = h / (p.Hq / p.Hkv);
  const int hi = p.causal ? min(kv_len, off + q0 + 128) : kv_len;
  const int lo = p.window > 0 ? max(0, off + q0 - p.window + 1) : 0;
  const int t_begin = lo / 128;
  const int n_iter = max((hi + 127) / 128 - t_begin, 0);

  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint8_t* smem_al = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t q_s = smem_base, do_s = q_s + Cfg::kTile;
  const uint32_t kv_s = do_s + Cfg::kTile;                       // stage: K tile then V tile

  if (threadIdx.x == 0) {
    abort_flag = 0;
    mbar_init(smem_u32(&qdo_full), 1);
    mbar_init(smem_u32(&qdo_ready), 8 * DCH);
    for (int i = 0; i < ST; ++i) { mbar_init(smem_u32(&kv_full[i]), 1); mbar_init(smem_u32(&kv_empty[i]), 1); }
    mbar_init(smem_u32(&s_full), 1);
    mbar_init(smem_u32(&dp_full), 1);
    mbar_init(smem_u32(&s_read), FA_BWD_WARPS);
    mbar_init(smem_u32(&ds_full), FA_BWD_WARPS);
    mbar_init(smem_u32(&acc_done), 1);
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&tmem_base_smem), FA_TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_smem;
  volatile int* abortp = &abort_flag;

  if (warp == 0) {
    if (elect_one_sync()) {
      bool ok = true;
      mbar_expect_tx(smem_u32(&qdo_full), 2 * Cfg::kTile);
#pragma unroll
      for (int c = 0; c < DCH; ++c) {
        tma_load_2d(q_s + c * CH, &p.q, smem_u32(&qdo_full), h * D + c * 64, q_begin + q0);
        tma_load_2d(do_s + c * CH, &p.dout, smem_u32(&qdo_full), h * D + c * 64, q_begin + q0);
      }
      int it = 0;
      for (; it < n_iter; ++it) {
        const int stage = it % ST;
        ok = mbar_wait_backoff(smem_u32(&kv_empty[stage]), ((it / ST) & 1u) ^ 1u, abortp, p.status, ST_TIMEOUT_SMEM_EMPTY);
        if (!ok) break;
        const uint32_t fb = smem_u32(&kv_full[stage]);
        const uint32_t dst = kv_s + stage * 2 * Cfg::kTile;
        const int y = k_begin + (t_begin + it) * 128;
        mbar_expect_tx(fb, 2 * Cfg::kTile);
#pragma unroll
        for (int c = 0; c < DCH; ++c) {
          tma_load_2d(dst + c * CH, &p.k, fb, kvh * D + c * 64, y);
          tma_load_2d(dst + Cfg::kTile + c * CH, &p.v, fb, kvh * D + c * 64, y);
        }
      }
      if (!ok) {
        auto drain = [&](uint64_t* bar, uint32_t parity) {
          const uint64_t t0 = globaltimer_ns();
          while (!mbar_try_wait(smem_u32(bar), parity))
            if (globaltimer_ns() - t0 > 50000000ull) break;
        };
        drain(&qdo_full, 0);
        for (int j = max(0, it - ST); j < it; ++j) drain(&kv_full[j % ST], (j / ST) & 1u);
      }
    }
  } else if (warp == 1) {
    if (elect_one_sync()) {
      constexpr uint32_t idesc_s = make_idesc_bf16(128, 128, 0, 0);
      constexpr uint32_t idesc_acc = make_idesc_bf16(128, D, 0, 1);
      auto wait = [&](uint64_t* bar, uint32_t parity, int code) { return mbar_wait_backoff(smem_u32(bar), parity, abortp, p.status, code); };
      bool ok = wait(&qdo_ready, 0, ST_TIMEOUT_SMEM_FULL);
      // Q K^T (which 0) or dO V^T (which 1)
      auto issue_scores = [&](int it, int which) {
        const uint32_t b_s = kv_s + (it % ST) * 2 * Cfg::kTile + which * Cfg::kTile;
#pragma unroll
        for (int k = 0; k < D / 16; ++k)
          umma_bf16_ts(tmem_base + which * TM_DP, tmem_base + (which ? TM_DO : TM_Q) + k * 8,
                       make_smem_desc_sw128(b_s + (k >> 2) * CH + (k & 3) * 32, 16, 1024), idesc_s, k > 0 ? 1u : 0u);
        umma_commit(smem_u32(which ? &dp_full : &s_full));
      };
      if (ok && n_iter > 0) {
        ok = wait(&kv_full[0], 0, ST_TIMEOUT_SMEM_FULL);
        if (ok) {
          tc_fence_after();
          issue_scores(0, 0);
          issue_scores(0, 1);
        }
      }
      for (int it = 0; it < n_iter && ok; ++it) {
        const bool more = it + 1 < n_iter;
        if (more) {
          ok = wait(&kv_full[(it + 1) % ST], ((it + 1) / ST) & 1u, ST_TIMEOUT_SMEM_FULL) && wait(&s_read, it & 1u, ST_TIMEOUT_TMEM_EMPTY);
          if (!ok) break;
          tc_fence_after();
          issue_scores(it + 1, 0);
        }
        ok = wait(&ds_full, it & 1u, ST_TIMEOUT_TMEM_FULL);
        if (!ok) break;
        tc_fence_after();
        const uint32_t k_s = kv_s + (it % ST) * 2 * Cfg::kTile;
#pragma unroll
        for (int k = 0; k < 8; ++k)   // 128 keys = 8 k-steps
          umma_bf16_ts(tmem_base + TM_DQ, tmem_base + TM_DP + packed_column(k), make_smem_desc_sw128(k_s + k * 2048, CH, 1024), idesc_acc,
                       (it > 0 || k > 0) ? 1u : 0u);
        umma_commit(smem_u32(&kv_empty[it % ST]));
        if (more) issue_scores(it + 1, 1);
      }
      if (ok) umma_commit(smem_u32(&acc_done));
    }
  } else if (warp >= 4) {
    const int qd = warp & 3;
    const int r = qd * 32 + lane;                  // query row of the tile
    const int wg = (warp >> 2) - 1;                // which 32 of the 128 key columns
    const int qi = q0 + r, qpos = off + qi;
    const uint32_t lane_addr = (uint32_t)(qd * 32) << 16;
    const uint32_t tm_s = tmem_base + wg * 32 + lane_addr, tm_p = tm_s + TM_DP;
    const uint64_t scale_l2 = pair(p.scale_log2, p.scale_log2), scale2 = pair(p.scale, p.scale);
    float nl = -INFINITY, nd = 0.f;                // a row past the end gets P = 0 everywhere
    if (qi < q_len) {
      const float* st = p.stat + ((long long)h * p.stat_tiles + (q_begin >> 7) + b + q_tile) * 256 + r;
      nl = st[0];
      nd = st[128];
    }
    const uint64_t nl2 = pair(nl, nl), nd2 = pair(nd, nd);
    // keys k_lo .. k_hi are seen from this query
    const int k_lo = p.window > 0 ? qpos - p.window + 1 : 0, k_hi = p.causal ? min(qpos, kv_len - 1) : kv_len - 1;
    bool ok = true;
    auto wait = [&](uint64_t* bar, uint32_t parity) -> bool {
      return __all_sync(0xffffffffu, mbar_wait_backoff(smem_u32(bar), parity, abortp, p.status, ST_TIMEOUT_TMEM_FULL));
    };
    if (wg < 2 * DCH) {      // Q and dO to tensor memory, one 64-column chunk a warpgroup
      ok = wait(&qdo_full, 0);
      if (ok) {
        const int which = wg / DCH, c = wg % DCH;
        const uint8_t* src = smem_al + which * Cfg::kTile + c * CH + r * 128;
        uint32_t v[32];
#pragma unroll
        for (int u = 0; u < 8; ++u) *reinterpret_cast<uint4*>(&v[u * 4]) = *reinterpret_cast<const uint4*>(src + ((u ^ (r & 7)) << 4));
        tmem_st_32x32(tmem_base + (which ? TM_DO : TM_Q) + c * 32 + lane_addr, v);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&qdo_ready));
      }
    }
    for (int it = 0; it < n_iter && ok; ++it) {
      const int k0 = (t_begin + it) * 128;
      ok = wait(&s_full, it & 1u);
      if (!ok) break;
      tc_fence_after();
      uint32_t prob[32], packed[16];
      tmem_ld_32x32(tm_s, prob);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&s_read));
      const bool need_mask = (k0 + 127 >= kv_len) || (p.causal && k0 + 127 > off + q0) ||
                             (p.window > 0 && k0 <= off + q0 + 127 - p.window);
      const uint32_t dead = need_mask ? outside_mask(k0 + wg * 32, k_lo, k_hi) : 0u;
      bwd_probabilities(prob, scale_l2, [&](int) { return nl2; }, dead, packed);
      ok = wait(&dp_full, it & 1u);
      if (!ok) break;
      tc_fence_after();
      uint32_t dv[32];
      tmem_ld_32x32(tm_p, dv);
      tmem_ld_wait();
      bwd_scores(prob, dv, scale2, [&](int) { return nd2; }, packed);
      tmem_st_32x16(tm_p, packed);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ds_full));
    }
    if (ok && n_iter > 0) ok = wait(&acc_done, 0);
    if (ok) {
      tc_fence_after();
      const bool row_ok = qi < q_len;
      __nv_bfloat16* dq_row = p.dq + ((long long)(q_begin + qi) * p.Hq + h) * D;
#pragma unroll 1
      for (int c = wg * (D / 64); c < (wg + 1) * (D / 64); ++c) {       // 16 columns at a time, a quarter of them a warpgroup
        uint32_t v[16];
        if (n_iter > 0) {
          tmem_ld_32x16(tmem_base + TM_DQ + lane_addr + c * 16, v);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = 0u;
        }
        if (row_ok) {
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            uint4 w;
            w.x = pack_bf16x2(__uint_as_float(v[u * 8 + 0]), __uint_as_float(v[u * 8 + 1]));
            w.y = pack_bf16x2(__uint_as_float(v[u * 8 + 2]), __uint_as_float(v[u * 8 + 3]));
            w.z = pack_bf16x2(__uint_as_float(v[u * 8 + 4]), __uint_as_float(v[u * 8 + 5]));
            w.w = pack_bf16x2(__uint_as_float(v[u * 8 + 6]), __uint_as_float(v[u * 8 + 7]));
            *reinterpret_cast<uint4*>(dq_row + c * 16 + u * 8) = w;
          }
        }
      }
      tc_fence_before();
    }
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, FA_TMEM_COLS);
  }
}

// Both passes in one launch: the CTAs of dK and dV, whose loops run over all queries of a group's heads, start first, and those of dQ fill the SMs that
// the last of them leave idle. In launches of their own 24 sequences of up to 640 tokens (14 / 2 heads, D 64) took 73 + 65 us, now 106; 5 of
// up to 6000 (32 / 8, D 128), which have no such tail, 1526 + 1334, now 2882.
template <int D>
__global__ void __launch_bounds__(FA_BWD_THREADS, 1) flash_bwd_kernel(const __grid_constant__ FlashBwdParams p, const dim3 grid_kv, const dim3 grid_q) {
  const unsigned n_kv = grid_kv.x * grid_kv.y * grid_kv.z;
  const bool kv = blockIdx.x < n_kv;
  const dim3 grid = kv ? grid_kv : grid_q;
  const unsigned lin = kv ? blockIdx.x : blockIdx.x - n_kv, yz = lin / grid.x;
  const dim3 block(lin - yz * grid.x, yz % grid.y, yz / grid.y);
  if (kv) flash_bwd_dkdv<D>(p, block, grid);
  else flash_bwd_dq<D>(p, block, grid);
}

// dv / dk = sum over the G query heads of a group of their fp32 partials (fixed order), rounded to bf16.
__global__ void flash_bwd_reduce_kernel(const float* __restrict__ part, int G, long long n, __nv_bfloat16* __restrict__ dv,
                                        __nv_bfloat16* __restrict__ dk) {
  const long long nvec = n >> 2;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < 2 * nvec; i += (long long)gridDim.x * blockDim.x) {
    const int which = i >= nvec;
    const long long j = which ? i - nvec : i;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int g = 0; g < G; ++g) {
      const float4 v = __ldcs(reinterpret_cast<const float4*>(part + ((long long)which * G + g) * n) + j);
      acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
    }
    uint2 o;
    o.x = pack_bf16x2(acc.x, acc.y);
    o.y = pack_bf16x2(acc.z, acc.w);
    reinterpret_cast<uint2*>(which ? dk : dv)[j] = o;
  }
}

template <int D>
static int launch_flash_bwd(const FlashBwdParams& p, dim3 grid_kv, dim3 grid_q, cudaStream_t stream) {
  constexpr int smem = FlashBwdCfg<D>::kSmemDkdv > FlashBwdCfg<D>::kSmemDq ? FlashBwdCfg<D>::kSmemDkdv : FlashBwdCfg<D>::kSmemDq;
  static bool attr_dev[64] = {};       // the shared-memory opt-in is a per-device function attribute
  int dev_i = 0;
  if (cudaGetDevice(&dev_i) != cudaSuccess || dev_i < 0 || dev_i >= 64) return -10;
  bool& attr = attr_dev[dev_i];
  if (!attr) {
    if (cudaFuncSetAttribute(flash_bwd_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return -10;
    attr = true;
  }
  const unsigned long long n_kv = (unsigned long long)grid_kv.x * grid_kv.y * grid_kv.z, n_q = (unsigned long long)grid_q.x * grid_q.y * grid_q.z;
  if (n_kv == 0 || n_q == 0 || n_kv + n_q > 0x7fffffffull) return -11;
  if (launch_kernel(flash_bwd_kernel<D>, dim3((unsigned)(n_kv + n_q)), dim3(FA_BWD_THREADS), smem, stream, p, grid_kv, grid_q) != cudaSuccess) return -11;
  if (p.dkv_part != nullptr) {
    const long long n = (long long)p.Tk * p.Hkv * D;
    long long blocks = (2 * (n >> 2) + 255) / 256;
    if (blocks > 148 * 8) blocks = 148 * 8;
    flash_bwd_reduce_kernel<<<(unsigned)blocks, 256, 0, stream>>>(p.dkv_part, p.Hq / p.Hkv, n, p.dv, p.dk);
  }
  return 0;
}

template <int D>
static int launch_flash_fwd(const FlashFwdParams& p, int max_seqlen_q, int B, cudaStream_t stream) {
  static bool attr_dev[64] = {}, two_tiles[64] = {};       // the shared-memory opt-in is a per-device function attribute
  int dev_i = 0;
  if (cudaGetDevice(&dev_i) != cudaSuccess || dev_i < 0 || dev_i >= 64) return -10;
  bool& attr = attr_dev[dev_i];
  if (!attr) {
    if (cudaFuncSetAttribute(flash_fwd_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, FlashCfg<D>::kSmemBytes) != cudaSuccess ||
        cudaFuncSetAttribute(flash_fwd2_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, Flash2Cfg<D>::kSmemBytes) != cudaSuccess)
      return -10;
    // The register shares of the roles have to add up to what a block is launched with. A compiler that gives the kernel fewer leaves all
    // sizes to the one-tile kernel.
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, flash_fwd2_kernel<D>) != cudaSuccess) return -13;
    two_tiles[dev_i] = fa.numRegs >= FA2_REGS_LAUNCH;
    attr = true;
  }
  static const bool one_tile = getenv("RB_FLASH_ONE_TILE") != nullptr;
  // Two query tiles per CTA share every K/V tile; a single tile's rows are better split over both warpgroups (flash_fwd_kernel).
  // Causal, TFLOP/s, dense / paged keys (in brackets with P in shared memory and a CTA per tile pair): 4 x 8192 tokens, 32 / 8
  // heads, D 128 1215 / 1000 (854 / 619); 8 x 2048 952 / 932 (475 / 417); 32 x 200 160 / 160 (67 / 66); 1 x 16384, 14 / 2 heads,
  // D 64 633 / 656 (506 / 333); 16 x 512 193 / 193 (82 / 80).
  if (max_seqlen_q > FA_BM && two_tiles[dev_i] && !one_tile) {
    dim3 grid((max_seqlen_q + 2 * FA_BM - 1) / (2 * FA_BM), p.Hq, B);
    return launch_kernel(flash_fwd2_kernel<D>, grid, dim3(FA2_THREADS), Flash2Cfg<D>::kSmemBytes, stream, p) == cudaSuccess ? 0 : -11;
  }
  dim3 grid((max_seqlen_q + FA_BM - 1) / FA_BM, p.Hq, B);
  return launch_kernel(flash_fwd_kernel<D>, grid, dim3(FA_THREADS), FlashCfg<D>::kSmemBytes, stream, p) == cudaSuccess ? 0 : -11;
}

}  // namespace rb

extern "C" {

// Packed varlen attention forward. Dense mode: k, v are [Tk, Hkv, D] views with row strides
// ldk, ldv (elements) and cu_k gives the key ranges. Paged mode: k, v are the cache
// [num_blocks, Hkv, 16, D] (kv_rows = num_blocks), keys of sequence b are the first seq_lens[b]
// slots of its block table and its queries are the LAST (cu_q[b+1]-cu_q[b]) positions.
// Rows of out are ldo apart. chunk > 0: a query sees the keys of its own run of `chunk` positions; gate: see FlashFwdParams.
int rb_flash_fwd_ex(const void* q, const void* k, const void* v, void* out, long long ldo, float* lse, const int* cu_q,
                    const int* cu_k, const int* seq_lens, const int* block_tables, int B, int Tq, int kv_rows,
                    int Hq, int Hkv, int D, int ldq, int ldk, int ldv, int max_seqlen_q, int max_blocks, int causal,
                    int window, int chunk, int paged, const float* gate, long long ld_gate, float gate_scale, float scale, int* status,
                    cudaStream_t stream) {
  using namespace rb;
  if (B <= 0 || Tq <= 0 || max_seqlen_q <= 0) return 0;
  if ((D != 64 && D != 128) || Hq % Hkv != 0 || ldo % 8 != 0 || (window > 0 && chunk > 0)) return -1;
  FlashFwdParams p;
  if (tma_map_2d_bf16(&p.q_map, q, Tq, (unsigned long long)Hq * D, ldq, FA_BM) != 0) return -20;
  if (!paged) {
    if (tma_map_2d_bf16(&p.k_map, k, kv_rows, (unsigned long long)Hkv * D, ldk, FA_BN) != 0) return -21;
    if (tma_map_2d_bf16(&p.v_map, v, kv_rows, (unsigned long long)Hkv * D, ldv, FA_BN) != 0) return -22;
  } else {
    const unsigned long long rows = (unsigned long long)kv_rows * Hkv * 16;
    if (tma_map_2d_bf16(&p.k_map, k, rows, D, D, 16) != 0) return -21;
    if (tma_map_2d_bf16(&p.v_map, v, rows, D, D, 16) != 0) return -22;
  }
  p.out = (__nv_bfloat16*)out;
  p.lse = lse;
  p.cu_q = cu_q;
  p.cu_k = cu_k;
  p.seq_lens = seq_lens;
  p.block_tables = block_tables;
  p.max_blocks = max_blocks;
  p.num_blocks = paged ? kv_rows : 0;
  p.Hq = Hq;
  p.Hkv = Hkv;
  p.Tq = Tq;
  p.causal = causal;
  p.window = window;
  p.chunk = chunk;
  p.gate = gate;
  p.ld_gate = ld_gate;
  p.gate_scale = gate_scale;
  p.ldo = ldo;
  p.paged = paged;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.status = status;
  int rc = D == 64 ? launch_flash_fwd<64>(p, max_seqlen_q, B, stream) : launch_flash_fwd<128>(p, max_seqlen_q, B, stream);
  if (rc != 0) return rc;
  return cudaGetLastError() == cudaSuccess ? 0 : -12;
}

int rb_flash_fwd(const void* q, const void* k, const void* v, void* out, float* lse, const int* cu_q,
                 const int* cu_k, const int* seq_lens, const int* block_tables, int B, int Tq, int kv_rows,
                 int Hq, int Hkv, int D, int ldq, int ldk, int ldv, int max_seqlen_q, int max_blocks, int causal,
                 int window, int paged, float scale, int* status, cudaStream_t stream) {
  return rb_flash_fwd_ex(q, k, v, out, (long long)Hq * D, lse, cu_q, cu_k, seq_lens, block_tables, B, Tq, kv_rows, Hq, Hkv, D, ldq, ldk, ldv,
                         max_seqlen_q, max_blocks, causal, window, 0, paged, nullptr, 0, 1.f, scale, status, stream);
}

// Latent attention, expanded form: see flash_latent_kernel. q [T, H*(DN+64)], k [S, H*DN], rot [S, 64], v [S, H*DV]; the
// queries of sequence b are rows cu_q[b]..cu_q[b+1] of q and out, its keys rows cu_k[b]..cu_k[b+1].
int rb_flash_latent(const void* q, const void* k, const void* rot, const void* v, void* out, const int* cu_q, const int* cu_k,
                    const float* sink, const float* gate, int B, int H, int T, int S, int max_q, int DN, int DV, int window,
                    float scale, int* status, cudaStream_t stream) {
  using namespace rb;
  if (B <= 0 || T <= 0 || S <= 0 || max_q <= 0) return 0;
  if ((DN != 64 && DN != 128) || (DV != 64 && DV != 128) || window < 1 || B > 65535 || H > 65535) return -1;
  FlashLatentParams p;
  const unsigned long long hq = (unsigned long long)H * (DN + 64), hk = (unsigned long long)H * DN, hv = (unsigned long long)H * DV;
  if (tma_map_2d_bf16(&p.q_map, q, T, hq, hq, FA_BM) != 0) return -20;
  if (tma_map_2d_bf16(&p.k_map, k, S, hk, hk, FA_BN) != 0) return -21;
  if (tma_map_2d_bf16(&p.r_map, rot, S, 64, 64, FA_BN) != 0) return -22;
  if (tma_map_2d_bf16(&p.v_map, v, S, hv, hv, FA_BN) != 0) return -23;
  p.out = (__nv_bfloat16*)out;
  p.cu_q = cu_q;
  p.cu_k = cu_k;
  p.sink = sink;
  p.gate = gate;
  p.H = H;
  p.window = window;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.status = status;
  int rc;
  if (DN == 128) rc = DV == 128 ? launch_flash_latent<128, 128>(p, max_q, B, stream) : launch_flash_latent<128, 64>(p, max_q, B, stream);
  else rc = DV == 128 ? launch_flash_latent<64, 128>(p, max_q, B, stream) : launch_flash_latent<64, 64>(p, max_q, B, stream);
  if (rc != 0) return rc;
  return cudaGetLastError() == cudaSuccess ? 0 : -12;
}

// Backward of rb_flash_fwd in dense mode. out, dout, dq are contiguous [Tq,Hq,D]; dk, dv contiguous
// [Tk,Hkv,D]; workspace (16-byte aligned) holds Hq * (Tq / 128 + B + 1) * 256 floats (row statistics by tiles of 128 queries). dkv_part (may be null): 2*(Hq/Hkv)*Tk*Hkv*D
// floats; when given, dK/dV run with one CTA per (key tile, query head) and are reduced over each group afterwards
// (few long sequences: the per-kv-head grid is too coarse to fill the SMs).
int rb_flash_bwd(const void* q, const void* k, const void* v, const void* out, const void* dout, const float* lse,
                 void* dq, void* dk, void* dv, const int* cu_q, const int* cu_k, float* workspace, float* dkv_part, int B, int Tq,
                 int Tk, int Hq, int Hkv, int D, int ldq, int ldk, int ldv, int max_seqlen_q, int max_seqlen_k,
                 int causal, int window, float scale, int* status, cudaStream_t stream) {
  using namespace rb;
  if (B <= 0 || Tq <= 0 || Tk <= 0) return 0;
  if ((D != 64 && D != 128) || Hq % Hkv != 0) return -1;
  FlashBwdParams p;
  const unsigned long long qc = (unsigned long long)Hq * D, kc = (unsigned long long)Hkv * D;
  if (tma_map_2d_bf16(&p.q, q, Tq, qc, ldq, 128) != 0) return -20;
  if (tma_map_2d_bf16(&p.dout, dout, Tq, qc, qc, 128) != 0) return -21;
  if (tma_map_2d_bf16(&p.k, k, Tk, kc, ldk, 128) != 0) return -22;
  if (tma_map_2d_bf16(&p.v, v, Tk, kc, ldv, 128) != 0) return -23;
  if (((unsigned long long)workspace & 15) != 0) return -1;
  p.stat = workspace;
  p.stat_tiles = Tq / 128 + B + 1;
  p.dkv_part = (Hq > Hkv) ? dkv_part : nullptr;
  p.dq = (__nv_bfloat16*)dq;
  p.dk = (__nv_bfloat16*)dk;
  p.dv = (__nv_bfloat16*)dv;
  p.cu_q = cu_q;
  p.cu_k = cu_k;
  p.Hq = Hq; p.Hkv = Hkv; p.Tq = Tq; p.Tk = Tk;
  p.causal = causal; p.window = window;
  p.scale = scale;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.status = status;
  const dim3 prep_grid((max_seqlen_q + 127) / 128, B, Hq);
  const auto prep = D == 64 ? flash_bwd_prep_kernel<64> : flash_bwd_prep_kernel<128>;
  if (launch_kernel(prep, prep_grid, dim3(256), 0, stream, (const __nv_bfloat16*)dout, (const __nv_bfloat16*)out, lse, workspace, cu_q, p.stat_tiles, Tq, Hq) !=
      cudaSuccess)
    return -11;
  dim3 grid_kv((max_seqlen_k + 127) / 128, p.dkv_part != nullptr ? Hq : Hkv, B), grid_q((max_seqlen_q + 127) / 128, Hq, B);
  int rc = D == 64 ? launch_flash_bwd<64>(p, grid_kv, grid_q, stream) : launch_flash_bwd<128>(p, grid_kv, grid_q, stream);
  if (rc != 0) return rc;
  return cudaGetLastError() == cudaSuccess ? 0 : -12;
}

}  // extern "C"
