// Products with few activation rows: C[M, N] = A[M, K] B[N, K]^T, the projections of a decode step. skinny_kernel for M <= 16,
// stream_kernel (below) for up to 64.
//
// What bounds both: reading the weights B once. A tcgen05 tile would spend 128 accumulator rows on M of them and give an
// output of a few hundred columns to a handful of CTAs, each of which pays barrier and tensor-memory set-up and a chain
// of staged tiles; in skinny_kernel every warp streams its own 16 weight rows straight from global memory into the fragments of
// mma.m16n8k16 (weights are the M side, tokens the N side) with two 32-byte loads per lane and 64 columns of K, up to
// eight of them in flight per lane, and nothing passes through shared memory but the partial sums.
//
// The K order inside an instruction is free as long as both operands agree: lane (g, t) loads the 16 consecutive values
// at k = 16 t of row g and feeds four to each of four instructions, so 32-byte loads need no shuffles (a load of 8 rows x 64 bytes
// occupies the load unit as long as one of 8 rows x 128 bytes: 16-byte loads were a fifth slower). Split of the work: a CTA's 8 warps cover `wr` row tiles x `wk` slices of K, and a cluster of S CTAs splits
// K further; slices meet in shared memory, the cluster's through distributed shared memory, always summed in the same
// order. K is cut until about 16 warps an SM have work or a slice is less than three loads long.
//
// With b_static the weights are known not to be written by the kernels before this one on the stream: their first loads
// are issued before the programmatic-launch wait and overlap the producer of A.
#include "common.cuh"
#include "gemm_epilogue.cuh"
#include "tma_host.h"

namespace rb {

struct SkinnyParams {
  const __nv_bfloat16* A;
  const __nv_bfloat16* B;
  void* C;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* residual;
  long long lda, ldb, ldc, ldr;
  int M, N, K;
  int log_wr, splits;          // row tiles per CTA (log2), CTAs per cluster
  int b_static, out_f32;
  int glu_half, glu_kind;      // glu_half > 0: B holds blocks of so many gate rows, then as many up rows
  float glu_limit;
  int norm_fold;
  float norm_eps;
  float softcap;
  int silu_cols, tail_col;
  float* tail;
  long long tail_ld;
};

struct Row16 {      // 16 consecutive bf16 values of a row
  uint32_t v[8];
};
__device__ __forceinline__ Row16 ld_stream(const void* p) {
  Row16 r;
  asm volatile("ld.global.L1::no_allocate.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]), "=r"(r.v[7])
               : "l"(p) : "memory");
  return r;
}
__device__ __forceinline__ Row16 ld_cached(const void* p) {
  Row16 r;
  asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]), "=r"(r.v[7])
               : "l"(p) : "memory");
  return r;
}
__device__ __forceinline__ Row16 no_row() { return {{0, 0, 0, 0, 0, 0, 0, 0}}; }
__device__ __forceinline__ void mma_16n8k16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float square_sum(const Row16& r, float s) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float2 f = unpack_bf16x2(r.v[i]);
    s = fmaf(f.x, f.x, s);
    s = fmaf(f.y, f.y, s);
  }
  return s;
}

// Everything behind the (scaled) sum of a plain product's element
__device__ __forceinline__ void finish_column(const SkinnyParams& p, int m, long long col, float v) {
  if (p.bias != nullptr) v += __bfloat162float(p.bias[col]);
  if (p.residual != nullptr) v += __bfloat162float(p.residual[m * p.ldr + col]);
  if (p.softcap > 0.f) v = p.softcap * tanhf(v * (1.f / p.softcap));
  if (p.tail != nullptr && col >= p.tail_col) {
    p.tail[m * p.tail_ld + (col - p.tail_col)] = v;
    return;
  }
  if (col < p.silu_cols) v = silu_fast(v);
  if (p.out_f32) reinterpret_cast<float*>(p.C)[m * p.ldc + col] = v;
  else reinterpret_cast<__nv_bfloat16*>(p.C)[m * p.ldc + col] = __float2bfloat16_rn(v);
}

// Four columns from col on (a multiple of 4; silu_cols and tail_col are multiples of 32); `quads`: by 8- and 16-byte accesses
__device__ __forceinline__ void store_quad(const SkinnyParams& p, int m, long long col, const float (&v)[4], int quads) {
  __nv_bfloat16* bf = reinterpret_cast<__nv_bfloat16*>(p.C) + m * p.ldc + col;
  float* fp = reinterpret_cast<float*>(p.C) + m * p.ldc + col;
  if (quads) {
    if (p.out_f32) *reinterpret_cast<float4*>(fp) = make_float4(v[0], v[1], v[2], v[3]);
    else *reinterpret_cast<uint2*>(bf) = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
    return;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (p.out_f32) fp[i] = v[i];
    else bf[i] = __float2bfloat16_rn(v[i]);
  }
}
__device__ __forceinline__ void finish_quad(const SkinnyParams& p, int m, long long col, float (&v)[4], int quads) {
  const bool tail = p.tail != nullptr && col >= p.tail_col;
  if (!quads || tail) {
#pragma unroll
    for (int i = 0; i < 4; ++i) finish_column(p, m, col + i, v[i]);
    return;
  }
  auto add = [&](const __nv_bfloat16* at) {
    const uint2 x = *reinterpret_cast<const uint2*>(at);
    const float2 lo = unpack_bf16x2(x.x), hi = unpack_bf16x2(x.y);
    v[0] += lo.x; v[1] += lo.y; v[2] += hi.x; v[3] += hi.y;
  };
  if (p.bias != nullptr) add(p.bias + col);
  if (p.residual != nullptr) add(p.residual + m * p.ldr + col);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (p.softcap > 0.f) v[i] = p.softcap * tanhf(v[i] * (1.f / p.softcap));
    if (col < p.silu_cols) v[i] = silu_fast(v[i]);
  }
  store_quad(p, m, col, v, quads);
}

constexpr int SK_THREADS = 256;

// NT: groups of 8 tokens
template <int NT>
__global__ void __launch_bounds__(SK_THREADS, 2) skinny_kernel(const __grid_constant__ SkinnyParams p) {
  constexpr int T = 8 * NT;
  constexpr int SK_UNROLL = 2;         // 64-column steps of K per batch of loads; two batches are in flight
  __shared__ __align__(16) float red[T * 160];      // partial sums [wk][T][16 wr + 4]: wk (16 wr + 4) <= 160
  __shared__ float ssq[8][T];
  __shared__ float rstd[T];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int wr = 1 << p.log_wr, wk = 8 >> p.log_wr, S = p.splits;
  const int rt = warp & (wr - 1), ks = warp >> p.log_wr;
  const int rank = blockIdx.x % S, block = blockIdx.x / S;
  const int R = 16 << p.log_wr, LD = R + 4;

  // the 16 weight rows of this warp
  int row0;
  if (p.glu_half > 0) {
    const int col = ((block * wr + rt) >> 1) * 16, j = col / p.glu_half;
    row0 = col < (p.N >> 1) ? j * 2 * p.glu_half + (rt & 1) * p.glu_half + (col - j * p.glu_half) : p.N;
  } else {
    row0 = (block * wr + rt) * 16;
  }
  const bool ok0 = row0 + g < p.N, ok1 = row0 + g + 8 < p.N;
  const __nv_bfloat16* b0 = p.B + (long long)(ok0 ? row0 + g : 0) * p.ldb;
  const __nv_bfloat16* b1 = p.B + (long long)(ok1 ? row0 + g + 8 : 0) * p.ldb;
  const int steps = (p.K + 63) >> 6, parts = wk * S, part = rank * wk + ks;
  const int s_begin = (int)((long long)steps * part / parts), s_end = (int)((long long)steps * (part + 1) / parts);

  Row16 w[2][SK_UNROLL][2];
  auto load_w = [&](Row16 (&dst)[SK_UNROLL][2], int s) {
#pragma unroll
    for (int u = 0; u < SK_UNROLL; ++u) {
      const int k = (s + u) * 64 + t * 16;
      const bool in = s + u < s_end && k < p.K;
      dst[u][0] = in && ok0 ? ld_stream(b0 + k) : no_row();
      dst[u][1] = in && ok1 ? ld_stream(b1 + k) : no_row();
    }
  };
  pdl_launch_dependents();
  // both batches: a slice of up to four steps then waits for nothing but its activations
  if (!p.b_static) pdl_wait();
  load_w(w[0], s_begin);
  load_w(w[1], s_begin + SK_UNROLL);
  if (p.b_static) pdl_wait();

  float acc[NT][4], sq[NT];
  const __nv_bfloat16* arow[NT];
  bool aok[NT];
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
    sq[n] = 0.f;
    aok[n] = n * 8 + g < p.M;
    arow[n] = p.A + (long long)(aok[n] ? n * 8 + g : 0) * p.lda;
  }
  const bool squares = p.norm_fold && rt == 0;
  auto load_x = [&](Row16 (&x)[NT], int s) {
    const int k = s * 64 + t * 16;
    const bool in = s < s_end && k < p.K;
#pragma unroll
    for (int n = 0; n < NT; ++n) x[n] = in && aok[n] ? ld_cached(arow[n] + k) : no_row();
  };
  auto multiply = [&](const Row16 (&v)[SK_UNROLL][2], int s) {
    Row16 x[SK_UNROLL][NT];
#pragma unroll
    for (int u = 0; u < SK_UNROLL; ++u) load_x(x[u], s + u);
#pragma unroll
    for (int u = 0; u < SK_UNROLL; ++u) {
#pragma unroll
      for (int n = 0; n < NT; ++n) {
#pragma unroll
        for (int i = 0; i < 8; i += 2)
          mma_16n8k16(acc[n], v[u][0].v[i], v[u][1].v[i], v[u][0].v[i + 1], v[u][1].v[i + 1], x[u][n].v[i], x[u][n].v[i + 1]);
        if (squares) sq[n] = square_sum(x[u][n], sq[n]);
      }
    }
  };
  for (int s = s_begin; s < s_end; s += 2 * SK_UNROLL) {
    multiply(w[0], s);
    if (s + 2 * SK_UNROLL < s_end) load_w(w[0], s + 2 * SK_UNROLL);
    if (s + SK_UNROLL < s_end) multiply(w[1], s + SK_UNROLL);
    if (s + 3 * SK_UNROLL < s_end) load_w(w[1], s + 3 * SK_UNROLL);
  }

  float* mine = red + ks * T * LD + rt * 16;
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    float* q = mine + (n * 8 + 2 * t) * LD + g;
    q[0] = acc[n][0];
    q[LD] = acc[n][1];
    q[8] = acc[n][2];
    q[LD + 8] = acc[n][3];
    if (squares) {
      float s = sq[n];
      s += __shfl_xor_sync(0xffffffffu, s, 1);
      s += __shfl_xor_sync(0xffffffffu, s, 2);
      if (t == 0) ssq[ks][n * 8 + g] = s;
    }
  }
  __syncthreads();
  if (wk > 1) {      // slices of this CTA
    for (int e = threadIdx.x; e < T * R; e += SK_THREADS) {
      const int m = e >> (4 + p.log_wr), r = e & (R - 1);
      float s = red[m * LD + r];
      for (int i = 1; i < wk; ++i) s += red[(i * T + m) * LD + r];
      red[m * LD + r] = s;
    }
  }
  if (p.norm_fold && threadIdx.x < T) {
    float s = 0.f;
    for (int i = 0; i < wk; ++i) s += ssq[i][threadIdx.x];
    ssq[0][threadIdx.x] = s;
  }
  if (S > 1) cluster_sync_all();
  else __syncthreads();
  if (p.norm_fold) {
    if (threadIdx.x < T) {
      float s = 0.f;
      for (int c = 0; c < S; ++c) s += S > 1 ? ld_dsmem_f1(mapa_cluster(smem_u32(&ssq[0][threadIdx.x]), c)) : ssq[0][threadIdx.x];
      rstd[threadIdx.x] = rsqrtf(s / (float)p.K + p.norm_eps);
    }
    __syncthreads();
  }
  auto total = [&](int m, int r) -> float {
    const float* at = red + m * LD + r;
    if (S == 1) return *at;
    float s = 0.f;
    for (int c = 0; c < S; ++c) s += ld_dsmem_f1(mapa_cluster(smem_u32(at), c));
    return s;
  };
  const int log_out = 4 + p.log_wr - (p.glu_half > 0 ? 1 : 0), RO = 1 << log_out;      // output columns of this CTA (the cluster)
  for (int e = threadIdx.x + rank * SK_THREADS; e < p.M << log_out; e += SK_THREADS * S) {
    const int m = e >> log_out, c = e & (RO - 1);
    const long long col = (long long)block * RO + c;
    const float f = p.norm_fold ? rstd[m] : 1.f;
    if (p.glu_half > 0) {
      if (col >= (p.N >> 1)) continue;
      const int r = (c >> 4) * 32 + (c & 15);
      reinterpret_cast<__nv_bfloat16*>(p.C)[m * p.ldc + col] =
          __float2bfloat16_rn(p.glu_kind == 1 ? clamped_glu_epi(total(m, r) * f, total(m, r + 16) * f, p.glu_limit)
                                              : swiglu_epi(total(m, r) * f, total(m, r + 16) * f));
      continue;
    }
    if (col >= p.N) continue;
    finish_column(p, m, col, total(m, c) * f);
  }
  if (S > 1) cluster_sync_all();       // the others may still read this CTA's sums
}

template <int NT>
static int launch_skinny(const SkinnyParams& p, int blocks, cudaStream_t stream) {
  const dim3 grid((unsigned)(blocks * p.splits));
  const cudaError_t rc = p.splits > 1 ? launch_kernel_cluster(skinny_kernel<NT>, grid, dim3(SK_THREADS), 0, stream, (unsigned)p.splits, p)
                                      : launch_kernel(skinny_kernel<NT>, grid, dim3(SK_THREADS), 0, stream, p);
  return rc == cudaSuccess ? 0 : -11;
}

// ------------------------------------------------------------------------------------------
// The same products for up to 64 rows: the weights are the 128-row side of tcgen05.mma (a CTA has 128 rows of B and all
// tokens), so no accumulator row is spent on padding and an output of a few hundred columns still gives work to many CTAs: K is cut
// over a cluster, whose fp32 partial tiles meet in distributed shared memory, four columns a load, always in the same order.
// What bounds it is reading B once: 16 KB boxes of weights in a ring, two CTAs an SM; with b_static the first of them are on
// their way before the kernel before this one has ended. The epilogue sums four groups of four columns a thread at a time: with one
// group, whose loads from the other CTAs and of the residual wait for each other, 4096 x 4096 at 64 rows took 17.3 us, not 14.0.
// Past 64 rows the partial tiles are what takes the time, and the one-CTA kernel is the better one (128 rows: 896 x 896 8.1 us there, 10.1
// here, 28672 x 4096 49.9 / 51.0). Warp 0 TMA, warp 1 products, warps 2-5 row sums of squares (a folded
// norm) while the ring turns, then all warps the epilogue.
// ------------------------------------------------------------------------------------------
struct StreamParams {
  CUtensorMap w_map, x_map;      // boxes 64 x 128 (64 x 64 with a gated unit) of B, 64 x tokens of A
  SkinnyParams e;
  int tokens, stages;            // M rounded up to 16; ring depth
  int quads;                     // output, residual and bias take four columns at a time
};
constexpr int ST_THREADS = 192, ST_MAX_TOKENS = 64, ST_ROWS = 128, ST_LD = ST_ROWS + 4, ST_MAX_STAGES = 8;

// S: CTAs of a cluster
template <int S>
__global__ void __launch_bounds__(ST_THREADS, 2) stream_kernel(const __grid_constant__ StreamParams sp, int* status) {
  const SkinnyParams& p = sp.e;
  extern __shared__ __align__(128) uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full[ST_MAX_STAGES], empty[ST_MAX_STAGES], acc_full;
  __shared__ float ssq[ST_MAX_TOKENS], rstd[ST_MAX_TOKENS];
  __shared__ uint32_t tmem_base_smem;
  __shared__ int abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = blockIdx.x % S, block = blockIdx.x / S;
  const int T = sp.tokens, stage_bytes = ST_ROWS * 128 + T * 128;
  const int num_kb = (p.K + 63) >> 6, kb0 = (int)((long long)num_kb * rank / S), n_kb = (int)((long long)num_kb * (rank + 1) / S) - kb0;
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_al = smem_raw + (smem_base - smem_u32(smem_raw));
  float* red = reinterpret_cast<float*>(smem_al);        // over the ring once it has run: [tokens][ST_LD]
  const uint32_t tmem_cols = T <= 32 ? 32u : 64u;

  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int i = 0; i < sp.stages; ++i) {
      mbar_init(smem_u32(&full[i]), 1);
      mbar_init(smem_u32(&empty[i]), p.norm_fold ? 5 : 1);       // the products (and the four warps that square)
    }
    mbar_init(smem_u32(&acc_full), 1);
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&tmem_base_smem), tmem_cols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_smem;
  volatile int* abortp = &abort_flag;
  pdl_launch_dependents();
  int issued = 0;      // stages filled by this thread (the elected one of warp 0)

  if (warp == 0) {
    if (elect_one_sync()) {
      int row = block * ST_ROWS, up = 0;
      if (p.glu_half > 0) {
        const int col = block * 64, j = col / p.glu_half;
        row = j * 2 * p.glu_half + (col - j * p.glu_half);
        up = row + p.glu_half;
      }
      auto load_w = [&](int i, int s) {
        const int k = (kb0 + i) * 64;
        const uint32_t fb = smem_u32(&full[s]), dst = smem_base + s * stage_bytes;
        mbar_expect_tx(fb, stage_bytes);
        tma_load_2d(dst, &sp.w_map, fb, k, row);
        if (p.glu_half > 0) tma_load_2d(dst + 64 * 128, &sp.w_map, fb, k, up);
      };
      auto load_x = [&](int i, int s) {
        tma_load_2d(smem_base + s * stage_bytes + ST_ROWS * 128, &sp.x_map, smem_u32(&full[s]), (kb0 + i) * 64, 0);
      };
      const int first = min(sp.stages, n_kb);
      if (!p.b_static) pdl_wait();
      for (int i = 0; i < first; ++i) load_w(i, i);
      if (p.b_static) pdl_wait();
      for (int i = 0; i < first; ++i) load_x(i, i);
      // (slot and phase go along: a division by the depth a stage stood in the way of one thread's loads)
      int i = first, s = 0;
      uint32_t ph = 0;
      for (; i < n_kb; ++i) {
        if (!mbar_wait_bounded(smem_u32(&empty[s]), ph, abortp, status, ST_TIMEOUT_SMEM_EMPTY)) break;
        load_w(i, s);
        load_x(i, s);
        if (++s == sp.stages) { s = 0; ph ^= 1u; }
      }
      issued = i;
    }
  } else if (warp == 1) {
    if (elect_one_sync()) {
      const uint32_t idesc = make_idesc_bf16(ST_ROWS, T, 0, 0);
      bool ok = true;
      pdl_wait();      // no stage is full before: the budget of the first wait is not spent on the kernel before this one
      int s = 0;
      uint32_t ph = 0;
      for (int i = 0; i < n_kb; ++i) {
        ok = mbar_wait_bounded(smem_u32(&full[s]), ph, abortp, status, ST_TIMEOUT_SMEM_FULL);
        if (!ok) break;
        tc_fence_after();
        const uint32_t w_s = smem_base + s * stage_bytes, x_s = w_s + ST_ROWS * 128;
#pragma unroll
        for (int k = 0; k < 4; ++k) umma_bf16_lo(tmem_base, smem_desc_lo(w_s, 16) + 2 * k, smem_desc_lo(x_s, 16) + 2 * k, idesc, (i > 0 || k > 0) ? 1u : 0u);
        umma_commit(smem_u32(&empty[s]));
        if (++s == sp.stages) { s = 0; ph ^= 1u; }
      }
      __threadfence_block();
      umma_commit(smem_u32(&acc_full));      // a wait that ran out has set the flag before
    }
  } else {
    const int tid = threadIdx.x - 64, q = warp & 3;
    pdl_wait();
    float sum = 0.f;
    if (p.norm_fold) {
      int s = 0;
      uint32_t ph = 0;
      for (int i = 0; i < n_kb; ++i) {
        const bool ok = mbar_wait_bounded(smem_u32(&full[s]), ph, abortp, status, ST_TIMEOUT_SMEM_FULL);
        if (!__all_sync(0xffffffffu, ok)) break;
        if (tid < T) {
          const uint8_t* x = smem_al + s * stage_bytes + ST_ROWS * 128 + tid * 128;
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const uint4 v = *reinterpret_cast<const uint4*>(x + ((u ^ (tid & 7)) << 4));
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const float2 f = unpack_bf16x2(w[j]);
              sum = fmaf(f.x, f.x, sum);
              sum = fmaf(f.y, f.y, sum);
            }
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&empty[s]));
        if (++s == sp.stages) { s = 0; ph ^= 1u; }
      }
      if (tid < T) ssq[tid] = sum;
    }
    bool ok = __all_sync(0xffffffffu, mbar_wait_bounded(smem_u32(&acc_full), 0, abortp, status, ST_TIMEOUT_TMEM_FULL));
    if (__any_sync(0xffffffffu, *abortp != 0)) ok = false;       // copies may still land in the ring
    // every warp has left the ring before one of them writes over it
    asm volatile("bar.sync 1, 128;" ::: "memory");
    if (ok) {
      tc_fence_after();
      for (int c0 = 0; c0 < T; c0 += 16) {
        uint32_t v[16];
        tmem_ld_32x16(tmem_base + c0 + ((uint32_t)(q * 32) << 16), v);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j) red[(c0 + j) * ST_LD + q * 32 + lane] = __uint_as_float(v[j]);
      }
      tc_fence_before();
    }
  }
  __syncthreads();
  if (*abortp != 0 && issued > 0) {      // given up: no copy may land in memory, no product read memory that has another use
    auto drain = [&](uint64_t* bar, uint32_t parity) {
      const uint64_t t0 = globaltimer_ns();
      while (!mbar_try_wait(smem_u32(bar), parity))
        if (globaltimer_ns() - t0 > 50000000ull) break;
    };
    for (int j = max(issued - sp.stages, 0); j < issued; ++j) drain(&full[j % sp.stages], (j / sp.stages) & 1u);
    drain(&acc_full, 0);
  }
  if (S > 1) cluster_sync_all();
  if (warp == 0) pdl_wait();
  if (p.norm_fold) {
    for (int t = threadIdx.x; t < p.M; t += ST_THREADS) {
      float s = 0.f;
      for (int c = 0; c < S; ++c) s += S > 1 ? ld_dsmem_f1(mapa_cluster(smem_u32(&ssq[t]), c)) : ssq[t];
      rstd[t] = rsqrtf(s / (float)p.K + p.norm_eps);
    }
    __syncthreads();
  }
  const int log_quads = p.glu_half > 0 ? 4 : 5;             // groups of four output columns of this block
  if (warp != 1 && *abortp == 0) {                          // (warp 1's lanes have not waited for the kernel before)
    constexpr int WORKERS = ST_THREADS - 32, U = S == 8 ? 2 : 4;       // U groups a thread have their loads in flight together
    const int worker = threadIdx.x < 32 ? threadIdx.x : threadIdx.x - 32, count = p.M << log_quads;
    uint32_t peer[S];
#pragma unroll
    for (int c = 0; c < S; ++c) peer[c] = S > 1 ? mapa_cluster(smem_u32(red), c) : smem_u32(red);
    auto sums = [&](float4 (&v)[U], int e0, int up) {       // of the groups e0 + u * WORKERS * S, in the order of the ranks
      float4 part[U][S];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int e = min(e0 + u * WORKERS * S, count - 1);
        const uint32_t at = ((e >> log_quads) * ST_LD + (e & ((1 << log_quads) - 1)) * 4 + up) * 4;
#pragma unroll
        for (int c = 0; c < S; ++c) part[u][c] = S > 1 ? ld_dsmem_f4(peer[c] + at) : *reinterpret_cast<const float4*>(reinterpret_cast<const uint8_t*>(red) + at);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        v[u] = part[u][0];
#pragma unroll
        for (int c = 1; c < S; ++c) { v[u].x += part[u][c].x; v[u].y += part[u][c].y; v[u].z += part[u][c].z; v[u].w += part[u][c].w; }
      }
    };
    for (int e0 = worker + rank * WORKERS; e0 < count; e0 += U * WORKERS * S) {
      float4 a[U], b[U];
      sums(a, e0, 0);
      if (p.glu_half > 0) sums(b, e0, 64);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int e = e0 + u * WORKERS * S;
        if (e >= count) break;
        const int m = e >> log_quads;
        const long long col = ((long long)block << (log_quads + 2)) + (e & ((1 << log_quads) - 1)) * 4;
        const float f = p.norm_fold ? rstd[m] : 1.f;
        float v[4] = {a[u].x * f, a[u].y * f, a[u].z * f, a[u].w * f};
        if (p.glu_half > 0) {
          const float w[4] = {b[u].x * f, b[u].y * f, b[u].z * f, b[u].w * f};
#pragma unroll
          for (int i = 0; i < 4; ++i) v[i] = p.glu_kind == 1 ? clamped_glu_epi(v[i], w[i], p.glu_limit) : swiglu_epi(v[i], w[i]);
          if (col < (p.N >> 1)) store_quad(p, m, col, v, sp.quads);
        } else if (col < p.N) {                             // (N is a multiple of 8)
          finish_quad(p, m, col, v, sp.quads);
        }
      }
    }
  }
  __syncthreads();
  if (S > 1) cluster_sync_all();       // the others may still read this CTA's sums
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, tmem_cols);
  }
}

template <int S>
static int launch_stream(const StreamParams& p, int grid, size_t smem, int* status, cudaStream_t stream) {
  static bool attr_dev[64] = {};       // the shared-memory opt-in is a per-device function attribute
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -10;
  if (!attr_dev[dev]) {
    if (cudaFuncSetAttribute(stream_kernel<S>, cudaFuncAttributeMaxDynamicSharedMemorySize, 112 * 1024) != cudaSuccess) return -10;
    attr_dev[dev] = true;
  }
  const cudaError_t rc = S > 1 ? launch_kernel_cluster(stream_kernel<S>, dim3(grid), dim3(ST_THREADS), smem, stream, (unsigned)S, p, status)
                                        : launch_kernel(stream_kernel<S>, dim3(grid), dim3(ST_THREADS), smem, stream, p, status);
  return rc == cudaSuccess ? 0 : -11;
}

}  // namespace rb

extern "C" {

void rb_skinny_set_pdl(int on) { rb::pdl_enabled() = on != 0; }

// C[M, N] = A[M, K] B[N, K]^T, M <= 16; K a multiple of 16, N of 8, rows 32-byte aligned. Epilogues as in rb_gemm_bf16_ex: bias,
// residual, fp32 output, gate|up unit (glu_half rows of each, alternating), folded RMS norm, soft cap, silu_cols, tail.
int rb_skinny(const void* A, const void* B, void* C, const void* bias, const void* residual, int M, int N, int K, long long lda,
              long long ldb, long long ldc, long long ldr, int out_f32, int glu_half, int glu_kind, float glu_limit, int norm_fold,
              float norm_eps, float softcap, int silu_cols, float* tail, int tail_col, long long tail_ld, int b_static,
              cudaStream_t stream) {
  using namespace rb;
  if (M <= 0 || M > 16 || N <= 0 || K <= 0 || N % 8 || K % 16 || lda % 16 || ldb % 16) return -1;
  if (((uintptr_t)A | (uintptr_t)B) & 31) return -1;
  if (glu_half > 0 && (glu_half % 16 || N % (2 * glu_half) || bias || residual || out_f32 || tail || silu_cols || softcap > 0.f)) return -1;
  if ((silu_cols || tail) && out_f32) return -1;
  // A CTA's row tiles share the T tokens that come through L1, so more tokens want more of them. K is cut in powers of two
  // while the whole grid fits the SMs at once (16 warps each) and what is cut has three 64-column steps: no slice is below one and a half.
  const int tiles = glu_half > 0 ? N / 16 : (N + 15) / 16, steps = (K + 63) / 64, nt = (M + 7) / 8;
  const int min_wr = nt > 1 || glu_half > 0 ? 2 : 1;
  int parts = 1;
  while (parts * 2 * min_wr <= 64 && tiles * parts * 2 <= 148 * 16 && steps >= 3 * parts) parts *= 2;
  const int wk = parts < 8 / min_wr ? parts : 8 / min_wr;
  SkinnyParams p;
  p.A = (const __nv_bfloat16*)A; p.B = (const __nv_bfloat16*)B; p.C = C;
  p.bias = (const __nv_bfloat16*)bias; p.residual = (const __nv_bfloat16*)residual;
  p.lda = lda; p.ldb = ldb; p.ldc = ldc; p.ldr = ldr;
  p.M = M; p.N = N; p.K = K;
  p.log_wr = wk == 1 ? 3 : wk == 2 ? 2 : wk == 4 ? 1 : 0;
  p.splits = parts / wk;
  p.b_static = b_static; p.out_f32 = out_f32;
  p.glu_half = glu_half; p.glu_kind = glu_kind; p.glu_limit = glu_limit;
  p.norm_fold = norm_fold; p.norm_eps = norm_eps; p.softcap = softcap;
  p.silu_cols = silu_cols; p.tail_col = tail_col; p.tail = tail; p.tail_ld = tail_ld;
  const int wr = 1 << p.log_wr, blocks = (tiles + wr - 1) / wr;
  return nt == 1 ? launch_skinny<1>(p, blocks, stream) : launch_skinny<2>(p, blocks, stream);
}

// The same for M <= 64 on the tensor cores (stream_kernel): K a multiple of 8, glu_half of 64, rows 16-byte aligned.
int rb_stream(const void* A, const void* B, void* C, const void* bias, const void* residual, int M, int N, int K, long long lda,
              long long ldb, long long ldc, long long ldr, int out_f32, int glu_half, int glu_kind, float glu_limit, int norm_fold,
              float norm_eps, float softcap, int silu_cols, float* tail, int tail_col, long long tail_ld, int b_static, int* status,
              cudaStream_t stream) {
  using namespace rb;
  if (M <= 0 || M > ST_MAX_TOKENS || N <= 0 || K <= 0 || N % 8 || K % 8) return -1;
  if (glu_half > 0 && (glu_half % 64 || N % (2 * glu_half) || bias || residual || out_f32 || tail || silu_cols || softcap > 0.f)) return -1;
  if ((silu_cols || tail) && out_f32) return -1;
  const int tiles = glu_half > 0 ? N / 128 : (N + 127) / 128, num_kb = (K + 63) / 64;
  StreamParams sp;
  SkinnyParams& p = sp.e;
  p.A = nullptr; p.B = nullptr; p.C = C;
  p.bias = (const __nv_bfloat16*)bias; p.residual = (const __nv_bfloat16*)residual;
  p.lda = lda; p.ldb = ldb; p.ldc = ldc; p.ldr = ldr;
  p.M = M; p.N = N; p.K = K;
  p.log_wr = 0; p.b_static = b_static; p.out_f32 = out_f32;
  p.glu_half = glu_half; p.glu_kind = glu_kind; p.glu_limit = glu_limit;
  p.norm_fold = norm_fold; p.norm_eps = norm_eps; p.softcap = softcap;
  p.silu_cols = silu_cols; p.tail_col = tail_col; p.tail = tail; p.tail_ld = tail_ld;
  sp.tokens = (M + 15) / 16 * 16;
  // K is cut in powers of two while the grid stays within one CTA an SM (the first cut beyond that only adds reduction) and a slice
  // keeps two 64-column blocks; the ring is as deep as two CTAs an SM allow.
  int splits = 1;
  while (splits < 8 && tiles * splits * 2 <= 148 && num_kb >= splits * 4) splits *= 2;
  p.splits = splits;
  const int stage = (ST_ROWS + sp.tokens) * 128, per = (num_kb + splits - 1) / splits;
  int stages = (108 * 1024) / stage;
  if (stages > ST_MAX_STAGES) stages = ST_MAX_STAGES;
  if (stages > per) stages = per;
  sp.stages = stages;
  const int red = sp.tokens * ST_LD * 4;
  const size_t smem = 1024 + (stages * stage > red ? stages * stage : red);
  int rc = tma_map_2d_bf16(&sp.w_map, B, N, K, ldb, glu_half > 0 ? 64 : ST_ROWS);
  if (rc != 0) return -20 + rc;
  rc = tma_map_2d_bf16(&sp.x_map, A, M, K, lda, sp.tokens);
  if (rc != 0) return -30 + rc;
  sp.quads = ldc % 4 == 0 && ((uintptr_t)C & (out_f32 ? 15 : 7)) == 0 && (residual == nullptr || (ldr % 4 == 0 && ((uintptr_t)residual & 7) == 0)) &&
             ((uintptr_t)bias & 7) == 0;
  const int grid = tiles * splits;
  return splits == 8   ? launch_stream<8>(sp, grid, smem, status, stream)
         : splits == 4 ? launch_stream<4>(sp, grid, smem, status, stream)
         : splits == 2 ? launch_stream<2>(sp, grid, smem, status, stream)
                       : launch_stream<1>(sp, grid, smem, status, stream);
}

}  // extern "C"
