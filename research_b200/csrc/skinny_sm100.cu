// Products with few activation rows: C[M, N] = A[M, K] B[N, K]^T for M <= 32, the projections of a decode step.
//
// What bounds it: reading the weights B once. A tcgen05 tile would spend 128 accumulator rows on M of them and give an
// output of a few hundred columns to a handful of CTAs, each of which pays barrier and tensor-memory set-up and a chain
// of staged tiles; here every warp streams its own 16 weight rows straight from global memory into the fragments of
// mma.m16n8k16 (weights are the M side, tokens the N side) with two 16-byte loads per lane and 32 columns of K, up to
// eight of them in flight per lane, and nothing passes through shared memory but the partial sums.
//
// The K order inside an instruction is free as long as both operands agree: lane (g, t) loads the 8 consecutive values
// at k = 8 t of row g and feeds the first four to one instruction, the last four to the next, so 16-byte loads need no
// shuffles. Split of the work: a CTA's 8 warps cover `wr` row tiles x `wk` slices of K, and a cluster of S CTAs splits
// K further; slices meet in shared memory, the cluster's through distributed shared memory, always summed in the same
// order. K is cut until about 16 warps an SM have work or a slice is three loads long.
//
// With b_static the weights are known not to be written by the kernels before this one on the stream: their first loads
// are issued before the programmatic-launch wait and overlap the producer of A.
#include "common.cuh"
#include "gemm_epilogue.cuh"

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

constexpr int SK_THREADS = 256;

// NT: groups of 8 tokens
template <int NT>
__global__ void __launch_bounds__(SK_THREADS, 2) skinny_kernel(const __grid_constant__ SkinnyParams p) {
  constexpr int T = 8 * NT;
  constexpr int SK_UNROLL = NT > 2 ? 1 : 2;         // 64-column steps of K per batch of loads; two batches are in flight
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
  if (p.b_static) load_w(w[0], s_begin);
  pdl_wait();
  if (!p.b_static) load_w(w[0], s_begin);

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
    load_w(w[1], s + SK_UNROLL);
    multiply(w[0], s);
    if (s + 2 * SK_UNROLL < s_end) load_w(w[0], s + 2 * SK_UNROLL);
    if (s + SK_UNROLL < s_end) multiply(w[1], s + SK_UNROLL);
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
    float v = total(m, c) * f;
    if (p.bias != nullptr) v += __bfloat162float(p.bias[col]);
    if (p.residual != nullptr) v += __bfloat162float(p.residual[m * p.ldr + col]);
    if (p.softcap > 0.f) v = p.softcap * tanhf(v * (1.f / p.softcap));
    if (p.tail != nullptr && col >= p.tail_col) {
      p.tail[m * p.tail_ld + (col - p.tail_col)] = v;
      continue;
    }
    if (col < p.silu_cols) v = silu_fast(v);
    if (p.out_f32) reinterpret_cast<float*>(p.C)[m * p.ldc + col] = v;
    else reinterpret_cast<__nv_bfloat16*>(p.C)[m * p.ldc + col] = __float2bfloat16_rn(v);
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

}  // namespace rb

extern "C" {

void rb_skinny_set_pdl(int on) { rb::pdl_enabled() = on != 0; }

// C[M, N] = A[M, K] B[N, K]^T, M <= 32; K and N multiples of 8, rows 16-byte aligned. Epilogues as in rb_gemm_bf16_ex: bias,
// residual, fp32 output, gate|up unit (glu_half rows of each, alternating), folded RMS norm, soft cap, silu_cols, tail.
int rb_skinny(const void* A, const void* B, void* C, const void* bias, const void* residual, int M, int N, int K, long long lda,
              long long ldb, long long ldc, long long ldr, int out_f32, int glu_half, int glu_kind, float glu_limit, int norm_fold,
              float norm_eps, float softcap, int silu_cols, float* tail, int tail_col, long long tail_ld, int b_static,
              cudaStream_t stream) {
  using namespace rb;
  if (M <= 0 || M > 32 || N <= 0 || K <= 0 || N % 8 || K % 16 || lda % 16 || ldb % 16) return -1;
  if (((uintptr_t)A | (uintptr_t)B) & 31) return -1;
  if (glu_half > 0 && (glu_half % 16 || N % (2 * glu_half) || bias || residual || out_f32 || tail || silu_cols || softcap > 0.f)) return -1;
  if ((silu_cols || tail) && out_f32) return -1;
  // A CTA's row tiles share the T tokens that come through L1, so more tokens want more of them. K is cut in powers of two
  // while the whole grid fits the SMs at once (16 warps each) and a slice keeps three steps.
  const int tiles = glu_half > 0 ? N / 16 : (N + 15) / 16, steps = (K + 63) / 64, nt = (M + 7) / 8;
  const int min_wr = nt > 2 ? 4 : (nt > 1 || glu_half > 0) ? 2 : 1;
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
  return nt == 1 ? launch_skinny<1>(p, blocks, stream) : nt == 2 ? launch_skinny<2>(p, blocks, stream) : launch_skinny<4>(p, blocks, stream);
}

}  // extern "C"
