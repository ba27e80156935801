// Plain matrix product on the CUDA cores, true 32-bit: out[m,n] = sum_k A[m,k] * W[n,k].
//
// This is the product of the float32 path and the reference twin of the tensor-core
// kernels.  Every output element is one chain of FFMAs over k in ascending order that
// starts from zero, whatever M is and whichever tile the element falls into, so a row's
// result does not depend on what else is in the batch.  (The reference's kernel sums
// 16-wide k tiles in ascending order too: src/hip_ops.hip:43-64.)
//
// Options, all of them orthogonal:
//   a_rows    gather: row m of A is A[a_rows[m], :]
//   grouped   W is [E, Nw, K]; M-tiles are listed in (tile_expert, tile_row0, tile_rows) and
//             each uses its own expert's matrix; rows are positions in an expert-sorted list
//   swiglu    W holds 2N rows, gate rows [0,N) then up rows [N,2N); out = silu(g) * u
//   bias      fp32 or bf16 vector of N, added after the sum
#include "common.cuh"

namespace {

constexpr int BM = 64;          // rows of a tile at most

struct GemmArgs {
  const void* A;
  const void* W;
  const void* bias;
  void* out;
  const int* a_rows;
  const int* tile_expert;
  const int* tile_row0;
  const int* tile_rows;
  const int* num_tiles;  // device scalar (grouped) or null
  long long lda, ldo;
  long long w_expert_stride;  // elements between experts' matrices
  int M, N, K;
  int bias_dt, out_dt;
  int swiglu;
  int act;                  // unary activation of the outputs (0: none; NV_EPI_* codes)
  float act_p0, act_p1;     // its two numbers (xIELU)
  int a_vec, w_vec;         // rows of A / W start on 16 bytes: copied in pieces of 16, else element by element
  int rows_alloc;           // rows of A that a stage has room for: 8, 16, 32 or 64
};

__device__ __forceinline__ void copy16(void* dst, const void* src, int bytes) {      // the rest of the 16 is zeroed
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void load4(const float* p, float (&v)[4]) {
  const float4 f = *(const float4*)p;
  v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
}
__device__ __forceinline__ void load4(const bf16* p, float (&v)[4]) {
  const uint2 u = *(const uint2*)p;
  v[0] = __uint_as_float(u.x << 16); v[1] = __uint_as_float(u.x & 0xffff0000u);
  v[2] = __uint_as_float(u.y << 16); v[3] = __uint_as_float(u.y & 0xffff0000u);
}

// A block makes up to 64 rows x (16 FT) features, FT features a lane.  What bounds it: with a few rows the chain of K
// dependent FFMAs of an output (4 cycles each; it may not be cut, see above) and the stream of W; with many the FFMA
// rate.  So W and A pass through a ring of ST stages of KC elements a row (cp.async: the loads of ST - 1 stages are
// under way while one is summed), blocks are narrow (N / 16 of them keep the multiprocessors busy for a handful of
// rows), and a thread's outputs are RT rows x FT features: four LDS.128 of W and eight of A feed 128 FFMAs in the widest
// form.  Rows are dealt to half-warps in steps of eight, so that RT is no larger than the tile's rows need (the lanes
// of a half-warp read one row of A together, its 16 rows of W lie 16 bytes apart modulo 128: no bank conflicts).
// Measured (float32, four layers of width 1,024 with 16 experts of 512; prompts of 75 and 333 tokens and eight decoded tokens
// of each, 225 products): 24.2 ms with tiles of 64 x 64 x 16 loaded element by element, 6.1 so; the whole 27.5 -> 7.1 ms.
// The widest form (64 x 64 outputs) is for many rows and features: 4,096 rows, 1,024 -> 4,096 in 931 us (1,535 in blocks of
// 32 features, 1,357 in the tiles of 64 x 64 x 16); 64 rows, 1,024 -> 32,000 154 (227, 215); 2,048 rows, 512 -> 1,024 86
// (127, 111).
// Tried and slower: blocks of 64 features where they leave multiprocessors idle (408 rows, 1,024 -> 1,024: 78 against 66
// us); tiles of 32 rows with shorter stages, 16 experts' 1,024 -> 2 x 512 in 203 against 186; for two rows blocks of eight
// features, the experts' 37 against 20; a loop around the product for tiles longer than a stage (every call a tenth).
template <typename T, int KC>
__device__ __forceinline__ void stage_row(char* dst, const T* src, int k0, int K, int c, bool ok, int vec) {
  constexpr int PER = 16 / sizeof(T);
  const int k = k0 + c * PER;
  if (vec) {
    const int left = ok ? min(max((K - k) * (int)sizeof(T), 0), 16) : 0;
    copy16(dst + c * 16, left ? (const void*)(src + k) : (const void*)src, left);
  } else {
#pragma unroll
    for (int i = 0; i < PER; ++i) ((T*)(dst + c * 16))[i] = ok && k + i < K ? src[k + i] : from_f32<T>(0.f);
  }
}

template <typename TA, typename TW, bool SWIGLU, int FT, int KC, int ST, int RT>
__device__ __forceinline__ void product_rows(const GemmArgs& g, char* sm, const TW* W, const long long* a_off, int row0,
                                             int rows_here, int col0) {
  constexpr int BN = 16 * FT, WR = (SWIGLU ? 2 : 1) * BN;
  constexpr int WROW = KC * sizeof(TW) + 16, AROW = KC * sizeof(TA) + 16;       // bytes; 16 of padding
  constexpr int WCH = KC * sizeof(TW) / 16, ACH = KC * sizeof(TA) / 16;
  const int tid = threadIdx.x, lane16 = tid % 16, group = tid / 16;
  const int stage_bytes = WR * WROW + g.rows_alloc * AROW;
  const int nk = (g.K + KC - 1) / KC;
  const TA* A = (const TA*)g.A;

  auto load_stage = [&](int it) {
    char* base = sm + (size_t)(it % ST) * stage_bytes;
    const int k0 = it * KC;
    for (int i = tid; i < WR * WCH; i += 128) {
      const int r = i / WCH, n = col0 + r % BN;
      const bool ok = n < g.N;
      stage_row<TW, KC>(base + r * WROW, W + (ok ? (size_t)(n + (r >= BN ? g.N : 0)) * g.K : 0), k0, g.K, i % WCH, ok, g.w_vec);
    }
    base += WR * WROW;
    for (int i = tid; i < rows_here * ACH; i += 128)
      stage_row<TA, KC>(base + i / ACH * AROW, A + a_off[i / ACH], k0, g.K, i % ACH, true, g.a_vec);
  };

  float acc[RT][FT] = {};
  float acc2[SWIGLU ? RT : 1][FT] = {};
  for (int it = 0; it < ST - 1; ++it) {
    if (it < nk) load_stage(it);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int it = 0; it < nk; ++it) {
    asm volatile("cp.async.wait_group %0;" ::"n"(ST - 2) : "memory");
    __syncthreads();                               // the stage is there, and everyone is through with the one before
    if (it + ST - 1 < nk) load_stage(it + ST - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (group >= rows_here) continue;
    const char* base = sm + (size_t)(it % ST) * stage_bytes;
    const char* wp = base + lane16 * WROW;
    const char* ap = base + WR * WROW + group * AROW;
    const int kn = min(KC, g.K - it * KC);         // (what a stage holds beyond K is zero up to a multiple of four)
#pragma unroll 4
    for (int k = 0; k < kn; k += 4) {
      float w[FT][4], w2[SWIGLU ? FT : 1][4];
#pragma unroll
      for (int f = 0; f < FT; ++f) {
        load4((const TW*)(wp + f * 16 * WROW) + k, w[f]);
        if (SWIGLU) load4((const TW*)(wp + (BN + f * 16) * WROW) + k, w2[f]);
      }
#pragma unroll
      for (int r = 0; r < RT; ++r) {
        float a[4];
        load4((const TA*)(ap + r * 8 * AROW) + k, a);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int f = 0; f < FT; ++f) {
            acc[r][f] = fmaf(a[i], w[f][i], acc[r][f]);
            if (SWIGLU) acc2[r][f] = fmaf(a[i], w2[f][i], acc2[r][f]);
          }
      }
    }
  }

#pragma unroll
  for (int r = 0; r < RT; ++r) {
    const int lrow = group + 8 * r;
    if (lrow >= rows_here) continue;
    const size_t orow = (size_t)(row0 + lrow) * g.ldo;
#pragma unroll
    for (int f = 0; f < FT; ++f) {
      const int n = col0 + lane16 + 16 * f;
      if (n >= g.N) continue;
      float v = acc[r][f];
      if (SWIGLU) v = pair_mul(g.swiglu, v, acc2[r][f], g.act_p0, g.act_p1);
      if (g.bias) v += ld_dt(g.bias, g.bias_dt, n);
      st_dt(g.out, g.out_dt, orow + n, epilogue_act(epi_at(g.act, n, g.act_p0), v, g.act_p0, g.act_p1));
    }
  }
}

template <typename TA, typename TW, bool SWIGLU, int FT, int KC, int ST>
__global__ void __launch_bounds__(128) gemm_plain_kernel(GemmArgs g) {
  extern __shared__ __align__(16) char sm[];
  __shared__ long long a_off[BM];
  grid_dep_wait();
  grid_dep_launch();
  int row0, rows_here;
  const TW* W = (const TW*)g.W;
  if (g.tile_expert) {
    if ((int)blockIdx.y >= *g.num_tiles) return;
    row0 = g.tile_row0[blockIdx.y];
    rows_here = min(g.tile_rows[blockIdx.y], g.rows_alloc);      // (a tile has no more rows than the product)
    W += (size_t)g.tile_expert[blockIdx.y] * g.w_expert_stride;
  } else {
    row0 = blockIdx.y * BM;
    rows_here = min(BM, g.M - row0);
  }
  if ((int)threadIdx.x < rows_here) {
    const int r = row0 + threadIdx.x;
    a_off[threadIdx.x] = (long long)(g.a_rows ? g.a_rows[r] : r) * g.lda;
  }
  __syncthreads();
  const int col0 = blockIdx.x * 16 * FT;
  if (rows_here <= 8) product_rows<TA, TW, SWIGLU, FT, KC, ST, 1>(g, sm, W, a_off, row0, rows_here, col0);
  else if (rows_here <= 16) product_rows<TA, TW, SWIGLU, FT, KC, ST, 2>(g, sm, W, a_off, row0, rows_here, col0);
  else if (rows_here <= 32) product_rows<TA, TW, SWIGLU, FT, KC, ST, 4>(g, sm, W, a_off, row0, rows_here, col0);
  else product_rows<TA, TW, SWIGLU, FT, KC, ST, 8>(g, sm, W, a_off, row0, rows_here, col0);
}

template <typename TA, typename TW, bool SWIGLU, int FT, int KC, int ST>
int launch_form(const GemmArgs& g, int m_tiles, cudaStream_t s) {
  const dim3 grid((g.N + 16 * FT - 1) / (16 * FT), m_tiles);
  const size_t w_bytes = (SWIGLU ? 2 : 1) * 16 * FT * (KC * sizeof(TW) + 16), a_bytes = g.rows_alloc * (KC * sizeof(TA) + 16);
  const size_t smem = ST * (w_bytes + a_bytes);
  auto* kernel = gemm_plain_kernel<TA, TW, SWIGLU, FT, KC, ST>;
  if (smem > 48 * 1024) NV_RETURN_IF(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  NV_RETURN_IF(launch_dep(kernel, grid, dim3(128), smem, s, g));
  NV_RETURN_LAST();
}

template <typename TA, typename TW>
int launch(const GemmArgs& g, int m_tiles, cudaStream_t s) {
  if (m_tiles == 0) return NV_OK;
  if (m_tiles > 65535) return NV_ERR_BAD_SIZE;
  // Wider blocks where there are enough of them for every multiprocessor (64 rows, 1,024 -> 1,024: 64 narrow blocks and not
  // 32 wide ones), the widest where there are two for each.
  constexpr int KC = sizeof(TA) == 2 && sizeof(TW) == 2 ? 64 : 32;
  const int sms = num_multiprocessors();
  const long long row_tiles = (g.M + BM - 1) / BM;
  const bool wide = g.M > (g.tile_expert ? BM - 1 : BM / 2) && (long long)((g.N + 31) / 32) * row_tiles >= sms;
  const bool widest = wide && (long long)((g.N + (g.swiglu ? 31 : 63)) / (g.swiglu ? 32 : 64)) * row_tiles >= 2 * sms;
  if (g.swiglu)
    return widest ? launch_form<TA, TW, true, 2, KC, 3>(g, m_tiles, s)
         : wide ? launch_form<TA, TW, true, 2, 64, 3>(g, m_tiles, s) : launch_form<TA, TW, true, 1, 128, 4>(g, m_tiles, s);
  return widest ? launch_form<TA, TW, false, 4, KC, 3>(g, m_tiles, s)
       : wide ? launch_form<TA, TW, false, 2, 64, 3>(g, m_tiles, s) : launch_form<TA, TW, false, 1, 128, 4>(g, m_tiles, s);
}

}  // namespace

// Rows per M-tile of the grouped form; the tile list given to nv_gemm_plain must be cut by this.
NV_API int nv_gemm_plain_tile_m() { return BM; }

NV_API int nv_gemm_plain(const void* A, int a_dt, long long lda, const int* a_rows,
                         const void* W, int w_dt, long long w_expert_stride,
                         const void* bias, int bias_dt,
                         void* out, int out_dt, long long ldo,
                         int M, int N, int K, int swiglu,
                         const int* tile_expert, const int* tile_row0, const int* tile_rows,
                         const int* num_tiles, int max_tiles, float act_p0, float act_p1, cudaStream_t stream) {
  if (!dt_ok(a_dt) || !dt_ok(w_dt) || !dt_ok(out_dt) || (bias && !dt_ok(bias_dt))) return NV_ERR_BAD_DTYPE;
  if (M < 0 || N <= 0 || K <= 0 || swiglu < 0 || swiglu > NV_EPI_LAST) return NV_ERR_BAD_SIZE;
  const int act = epi_unary(swiglu);
  swiglu = epi_pair(swiglu);
  GemmArgs g;
  g.act = act;
  g.act_p0 = act_p0;
  g.act_p1 = act_p1;
  g.A = A; g.W = W; g.bias = bias; g.out = out; g.a_rows = a_rows;
  g.tile_expert = tile_expert; g.tile_row0 = tile_row0; g.tile_rows = tile_rows; g.num_tiles = num_tiles;
  g.lda = lda; g.ldo = ldo; g.w_expert_stride = w_expert_stride;
  g.M = M; g.N = N; g.K = K; g.bias_dt = bias_dt; g.out_dt = out_dt; g.swiglu = swiglu;
  const int m_tiles = tile_expert ? max_tiles : (M + BM - 1) / BM;
  const size_t ea = a_dt == NV_DT_F32 ? 4 : 2, ew = w_dt == NV_DT_F32 ? 4 : 2;
  g.a_vec = (uintptr_t)A % 16 == 0 && lda * ea % 16 == 0;
  g.w_vec = (uintptr_t)W % 16 == 0 && K * ew % 16 == 0 && w_expert_stride * ew % 16 == 0;
  g.rows_alloc = M <= 8 ? 8 : M <= 16 ? 16 : M <= 32 ? 32 : BM;
  if (a_dt == NV_DT_F32 && w_dt == NV_DT_F32) return launch<float, float>(g, m_tiles, stream);
  if (a_dt == NV_DT_F32 && w_dt == NV_DT_BF16) return launch<float, bf16>(g, m_tiles, stream);
  if (a_dt == NV_DT_BF16 && w_dt == NV_DT_F32) return launch<bf16, float>(g, m_tiles, stream);
  return launch<bf16, bf16>(g, m_tiles, stream);
}
