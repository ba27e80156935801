// Plain matrix product on the CUDA cores, true 32-bit: out[m,n] = sum_k A[m,k] * W[n,k].
//
// This is the product of the float32 path, of float32 rows with a short matrix (gates), and the reference twin of the
// tensor-core kernels.  The order of a sum is a function of K alone: K is cut into eight ranges of class_len(K) elements (a
// multiple of 32), a range is one chain of FFMAs over k in ascending order that starts from zero, and with c0 .. c7 the
// ranges' sums an output is ((c0 + c1) + c2) + ... + c7.  So a row's result does not depend on what else is in the batch,
// whichever of the kernels below takes it, and ranges can be worked out side by side.  (The reference's kernel sums 16-wide
// k tiles in ascending order: src/hip_ops.hip:43-64.)
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
constexpr int CLASSES = 8;      // ranges of K whose sums are chains of their own
constexpr int STEP = 32;        // elements of K per stage of the tile kernel's ring; a range is a multiple of it
constexpr int ST = 3;           // stages of the tile kernel's ring
constexpr int FEW_ROWS = 16;    // rows that the kernel of a handful of rows takes
constexpr int FEW_STEP = 64;    // elements of K per stage there
constexpr int FEW_ST = 2;

__host__ __device__ __forceinline__ int class_len(int K) {
  return (K + CLASSES * STEP - 1) / (CLASSES * STEP) * STEP;
}

__device__ __forceinline__ float in_order(const float (&c)[CLASSES]) {
  float v = c[0];
#pragma unroll
  for (int i = 1; i < CLASSES; ++i) v += c[i];
  return v;
}

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
  int rows_alloc;           // rows of A that a stage has room for, and the rows of a dense tile
  int early;                // W may be read before the kernel in front has finished: that kernel does not write it
};

__device__ __forceinline__ void copy16(void* dst, const void* src, int bytes) {      // the rest of the 16 is zeroed
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void copies_end() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void load4(const float* p, float (&v)[4]) {
  const float4 f = *(const float4*)p;
  v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
}
__device__ __forceinline__ void load4(const bf16* p, float (&v)[4]) {
  const uint2 u = *(const uint2*)p;
  v[0] = __uint_as_float(u.x << 16); v[1] = __uint_as_float(u.x & 0xffff0000u);
  v[2] = __uint_as_float(u.y << 16); v[3] = __uint_as_float(u.y & 0xffff0000u);
}

// The c-th 16 bytes of a row's elements k0 .. (those from k_end on as zeros; `ok` false: all of them).
template <typename T>
__device__ __forceinline__ void stage_row(char* dst, const T* src, int k0, int k_end, int c, bool ok, int vec) {
  constexpr int PER = 16 / sizeof(T);
  const int k = k0 + c * PER;
  if (vec) {
    const int left = ok ? min(max((k_end - k) * (int)sizeof(T), 0), 16) : 0;
    copy16(dst + c * 16, left ? (const void*)(src + k) : (const void*)src, left);
  } else {
#pragma unroll
    for (int i = 0; i < PER; ++i) ((T*)(dst + c * 16))[i] = ok && k + i < k_end ? src[k + i] : from_f32<T>(0.f);
  }
}

__device__ __forceinline__ void finish_store(const GemmArgs& g, int row, int n, float v) {
  if (g.bias) v += ld_dt(g.bias, g.bias_dt, n);
  st_dt(g.out, g.out_dt, (size_t)row * g.ldo + n, epilogue_act(epi_at(g.act, n, g.act_p0), v, g.act_p0, g.act_p1));
}

// ------------------------------------------------------------------ tiles of up to 64 rows
// A block makes up to 64 rows x (16 FT) features, FT features (pairs: FT gate and FT up rows) a lane; W and A pass through a
// ring of ST stages of STEP elements a row.  Rows are dealt to half-warps in steps of eight, so that RT is no larger than
// the tile's rows need (the lanes of a half-warp read one row of A together, its 16 rows of W lie 16 bytes apart modulo 128:
// no bank conflicts).  What bounds it: the FFMA rate, at 45 % of it where there are many blocks (what is missing is latency of
// shared memory and of the ring: four blocks of the wide form live on a multiprocessor, and with three, or with stages of 64
// elements, which leave room for fewer blocks, it is a tenth to a fifth slower; threads of 8 x 8 outputs, two a multiprocessor,
// were slower still).  CL = 1: a block takes the ranges of K one after the other.  CL = 4: four blocks of a cluster
// share a tile, block q takes ranges 2q and 2q + 1, and the sums meet through distributed shared memory.
template <typename TA, typename TW, bool SWIGLU, int FT, int CL, int RT>
__device__ __forceinline__ void tile_product(const GemmArgs& g, char* sm, const TW* W, const long long* a_off, int row0,
                                             int rows_here, int col0, int cta) {
  constexpr int FW = SWIGLU ? 2 * FT : FT;         // rows of W a lane
  constexpr int BN = 16 * FT, WR = 16 * FW;
  constexpr int WROW = STEP * sizeof(TW) + 16, AROW = STEP * sizeof(TA) + 16;       // bytes; 16 of padding
  constexpr int WCH = STEP * sizeof(TW) / 16, ACH = STEP * sizeof(TA) / 16;
  const int tid = threadIdx.x, lane16 = tid % 16, group = tid / 16;
  const int stage_bytes = WR * WROW + g.rows_alloc * AROW;
  const TA* A = (const TA*)g.A;
  const int L = class_len(g.K);
  const int k_first = CL == 4 ? 2 * cta * L : 0, k_last = CL == 4 ? min(g.K, k_first + 2 * L) : g.K;

  int lk = k_first, slot = 0;                      // the next stage to ask for
  auto load_stage = [&] {
    if (lk < k_last) {
      char* base = sm + (size_t)slot * stage_bytes;
#pragma unroll
      for (int i0 = 0; i0 < WR * WCH; i0 += 128) {
        const int i = i0 + tid, r = i / WCH, n = col0 + r % BN;
        const bool ok = n < g.N;
        if (WR * WCH % 128 == 0 || i < WR * WCH)
          stage_row<TW>(base + r * WROW, W + (ok ? (size_t)(n + (r >= BN ? g.N : 0)) * g.K : 0), lk, g.K, i % WCH, ok, g.w_vec);
      }
      base += WR * WROW;
      for (int i = tid; i < rows_here * ACH; i += 128)
        stage_row<TA>(base + i / ACH * AROW, A + a_off[i / ACH], lk, g.K, i % ACH, true, g.a_vec);
      slot = slot + 1 == ST ? 0 : slot + 1;
      lk += STEP;
    }
    copies_end();
  };

  // CL = 1: `sum` is the ranges' so far, in order; CL = 4: range 2q's, and `acc` in the end range 2q + 1's
  float sum[RT][FW] = {}, acc[RT][FW] = {};
  for (int i = 0; i < ST - 1; ++i) load_stage();
  int at = 0, turn = k_first + L;
#pragma unroll 1
  for (int k0 = k_first; k0 < k_last; k0 += STEP) {
    copies_wait<ST - 2>();
    __syncthreads();                               // the stage is there, and everyone is through with the one before
    load_stage();
    const char* base = sm + (size_t)at * stage_bytes;
    at = at + 1 == ST ? 0 : at + 1;
    if (group >= rows_here) continue;
    if (k0 == turn) {
      turn += L;
#pragma unroll
      for (int r = 0; r < RT; ++r)
#pragma unroll
        for (int f = 0; f < FW; ++f) { sum[r][f] += acc[r][f]; acc[r][f] = 0.f; }
    }
    const char* wp = base + lane16 * WROW;
    const char* ap = base + WR * WROW + group * AROW;
#pragma unroll 2
    for (int k = 0; k < STEP; k += 4) {            // (what a stage holds beyond K is zero)
      float w[FW][4];
#pragma unroll
      for (int f = 0; f < FW; ++f) load4((const TW*)(wp + f * 16 * WROW) + k, w[f]);
#pragma unroll
      for (int r = 0; r < RT; ++r) {
        float a[4];
        load4((const TA*)(ap + r * 8 * AROW) + k, a);
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
          for (int f = 0; f < FW; ++f) acc[r][f] = fmaf(a[e], w[f][e], acc[r][f]);
      }
    }
  }
  copies_wait<0>();

  auto put = [&](int r, const float (&v)[FW]) {
    const int lrow = group + 8 * r;
    if (lrow >= rows_here) return;
#pragma unroll
    for (int f = 0; f < FT; ++f) {
      const int n = col0 + lane16 + 16 * f;
      if (n < g.N) finish_store(g, row0 + lrow, n, SWIGLU ? pair_mul(g.swiglu, v[f], v[f + FW - FT], g.act_p0, g.act_p1) : v[f]);
    }
  };
  if (CL == 1) {
#pragma unroll
    for (int r = 0; r < RT; ++r) {
      float v[FW];
#pragma unroll
      for (int f = 0; f < FW; ++f) v[f] = sum[r][f] + acc[r][f];
      put(r, v);
    }
    return;
  }
  __syncthreads();                                 // everyone is through with the ring
  float* buf = (float*)sm;
  const bool second = turn > k_first + L;          // there was a second range (else `acc` is the first)
#pragma unroll
  for (int r = 0; r < RT; ++r)
#pragma unroll
    for (int f = 0; f < FW; ++f) {
      buf[(r * FW + f) * 128 + tid] = second ? sum[r][f] : acc[r][f];
      buf[((RT + r) * FW + f) * 128 + tid] = second ? acc[r][f] : 0.f;
    }
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
#pragma unroll
  for (int r = 0; r < RT; ++r) {                   // rows are shared out among the blocks
    if (r % 4 != cta) continue;
    float v[FW];
#pragma unroll
    for (int f = 0; f < FW; ++f) {
      float c[CLASSES];
#pragma unroll
      for (int i = 0; i < CLASSES; ++i) {
        uint32_t there;
        const uint32_t at = (uint32_t)__cvta_generic_to_shared(buf + ((i % 2 * RT + r) * FW + f) * 128 + tid);
        asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(at), "r"(i / 2));
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(c[i]) : "r"(there) : "memory");
      }
      v[f] = in_order(c);
    }
    put(r, v);
  }
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <typename TA, typename TW, bool SWIGLU, int FT, int CL>
__global__ void __launch_bounds__(128, (SWIGLU ? 2 : 1) * FT >= 4 ? 4 : 5) gemm_plain_kernel(GemmArgs g) {
  extern __shared__ __align__(16) char sm[];
  __shared__ long long a_off[BM];
  grid_dep_wait();
  grid_dep_launch();
  int row0, rows_here;
  const TW* W = (const TW*)g.W;
  if (g.tile_expert) {
    if ((int)blockIdx.y >= *g.num_tiles) return;               // (all blocks of a cluster alike)
    row0 = g.tile_row0[blockIdx.y];
    rows_here = min(g.tile_rows[blockIdx.y], g.rows_alloc);      // (a tile has no more rows than the product)
    W += (size_t)g.tile_expert[blockIdx.y] * g.w_expert_stride;
  } else {
    row0 = blockIdx.y * g.rows_alloc;
    rows_here = min(g.rows_alloc, g.M - row0);
  }
  if ((int)threadIdx.x < rows_here) {
    const int r = row0 + threadIdx.x;
    a_off[threadIdx.x] = (long long)(g.a_rows ? g.a_rows[r] : r) * g.lda;
  }
  __syncthreads();
  const int col0 = (int)blockIdx.x / CL * 16 * FT, cta = blockIdx.x % CL;
  if (rows_here <= 8) tile_product<TA, TW, SWIGLU, FT, CL, 1>(g, sm, W, a_off, row0, rows_here, col0, cta);
  else if (rows_here <= 16) tile_product<TA, TW, SWIGLU, FT, CL, 2>(g, sm, W, a_off, row0, rows_here, col0, cta);
  else if (rows_here <= 32) tile_product<TA, TW, SWIGLU, FT, CL, 4>(g, sm, W, a_off, row0, rows_here, col0, cta);
  else tile_product<TA, TW, SWIGLU, FT, CL, 8>(g, sm, W, a_off, row0, rows_here, col0, cta);
}

// ------------------------------------------------------------------ a handful of rows
// What bounds it: the stream of W, and for one product the way from the launch to the first sums.  A block makes up to 16
// rows x 16 rows of W (8 pairs); its eight warps take a range of K each, so the chain of an output is K / 8 FFMAs, through
// rings of their own that no other warp waits for.  A dense product of weights asks for its first stages of W before the kernel in
// front of it has finished.  Measured (float32, two rows, cold weights, the launch included): 1,024 -> 1,536 14.4 us with one
// chain over K and 16 features a block, 9.2 so; 2,048 -> 2,048 22.6 and 12.3; eight pairs of 16 experts, SwiGLU 1,024 -> 512
// 20.5 and 16.4.  In a chain of decode steps (two rows, four layers of width 1,024 with experts of 512) a product of rows took
// 14 to 22 us and takes 9 to 12; the relative error against float64 falls from 5.7e-7 to 2.1e-7 (chains an eighth as long).
template <typename TA, typename TW, bool SWIGLU, int RT>
__device__ __forceinline__ void few_product(const GemmArgs& g, char* sm, const TW* W, const long long* a_off, int row0,
                                            int rows_here, int col0, bool early) {
  constexpr int WR = 16, BN = SWIGLU ? 8 : 16;
  constexpr int WROW = FEW_STEP * sizeof(TW) + 16, AROW = FEW_STEP * sizeof(TA) + 16;
  constexpr int WCH = FEW_STEP * sizeof(TW) / 16, ACH = FEW_STEP * sizeof(TA) / 16;
  const int tid = threadIdx.x, c = tid / 32, lane = tid % 32, wl = lane % 16, rg = lane / 16;
  const int stage_bytes = WR * WROW + g.rows_alloc * AROW;
  char* ring = sm + (size_t)c * FEW_ST * stage_bytes;
  const TA* A = (const TA*)g.A;
  const int L = class_len(g.K), k_first = c * L, k_end = min(g.K, k_first + L);
  const int nk = (max(0, k_end - k_first) + FEW_STEP - 1) / FEW_STEP;
  auto load_w = [&](int it) {
    char* base = ring + (size_t)(it % FEW_ST) * stage_bytes;
#pragma unroll
    for (int i0 = 0; i0 < WR * WCH; i0 += 32) {
      const int i = i0 + lane, r = i / WCH, n = col0 + r % BN;
      const bool ok = n < g.N;
      stage_row<TW>(base + r * WROW, W + (ok ? (size_t)(n + (SWIGLU && r >= BN ? g.N : 0)) * g.K : 0), k_first + it * FEW_STEP, k_end,
                    i % WCH, ok, g.w_vec);
    }
  };
  auto load_a = [&](int it) {
    char* base = ring + (size_t)(it % FEW_ST) * stage_bytes + WR * WROW;
    for (int i = lane; i < rows_here * ACH; i += 32)
      stage_row<TA>(base + i / ACH * AROW, A + a_off[i / ACH], k_first + it * FEW_STEP, k_end, i % ACH, true, g.a_vec);
  };
  if (early) {                                     // (the kernel's first lines asked for the stages of W)
    grid_dep_wait();
    grid_dep_launch();
  }
#pragma unroll
  for (int it = 0; it < FEW_ST; ++it) {
    if (it < nk) {
      if (!early) load_w(it);
      load_a(it);
    }
    copies_end();
  }
  float acc[RT] = {};
#pragma unroll 1
  for (int it = 0; it < nk; ++it) {
    copies_wait<FEW_ST - 1>();
    __syncwarp();
    const char* base = ring + (size_t)(it % FEW_ST) * stage_bytes;
    const TW* wp = (const TW*)(base + wl * WROW);
    const char* ap = base + WR * WROW + rg * AROW;
    const int kn = min(FEW_STEP, k_end - k_first - it * FEW_STEP);
#pragma unroll 4
    for (int k = 0; k < kn; k += 4) {
      float w[4];
      load4(wp + k, w);
#pragma unroll
      for (int r = 0; r < RT; ++r) {
        float a[4];
        load4((const TA*)(ap + r * 2 * AROW) + k, a);
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[r] = fmaf(a[i], w[i], acc[r]);
      }
    }
    __syncwarp();
    if (it + FEW_ST < nk) {
      load_w(it + FEW_ST);
      load_a(it + FEW_ST);
    }
    copies_end();
  }
  copies_wait<0>();
  __syncthreads();
  float* part = (float*)sm;                        // [class][row][16]
#pragma unroll
  for (int r = 0; r < RT; ++r) part[(c * 2 * RT + rg + 2 * r) * 16 + wl] = acc[r];
  __syncthreads();
  const int row = tid / BN, f = tid % BN, n = col0 + f;
  if (row >= rows_here || n >= g.N) return;
  auto sum = [&](int wrow) {
    float v[CLASSES];
#pragma unroll
    for (int i = 0; i < CLASSES; ++i) v[i] = part[(i * 2 * RT + row) * 16 + wrow];
    return in_order(v);
  };
  finish_store(g, row0 + row, n, SWIGLU ? pair_mul(g.swiglu, sum(f), sum(8 + f), g.act_p0, g.act_p1) : sum(f));
}

template <typename TA, typename TW, bool SWIGLU>
__global__ void __launch_bounds__(256) gemm_few_kernel(GemmArgs g) {
  extern __shared__ __align__(16) char sm[];
  __shared__ long long a_off[FEW_ROWS];
  int row0 = 0, rows_here = g.M;
  const TW* W = (const TW*)g.W;
  const int col0 = blockIdx.x * (SWIGLU ? 8 : 16);
  const bool early = g.early && !g.tile_expert && !g.a_rows && g.w_vec;
  if (early) {
    constexpr int WROW = FEW_STEP * sizeof(TW) + 16, AROW = FEW_STEP * sizeof(TA) + 16, WCH = FEW_STEP * sizeof(TW) / 16;
    const int c = threadIdx.x / 32, lane = threadIdx.x % 32, L = class_len(g.K), k_end = min(g.K, (c + 1) * L);
    const int stage_bytes = 16 * WROW + g.rows_alloc * AROW;
#pragma unroll
    for (int it = 0; it < FEW_ST; ++it)
#pragma unroll
      for (int i0 = 0; i0 < 16 * WCH; i0 += 32) {
        const int i = i0 + lane, r = i / WCH, n = col0 + (SWIGLU ? r % 8 : r);
        const bool ok = n < g.N;
        if (c * L + it * FEW_STEP < k_end)
          stage_row<TW>(sm + (size_t)(c * FEW_ST + it) * stage_bytes + r * WROW,
                        W + (ok ? (size_t)(n + (SWIGLU && r >= 8 ? g.N : 0)) * g.K : 0), c * L + it * FEW_STEP, k_end, i % WCH, ok, 1);
      }
    if ((int)threadIdx.x < rows_here) a_off[threadIdx.x] = (long long)threadIdx.x * g.lda;
  } else {
    grid_dep_wait();
    grid_dep_launch();
    if (g.tile_expert) {
      if ((int)blockIdx.y >= *g.num_tiles) return;
      row0 = g.tile_row0[blockIdx.y];
      rows_here = min(g.tile_rows[blockIdx.y], g.rows_alloc);
      W += (size_t)g.tile_expert[blockIdx.y] * g.w_expert_stride;
    }
    if ((int)threadIdx.x < rows_here) {
      const int r = row0 + threadIdx.x;
      a_off[threadIdx.x] = (long long)(g.a_rows ? g.a_rows[r] : r) * g.lda;
    }
  }
  __syncthreads();
  if (rows_here <= 2) few_product<TA, TW, SWIGLU, 1>(g, sm, W, a_off, row0, rows_here, col0, early);
  else if (rows_here <= 4) few_product<TA, TW, SWIGLU, 2>(g, sm, W, a_off, row0, rows_here, col0, early);
  else if (rows_here <= 8) few_product<TA, TW, SWIGLU, 4>(g, sm, W, a_off, row0, rows_here, col0, early);
  else few_product<TA, TW, SWIGLU, 8>(g, sm, W, a_off, row0, rows_here, col0, early);
}

template <typename TA, typename TW, bool SWIGLU, int FT, int CL>
int launch_tiles(const GemmArgs& g, int m_tiles, cudaStream_t s) {
  size_t smem = ST * ((size_t)(SWIGLU ? 32 : 16) * FT * (STEP * sizeof(TW) + 16) + g.rows_alloc * (STEP * sizeof(TA) + 16));
  // (a cluster's blocks put two sums of 128 threads x (rows / 8) x FW outputs where the ring was)
  const size_t sums = (size_t)2 * ((g.rows_alloc + 7) / 8) * (SWIGLU ? 2 * FT : FT) * 128 * sizeof(float);
  if (CL > 1 && sums > smem) smem = sums;
  auto* kernel = gemm_plain_kernel<TA, TW, SWIGLU, FT, CL>;
  if (smem > 48 * 1024) NV_RETURN_IF(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const dim3 grid((g.N + 16 * FT - 1) / (16 * FT) * CL, m_tiles);
  NV_RETURN_IF(launch_dep_clusters(CL, kernel, grid, dim3(128), smem, s, g));
  NV_RETURN_LAST();
}

template <typename TA, typename TW, bool SWIGLU>
int launch_few(const GemmArgs& g, int m_tiles, cudaStream_t s) {
  const size_t smem = CLASSES * FEW_ST * (16 * (FEW_STEP * sizeof(TW) + 16) + g.rows_alloc * (FEW_STEP * sizeof(TA) + 16));
  auto* kernel = gemm_few_kernel<TA, TW, SWIGLU>;
  if (smem > 48 * 1024) NV_RETURN_IF(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int per = SWIGLU ? 8 : 16;
  NV_RETURN_IF(launch_dep(kernel, dim3((g.N + per - 1) / per, m_tiles), dim3(256), smem, s, g));
  NV_RETURN_LAST();
}

template <typename TA, typename TW>
int launch(GemmArgs g, int max_tiles, cudaStream_t s) {
  const bool grouped = g.tile_expert != nullptr;
  const int sms = num_multiprocessors();
  g.rows_alloc = g.M <= 2 ? 2 : g.M <= 4 ? 4 : g.M <= 8 ? 8 : g.M <= 16 ? 16 : g.M <= 32 ? 32 : BM;
  const long long m_tiles = grouped ? max_tiles : (g.M + BM - 1) / BM;
  if (m_tiles == 0) return NV_OK;
  if (m_tiles > 65535) return NV_ERR_BAD_SIZE;
  // Which blocks: by their number, every form measured at 1 to 3,000 rows, 64 to 32,000 features and K of 64 to 4,096 (us below:
  // WHOLE_WIDE, SPLIT_WIDE, WHOLE_NARROW, SPLIT_NARROW, float32, K = 1,024 unless said).  Five narrow blocks live on a multiprocessor
  // and four wide ones.  A grouped product is taken for its list's most tiles.
  const long long wide = (g.N + (g.swiglu ? 31 : 63)) / (g.swiglu ? 32 : 64) * m_tiles;
  const long long narrow = (g.N + (g.swiglu ? 15 : 31)) / (g.swiglu ? 16 : 32) * m_tiles;
  // Up to 16 rows: the kernel of a handful of rows, whose eight warps want a K for each of them (eight rows, 128 -> 1,024: 2.5, 3.5
  // in tiles; nine rows, 64 -> 2,048: 4.1 and 3.0), but float32 rows from nine on only where there are few blocks (16 rows -> 8,000:
  // 36, SPLIT_WIDE 20; -> 32,000: 123, WHOLE_WIDE 62; -> 1,024: 9 either way).
  if (g.M <= FEW_ROWS && (g.K >= 128 || g.M <= 4) && (sizeof(TA) == 2 || g.M <= 8 || narrow < sms))
    return g.swiglu ? launch_few<TA, TW, true>(g, m_tiles, s) : launch_few<TA, TW, false>(g, m_tiles, s);
  // Narrow blocks that share K among a cluster, while they run in one wave (192 rows, 1,536: 68, 42, 43, 30; 320 rows, 1,024, 640
  // blocks: 68, 43, 58, 30; 50 rows, 256 -> 512: 27, 13, 15, 7).  Beyond that wide ones while they are three and a half a
  // multiprocessor: the fourth costs what a wave costs (408 rows, 1,024: 69, 43, 59, 46; 512 rows, 512 blocks: 68, 44, 59, 50; 576
  // rows, 576 blocks: 69, 57, 59, 54).  Then narrow ones, which leave less of a last wave (640 rows, 1,024: 91, 64, 74, 57; 896 rows:
  // 93, 79, 104, 76), until those are three and a half waves; from there wide ones again up to three and a quarter whole blocks a
  // multiprocessor (1,500 rows, 1,024: 145, 114, 121, 120; 640 rows, 2,048 -> 2,048: 277, 180, 202, 195), after which whole K fills
  // the multiprocessors as well and needs no exchange (1,500 rows, 1,536: 148, 162, 168, 174).  Many experts of a few rows each
  // gain from this last rule with a long K only (20 pairs of 16 experts, 512 -> 1,024: 13.6, 13.1, 10.4, 14.3).
  const bool one_wave = 4 * narrow <= 5 * sms;
  if (g.K >= 512) {
    if (!one_wave && (8 * wide <= 7 * sms || (2 * narrow > 7 * sms && 4 * wide <= 13 * sms && (g.K >= 1024 || !grouped))))
      return g.swiglu ? launch_tiles<TA, TW, true, 2, 4>(g, m_tiles, s) : launch_tiles<TA, TW, false, 4, 4>(g, m_tiles, s);
    if (2 * narrow <= 7 * sms)
      return g.swiglu ? launch_tiles<TA, TW, true, 1, 4>(g, m_tiles, s) : launch_tiles<TA, TW, false, 2, 4>(g, m_tiles, s);
    if (narrow >= 4 * sms)
      return g.swiglu ? launch_tiles<TA, TW, true, 2, 1>(g, m_tiles, s) : launch_tiles<TA, TW, false, 4, 1>(g, m_tiles, s);
  } else {
    if ((g.K >= 256 && one_wave) || (g.K >= 128 && 4 * narrow <= sms))
      return g.swiglu ? launch_tiles<TA, TW, true, 1, 4>(g, m_tiles, s) : launch_tiles<TA, TW, false, 2, 4>(g, m_tiles, s);
    // With a short K a block is mostly its epilogue: blocks of 16 features while there are no more than two a multiprocessor (64
    // rows, 64 -> 2,048: 6, narrow 8; 200 rows, 128 -> 1,024, bfloat16: 8, narrow 11 and split 12), else narrow ones (6,737 rows, 64 ->
    // 2,048: 118, 306, 92, 278).
    if (!g.swiglu && narrow <= sms) return launch_tiles<TA, TW, false, 1, 1>(g, m_tiles, s);
  }
  return g.swiglu ? launch_tiles<TA, TW, true, 1, 1>(g, m_tiles, s) : launch_tiles<TA, TW, false, 2, 1>(g, m_tiles, s);
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
                         const int* num_tiles, int max_tiles, float act_p0, float act_p1, int early, cudaStream_t stream) {
  // early: the kernel in front on the stream does not write W (a layer's weights), which may then be read before it has ended
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
  g.M = M; g.N = N; g.K = K; g.bias_dt = bias_dt; g.out_dt = out_dt; g.swiglu = swiglu; g.early = early;
  const size_t ea = a_dt == NV_DT_F32 ? 4 : 2, ew = w_dt == NV_DT_F32 ? 4 : 2;
  g.a_vec = (uintptr_t)A % 16 == 0 && lda * ea % 16 == 0;
  g.w_vec = (uintptr_t)W % 16 == 0 && K * ew % 16 == 0 && w_expert_stride * ew % 16 == 0;
  if (a_dt == NV_DT_F32 && w_dt == NV_DT_F32) return launch<float, float>(g, max_tiles, stream);
  if (a_dt == NV_DT_F32 && w_dt == NV_DT_BF16) return launch<float, bf16>(g, max_tiles, stream);
  if (a_dt == NV_DT_BF16 && w_dt == NV_DT_F32) return launch<bf16, float>(g, max_tiles, stream);
  return launch<bf16, bf16>(g, max_tiles, stream);
}
