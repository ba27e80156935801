// The two products of a mixture of experts for a handful of (row, expert) pairs (one to four rows while decoding), with
// the routing inside the first of them.
//
// So few pairs need no permutation: a unit of work is sixteen features of one pair's expert (or of one chunk of the shared
// expert, for all rows at once), its row is the batch's own, and its result goes to row t * (K + C) + k of the output.
// What bounds them is the stream of the experts' weights and the chain of kernels around it.  The tcgen05 products took
// eight launches for this (routing, row copy, two products of the routed experts and two of the shared one's chunks, their K
// split, and a pass each to add the parts).  Here a block of sixteen warps walks units as the product of a handful of
// rows does (skinny_gemm.cu: a warp's share of K is every sixteenth step of 32 elements, mma.sync.m16n8k16 on 16-byte pieces
// of a lane's own), with the pieces on their way through shared memory up to four rounds ahead (cp.async; a lane waits for its
// own only) and the rows there from the start.  The shared expert's units come first: the first of them is asked for before the
// kernel in front has finished, and a seventeenth warp routes the rows meanwhile, in every block by itself, so that no
// block waits for another.
// Measured inside a decode step of one row (60 experts of 1,408 x 2,048, four chosen, four chunks of the shared one): routing
// and experts 38 -> 28 us a layer, the step 1.98 -> 1.71 ms.  With the pieces in registers, two rounds of them, instead of
// the ring, and the rows read from L2 at every unit, 36 us: a unit's rows were waited for.
#include "common.cuh"
#include "moe_route.cuh"

namespace {

constexpr int FX_WARPS = 16;
constexpr int FX_LOADS = 4;             // 16-byte pieces of the weights of a lane per round
constexpr int FX_THREADS = FX_WARPS * 32;     // of the products
constexpr int FX_SMEM = 192 * 1024;     // of dynamic shared memory
constexpr int FX_PAIRS = 64;            // at most so many pairs

struct FxArgs {
  const bf16* x;          // first product: the rows; second: the first one's outputs, [T * KT, K_in]
  const bf16* w;          // [E + C][(gated ? 2 : 1) * N][K_in]
  void* out;              // [T * KT, N]
  int* idx;               // [T, KT]: written by the first product, read by the second
  float* score;
  const float* logits;    // [T, E], rows ld apart (first product)
  long long ld;
  const float* gate_logit;
  long long gate_ld;
  RouteRule rule;
  int renorm;
  long long ldx;
  int T, E, K, C, N, K_in, out_dt, first, stages;
  int act, pair;
  float act_p0, act_p1;
};

__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                          uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
               "{%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

struct FxUnit {
  const bf16* w;          // the expert's matrix
  int x0, x_step;         // row 0 of the unit's rows, and from one of them to the next
  int rows, n0, out0;     // rows; first feature; output row of row 0 (the next ones KT further)
};

// (a call, so that the routing's registers are not the products')
__device__ __noinline__ void route_here(const FxArgs& a, double* scratch, int lane, int* chosen, float* weight) {
  const int KT = a.K + a.C;
  for (int t = 0; t < a.T; ++t)
    route_row(a.logits + t * a.ld, a.E, a.K, a.renorm, scratch, lane, chosen + t * KT, weight + t * KT, a.C,
              a.gate_logit ? a.gate_logit + t * a.gate_ld : nullptr, a.rule);
}

template <bool GATED>
__global__ void __launch_bounds__((FX_WARPS + 1) * 32, 1) few_experts_kernel(const __grid_constant__ FxArgs a) {
  constexpr int NA = GATED ? 2 : 1;                   // accumulators: gate and up
  constexpr int BATCH = FX_LOADS / (2 * NA);          // steps of 32 elements of K per round of loads
  extern __shared__ __align__(16) uint8_t fx_smem[];  // [stages][FX_LOADS][FX_THREADS] pieces, the rows, the routing's scratch
  __shared__ __align__(16) float part[2][FX_WARPS][NA][32][4];
  __shared__ int chosen[FX_PAIRS];
  __shared__ float weight[FX_PAIRS];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, KT = a.K + a.C;
  const int groups = (a.N + 15) / 16, shared_units = a.C * groups, total = shared_units + a.T * a.K * groups;

  const int x_rows = a.first ? a.T : a.T * KT;
  uint4* ring = (uint4*)fx_smem;
  uint4* xs = ring + (size_t)a.stages * FX_LOADS * FX_THREADS;
  if (warp == FX_WARPS) {
    // ---------------------------------------------------------------- routing
    grid_dep_wait();
    grid_dep_launch();
    if (a.first) {
      route_here(a, (double*)(xs + (size_t)x_rows * (a.K_in / 8)), lane, chosen, weight);
      __syncwarp();
      if (blockIdx.x == 0)
        for (int i = lane; i < a.T * KT; i += 32) {
          a.idx[i] = chosen[i];
          a.score[i] = weight[i];
        }
    } else {
      for (int i = lane; i < a.T * KT; i += 32) chosen[i] = a.idx[i];
    }
    __syncwarp();
    asm volatile("bar.arrive 2, %0;" ::"n"(FX_THREADS + 32) : "memory");
    return;
  }

  // ---------------------------------------------------------------- the products
  const int g = lane / 4, c = lane % 4;               // fragment row / column group of this lane
  const int steps = a.K_in / 32;                      // this warp takes steps warp, warp + 16, ...
  const int my_steps = steps > warp ? (steps - warp + FX_WARPS - 1) / FX_WARPS : 0;
  const int rounds = max(1, ((steps + FX_WARPS - 1) / FX_WARPS + BATCH - 1) / BATCH);   // the same for every warp
  const long long w_expert = (long long)NA * a.N * a.K_in;
  bool routed = false;                                // this warp has waited for the choices
  auto unit_of = [&](int u) {
    FxUnit n;
    if (u < shared_units) {
      const int ch = u / groups;
      n.w = a.w + (a.E + ch) * w_expert;
      n.x0 = a.first ? 0 : a.K + ch;
      n.x_step = a.first ? 1 : KT;
      n.rows = a.T;
      n.n0 = (u - ch * groups) * 16;
      n.out0 = a.K + ch;
      return n;
    }
    if (!routed) {
      asm volatile("bar.sync 2, %0;" ::"n"(FX_THREADS + 32) : "memory");
      routed = true;
    }
    const int p = (u - shared_units) / groups, t = p / a.K, k = p - t * a.K;
    n.w = a.w + chosen[t * KT + k] * w_expert;
    n.x0 = a.first ? t : t * KT + k;
    n.x_step = 0;
    n.rows = 1;
    n.n0 = (u - shared_units - p * groups) * 16;
    n.out0 = t * KT + k;
    return n;
  };
  auto issue = [&](const FxUnit& n, int r, int stage) {
    const int f_lo = min(n.n0 + g, a.N - 1), f_hi = min(n.n0 + g + 8, a.N - 1);
    const uint32_t to = (uint32_t)__cvta_generic_to_shared(ring + (size_t)stage * FX_LOADS * FX_THREADS + threadIdx.x);
#pragma unroll
    for (int b = 0; b < BATCH; ++b) {
      const int i = r * BATCH + b;
      if (i < my_steps) {
        const int at = (warp + i * FX_WARPS) * 32 + c * 8;
#pragma unroll
        for (int s = 0; s < NA; ++s) {
          const uint32_t p = to + (b * NA + s) * 2 * FX_THREADS * 16;
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(p), "l"(n.w + (long long)(s * a.N + f_lo) * a.K_in + at) : "memory");
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(p + FX_THREADS * 16), "l"(n.w + (long long)(s * a.N + f_hi) * a.K_in + at) : "memory");
        }
      }
    }
  };
  float acc[NA][4];
  auto clear = [&] {
#pragma unroll
    for (int s = 0; s < NA; ++s) acc[s][0] = acc[s][1] = acc[s][2] = acc[s][3] = 0.f;
  };
  int done = 0;
  auto compute = [&](const FxUnit& n, int r, int stage) {
    const uint4* own = ring + (size_t)stage * FX_LOADS * FX_THREADS + threadIdx.x;
    const uint4* xp = xs + (size_t)(n.x0 + (g < n.rows ? g : 0) * n.x_step) * (a.K_in / 8) + c;
#pragma unroll
    for (int b = 0; b < BATCH; ++b) {
      const int i = r * BATCH + b;
      if (i < my_steps) {
        const uint4 xv = g < n.rows ? xp[(warp + i * FX_WARPS) * 4] : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int s = 0; s < NA; ++s) {
          const uint4 wl = own[(b * NA + s) * 2 * FX_THREADS], wh = own[((b * NA + s) * 2 + 1) * FX_THREADS];
          mma_16816(acc[s], wl.x, wh.x, wl.y, wh.y, xv.x, xv.y);
          mma_16816(acc[s], wl.z, wh.z, wl.w, wh.w, xv.z, xv.w);
        }
      }
    }
    if (r + 1 < rounds) return;
    // the unit is complete: the warps' sums are added in warp order (the halves of `part` take turns, see skinny_gemm.cu)
    float(*p)[NA][32][4] = part[done & 1];
    ++done;
#pragma unroll
    for (int s = 0; s < NA; ++s) *(float4*)p[warp][s][lane] = make_float4(acc[s][0], acc[s][1], acc[s][2], acc[s][3]);
    clear();
    asm volatile("bar.sync 1, %0;" ::"n"(FX_THREADS) : "memory");
    if (threadIdx.x < 128) {
      const int l = threadIdx.x / 4, j = threadIdx.x % 4;
      const int feat = n.n0 + l / 4 + 8 * (j / 2), row = 2 * (l % 4) + (j % 2);
      if (feat < a.N && row < n.rows) {
        float v[NA];
#pragma unroll
        for (int s = 0; s < NA; ++s) {
          v[s] = 0.f;
#pragma unroll
          for (int wi = 0; wi < FX_WARPS; ++wi) v[s] += p[wi][s][l][j];
        }
        const float o = GATED ? pair_mul(a.pair, v[0], v[NA - 1], a.act_p0, a.act_p1)
                              : epilogue_act(epi_at(a.act, feat, a.act_p0), v[0], a.act_p0, a.act_p1);
        st_dt(a.out, a.out_dt, (size_t)(n.out0 + row * KT) * a.N + feat, o);
      }
    }
  };

  // rounds are asked for `stages - 1` ahead of the one that is worked on, also across units
  clear();
  int iu = blockIdx.x, ir = 0, islot = 0, asked = 0;
  FxUnit ahead;
  auto ask = [&] {
    if (iu < total) {
      if (ir == 0) ahead = unit_of(iu);
      issue(ahead, ir, islot);
      if (++ir == rounds) { ir = 0; iu += gridDim.x; }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    islot = islot + 1 == a.stages ? 0 : islot + 1;
    ++asked;
  };
  while (asked < a.stages - 1 && iu < shared_units) ask();        // (no choice of the routing is needed for these)
  grid_dep_wait();                                    // now the rows, and with them the rest
  const int per = a.K_in / 8, x_all = x_rows * per;
  for (int i0 = threadIdx.x; i0 < x_all; i0 += 4 * FX_THREADS) {
    uint4 v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int i = min(i0 + j * FX_THREADS, x_all - 1), r = i / per;
      v[j] = *((const uint4*)(a.x + r * a.ldx) + (i - r * per));
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (i0 + j * FX_THREADS < x_all) xs[i0 + j * FX_THREADS] = v[j];
  }
  asm volatile("bar.sync 1, %0;" ::"n"(FX_THREADS) : "memory");
  while (asked < a.stages - 1) ask();
  int slot = 0;
  for (int u = blockIdx.x; u < total; u += gridDim.x) {
    const FxUnit n = unit_of(u);
    for (int r = 0; r < rounds; ++r) {
      if (a.stages == 5) asm volatile("cp.async.wait_group 3;" ::: "memory");
      else if (a.stages == 4) asm volatile("cp.async.wait_group 2;" ::: "memory");
      else asm volatile("cp.async.wait_group 1;" ::: "memory");
      ask();              // (into the slot of the round before this one: a lane reads its own pieces only)
      compute(n, r, slot);
      slot = slot + 1 == a.stages ? 0 : slot + 1;
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  // (a block without routed units still meets the routing warp's arrival)
  if (!routed) asm volatile("bar.sync 2, %0;" ::"n"(FX_THREADS + 32) : "memory");
}

}  // namespace

namespace {
// Rounds of pieces that fit beside the rows of the larger of the two products (0: not three of them).
int fx_stages(int T, int E, int K, int C, int H, int I, int groups) {
  const long long first = (long long)T * H * 2 + (long long)(E + groups) * 8, second = (long long)T * (K + C) * I * 2;
  const long long room = FX_SMEM - (first > second ? first : second);
  const long long n = room / (FX_LOADS * FX_THREADS * 16);
  return n < 3 ? 0 : n > 5 ? 5 : (int)n;
}
}  // namespace

// Whether the two kernels take a layer of these sizes: K, C experts per row of E, T rows, hidden H, inner I.
NV_API int nv_few_experts_usable(int T, int E, int K, int C, int H, int I, int groups) {
  return T >= 1 && T <= 8 && T * (K + C) <= FX_PAIRS && K >= 1 && K <= 32 && K <= E && C >= 0 && C <= 32 && H % 32 == 0 &&
         I % 32 == 0 && fx_stages(T, E, K, C, H, I, groups) >= 3;
}

// First product (`first`): routes the T rows of `logits` (see route_row), writes idx and score [T, K + C], and
// out[t * (K + C) + k, :] (bfloat16 or float32, [T (K + C), N]) = the expert's first product of row t of x.  gated: w holds N gate
// and N up rows an expert, paired as `act` says.  Second product: x is the first one's output, w [E + C, N, K_in].
NV_API int nv_few_experts(const void* x, long long ldx, const void* w, void* out, int out_dt, int* idx, float* score,
                          const float* logits, long long ld, const float* gate_logit, long long gate_ld, int renorm, int T, int E,
                          int K, int C, int N, int K_in, int first, int epi, float act_p0, float act_p1, int mode,
                          const float* choice_bias, float weight_scale, int groups, int keep, cudaStream_t stream) {
  if (!dt_ok(out_dt)) return NV_ERR_BAD_DTYPE;
  if (!route_groups_ok(E, K, groups, keep) || mode < 0 || mode > 1 || epi < 0 || epi > NV_EPI_LAST) return NV_ERR_BAD_SIZE;
  if (!nv_few_experts_usable(T, E, K, C, first ? K_in : 32, first ? 32 : K_in, groups) || N <= 0 || ldx % 8 || ((uintptr_t)x & 15) || ((uintptr_t)w & 15))
    return NV_ERR_UNSUPPORTED;
  FxArgs a;
  a.x = (const bf16*)x; a.w = (const bf16*)w; a.out = out; a.idx = idx; a.score = score; a.logits = logits; a.ld = ld;
  a.gate_logit = C ? gate_logit : nullptr; a.gate_ld = gate_ld;
  a.rule = RouteRule{mode, choice_bias, weight_scale, groups, keep};
  a.renorm = renorm; a.ldx = ldx; a.T = T; a.E = E; a.K = K; a.C = C; a.N = N; a.K_in = K_in; a.out_dt = out_dt; a.first = first;
  a.act = epi_unary(epi); a.pair = epi_pair(epi); a.act_p0 = act_p0; a.act_p1 = act_p1;
  const long long units = (long long)(C + T * K) * ((N + 15) / 16);
  const int sms = num_multiprocessors();
  const dim3 grid((unsigned)(units < sms ? units : sms)), block((FX_WARPS + 1) * 32);
  a.stages = fx_stages(T, E, K, C, first ? K_in : 0, first ? 0 : K_in, groups);
  const size_t smem = (size_t)a.stages * FX_LOADS * FX_THREADS * 16 + (size_t)(first ? T : T * (K + C)) * K_in * 2 +
                      (first ? (size_t)(E + groups) * sizeof(double) : 0);
  auto* kernel = a.pair ? few_experts_kernel<true> : few_experts_kernel<false>;
  NV_RETURN_IF(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FX_SMEM));
  NV_RETURN_IF(launch_dep(kernel, grid, block, smem, stream, a));
  NV_RETURN_LAST();
}
