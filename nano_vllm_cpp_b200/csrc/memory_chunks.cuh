// Matrix memories over many rows, in chunks of eight: the delta rule (one decay per head, or per head and key channel)
// and the matrix LSTM.  Included by seq_mix_ops.cu, whose row-by-row scan (col_scan_kernel) keeps the steps of many short
// entries (memory_chunks_pay in ops.py) and the float32 runs, whose sums do not depend on how a sequence is cut into steps.
//
// What bounds the scan is that a row's product with the memory has to be known before the next row changes the memory:
// a barrier, two shuffled sums and a hundred and sixty FMAs a lane for every row, one after the other (2,048 rows of one
// sequence: 0.36 us a row).  With S0 the memory before a chunk, D_i the product of the decays of rows 1 .. i,
//
//     u_i = beta_i (v_i - S0^T (D_i k_i) - sum_{j<i} kk_ij u_j),     kk_ij = sum_r k_i[r] k_j[r] D_i[r] / D_j[r]
//     o_i = S0^T (D_i q_i) + sum_{j<=i} qk_ij u_j,                   qk_ij = sum_r q_i[r] k_j[r] D_i[r] / D_j[r]
//     S   = D_n S0 + sum_j (k_j D_n / D_j) u_j^T
//
// so all eight products with the memory are independent, and what is left of the chain is eight steps of one FMA.  The
// quotients D_i / D_j are products of the decays in between (no division, nothing overflows).  All sums are float32.
// chunk_prepare_kernel makes D_i k_i, D_i q_i, k_j D_n / D_j and the two triangles once per chunk and head;
// chunk_scan_kernel walks a sequence's chunks with the memory in registers: four (or two) columns in sixteen lanes, eight rows of
// each a lane at 128.  A 16-byte read of shared memory takes a warp four cycles of its multiprocessor's port however many
// lanes read the same, so what matters is how many FMAs such a read feeds (16 here; with a column in eight lanes
// and one column a lane the port was the kernel's time).  The eight sums of a column's chunk end, after eight shuffles, with
// lane i holding row i's.  The matrix LSTM is the same without the first product and with weights exp(F_i - F_j + i_j - m_i) for
// the quotients (F the running sum of the log forget gates, m_i the running maximum).
// Measured (heads of 128 x 128, preparation, gates and head norm included): 1,500 rows of one sequence, 8 heads: delta rule
// 576 -> 281 us, matrix LSTM 531 -> 277; eight sequences of 200 to 2,048 rows, 16 heads, a decay per channel: 1,870 -> 734 us
// (825 before two FMAs went into one instruction and the longest sequences first).  Against float64
// the states are off by no more than row by row (tests/test_memory_chunks_gpu.py).

constexpr int MC_R = 8;                                   // rows of a chunk
constexpr int MC_RING = 3;                                // chunks in shared memory
constexpr int MC_TRI = 144;                               // floats behind a record's rows: kk[8][8], qk[8][8], beta[8], pad

// A chunk's record: delta rule [3][8][DK] + [DK] (D k, D q, k D_n / D, D_n), LSTM [2][8][DK] (q, k), then MC_TRI floats
// (LSTM: f[8], i[8] in place of kk).
__host__ __device__ constexpr int mc_rows(int DK, bool lstm) { return (lstm ? 16 : 25) * DK; }
__host__ __device__ constexpr int mc_record(int DK, bool lstm) { return mc_rows(DK, lstm) + MC_TRI; }
// Entry e's chunks stand at records cu_rows[e] / 8 + e and on: room for every entry's last, shorter chunk.
__host__ __device__ inline long long mc_records(int T, int S) { return T / MC_R + S; }

struct ChunkArgs {
  const int* cu_rows;
  int S_entries;
  const float* qk;          // rows that hold q and k
  long long qk_ld;
  int q0, k0, G;
  const void* gates;        // delta rule: beta; LSTM: i, f
  int gates_dt;
  long long gates_ld;
  int ga0, gb0;             // LSTM: i, f; delta rule: beta, and (one decay per head) the decay's pre-activation
  const float* dec;         // a decay per channel: pre-activations [T, dec_ld], head h's at dec0 + h dk; else null
  long long dec_ld;
  int dec0;
  const float* A_log;
  const float* dt_bias;
  float cap;
  float* rec;               // [records][H][mc_record]
  int H, dk;
};

template <int DK, bool LSTM>
__global__ void __launch_bounds__(DK) chunk_prepare_kernel(ChunkArgs a) {
  constexpr int NW = DK / 32;
  __shared__ float part[NW][64];
  const int x = blockIdx.x, h = blockIdx.y, r = threadIdx.x, lane = r % 32;
  int lo = 0, hi = a.S_entries - 1;                       // the last entry whose chunks start at or before x
  while (lo < hi) {
    const int mid = (lo + hi + 1) / 2;
    if (a.cu_rows[mid] / MC_R + mid <= x) lo = mid;
    else hi = mid - 1;
  }
  const int begin = a.cu_rows[lo], row0 = begin + (x - (begin / MC_R + lo)) * MC_R;
  const int n = min(MC_R, a.cu_rows[lo + 1] - row0);
  if (n <= 0) return;
  const int dk = a.dk, gh = h / (a.H / a.G);
  const bool in = r < dk;
  float* rec = a.rec + ((long long)x * a.H + h) * mc_record(DK, LSTM);
  float* tri = rec + mc_rows(DK, LSTM);
  float q[MC_R], k[MC_R], val[64];
#pragma unroll
  for (int i = 0; i < MC_R; ++i) {
    const float* p = a.qk + (size_t)(row0 + i) * a.qk_ld + gh * dk + r;
    q[i] = in && i < n ? p[a.q0] : 0.f;
    k[i] = in && i < n ? p[a.k0] : 0.f;
  }
  if (LSTM) {
#pragma unroll
    for (int i = 0; i < MC_R; ++i) {
      rec[i * DK + r] = q[i];
      rec[(MC_R + i) * DK + r] = k[i];
#pragma unroll
      for (int j = 0; j < MC_R; ++j) {
        if (j < i) val[i * (i - 1) / 2 + j] = 0.f;
        if (j <= i) val[28 + i * (i + 1) / 2 + j] = q[i] * k[j];
      }
    }
  } else {
    float d[MC_R];
    const float rate = expf(a.A_log[h]), bias = a.dec ? (in ? a.dt_bias[h * dk + r] : 0.f) : a.dt_bias[h];
#pragma unroll
    for (int i = 0; i < MC_R; ++i) {
      d[i] = 1.f;
      if (i < n && (in || !a.dec))
        d[i] = expf(-rate * softplusf_((a.dec ? a.dec[(size_t)(row0 + i) * a.dec_ld + a.dec0 + h * dk + r]
                                              : ((const float*)a.gates)[(size_t)(row0 + i) * a.gates_ld + a.gb0 + h]) + bias));
    }
    float c = 1.f;
#pragma unroll
    for (int i = 0; i < MC_R; ++i) {
      c *= d[i];
      rec[i * DK + r] = k[i] * c;
      rec[(MC_R + i) * DK + r] = q[i] * c;
    }
    rec[3 * MC_R * DK + r] = c;
    c = 1.f;
#pragma unroll
    for (int j = MC_R - 1; j >= 0; --j) {
      rec[(2 * MC_R + j) * DK + r] = k[j] * c;
      c *= d[j];
    }
#pragma unroll
    for (int j = 0; j < MC_R; ++j) {
      float w = k[j];
      val[28 + j * (j + 1) / 2 + j] = q[j] * w;
#pragma unroll
      for (int i = j + 1; i < MC_R; ++i) {
        w *= d[i];
        val[i * (i - 1) / 2 + j] = k[i] * w;
        val[28 + i * (i + 1) / 2 + j] = q[i] * w;
      }
    }
  }
  // 64 sums over the channels: after five exchanges a lane holds two of its warp's
#pragma unroll
  for (int off = 16, half = 32; off > 0; off >>= 1, half >>= 1) {
    const bool up = lane & off;
#pragma unroll
    for (int v = 0; v < half; ++v) {
      const float send = up ? val[v] : val[v + half];
      val[v] = (up ? val[v + half] : val[v]) + __shfl_xor_sync(0xffffffffu, send, off);
    }
  }
  // (lane bit 4 chose between halves of 64, bit 3 of 32, ...: its two sums are 2 lane and 2 lane + 1)
  part[r / 32][2 * lane] = val[0];
  part[r / 32][2 * lane + 1] = val[1];
  __syncthreads();
  for (int t = r; t < MC_TRI; t += DK) {
    float v = 0.f;
    if (t < 128) {
      const int i = t % 64 / 8, j = t % 8;
      if (t >= 64 ? j <= i : (j < i && !LSTM)) {
        const int at = t >= 64 ? 28 + i * (i + 1) / 2 + j : i * (i - 1) / 2 + j;
#pragma unroll
        for (int w = 0; w < NW; ++w) v += part[w][at];
      } else if (LSTM && t < 16) {
        const int row = row0 + t % 8;
        const float* g = (const float*)a.gates + (size_t)row * a.gates_ld;
        if (t < 8) v = t < n ? logsigmoidf_(a.cap * tanhf(g[a.gb0 + h] / a.cap)) : 0.f;
        else v = t - 8 < n ? a.cap * tanhf(g[a.ga0 + h] / a.cap) : -1e30f;
      }
    } else if (!LSTM && t < 128 + n) {
      v = sigmoidf_(ld_dt(a.gates, a.gates_dt, (size_t)(row0 + t - 128) * a.gates_ld + a.ga0 + h));
    }
    tri[t] = v;
  }
}

struct ChunkScanArgs {
  const int* cu_rows;
  const int* entry_slot;
  const float* rec;
  float* S;                 // [slots][H, dk, dv]
  long long S_stride;
  float* n;                 // LSTM: [slots][H, dk]
  long long n_stride;
  const float* m;           // LSTM: [slots][H]; the new maximum goes to raw (head_finish_kernel takes it from there)
  long long m_stride;
  const float* vsrc;
  long long v_ld;
  int v0;
  float q_scale;
  float* raw;               // [T, H, RW]
  int RW, H, dk, dv;
};

// Of eight sums a lane (x[i]: this lane's part of row i's), row (l mod 8)'s, summed over the sixteen lanes.
__device__ __forceinline__ float own_row_sum(const float (&x)[MC_R], int l) {
  float y[4], z[2];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float send = l & 4 ? x[i] : x[i + 4];
    y[i] = (l & 4 ? x[i + 4] : x[i]) + __shfl_xor_sync(0xffffffffu, send, 4);
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const float send = l & 2 ? y[i] : y[i + 2];
    z[i] = (l & 2 ? y[i + 2] : y[i]) + __shfl_xor_sync(0xffffffffu, send, 2);
  }
  const float send = l & 1 ? z[0] : z[1];
  const float w = (l & 1 ? z[1] : z[0]) + __shfl_xor_sync(0xffffffffu, send, 1);
  return w + __shfl_xor_sync(0xffffffffu, w, 8);
}

// Two float32 FMAs, each rounded as one, in one instruction.
__device__ __forceinline__ void fma2(float2& d, float2 a, float2 b, float2 c) {
  unsigned long long r, x = *(unsigned long long*)&a, y = *(unsigned long long*)&b, z = *(unsigned long long*)&c;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(x), "l"(y), "l"(z));
  d = *(float2*)&r;
}

constexpr int MC_LANES = 16;                              // lanes of a column

// CT: columns of a lane.
template <int DK, bool LSTM, int WARPS, int CT>
__global__ void __launch_bounds__(32 * WARPS) chunk_scan_kernel(ChunkScanArgs a) {
  constexpr int REC = mc_record(DK, LSTM), NP = DK / 64;      // a lane's rows: NP pieces of four, 64 apart
  extern __shared__ __align__(16) float ring[];
  const int h = blockIdx.y, tid = threadIdx.x, l = tid % MC_LANES, row = l % MC_R, group = tid / MC_LANES;
  // Longest sequences first: a sequence is one walk however many blocks share its columns, so the last to begin should be
  // short (eight sequences of 200 to 2,048 rows in order of their numbers left some multiprocessors three of the longest).
  int e = blockIdx.z;
  if (gridDim.z <= 32 * WARPS) {
    __shared__ int chosen;
    const int S_n = gridDim.z;
    if (tid < S_n) {
      const int mine = a.cu_rows[tid + 1] - a.cu_rows[tid];
      int rank = 0;
      for (int j = 0; j < S_n; ++j) {
        const int other = a.cu_rows[j + 1] - a.cu_rows[j];
        rank += other > mine || (other == mine && j < tid);
      }
      if (rank == e) chosen = tid;
    }
    __syncthreads();
    e = chosen;
  }
  const int dk = a.dk, dv = a.dv, ncols = LSTM ? dv + 1 : dv;
  const int col = (blockIdx.x * 2 * WARPS + group) * CT;
  const int row0 = a.cu_rows[e], rows = a.cu_rows[e + 1] - row0, chunks = (rows + MC_R - 1) / MC_R;
  const int slot = a.entry_slot[e];
  const float* rec = a.rec + ((long long)(row0 / MC_R + e) * a.H + h) * REC;
  const size_t rec_step = (size_t)a.H * REC;
  auto fetch = [&](int c) {
    if (c < chunks)
      for (int i = tid; i < REC / 4; i += 32 * WARPS)
        cp_async16(ring + (c % MC_RING) * REC + 4 * i, rec + c * rec_step + 4 * i);
    cp_async_commit();
  };
  for (int c = 0; c < MC_RING - 1; ++c) fetch(c);

  float2 S[NP][2][CT];                             // rows 4 (l + 16 p) + 0, 1 and + 2, 3 of every column
  auto place = [&](int t, int r) -> float* {
    return LSTM && col + t == dv ? a.n + (size_t)slot * a.n_stride + (size_t)h * dk + r
                                 : a.S + (size_t)slot * a.S_stride + ((size_t)h * dk + r) * dv + col + t;
  };
#pragma unroll
  for (int p = 0; p < NP; ++p)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int r = 4 * (l + MC_LANES * p) + 2 * i;
#pragma unroll
      for (int t = 0; t < CT; ++t)
        S[p][i][t] = make_float2(col + t < ncols && r < dk ? *place(t, r) : 0.f,
                                 col + t < ncols && r + 1 < dk ? *place(t, r + 1) : 0.f);
    }
  float m0 = LSTM ? a.m[(size_t)slot * a.m_stride + h] : 0.f;
  const float* vp = a.vsrc + (size_t)(row0 + row) * a.v_ld + a.v0 + (size_t)h * dv + col;
  float v_next[CT];
  auto fetch_v = [&](int c) {
#pragma unroll
    for (int t = 0; t < CT; ++t)
      v_next[t] = c * MC_R + row < rows ? (col + t < dv ? vp[(size_t)c * MC_R * a.v_ld + t] : 1.f) : 0.f;
  };
  fetch_v(0);
  float* out = a.raw + ((size_t)(row0 + row) * a.H + h) * a.RW + col;

  for (int c = 0; c < chunks; ++c) {
    cp_async_wait<MC_RING - 2>();
    __syncthreads();                               // the chunk's record is there, and everyone is through with the last one
    fetch(c + MC_RING - 1);
    const float* rc = ring + (c % MC_RING) * REC;
    const float4* q4 = (const float4*)(rc + (LSTM ? 0 : MC_R * DK)) + l;
    const float4* k4 = (const float4*)rc + l;                                       // delta rule: D k
    const float4* t4 = (const float4*)(rc + (LSTM ? 1 : 2) * MC_R * DK) + l;        // what the values are multiplied by
    const float* tri = rc + mc_rows(DK, LSTM);
    float v[CT];
#pragma unroll
    for (int t = 0; t < CT; ++t) v[t] = v_next[t];
    fetch_v(c + 1);

    float pk[CT][MC_R], pq[CT][MC_R];
#pragma unroll
    for (int i = 0; i < MC_R; ++i) {
      float2 sk[CT], sq[CT];
#pragma unroll
      for (int t = 0; t < CT; ++t) sk[t] = sq[t] = make_float2(0.f, 0.f);
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        const float4 qq = q4[i * (DK / 4) + MC_LANES * p];
        float4 kk = make_float4(0.f, 0.f, 0.f, 0.f);
        if (!LSTM) kk = k4[i * (DK / 4) + MC_LANES * p];
#pragma unroll
        for (int t = 0; t < CT; ++t) {
          fma2(sq[t], S[p][0][t], make_float2(qq.x, qq.y), sq[t]);
          fma2(sq[t], S[p][1][t], make_float2(qq.z, qq.w), sq[t]);
          if (!LSTM) {
            fma2(sk[t], S[p][0][t], make_float2(kk.x, kk.y), sk[t]);
            fma2(sk[t], S[p][1][t], make_float2(kk.z, kk.w), sk[t]);
          }
        }
      }
#pragma unroll
      for (int t = 0; t < CT; ++t) { pq[t][i] = sq[t].x + sq[t].y; pk[t][i] = sk[t].x + sk[t].y; }
    }
    float qkr[MC_R], u[CT][MC_R], o[CT], scale = 1.f, keep = 1.f;
    *(float4*)qkr = *(const float4*)(tri + 64 + 8 * row);
    *(float4*)(qkr + 4) = *(const float4*)(tri + 64 + 8 * row + 4);
    if (LSTM) {
      float f[MC_R], g[MC_R];
#pragma unroll
      for (int i = 0; i < MC_R; i += 4) {
        *(float4*)(f + i) = *(const float4*)(tri + i);
        *(float4*)(g + i) = *(const float4*)(tri + 8 + i);
      }
      float F = 0.f, mine = 0.f;                   // F: running sum of the log forget gates; this lane's row's
#pragma unroll
      for (int j = 0; j < MC_R; ++j) { F += f[j]; f[j] = F; if (j <= row) mine = F; }
      float m = mine + m0;
#pragma unroll
      for (int j = 0; j < MC_R; ++j) if (j <= row) m = fmaxf(m, mine - f[j] + g[j]);
#pragma unroll
      for (int j = 0; j < MC_R; ++j) g[j] = j <= row ? expf(mine - f[j] + g[j] - m) : 0.f;      // row j's weight in this row
      keep = expf(mine + m0 - m);
#pragma unroll
      for (int t = 0; t < CT; ++t) o[t] = keep * own_row_sum(pq[t], l);
#pragma unroll
      for (int j = 0; j < MC_R; ++j) {
        const float w7 = __shfl_sync(0xffffffffu, g[j], MC_R - 1, MC_LANES);
#pragma unroll
        for (int t = 0; t < CT; ++t) {
          const float vj = __shfl_sync(0xffffffffu, v[t], j, MC_LANES);
          if (j <= row) o[t] = fmaf(g[j] * qkr[j], vj, o[t]);        // (a later row's value may not be finite)
          u[t][j] = w7 * vj;
        }
      }
      if (blockIdx.x == 0 && tid < MC_R && c * MC_R + row < rows) out[dv + 1] = m;
      m0 = __shfl_sync(0xffffffffu, m, MC_R - 1, MC_LANES);
      keep = __shfl_sync(0xffffffffu, keep, MC_R - 1, MC_LANES);
      scale = a.q_scale;
    } else {
      float kkr[MC_R], acc[CT];
      *(float4*)kkr = *(const float4*)(tri + 8 * row);
      *(float4*)(kkr + 4) = *(const float4*)(tri + 8 * row + 4);
      const float beta = tri[128 + row];
#pragma unroll
      for (int t = 0; t < CT; ++t) { acc[t] = v[t] - own_row_sum(pk[t], l); o[t] = own_row_sum(pq[t], l); }
#pragma unroll
      for (int j = 0; j < MC_R; ++j)
#pragma unroll
        for (int t = 0; t < CT; ++t) {
          u[t][j] = __shfl_sync(0xffffffffu, beta * acc[t], j, MC_LANES);       // (rows before j have taken theirs off)
          acc[t] = fmaf(-kkr[j], u[t][j], acc[t]);
          if (j <= row) o[t] = fmaf(qkr[j], u[t][j], o[t]);          // (0 times a later row's infinity would be NaN)
        }
    }
    if (l < MC_R && c * MC_R + row < rows) {
#pragma unroll
      for (int t = 0; t < CT; ++t)
        if (col + t < ncols) out[t] = o[t] * scale;
    }
    out += (size_t)MC_R * a.H * a.RW;
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      float4 dd = make_float4(keep, keep, keep, keep);
      if (!LSTM) dd = ((const float4*)(rc + 3 * MC_R * DK) + l)[MC_LANES * p];
#pragma unroll
      for (int t = 0; t < CT; ++t) {
        S[p][0][t].x *= dd.x; S[p][0][t].y *= dd.y; S[p][1][t].x *= dd.z; S[p][1][t].y *= dd.w;
      }
#pragma unroll
      for (int j = 0; j < MC_R; ++j) {
        const float4 kk = t4[j * (DK / 4) + MC_LANES * p];
#pragma unroll
        for (int t = 0; t < CT; ++t) {
          const float2 uu = make_float2(u[t][j], u[t][j]);
          fma2(S[p][0][t], make_float2(kk.x, kk.y), uu, S[p][0][t]);
          fma2(S[p][1][t], make_float2(kk.z, kk.w), uu, S[p][1][t]);
        }
      }
    }
  }
  cp_async_wait<0>();
#pragma unroll
  for (int p = 0; p < NP; ++p)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int r = 4 * (l + MC_LANES * p) + 2 * i;
#pragma unroll
      for (int t = 0; t < CT; ++t)
        if (col + t < ncols) {
          if (r < dk) *place(t, r) = S[p][i][t].x;
          if (r + 1 < dk) *place(t, r + 1) = S[p][i][t].y;
        }
    }
}

// Ordinary launches: as programmatic dependents the scan's few blocks were placed while the preparation still ran, four
// to a multiprocessor, and stayed there for the whole walk (1,500 rows of 8 heads: 790 instead of 340 us).
template <int DK, bool LSTM, int WARPS, int CT>
int launch_chunk_scan(const ChunkScanArgs& a, int S, cudaStream_t s) {
  const int ncols = LSTM ? a.dv + 1 : a.dv, per = 2 * WARPS * CT;
  const size_t smem = sizeof(float) * MC_RING * mc_record(DK, LSTM);
  auto* kernel = chunk_scan_kernel<DK, LSTM, WARPS, CT>;
  if (smem > 48 * 1024) NV_RETURN_IF(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  kernel<<<dim3((ncols + per - 1) / per, a.H, S), 32 * WARPS, smem, s>>>(a);
  NV_RETURN_LAST();
}

template <int DK, bool LSTM>
int launch_chunks(const ChunkArgs& p, const ChunkScanArgs& a, int T, cudaStream_t s) {
  const int S = p.S_entries;
  if (mc_records(T, S) > 0x7fffffff || a.H > 65535 || S > 65535) return NV_ERR_BAD_SIZE;
  chunk_prepare_kernel<DK, LSTM><<<dim3((unsigned)mc_records(T, S), a.H), DK, 0, s>>>(p);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return (int)e;
  // Blocks of 32 columns share a record between four warps of four columns a lane.  Where they would not give every
  // multiprocessor one, a warp's instructions are the time of a chunk (1,130 of them, two cycles each, on one of four
  // schedulers): two columns a lane halve them, at the price of reading the record twice as often, and four warps still share it
  // (1,500 rows of one sequence, preparation and head norm included, 8 heads: delta rule 298 us with one warp of four columns a
  // block, 263 so; matrix LSTM 309 and 272; 16 heads, a decay per channel, 328 and 280).  The LSTM's shorter chunks stay with the one
  // warp where the halves are more than the multiprocessors (four sequences of 500, 8 heads: 152 and 155).
  const int sms = num_multiprocessors();
  const long long wide = (long long)S * a.H * ((a.dv + 31) / 32), half = (long long)S * a.H * ((a.dv + 15) / 16);
  if (wide >= sms) return launch_chunk_scan<DK, LSTM, 4, 4>(a, S, s);
  return LSTM && half > sms ? launch_chunk_scan<DK, LSTM, 1, 4>(a, S, s) : launch_chunk_scan<DK, LSTM, 4, 2>(a, S, s);
}

template <bool LSTM>
int launch_chunks_of(const ChunkArgs& p, const ChunkScanArgs& a, int T, cudaStream_t s) {
  if (a.dk <= 64) return launch_chunks<64, LSTM>(p, a, T, s);
  if (a.dk <= 128) return launch_chunks<128, LSTM>(p, a, T, s);
  return NV_ERR_UNSUPPORTED;
}
