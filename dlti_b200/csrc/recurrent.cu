// Linear recurrences with an outer-product update, one state matrix per head:
//     S_t = a_t S_(t-1) + k_t (s_t v_t)^T,      o_t = S_t^T q_t + D v_t        (S is N x P, fp32)
// Mamba-2:    k = B, q = C (shared by the heads of a group), v = x, s_t = dt, a_t = exp(-exp(A_log) dt), D per head
// lightning:  a_t = one constant per head, s_t = 1, D = 0, silu on q, k, v as they are loaded
// mLSTM:      a_t = exp(f_t + m_(t-1) - m_t), s_t = exp(i_t - m_t) with log gates i_t, f_t and the running maximum
//             m_t = max(f_t + m_(t-1), i_t), m_0 = 0; n_t = a_t n_(t-1) + s_t k_t and o_t is divided by
//             max(|n_t . q_t|, exp(-m_t)) + 1e-6. n and m are state too; every slice of 32 columns of P, which is a CTA of
//             its own, keeps them for itself: vec [slots, heads, slices, N + 1] = n, then m.
// States live in slots [slots, heads, N, P] and are carried from step to step; a sequence whose step starts at position
// 0 starts from zero whatever its slot holds.
#include "recurrent.cuh"
#include "mma_sync.cuh"

namespace {

struct ScanParams {
  const void *q, *k, *v;
  long long q_ld, k_ld, v_ld;
  int rep;                                 // heads per q/k group
  int silu;
  const float* decay;                  // [heads] or null
  const void* dt; long long dt_ld;         // raw step sizes [rows, heads] (T) when decay is null
  const float *dt_bias, *A_log, *D;        // [heads]; D may be null
  float* state;
  const int *sslot, *ctx, *cu;
  int nd, seq0, heads, N, P;
  void* out; long long o_ld;
  // tail job: new convolution state = last conv_rows inputs of every sequence
  const void* conv_src; long long conv_ld; int conv_col, conv_rows, conv_C;
  void* conv_state;
  // mLSTM: raw gates [rows, >= 2 heads] fp32 (input gates, then forget gates), biases in the same order, soft cap, factor on q
  const float *gates, *gate_b; long long g_ld;
  float cap, q_scale;
  float* vec;
  // chunked form in segments: tokens of a segment (a multiple of 64), segments of the longest sequence, see SegEntry
  int seg_len, segs;
  float* seg_ws;
};

// log gates of an mLSTM head: cap tanh(z / cap), for the forget gate the logarithm of its sigmoid
__device__ __forceinline__ float log_in_gate(float z, float cap) { return cap * tanhf(z / cap); }
__device__ __forceinline__ float log_forget_gate(float z, float cap) { return -softplus_f(-cap * tanhf(z / cap)); }
__device__ __forceinline__ float silu_f(float z) { return z / (1.f + expf(-z)); }

// One token per sequence (decode rows). What bounds it is the state, read and written once; the token-by-token form below spends a
// CTA of its own, with its three barriers and its loads of q and k, on every 32 columns. Here a lane owns V consecutive columns, so
// the CTAs of an SM have 64 KB of the state in flight or more. States that come from HBM, us with the token-by-token form -> now: 8 heads of
// 128 x 256 (mLSTM) 1 row 4.1 -> 3.6, 4 rows 5.6 -> 5.7, 16 rows 14.0 -> 9.0, 64 rows 47 -> 28; 64 heads of 128 x 64 1 row 3.5 -> 2.7, 4 rows 6.2 ->
// 5.4, 16 rows 18.7 -> 15.0, 64 rows 75 -> 47 (268 MB read and written). The order of all sums is that of the token-by-token form. The
// next kernel may start after the wait, not before it (griddep_pass): 256 CTAs take 5.7 instead of 6.3 us, as if the CTAs that already wait
// on the SMs made these spread less evenly.
template <typename T, int NR, int V, bool ML>
__global__ void __launch_bounds__(256, step_ctas(NR, V)) scan_step_kernel(const ScanParams p, int blocks, int conv_parts) {
  griddep_wait();
  griddep_launch();
  const int s = p.seq0 + blockIdx.z;
  if ((int)blockIdx.x >= blocks) {
    if (blockIdx.y == 0) conv_tail<T>(p, s, blockIdx.x - blocks, conv_parts);
    return;
  }
  __shared__ float sk[8 * NR], sq[8 * NR], part[8][32 * V], nq[8], sc[3];          // sc: factor of the update, decay, exp(-m)
  const int h = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, grp = h / p.rep;
  const int c0 = blockIdx.x * 32 * V, col = c0 + lane * V;
  const int slot = p.sslot[s];
  const bool live = slot >= 0 && p.ctx[s] > 1, colok = col < p.P;                  // P is a multiple of V
  const long long row = s, head = (long long)(slot < 0 ? 0 : slot) * p.heads + h;
  float* st = p.state + (head * p.N + warp * NR) * p.P + col;
  float S[NR][V];
#pragma unroll
  for (int i = 0; i < NR; ++i) {
    const bool ok = live && colok && warp * NR + i < p.N;
    if constexpr (V == 2) {
      const float2 x = ok ? *reinterpret_cast<const float2*>(st + (long long)i * p.P) : make_float2(0.f, 0.f);
      S[i][0] = x.x; S[i][1] = x.y;
    } else {
      S[i][0] = ok ? st[(long long)i * p.P] : 0.f;
    }
  }
  const T* q = reinterpret_cast<const T*>(p.q) + row * p.q_ld + (long long)grp * p.N;
  const T* k = reinterpret_cast<const T*>(p.k) + row * p.k_ld + (long long)grp * p.N;
  const T* v = reinterpret_cast<const T*>(p.v) + row * p.v_ld + (long long)h * p.P;
  auto plain = [&](T x) {
    float f = Cvt<T>::to_f(x);
    if (p.silu) f = Cvt<T>::to_f(Cvt<T>::from_f(silu_f(f)));
    return f;
  };
  constexpr int GATES = 224;                               // in a warp without loads of q and k (up to 128 rows), which would wait for the gates
  constexpr int NV = (NR + 31) / 32;                       // entries of n per lane
  const int slices = (p.P + 31) / 32;                      // every slice of 32 columns has its own n and m; they are equal
  float nv[NV], m = 0.f;
  float* vec = ML ? p.vec + (head * slices + blockIdx.x * V) * (p.N + 1) : nullptr;
  if constexpr (ML) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int r = warp * NR + lane + 32 * i;
      nv[i] = (live && lane + 32 * i < NR && r < p.N) ? vec[r] : 0.f;
    }
  }
  if (threadIdx.x == GATES) {
    if constexpr (ML) {
      if (live) m = vec[p.N];
      const float zi = p.gates[row * p.g_ld + h] + p.gate_b[h], zf = p.gates[row * p.g_ld + p.heads + h] + p.gate_b[p.heads + h];
      const float f = log_forget_gate(zf, p.cap) + m, i = log_in_gate(zi, p.cap);
      m = fmaxf(f, i);
      sc[0] = expf(i - m);
      sc[1] = decay_of(f - m);
      sc[2] = expf(-m);
    } else if (p.decay) {
      sc[0] = 1.f;
      sc[1] = p.decay[h];
    } else {
      const float step = softplus_f(Cvt<T>::to_f(reinterpret_cast<const T*>(p.dt)[row * p.dt_ld + h]) + p.dt_bias[h]);
      sc[0] = step;
      sc[1] = decay_of(-expf(p.A_log[h]) * step);
    }
  }
  for (int i = threadIdx.x; i < 8 * NR; i += 256) {
    sk[i] = i < p.N ? plain(k[i]) : 0.f;
    sq[i] = i < p.N ? plain(q[i]) : 0.f;
  }
  float vv[V];
#pragma unroll
  for (int j = 0; j < V; ++j) vv[j] = colok ? plain(v[col + j]) : 0.f;
  __syncthreads();
  const float step = sc[0], a = sc[1];
  float acc[V];
#pragma unroll
  for (int j = 0; j < V; ++j) {
    vv[j] *= step;
    acc[j] = 0.f;
  }
  if constexpr (ML) {
    float d = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i)
      if (lane + 32 * i < NR) {
        nv[i] = fmaf(a, nv[i], step * sk[warp * NR + lane + 32 * i]);
        d = fmaf(sq[warp * NR + lane + 32 * i], nv[i], d);
      }
    d = warp_sum(d);
    if (lane == 0) nq[warp] = d;
  }
#pragma unroll
  for (int i = 0; i < NR; ++i)
#pragma unroll
    for (int j = 0; j < V; ++j) {
      S[i][j] = fmaf(a, S[i][j], sk[warp * NR + i] * vv[j]);
      acc[j] = fmaf(sq[warp * NR + i], S[i][j], acc[j]);
    }
#pragma unroll
  for (int j = 0; j < V; ++j) part[warp][lane * V + j] = acc[j];
  if (slot >= 0 && colok) {
#pragma unroll
    for (int i = 0; i < NR; ++i) {
      if (warp * NR + i >= p.N) break;
      if constexpr (V == 2) *reinterpret_cast<float2*>(st + (long long)i * p.P) = make_float2(S[i][0], S[i][1]);
      else st[(long long)i * p.P] = S[i][0];
    }
  }
  if constexpr (ML) {
    if (slot >= 0) {
#pragma unroll
      for (int x = 0; x < V; ++x) {
        if ((int)blockIdx.x * V + x >= slices) break;
#pragma unroll
        for (int i = 0; i < NV; ++i) {
          const int r = warp * NR + lane + 32 * i;
          if (lane + 32 * i < NR && r < p.N) vec[x * (p.N + 1) + r] = nv[i];
        }
        if (threadIdx.x == GATES) vec[x * (p.N + 1) + p.N] = m;
      }
    }
  }
  __syncthreads();
  const int c = threadIdx.x;
  if (c < 32 * V && c0 + c < p.P) {
    float o = (p.D ? p.D[h] : 0.f) * plain(v[c0 + c]);
#pragma unroll
    for (int w = 0; w < 8; ++w) o += part[w][c];
    if constexpr (ML) {
      float d = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) d += nq[w];
      o = o * p.q_scale / (fmaxf(fabsf(d * p.q_scale), sc[2]) + 1e-6f);
    }
    reinterpret_cast<T*>(p.out)[row * p.o_ld + (long long)h * p.P + c0 + c] = Cvt<T>::from_f(o);
  }
}

template <typename T, int NR, int V, bool ML>
int launch_step(const ScanParams& p, int nseq, cudaStream_t st) {
  const int blocks = (p.P + 32 * V - 1) / (32 * V), conv_parts = p.conv_state ? (p.conv_C + 2047) / 2048 : 0;
  DLTI_CUDA_CHECK(dlti_launch_pdl(p.nd, scan_step_kernel<T, NR, V, ML>, dim3(blocks + conv_parts, p.heads, nseq), dim3(256), 0, st, p, blocks, conv_parts));
  dlti_count_launch();
  return 0;
}
template <typename T, int NR, bool ML>
int dispatch_step(const ScanParams& p, int nseq, cudaStream_t st) {
  const int V = step_columns(NR, p.P, (long long)p.heads * nseq, p.state);
  if constexpr (NR <= 32) if (V == 2) return launch_step<T, NR, 2, ML>(p, nseq, st);
  return launch_step<T, NR, 1, ML>(p, nseq, st);
}

// Token-by-token form. CTA = (32 columns of P, head, sequence), 8 warps: lane = column, a warp owns the NR consecutive
// rows [warp * NR, ...), so q and k are warp-uniform shared-memory reads. TT tokens are staged at a time; the warps'
// partial outputs are summed once per stage.
constexpr int TT = 8;
template <typename T, int NR, bool ML>
__global__ void __launch_bounds__(256) scan_kernel(const ScanParams p, int slices, int conv_parts) {
  const int s = p.seq0 + blockIdx.z;
  if ((int)blockIdx.x >= slices) {
    if (blockIdx.y == 0) conv_tail<T>(p, s, blockIdx.x - slices, conv_parts);
    return;
  }
  __shared__ float sk[TT][8 * NR], sq[TT][8 * NR], sv[TT][32], part[TT][8][32], sstep[TT], sdecay[TT];
  __shared__ float nq[TT][8], floor_s[TT];                 // mLSTM: the warps' parts of n . q; exp(-m)
  long long row0;
  int n, start;
  seq_rows(p, s, row0, n, start);
  const int h = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int col = blockIdx.x * 32 + lane, grp = h / p.rep;
  const int slot = p.sslot[s];
  const bool colok = col < p.P;
  float* st = p.state + (((long long)(slot < 0 ? 0 : slot) * p.heads + h) * p.N) * p.P + col;
  float S[NR];
#pragma unroll
  for (int i = 0; i < NR; ++i) {
    const int r = warp * NR + i;
    S[i] = (slot >= 0 && start > 0 && colok && r < p.N) ? st[(long long)r * p.P] : 0.f;
  }
  const float Dh = p.D ? p.D[h] : 0.f;
  const float cdec = p.decay ? p.decay[h] : 0.f;
  constexpr int NV = (NR + 31) / 32;                       // entries of n per lane
  float nv[NV], m = 0.f;
  float* vec = ML ? p.vec + (((long long)(slot < 0 ? 0 : slot) * p.heads + h) * slices + blockIdx.x) * (p.N + 1) : nullptr;
  if constexpr (ML) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int r = warp * NR + lane + 32 * i;
      nv[i] = (slot >= 0 && start > 0 && lane + 32 * i < NR && r < p.N) ? vec[r] : 0.f;
    }
    if (slot >= 0 && start > 0) m = vec[p.N];
  }
  const T* q = reinterpret_cast<const T*>(p.q) + (long long)grp * p.N;
  const T* k = reinterpret_cast<const T*>(p.k) + (long long)grp * p.N;
  const T* v = reinterpret_cast<const T*>(p.v) + (long long)h * p.P;
  for (int t0 = 0; t0 < n; t0 += TT) {
    const int nt = min(TT, n - t0);
    __syncthreads();
    for (int i = threadIdx.x; i < nt * 8 * NR; i += 256) {
      const int t = i / (8 * NR), r = i - t * (8 * NR);
      const long long row = row0 + t0 + t;
      float kv = 0.f, qv = 0.f;
      if (r < p.N) {
        kv = Cvt<T>::to_f(k[row * p.k_ld + r]);
        qv = Cvt<T>::to_f(q[row * p.q_ld + r]);
        if (p.silu) { kv = Cvt<T>::to_f(Cvt<T>::from_f(silu_f(kv))); qv = Cvt<T>::to_f(Cvt<T>::from_f(silu_f(qv))); }
      }
      sk[t][r] = kv;
      sq[t][r] = qv;
    }
    if (warp < nt) {
      const long long row = row0 + t0 + warp;
      float x = colok ? Cvt<T>::to_f(v[row * p.v_ld + col]) : 0.f;
      if (p.silu) x = Cvt<T>::to_f(Cvt<T>::from_f(silu_f(x)));
      sv[warp][lane] = x;
      if (ML) {
        if (lane < 2) {
          const float z = p.gates[row * p.g_ld + lane * p.heads + h] + p.gate_b[lane * p.heads + h];
          if (lane == 0) sstep[warp] = log_in_gate(z, p.cap);
          else sdecay[warp] = log_forget_gate(z, p.cap);
        }
      } else if (lane == 0) {
        if (p.decay) {
          sstep[warp] = 1.f;
          sdecay[warp] = cdec;
        } else {
          const float step = softplus_f(Cvt<T>::to_f(reinterpret_cast<const T*>(p.dt)[row * p.dt_ld + h]) + p.dt_bias[h]);
          sstep[warp] = step;
          sdecay[warp] = decay_of(-expf(p.A_log[h]) * step);
        }
      }
    }
    __syncthreads();
    if constexpr (ML) {
      if (threadIdx.x == 0)                                // log gates -> factors, one token after the other
        for (int t = 0; t < nt; ++t) {
          const float f = sdecay[t] + m, i = sstep[t];
          m = fmaxf(f, i);
          sdecay[t] = decay_of(f - m);
          sstep[t] = expf(i - m);
          floor_s[t] = expf(-m);
        }
      __syncthreads();
    }
    for (int t = 0; t < nt; ++t) {
      const float a = sdecay[t];
      const float vv = sv[t][lane] * sstep[t];
      float acc = 0.f;
      if constexpr (ML) {
        float d = 0.f;
#pragma unroll
        for (int i = 0; i < NV; ++i)
          if (lane + 32 * i < NR) {
            nv[i] = fmaf(a, nv[i], sstep[t] * sk[t][warp * NR + lane + 32 * i]);
            d = fmaf(sq[t][warp * NR + lane + 32 * i], nv[i], d);
          }
        d = warp_sum(d);
        if (lane == 0) nq[t][warp] = d;
      }
#pragma unroll
      for (int i = 0; i < NR; ++i) {
        S[i] = fmaf(a, S[i], sk[t][warp * NR + i] * vv);
        acc = fmaf(sq[t][warp * NR + i], S[i], acc);
      }
      part[t][warp][lane] = acc;
    }
    __syncthreads();
    if (warp < nt && colok) {
      float o = Dh * sv[warp][lane];
#pragma unroll
      for (int w = 0; w < 8; ++w) o += part[warp][w][lane];
      if constexpr (ML) {
        float d = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) d += nq[warp][w];
        o = o * p.q_scale / (fmaxf(fabsf(d * p.q_scale), floor_s[warp]) + 1e-6f);
      }
      reinterpret_cast<T*>(p.out)[(row0 + t0 + warp) * p.o_ld + (long long)h * p.P + col] = Cvt<T>::from_f(o);
    }
  }
  if (slot >= 0 && colok) {
#pragma unroll
    for (int i = 0; i < NR; ++i) {
      const int r = warp * NR + i;
      if (r < p.N) st[(long long)r * p.P] = S[i];
    }
  }
  if constexpr (ML) {
    if (slot >= 0) {
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const int r = warp * NR + lane + 32 * i;
        if (lane + 32 * i < NR && r < p.N) vec[r] = nv[i];
      }
      if (threadIdx.x == 0) vec[p.N] = m;
    }
  }
}

template <typename T, bool ML>
int launch_scan(const ScanParams& p, int nseq, cudaStream_t st) {
  const int slices = (p.P + 31) / 32;
  const int conv_parts = p.conv_state ? (p.conv_C + 2047) / 2048 : 0;
  const dim3 grid(slices + conv_parts, p.heads, nseq);
  const bool single = p.seq0 + nseq <= p.nd;   // decode rows
#define SCAN_CASE(NR)                                                                      \
  if (p.N <= 8 * NR) {                                                                     \
    if (single) return dispatch_step<T, NR, ML>(p, nseq, st);                              \
    scan_kernel<T, NR, ML><<<grid, 256, 0, st>>>(p, slices, conv_parts);                   \
    dlti_count_launch();                                                                   \
    return (int)cudaGetLastError();                                                        \
  }
  SCAN_CASE(4) SCAN_CASE(8) SCAN_CASE(16) SCAN_CASE(32) SCAN_CASE(64)
#undef SCAN_CASE
  dlti_set_error("linear_scan: states of up to 512 rows");
  return DLTI_ERR_TOO_LARGE;
}

// Chunked form for prompts, bf16: CTA = (32 columns of P, head, sequence), 64 tokens a chunk. With L_t the running sum of
// log2 a within the chunk and d_s = step size,
//     o_t   = 2^(L_t) S^T q_t + sum_(s <= t) [2^(L_t - L_s) d_s (k_s . q_t)] v_s
//     S'    = 2^(L_63) S + sum_s k_s [2^(L_63 - L_s) d_s v_s]^T
// q, k, v are exact bf16 operands; the three fp32 operands (S, the bracketed weights, the bracketed values) enter the
// tensor-core products as hi + lo bf16 pairs, so the recurrence keeps 16+ mantissa bits everywhere.
// Warps 0-3 compute the outputs (16 tokens each) from the S operand in shared memory; warps 4-7 meanwhile advance S, which
// lives in their fp32 accumulators (NT / 4 rows each), and publish it as the next operand once warps 0-3 have read the old
// one. Warp 4 also prepares the next chunk's decay vectors. One CTA-wide barrier per chunk.
//
// mLSTM: with F_t the running sum of log2 forget gates, a_s = log2 i_s - F_s and A_t = max(m, a_0 ... a_t) (m: the running
// maximum before the chunk, in log2) the maximum after token t is F_t + A_t, so the weight of s in t is 2^(a_s - A_t), that
// of the old state 2^(m - A_t): the same products with -A in the place of L and 2^a in that of the step sizes. n is one more
// column of the state product (its operand: the scaling factors themselves, hi in column 0 and lo in column 1), and
// n . q the row sums of the bracketed weights plus one more column of S^T q.
//
// One sequence gives only heads * P / 32 CTAs, each a chain of n / 64 chunks. Where that leaves SMs without work, the sequence is
// cut into segments of whole chunks: a first launch (SEG_STATE) runs the state half alone, one chain over every segment but the
// last, and leaves the state before each segment in a SegEntry; the second (SEG_FULL) runs all segments side by side from
// there. The chain has the products and sums of the form without segments, in their order, so the results are the same bit by bit.
// (Segments that each start from zero and are folded with their decays shorten the chain, but round in another order.) The state half is
// under half of the work of a chunk, and the chain has its eight warps to itself: half of the columns each, a ninth prepares the vectors.
// One prompt of 8192 tokens, 16 heads of 128 x 128 (64 CTAs, 4 segments): 324 -> 228 us in both launches together; a chunk costs the
// chain 1.0 us, the whole form 2.5.
constexpr int WHOLE = 0, SEG_STATE = 1, SEG_FULL = 2;
constexpr int CQ = 64, CP = 32, CPP = CP + 8;
template <int NT, int MODE>
struct ChunkSmem {                                               // a stage holds q (not in the chain of SEG_STATE), k and v of a chunk
  static constexpr int NP = NT + 8, STAGES = MODE == SEG_STATE ? 4 : 2;
  static constexpr int QK = CQ * NP * 2, V = CQ * CPP * 2, K_AT = MODE == SEG_STATE ? 0 : QK, V_AT = K_AT + QK, STAGE = V_AT + V;          // bytes
  static constexpr int W = STAGES * STAGE, S = W + 2 * V, VEC = S + (MODE == SEG_STATE ? 0 : 2 * NT * CPP * 2), VECS = 6 * CQ, NB = VEC + 2 * VECS * 4;
  static constexpr int BYTES = NB, BYTES_ML = NB + 2 * NT * 2;     // mLSTM: n as hi, lo
};
struct ChunkVec {                                                // one chunk's vectors, 64 each
  float *L, *step, *E, *F;                                       // L; d; 2^(L_63 - L_s) d; 2^(L_e - L_s) d, e = end of s's 16-block
  float *floor, *m;                                              // mLSTM: exp(-m_t); m before the chunk. L = -A, step = a
};
// The state after a segment as the registers hold it, fp32: S [NT][32], n [NT][2] (its hi and lo column), m in log2. The entry of a
// sequence's last segment holds the state that the sequence brought: nothing may read p.state in the second launch, which renews it.
template <int NT>
struct SegEntry { static constexpr int N = NT * CP, M = N + 2 * NT, FLOATS = M + 4; };
constexpr int chunk_threads(int mode) { return mode == SEG_STATE ? 288 : 256; }
template <int NT, bool ML, int MODE>
__global__ void __launch_bounds__(chunk_threads(MODE), NT <= 128 ? 2 : 1) scan_chunk_kernel(const ScanParams p, int slices, int conv_parts) {
  using L = ChunkSmem<NT, MODE>;
  using bf16 = __nv_bfloat16;
  const int sq = MODE == SEG_FULL ? blockIdx.z / p.segs : blockIdx.z, seg = MODE == SEG_FULL ? blockIdx.z - sq * p.segs : 0, s = p.seq0 + sq;
  const int h = blockIdx.y, slice = blockIdx.x;
  if (h >= p.heads) {                                            // behind all others: see launch_chunk_mode
    const int part = (h - p.heads) * slices + slice;
    if (seg == 0 && part < conv_parts) conv_tail<bf16>(p, s, part, conv_parts);
    return;
  }
  extern __shared__ __align__(128) uint8_t smem[];
  const uint32_t sb = smem_u32(smem);
  long long row0;
  int n, start;
  seq_rows(p, s, row0, n, start);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c0 = slice * CP, ncol = min(CP, p.P - c0), grp = h / p.rep;
  const int slot = p.sslot[s];
  const int last_seg = MODE == WHOLE ? 0 : min((n - 1) / p.seg_len, p.segs - 1);       // the tokens [tb, te) are this CTA's
  if (MODE != WHOLE && (n <= 0 || seg > last_seg || (MODE == SEG_STATE && last_seg == 0))) return;
  const int tb = MODE == SEG_FULL ? seg * p.seg_len : 0;
  const int te = MODE == SEG_STATE ? last_seg * p.seg_len : (seg == last_seg ? n : tb + p.seg_len);
  auto entry = [&](int i) { return p.seg_ws + ((((long long)sq * p.segs + i) * p.heads + h) * slices + slice) * SegEntry<NT>::FLOATS; };
  const bf16* q = reinterpret_cast<const bf16*>(p.q) + row0 * p.q_ld + (long long)grp * p.N;
  const bf16* k = reinterpret_cast<const bf16*>(p.k) + row0 * p.k_ld + (long long)grp * p.N;
  const bf16* v = reinterpret_cast<const bf16*>(p.v) + row0 * p.v_ld + (long long)h * p.P + c0;
  const float Dh = p.D ? p.D[h] : 0.f;
  auto vec = [&](int i) {
    float* f = reinterpret_cast<float*>(smem + L::VEC) + (i & 1) * L::VECS;
    return ChunkVec{f, f + CQ, f + 2 * CQ, f + 3 * CQ, f + 4 * CQ, f + 5 * CQ};
  };
  auto load = [&](int stage, int t0) {
    if (MODE == SEG_STATE && warp == 8) return;
    constexpr int STEP = 256 / (NT / 8);                         // rows per pass
    const uint32_t base = sb + stage * L::STAGE;
    const int r0 = threadIdx.x / (NT / 8), c = threadIdx.x % (NT / 8);
    const bool cok = c * 8 < p.N;
    const bf16* qp = q + (t0 + r0) * p.q_ld + c * 8;             // never dereferenced where a row or column is out of range
    const bf16* kp = k + (t0 + r0) * p.k_ld + c * 8;
    const uint32_t dst = base + (r0 * L::NP + c * 8) * 2;
#pragma unroll
    for (int i = 0; i < CQ / STEP; ++i) {
      const bool ok = cok && t0 + r0 + i * STEP < n;
      if (MODE != SEG_STATE) cp_async16(dst + i * STEP * L::NP * 2, ok ? qp : q, ok);
      cp_async16(dst + i * STEP * L::NP * 2 + L::K_AT, ok ? kp : k, ok);
      qp += STEP * p.q_ld;
      kp += STEP * p.k_ld;
    }
    const int r = threadIdx.x / (CP / 8), cv = threadIdx.x % (CP / 8);     // 64 rows x 4 pieces
    const bool ok = t0 + r < n && cv * 8 < ncol;
    cp_async16(base + L::V_AT + (r * CPP + cv * 8) * 2, ok ? v + (t0 + r) * p.v_ld + cv * 8 : v, ok);
    cp_async_commit();
  };
  // in a ring of more than two every chunk commits one group, also where nothing is left to load
  auto load_ahead = [&](int it, int t0) {
    if (t0 + (L::STAGES - 1) * CQ < te) load((it + L::STAGES - 1) & (L::STAGES - 1), t0 + (L::STAGES - 1) * CQ);
    else if (L::STAGES > 2) cp_async_commit();
  };
#pragma unroll
  for (int i = 0; i < L::STAGES - 1; ++i) load_ahead(i - (L::STAGES - 1), tb + (i - (L::STAGES - 1)) * CQ);

  const bool have = slot >= 0 && start > 0;
  constexpr float LOG2E = 1.4426950408889634f;
  const float eA = ML || p.decay ? 0.f : expf(p.A_log[h]) * LOG2E;
  const float la_c = !ML && p.decay ? fmaxf(logf(p.decay[h]), -80.f) * LOG2E : 0.f;
  const float bias = ML ? p.gate_b[h] : (p.decay ? 0.f : p.dt_bias[h]);
  const float bias_f = ML ? p.gate_b[p.heads + h] : 0.f;
  float* vecs = ML ? p.vec + (((long long)(slot < 0 ? 0 : slot) * p.heads + h) * slices + slice) * (p.N + 1) : nullptr;
  float m = 0.f;                                                 // warp PREP, mLSTM: log2 of the running maximum
  // warp PREP: step sizes and decays of the chunk at t0, two consecutive tokens a lane
  auto raw_dt = [&](int t0, float (&d)[4]) {                     // mLSTM: input gates, then forget gates
#pragma unroll
    for (int y = 0; y < 2; ++y) {
      const int t = t0 + 2 * lane + y;
      if constexpr (ML) {
        d[y] = t < n ? p.gates[(row0 + t) * p.g_ld + h] + bias : 0.f;
        d[2 + y] = t < n ? p.gates[(row0 + t) * p.g_ld + p.heads + h] + bias_f : 0.f;
      } else
      d[y] = (!p.decay && t < n) ? __bfloat162float(reinterpret_cast<const bf16*>(p.dt)[(row0 + t) * p.dt_ld + h]) + bias : 0.f;
    }
  };
  auto prepare_ml = [&](int i, int t0, const float (&d)[4]) {
    float f[2], a[2];
#pragma unroll
    for (int y = 0; y < 2; ++y) f[y] = t0 + 2 * lane + y < n ? log_forget_gate(d[2 + y], p.cap) * LOG2E : 0.f;
    f[1] += f[0];
    float x = f[1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    const float F1 = x, F0 = x - f[1] + f[0];
#pragma unroll
    for (int y = 0; y < 2; ++y) a[y] = t0 + 2 * lane + y < n ? log_in_gate(d[y], p.cap) * LOG2E - (y ? F1 : F0) : -INFINITY;
    x = fmaxf(a[0], a[1]);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x = fmaxf(x, y);
    }
    float before = __shfl_up_sync(0xffffffffu, x, 1);
    before = lane == 0 ? m : fmaxf(m, before);
    const float A0 = fmaxf(before, a[0]), A1 = fmaxf(A0, a[1]);
    const float last = __shfl_sync(0xffffffffu, A1, 31), Ae = __shfl_sync(0xffffffffu, A1, lane | 7);
    const ChunkVec cv = vec(i);
    *reinterpret_cast<float2*>(cv.L + 2 * lane) = make_float2(-A0, -A1);
    *reinterpret_cast<float2*>(cv.step + 2 * lane) = make_float2(a[0], a[1]);
    *reinterpret_cast<float2*>(cv.E + 2 * lane) = make_float2(ex2(a[0] - last), ex2(a[1] - last));
    *reinterpret_cast<float2*>(cv.F + 2 * lane) = make_float2(ex2(a[0] - Ae), ex2(a[1] - Ae));
    *reinterpret_cast<float2*>(cv.floor + 2 * lane) = make_float2(ex2(-(F0 + A0)), ex2(-(F1 + A1)));
    if (lane == 0) *cv.m = m;
    m = __shfl_sync(0xffffffffu, F1, 31) + last;
  };
  auto prepare = [&](int i, int t0, const float (&d)[4]) {
    float step[2], l[2];
#pragma unroll
    for (int y = 0; y < 2; ++y) {
      const bool ok = t0 + 2 * lane + y < n;
      step[y] = !ok ? 0.f : (p.decay ? 1.f : softplus_f(d[y]));
      l[y] = !ok ? 0.f : (p.decay ? la_c : -eA * step[y]);
    }
    l[1] += l[0];
    float x = l[1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    const float before = x - l[1];
    const float total = __shfl_sync(0xffffffffu, x, 31);
    const float le = __shfl_sync(0xffffffffu, x, lane | 7);      // end of this 16-token block
    const float l0 = before + l[0], l1 = x;
    const ChunkVec cv = vec(i);
    *reinterpret_cast<float2*>(cv.L + 2 * lane) = make_float2(l0, l1);
    *reinterpret_cast<float2*>(cv.step + 2 * lane) = make_float2(step[0], step[1]);
    *reinterpret_cast<float2*>(cv.E + 2 * lane) = make_float2(ex2(total - l0) * step[0], ex2(total - l1) * step[1]);
    *reinterpret_cast<float2*>(cv.F + 2 * lane) = make_float2(ex2(le - l0) * step[0], ex2(le - l1) * step[1]);
  };
  float d[4] = {0.f, 0.f, 0.f, 0.f};
  // the warp that prepares the vectors: see above; the gates of an mLSTM are more than the slack of warp 0
  constexpr int PREP = MODE == SEG_STATE ? 8 : (ML ? 4 : 0);
  if (warp == PREP) {
    if constexpr (ML) {
      if (MODE == SEG_FULL && last_seg > 0) m = entry(seg > 0 ? seg - 1 : last_seg)[SegEntry<NT>::M];
      else if (have) m = vecs[p.N] * LOG2E;
      if (MODE == SEG_STATE && lane == 0) entry(last_seg)[SegEntry<NT>::M] = m;
    }
    raw_dt(tb, d);
    if constexpr (ML) prepare_ml(0, tb, d);
    else prepare(0, tb, d);
    raw_dt(tb + CQ, d);
  }
  auto prepare_next = [&](int it, int t0) {                      // the vectors of the chunk after the one at t0
    if (warp != PREP || t0 + CQ >= te) return;
    if constexpr (ML) prepare_ml(it + 1, t0 + CQ, d);
    else prepare(it + 1, t0 + CQ, d);
    raw_dt(t0 + 2 * CQ, d);
  };

  if (MODE == SEG_STATE && warp == PREP) {
    int it = 0, ends = p.seg_len, i = 0;                         // end and number of the segment
    for (int t0 = tb; t0 < te; t0 += CQ, ++it) {
      __syncthreads();
      if (t0 + CQ == ends) {
        if (ML && lane == 0) entry(i)[SegEntry<NT>::M] = m;
        ends += p.seg_len;
        ++i;
      }
      prepare_next(it, t0);
    }
    return;
  }
  if (MODE != SEG_STATE && warp < 4) {
    // ---- outputs of 16 tokens per chunk ----
    const int scol = (lane & 3) * 2, tr = warp * 16 + (lane >> 2);
    int it = 0;
    for (int t0 = tb; t0 < te; t0 += CQ, ++it) {
      cp_async_wait<L::STAGES - 2>();
      __syncthreads();                                           // tile, vectors and S operand of this chunk are there
      load_ahead(it, t0);
      const uint32_t base = sb + (it & 1) * L::STAGE;
      const ChunkVec cv = vec(it);
      uint32_t qf[NT / 16][4];
      {
        const uint32_t qa = base + ((warp * 16 + (lane & 15)) * L::NP + (lane >> 4) * 8) * 2;
#pragma unroll
        for (int kk = 0; kk < NT / 16; ++kk) ldsm4(qf[kk], qa + kk * 32);
      }
      float o[CP / 8][4];
#pragma unroll
      for (int j = 0; j < CP / 8; ++j)
#pragma unroll
        for (int x = 0; x < 4; ++x) o[j][x] = 0.f;
      {
        const uint32_t sa = sb + L::S + ((lane & 15) * CPP + (lane >> 4) * 8) * 2;
#pragma unroll
        for (int kk = 0; kk < NT / 16; ++kk)
#pragma unroll
          for (int x = 0; x < 2; ++x)                            // hi, lo
#pragma unroll
            for (int j = 0; j < CP / 16; ++j) {
              uint32_t b[4];
              ldsm4_t(b, sa + x * (NT * CPP * 2) + (kk * 16 * CPP + j * 16) * 2);
              mma_bf16(o[2 * j], qf[kk], b[0], b[1]);
              mma_bf16(o[2 * j + 1], qf[kk], b[2], b[3]);
            }
      }
      float nq[4] = {};                                          // mLSTM: columns 0 and 1 (lanes 4 r): n . q, hi and lo part of n
      if constexpr (ML) {
        const uint8_t* nb = smem + L::NB + ((lane >> 2) & 1) * (NT * 2) + scol * 2;
#pragma unroll
        for (int kk = 0; kk < NT / 16; ++kk) {
          uint32_t b0 = *reinterpret_cast<const uint32_t*>(nb + kk * 32), b1 = *reinterpret_cast<const uint32_t*>(nb + kk * 32 + 16);
          if (lane >= 8) b0 = b1 = 0;
          mma_bf16(nq, qf[kk], b0, b1);
        }
      }
      asm volatile("bar.arrive 2, 256;" ::: "memory");           // the old S operand has been read
      const float lt[2] = {cv.L[tr], cv.L[tr + 8]};
      const float m0 = ML ? *cv.m : 0.f;
      const float el[2] = {ex2(lt[0] + m0), ex2(lt[1] + m0)};
      float rs[2] = {0.f, 0.f};                                  // mLSTM: row sums of the weights
#pragma unroll
      for (int j = 0; j < CP / 8; ++j)
#pragma unroll
        for (int x = 0; x < 4; ++x) o[j][x] *= el[x >> 1];
      for (int kb = 0; kb <= warp; ++kb) {                       // 16 keys at a time up to the diagonal
        float g0[4] = {}, g1[4] = {};
        const uint32_t ka = base + L::QK + ((kb * 16 + (lane & 7) + ((lane >> 4) << 3)) * L::NP + ((lane >> 3) & 1) * 8) * 2;
#pragma unroll
        for (int kk = 0; kk < NT / 16; ++kk) {
          uint32_t b[4];
          ldsm4(b, ka + kk * 32);
          mma_bf16(g0, qf[kk], b[0], b[1]);
          mma_bf16(g1, qf[kk], b[2], b[3]);
        }
        if (kb < warp) {                                         // all keys precede all tokens: factored through the block's end
          const float le = cv.L[kb * 16 + 15];
          const float f0 = ex2(lt[0] - le), f1 = ex2(lt[1] - le);
          const float2 a = *reinterpret_cast<const float2*>(cv.F + kb * 16 + scol), b = *reinterpret_cast<const float2*>(cv.F + kb * 16 + 8 + scol);
          g0[0] *= a.x * f0; g0[1] *= a.y * f0; g0[2] *= a.x * f1; g0[3] *= a.y * f1;
          g1[0] *= b.x * f0; g1[1] *= b.y * f0; g1[2] *= b.x * f1; g1[3] *= b.y * f1;
        } else {
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            const int t = tr + 8 * (x >> 1);
            const int u0 = kb * 16 + scol + (x & 1), u1 = u0 + 8;
            if constexpr (ML) {
              g0[x] = u0 <= t ? g0[x] * ex2(lt[x >> 1] + cv.step[u0]) : 0.f;
              g1[x] = u1 <= t ? g1[x] * ex2(lt[x >> 1] + cv.step[u1]) : 0.f;
            } else {
              g0[x] = u0 <= t ? g0[x] * cv.step[u0] * ex2(lt[x >> 1] - cv.L[u0]) : 0.f;
              g1[x] = u1 <= t ? g1[x] * cv.step[u1] * ex2(lt[x >> 1] - cv.L[u1]) : 0.f;
            }
          }
        }
        if constexpr (ML) {
#pragma unroll
          for (int x = 0; x < 4; ++x) rs[x >> 1] += g0[x] + g1[x];
        }
        uint32_t hi[4], lo[4];
        split_pair(g0[0], g0[1], hi[0], lo[0]);
        split_pair(g0[2], g0[3], hi[1], lo[1]);
        split_pair(g1[0], g1[1], hi[2], lo[2]);
        split_pair(g1[2], g1[3], hi[3], lo[3]);
        const uint32_t va = base + 2 * L::QK + ((kb * 16 + (lane & 15)) * CPP + (lane >> 4) * 8) * 2;
#pragma unroll
        for (int j = 0; j < CP / 16; ++j) {
          uint32_t b[4];
          ldsm4_t(b, va + j * 32);
          mma_bf16(o[2 * j], hi, b[0], b[1]);
          mma_bf16(o[2 * j + 1], hi, b[2], b[3]);
          mma_bf16(o[2 * j], lo, b[0], b[1]);
          mma_bf16(o[2 * j + 1], lo, b[2], b[3]);
        }
      }
      const bf16* sv = reinterpret_cast<const bf16*>(smem + (it & (L::STAGES - 1)) * L::STAGE + L::V_AT);
#pragma unroll
      for (int y = 0; y < 2; ++y) {
        const int t = tr + 8 * y;
        float f = 1.f;
        if constexpr (ML) {
          rs[y] += __shfl_xor_sync(0xffffffffu, rs[y], 1);
          rs[y] += __shfl_xor_sync(0xffffffffu, rs[y], 2);
          const float old = __shfl_sync(0xffffffffu, nq[2 * y] + nq[2 * y + 1], lane & ~3);
          f = p.q_scale / (fmaxf(fabsf(p.q_scale * (el[y] * old + rs[y])), cv.floor[t]) + 1e-6f);
        }
        if (t0 + t < n) {
          bf16* orow = reinterpret_cast<bf16*>(p.out) + (row0 + t0 + t) * p.o_ld + (long long)h * p.P + c0;
#pragma unroll
          for (int j = 0; j < CP / 8; ++j) {
            const int c = j * 8 + scol;
            if (c >= ncol) continue;
            const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(sv + t * CPP + c));
            if constexpr (ML) *reinterpret_cast<__nv_bfloat162*>(orow + c) = __floats2bfloat162_rn(o[j][2 * y] * f, o[j][2 * y + 1] * f);
            else *reinterpret_cast<__nv_bfloat162*>(orow + c) = __floats2bfloat162_rn(o[j][2 * y] + Dh * x.x, o[j][2 * y + 1] + Dh * x.y);
          }
        }
      }
      prepare_next(it, t0);
    }
    return;
  }

  // ---- state ----
  // NT / 4 rows a warp, in the chain of SEG_STATE half of the columns
  constexpr int STATE_THREADS = MODE == SEG_STATE ? 256 : 128, JN = MODE == SEG_STATE ? 1 : 2;     // JN: groups of 16 columns
  const int sw = MODE == SEG_STATE ? warp & 3 : warp - 4, jc = MODE == SEG_STATE ? (warp >> 2) * 16 : 0;
  constexpr int MT = NT / 64;                                    // 16-row state tiles of a warp
  float S[MT][2 * JN][4];
  float* st = p.state + (((long long)(slot < 0 ? 0 : slot) * p.heads + h) * p.N) * p.P + c0;
  const int srow = sw * (NT / 4) + (lane >> 2), scol = (lane & 3) * 2, col0 = jc + scol;
  float ns[ML ? MT : 1][4];                                      // mLSTM: columns 0 (from hi) and 1 (from lo) in lanes 4 r; n is their sum
  auto publish = [&]() {                                         // S as hi / lo operands
    if constexpr (ML) {
      if ((lane & 3) == 0)
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
          for (int y = 0; y < 2; ++y) {
            const float x = ns[i][2 * y] + ns[i][2 * y + 1];
            const bf16 hi = __float2bfloat16(x);
            bf16* nb = reinterpret_cast<bf16*>(smem + L::NB) + srow + i * 16 + 8 * y;
            nb[0] = hi;
            nb[NT] = __float2bfloat16(x - __bfloat162float(hi));
          }
    }
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int j = 0; j < 2 * JN; ++j)
#pragma unroll
        for (int y = 0; y < 2; ++y) {
          uint32_t hi, lo;
          split_pair(S[i][j][2 * y], S[i][j][2 * y + 1], hi, lo);
          const int off = ((srow + i * 16 + 8 * y) * CPP + j * 8 + col0) * 2;
          *reinterpret_cast<uint32_t*>(smem + L::S + off) = hi;
          *reinterpret_cast<uint32_t*>(smem + L::S + NT * CPP * 2 + off) = lo;
        }
  };
  // the state before the segment: carried, or the entry of the segment before it
  auto each = [&](auto f) {
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int j = 0; j < 2 * JN; ++j)
#pragma unroll
        for (int x = 0; x < 4; ++x) f(S[i][j][x], srow + i * 16 + 8 * (x >> 1), j * 8 + col0 + (x & 1));
  };
  auto each_n = [&](auto f) {
    if constexpr (ML)
#pragma unroll
      for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int y = 0; y < 2; ++y) f(ns[i][2 * y], ns[i][2 * y + 1], srow + i * 16 + 8 * y);
  };
  auto save = [&](int i) {
    float* e = entry(i);
    each([&](float& x, int r, int c) { e[r * CP + c] = x; });
    each_n([&](float& a, float& b, int r) {
      if ((lane & 3) == 0 && jc == 0) *reinterpret_cast<float2*>(e + SegEntry<NT>::N + 2 * r) = make_float2(a, b);
    });
  };
  if (MODE == SEG_FULL && last_seg > 0) {
    const float* e = entry(seg > 0 ? seg - 1 : last_seg);
    each([&](float& x, int r, int c) { x = e[r * CP + c]; });
    each_n([&](float& a, float& b, int r) {
      const float2 u = (lane & 3) == 0 ? *reinterpret_cast<const float2*>(e + SegEntry<NT>::N + 2 * r) : make_float2(0.f, 0.f);
      a = u.x;
      b = u.y;
    });
  } else {
    each([&](float& x, int r, int c) { x = have && r < p.N && c < ncol ? st[(long long)r * p.P + c] : 0.f; });
    each_n([&](float& a, float& b, int r) { a = have && (lane & 3) == 0 && r < p.N ? vecs[r] : 0.f; b = 0.f; });
    if (MODE == SEG_STATE) save(last_seg);
  }
  if (MODE != SEG_STATE) publish();
  int it = 0, ends = p.seg_len, seg_i = 0;                       // SEG_STATE: end and number of the segment
  for (int t0 = tb; t0 < te; t0 += CQ, ++it) {
    cp_async_wait<L::STAGES - 2>();
    __syncthreads();
    load_ahead(it, t0);
    const uint32_t base = sb + (it & (L::STAGES - 1)) * L::STAGE;
    const ChunkVec cv = vec(it);
    const bf16* sv = reinterpret_cast<const bf16*>(smem + (it & (L::STAGES - 1)) * L::STAGE + L::V_AT);
#pragma unroll
    for (int i = 0; i < CQ * CP / 2 / STATE_THREADS; ++i) {      // scaled values as hi / lo operands
      const int r = (threadIdx.x & (STATE_THREADS - 1)) / (CP / 2) + i * (STATE_THREADS / (CP / 2)), c = 2 * (threadIdx.x % (CP / 2));
      const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(sv + r * CPP + c));
      const float e = cv.E[r];
      uint32_t hi, lo;
      split_pair(x.x * e, x.y * e, hi, lo);
      *reinterpret_cast<uint32_t*>(smem + L::W + (r * CPP + c) * 2) = hi;
      *reinterpret_cast<uint32_t*>(smem + L::W + L::V + (r * CPP + c) * 2) = lo;
    }
    const float keep = ex2(cv.L[CQ - 1] + (ML ? *cv.m : 0.f));
#pragma unroll
    for (int i = 0; i < MT; ++i) {
#pragma unroll
      for (int j = 0; j < 2 * JN; ++j)
#pragma unroll
        for (int x = 0; x < 4; ++x) S[i][j][x] *= keep;
      if constexpr (ML)
#pragma unroll
        for (int x = 0; x < 4; ++x) ns[i][x] *= keep;
    }
    asm volatile("bar.sync 1, %0;" ::"n"(STATE_THREADS) : "memory");       // scaled values written
#pragma unroll
    for (int kb = 0; kb < CQ / 16; ++kb) {
      uint32_t w[2][JN][4];
      const uint32_t wa = sb + L::W + ((kb * 16 + (lane & 15)) * CPP + jc + (lane >> 4) * 8) * 2;
#pragma unroll
      for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int j = 0; j < JN; ++j) ldsm4_t(w[x][j], wa + x * L::V + j * 32);
      uint32_t e0 = 0, e1 = 0;                                   // mLSTM: factors of keys 16 kb .. as columns 0 (hi) and 1 (lo)
      if constexpr (ML) {
        const float2 u = *reinterpret_cast<const float2*>(cv.E + kb * 16 + scol), v2 = *reinterpret_cast<const float2*>(cv.E + kb * 16 + 8 + scol);
        uint32_t lo0, lo1;
        split_pair(u.x, u.y, e0, lo0);
        split_pair(v2.x, v2.y, e1, lo1);
        if (lane >= 4) { e0 = lane < 8 ? lo0 : 0; e1 = lane < 8 ? lo1 : 0; }
      }
#pragma unroll
      for (int i = 0; i < MT; ++i) {
        // A = K^T: rows n, columns s, read transposed from K [s][n]
        uint32_t a[4];
        ldsm4_t(a, base + L::K_AT + ((kb * 16 + (lane & 7) + ((lane >> 4) << 3)) * L::NP + sw * (NT / 4) + i * 16 + ((lane >> 3) & 1) * 8) * 2);
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
          for (int j = 0; j < JN; ++j) {
            mma_bf16(S[i][2 * j], a, w[x][j][0], w[x][j][1]);
            mma_bf16(S[i][2 * j + 1], a, w[x][j][2], w[x][j][3]);
          }
        if constexpr (ML) mma_bf16(ns[i], a, e0, e1);
      }
    }
    if (MODE == SEG_STATE) {
      if (t0 + CQ == ends) {
        save(seg_i++);
        ends += p.seg_len;
      }
      continue;
    }
    prepare_next(it, t0);
    asm volatile("bar.sync 2, 256;" ::: "memory");               // warps 0-3 have read the old operand
    publish();
  }
  if (MODE != SEG_STATE && slot >= 0 && seg == last_seg) {
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int j = 0; j < 2 * JN; ++j)
#pragma unroll
        for (int y = 0; y < 2; ++y) {
          const int r = srow + i * 16 + 8 * y, c = j * 8 + col0;
          if (r < p.N && c < ncol) {
            st[(long long)r * p.P + c] = S[i][j][2 * y];
            st[(long long)r * p.P + c + 1] = S[i][j][2 * y + 1];
          }
        }
    if constexpr (ML) {
      if ((lane & 3) == 0)
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
          for (int y = 0; y < 2; ++y) {
            const int r = srow + i * 16 + 8 * y;
            if (r < p.N) vecs[r] = ns[i][2 * y] + ns[i][2 * y + 1];
          }
      if (warp == PREP && lane == 0) vecs[p.N] = m * (1.f / LOG2E);
    }
  }
}

// Segments per sequence: as many as fill the SMs with the CTAs that fit one of them side by side (two up to 128 rows of a state, one
// above: shared memory), of at least 8 chunks. Two CTAs of an SM slow each other down, so that more than one per SM has to come with
// three segments or more, or with a long sequence. 8192 tokens in 1 / 2 / 3 / 4 / 8 segments, us, heads of 128 x 128: 32 CTAs 339 / 243 / 208 /
// 189 / 185, 64 CTAs 341 / 247 / 263 / 230 / 253, 96 CTAs 344 / 329 / 267 / 359 / 321, 128 CTAs 343 / 327 / 431 / 364 / 386, with q and k shared by
// all heads 383 / 368; 128 CTAs with 4096 tokens 169 / 171, with 1024 52 / 60. Heads of 256 x 256, 4096 tokens: 64 CTAs 266 / 192 / 251, 96
// CTAs 267 / 325 / 261.
inline int scan_segments(int longest, int nseq, int heads, int N, int P) {
  const long long ctas = (long long)((P + CP - 1) / CP) * heads * nseq, sms = dlti_num_sms();
  const long long room = (N <= 128 ? 2 : 1) * sms / (ctas > 0 ? ctas : 1);
  const int most = longest / (8 * CQ);
  int segs = (int)(room < most ? room : most);
  segs = segs < 16 ? segs : 16;
  return segs > 2 || (segs == 2 && (2 * ctas <= sms || (room == 2 && longest >= 80 * CQ))) ? segs : 1;
}

template <int NT, bool ML, int MODE>
int launch_chunk_mode(const ScanParams& p, int nseq, int conv_parts, cudaStream_t st) {
  static bool done[64] = {};
  const int bytes = ML ? ChunkSmem<NT, MODE>::BYTES_ML : ChunkSmem<NT, MODE>::BYTES;
  int dev = 0;
  DLTI_CUDA_CHECK(cudaGetDevice(&dev));
  if (!done[dev & 63]) {
    DLTI_CUDA_CHECK(cudaFuncSetAttribute(scan_chunk_kernel<NT, ML, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    done[dev & 63] = true;
  }
  const int slices = (p.P + CP - 1) / CP;
  // The few CTAs of the convolution's state come last: as a share of every head they would be CTAs that leave at once, and of the others some SMs
  // get two and some none (8192 tokens, 64 heads of 128 x 64 that share q and k: 508 us whole instead of 383). Head and slice stay indices of
  // the grid: divided from one index they cost 5 to 10 %.
  scan_chunk_kernel<NT, ML, MODE><<<dim3(slices, p.heads + (conv_parts + slices - 1) / slices, nseq * (MODE == SEG_FULL ? p.segs : 1)), chunk_threads(MODE), bytes, st>>>(p, slices, conv_parts);
  dlti_count_launch();
  return (int)cudaGetLastError();
}
template <int NT, bool ML>
int launch_chunk(const ScanParams& p, int nseq, cudaStream_t st) {
  const int conv_parts = p.conv_state ? (p.conv_C + 2047) / 2048 : 0;
  if (p.segs <= 1) return launch_chunk_mode<NT, ML, WHOLE>(p, nseq, conv_parts, st);
  if (int rc = launch_chunk_mode<NT, ML, SEG_STATE>(p, nseq, 0, st)) return rc;
  return launch_chunk_mode<NT, ML, SEG_FULL>(p, nseq, conv_parts, st);
}
inline int segment_floats(int N) { return N <= 64 ? SegEntry<64>::FLOATS : (N <= 128 ? SegEntry<128>::FLOATS : SegEntry<256>::FLOATS); }
// segments of at most `longest` rows a sequence in ws (null: none)
inline void set_segments(ScanParams& p, int longest, int nseq, float* ws) {
  const int segs = ws ? scan_segments(longest, nseq, p.heads, p.N, p.P) : 1;
  if (segs <= 1 || (long long)nseq * segs > 65535) return;
  p.seg_len = ((longest + segs - 1) / segs + CQ - 1) / CQ * CQ;
  p.segs = (longest + p.seg_len - 1) / p.seg_len;
  p.seg_ws = ws;
}

// x = silu(x) in place, rounded to T. A thread takes the same 8 columns of SILU_ROWS rows, with all its loads in flight: 8192 x 6144
// (201 MB read and written) in 47 instead of 58 us.
constexpr int SILU_ROWS = 4;
template <typename T>
__global__ void __launch_bounds__(256) silu_rows_kernel(T* __restrict__ x, long long ld, long long rows, int n) {
  const int c = (blockIdx.y * 256 + threadIdx.x) * 8;
  if (c >= n) return;
  const long long t0 = (long long)blockIdx.x * SILU_ROWS;
  int4 v[SILU_ROWS];
#pragma unroll
  for (int r = 0; r < SILU_ROWS; ++r)
    if (t0 + r < rows) v[r] = *reinterpret_cast<const int4*>(x + (t0 + r) * ld + c);
#pragma unroll
  for (int r = 0; r < SILU_ROWS; ++r) {
    if (t0 + r >= rows) break;
    uint32_t* u = reinterpret_cast<uint32_t*>(&v[r]);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = Cvt<T>::unpack2(u[j]);
      u[j] = Cvt<T>::pack2(f.x / (1.f + __expf(-f.x)), f.y / (1.f + __expf(-f.y)));
    }
    *reinterpret_cast<int4*>(x + (t0 + r) * ld + c) = v[r];
  }
}

}  // namespace

// Sequences [seq0, seq0 + nseq) of the step (the first nd sequences are single rows, sequence nd + i has the rows
// nd + cu[i] ... nd + cu[i + 1]). conv_state: optional tail job, see conv_tail.
DLTI_API int dlti_linear_scan(const void* q, long long q_ld, const void* k, long long k_ld, const void* v, long long v_ld, int rep,
                              int silu, const float* decay, const void* dt, long long dt_ld, const float* dt_bias,
                              const float* A_log, const float* D, float* state, const int* sslot, const int* ctx, const int* cu, int nd,
                              int seq0, int nseq, int heads, int N, int P, void* out, long long o_ld, const void* conv_src,
                              long long conv_ld, int conv_col, int conv_rows, int conv_C, void* conv_state, int dtype,
                              cudaStream_t st) {
  if (nseq <= 0) return 0;
  if (heads < 1 || rep < 1 || N < 1 || P < 1 || nseq > 65535 || (!decay && (!dt || !dt_bias || !A_log))) return DLTI_ERR_BAD_ARG;
  if (conv_rows <= 0) conv_state = nullptr;
  ScanParams p{q, k, v, q_ld, k_ld, v_ld, rep, silu, decay, dt, dt_ld, dt_bias, A_log, D, state, sslot, ctx, cu,
               nd, seq0, heads, N, P, out, o_ld, conv_src, conv_ld, conv_col, conv_rows, conv_C, conv_state};
  if (dtype == DLTI_BF16) return launch_scan<__nv_bfloat16, false>(p, nseq, st);
  if (dtype == DLTI_FP32) return launch_scan<float, false>(p, nseq, st);
  return DLTI_ERR_UNSUPPORTED;
}

// The chunked tensor-core form of the same for prompt sequences: bf16, N and P multiples of 8, N <= 256, q / k / v rows
// 16-byte aligned, no silu (see dlti_silu_rows).
// longest and ws: rows of the longest of these sequences, and dlti_scan_workspace floats for cutting it into segments (null: whole).
DLTI_API int dlti_linear_scan_split(const void* q, long long q_ld, const void* k, long long k_ld, const void* v, long long v_ld, int rep,
                                      const float* decay, const void* dt, long long dt_ld, const float* dt_bias, const float* A_log,
                                      const float* D, float* state, const int* sslot, const int* ctx, const int* cu, int nd, int seq0,
                                      int nseq, int heads, int N, int P, void* out, long long o_ld, const void* conv_src,
                                      long long conv_ld, int conv_col, int conv_rows, int conv_C, void* conv_state, int longest, float* ws,
                                    cudaStream_t st) {
  if (nseq <= 0) return 0;
  if (heads < 1 || rep < 1 || nseq > 65535 || (!decay && (!dt || !dt_bias || !A_log))) return DLTI_ERR_BAD_ARG;
  if (N % 8 || P % 8 || q_ld % 8 || k_ld % 8 || v_ld % 8 || o_ld % 2 ||
      ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v)) & 15)) {
    dlti_set_error("linear_scan_chunked: 16-byte aligned rows, N and P multiples of 8");
    return DLTI_ERR_BAD_ARG;
  }
  if (conv_rows <= 0) conv_state = nullptr;
  ScanParams p{q, k, v, q_ld, k_ld, v_ld, rep, 0, decay, dt, dt_ld, dt_bias, A_log, D, state, sslot, ctx, cu,
               nd, seq0, heads, N, P, out, o_ld, conv_src, conv_ld, conv_col, conv_rows, conv_C, conv_state};
  set_segments(p, longest, nseq, ws);
  if (N <= 64) return launch_chunk<64, false>(p, nseq, st);
  if (N <= 128) return launch_chunk<128, false>(p, nseq, st);
  if (N <= 256) return launch_chunk<256, false>(p, nseq, st);
  dlti_set_error("linear_scan_chunked: states of up to 256 rows");
  return DLTI_ERR_TOO_LARGE;
}

DLTI_API int dlti_linear_scan_chunked(const void* q, long long q_ld, const void* k, long long k_ld, const void* v, long long v_ld, int rep,
                                      const float* decay, const void* dt, long long dt_ld, const float* dt_bias, const float* A_log,
                                      const float* D, float* state, const int* sslot, const int* ctx, const int* cu, int nd, int seq0,
                                      int nseq, int heads, int N, int P, void* out, long long o_ld, const void* conv_src,
                                      long long conv_ld, int conv_col, int conv_rows, int conv_C, void* conv_state, cudaStream_t st) {
  return dlti_linear_scan_split(q, q_ld, k, k_ld, v, v_ld, rep, decay, dt, dt_ld, dt_bias, A_log, D, state, sslot, ctx, cu, nd, seq0, nseq, heads,
                                N, P, out, o_ld, conv_src, conv_ld, conv_col, conv_rows, conv_C, conv_state, 0, nullptr, st);
}

// floats of workspace with which the chunked forms cut sequences of up to `longest` rows into segments (0: they would not)
DLTI_API long long dlti_scan_workspace(int longest, int nseq, int heads, int N, int P) {
  if (nseq < 1 || heads < 1 || P < 1 || N < 1 || N > 256) return 0;
  const int segs = scan_segments(longest, nseq, heads, N, P);
  return segs > 1 ? (long long)nseq * segs * heads * ((P + CP - 1) / CP) * segment_floats(N) : 0;
}

// mLSTM over the sequences [seq0, seq0 + nseq): q, k rows heads * N, v rows heads * P wide; gates / gate_b: see ScanParams; state
// [slots, heads, N, P], vec [slots, heads, ceil(P / 32), N + 1]. chunked: the tensor-core form (bf16, N and P multiples of 8,
// N <= 256, 16-byte aligned rows), else token by token (N <= 512).
// longest, ws: see dlti_linear_scan_split.
DLTI_API int dlti_mlstm_scan_split(const void* q, long long q_ld, const void* k, long long k_ld, const void* v, long long v_ld, const float* gates,
                             long long g_ld, const float* gate_b, float cap, float q_scale, float* state, float* vec, const int* sslot,
                             const int* ctx, const int* cu, int nd, int seq0, int nseq, int heads, int N, int P, void* out, long long o_ld,
                             int chunked, int dtype, int longest, float* ws, cudaStream_t st) {
  if (nseq <= 0) return 0;
  if (heads < 1 || N < 1 || P < 1 || nseq > 65535 || !gates || !gate_b || !(cap > 0.f)) return DLTI_ERR_BAD_ARG;
  ScanParams p{};
  p.q = q; p.k = k; p.v = v; p.q_ld = q_ld; p.k_ld = k_ld; p.v_ld = v_ld; p.rep = 1;
  p.gates = gates; p.g_ld = g_ld; p.gate_b = gate_b; p.cap = cap; p.q_scale = q_scale; p.state = state; p.vec = vec;
  p.sslot = sslot; p.ctx = ctx; p.cu = cu; p.nd = nd; p.seq0 = seq0; p.heads = heads; p.N = N; p.P = P; p.out = out; p.o_ld = o_ld;
  if (!chunked) {
    if (dtype == DLTI_BF16) return launch_scan<__nv_bfloat16, true>(p, nseq, st);
    if (dtype == DLTI_FP32) return launch_scan<float, true>(p, nseq, st);
    return DLTI_ERR_UNSUPPORTED;
  }
  if (dtype != DLTI_BF16 || N % 8 || P % 8 || N > 256 || q_ld % 8 || k_ld % 8 || v_ld % 8 || o_ld % 2 ||
      ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v)) & 15)) {
    dlti_set_error("mlstm_scan, chunked: bf16, 16-byte aligned rows, N and P multiples of 8, N <= 256");
    return DLTI_ERR_BAD_ARG;
  }
  set_segments(p, longest, nseq, ws);
  if (N <= 64) return launch_chunk<64, true>(p, nseq, st);
  if (N <= 128) return launch_chunk<128, true>(p, nseq, st);
  return launch_chunk<256, true>(p, nseq, st);
}

DLTI_API int dlti_mlstm_scan(const void* q, long long q_ld, const void* k, long long k_ld, const void* v, long long v_ld, const float* gates,
                             long long g_ld, const float* gate_b, float cap, float q_scale, float* state, float* vec, const int* sslot,
                             const int* ctx, const int* cu, int nd, int seq0, int nseq, int heads, int N, int P, void* out, long long o_ld,
                             int chunked, int dtype, cudaStream_t st) {
  return dlti_mlstm_scan_split(q, q_ld, k, k_ld, v, v_ld, gates, g_ld, gate_b, cap, q_scale, state, vec, sslot, ctx, cu, nd, seq0, nseq, heads,
                               N, P, out, o_ld, chunked, dtype, 0, nullptr, st);
}

DLTI_API int dlti_silu_rows(void* x, long long ld, long long rows, int n, int dtype, cudaStream_t st) {
  if (rows <= 0 || n <= 0) return 0;
  if (dtype != DLTI_BF16) return DLTI_ERR_UNSUPPORTED;
  if (n % 8 || ld % 8 || (reinterpret_cast<uintptr_t>(x) & 15)) return DLTI_ERR_BAD_ARG;
  if (rows > 0x7fffffffLL * SILU_ROWS || n > 65535 * 2048) return DLTI_ERR_TOO_LARGE;
  silu_rows_kernel<__nv_bfloat16><<<dim3((unsigned)((rows + SILU_ROWS - 1) / SILU_ROWS), (n / 8 + 255) / 256), 256, 0, st>>>((__nv_bfloat16*)x, ld, rows, n);
  dlti_count_launch();
  return (int)cudaGetLastError();
}
