// The matrix-state recurrences of recurrent.cu for prompt portions, in chunks of 64 tokens.
//
// Walking a portion token by token is a chain of T dependent steps per head.  Here the chain has one
// link per chunk.  With L_i the running sum, inside the chunk, of the logarithms of the decays up to
// and including token i (one per key channel; for the decayed sum L_i = (i + 1) log a), k and q as
// the recurrence uses them (unit length, or silu), S_0 the state before the chunk:
//
//   every write u_j reaches token i >= j weakened by exp(L_i - L_j) <= 1:
//     S_i = diag(exp L_i) S_0 + sum_{j<=i} diag(exp(L_i - L_j)) k_j u_j^T
//   decayed sum: u_j = v_j.   Delta rule: u_j = beta_j (v_j - k_j^T diag(g_j) S_{j-1}), which, with
//     A_jm = sum_c k_j[c] k_m[c] exp(L_j[c] - L_m[c])  (m < j),    T = I + diag(beta) A,
//     is the triangular system  T U = diag(beta) (V - (K * exp L) S_0),  so
//     U = Uv - W S_0  with  Uv = T^-1 diag(beta) V  and  W = T^-1 diag(beta) (K * exp L),
//     two matrices that do not depend on the state.
//   read-out: o_i = (q_i * exp L_i)^T S_0 + sum_{j<=i} B_ij u_j,   B_ij = sum_c q_i[c] k_j[c] exp(L_i[c] - L_j[c])
//   state after the chunk of n tokens: S = diag(exp L_{n-1}) S_0 + (K * exp(L_{n-1} - L))^T U
//
// Time mixing (kRuleWkv) is the decayed sum with a decay per channel and a read-out before the token's own write:
//   o_i = (q_i * exp L_(i-1))^T S_0 + sum_{j<i} B_ij v_j + B_ii v_i,  B_ij = sum_c q_i[c] k_j[c] exp(L_(i-1)[c] - L_j[c]),
//   B_ii = sum_c q_i[c] b[c] k_i[c] with the bonus b;  `wkv_prepare` makes these operands, what follows is the decayed sum's.  Retention
// (kRuleRetention) is the decayed sum whose q and k are rotated as they are read.  The decayed sums' operands are made by
// `decay_prepare`.
//
// Only differences L_i - L_j with i >= j are ever exponentiated, so nothing overflows however strong
// the decay.  A first launch (`delta_prepare`, `decay_prepare`, `wkv_prepare`) makes W, Uv, B, Q * exp L,
// K * exp(L_end - L) and exp L_end for every (chunk, head) in parallel.  What follows keeps the chain from chunk to
// chunk as short as it can be and does everything else in parallel over chunks: for the decayed sums the chain is
// element-wise, for the delta rule two products with the state a chunk.  All arithmetic is float on the
// CUDA cores: scores, decays, the triangular solve and the state stay 32-bit in both storage types.
// Chunks start at the portion's first token; results do not depend on where a portion is cut beyond
// rounding.
#include "recurrence_rules.cuh"
#include <algorithm>
#include <type_traits>

namespace pmm {

constexpr int kChunk = 64;
constexpr int kPrepThreads = 256;

__device__ __forceinline__ float sigmoid_c(float x) { return 1.f / (1.f + expf(-x)); }

struct ChunkArgs {
  const void* q; long long ld_q;        // [T, Hk*d]
  const void* k; long long ld_k;
  const void* v; long long ld_v;        // [T, H*dv]
  const void* beta; long long ld_beta;  // delta: [T, H]
  const void* a; long long ld_a;        // delta: [T, H*d]
  const float* dt_bias; const float* a_log; const float* decay;   // wkv: dt_bias is the bias of a, a is float
  const float* bonus;                   // wkv: [H*d]
  float k_scale;                        // retention
  RecRotation rot;                      // retention
  const int* cu; int n_seq;
  int H, Hk, d, dv;
  float unit_eps, q_scale;
  // per (chunk, head), chunk-major: W [C, d] (delta), Uv [C, dv], B [C, C], Qg [C, d], Ke [C, d], Eg [d]
  float *W, *Uv, *B, *Qg, *Ke, *Eg;
  int tile0;                            // first column tile of the launch (a grid holds 65,535)
  int with_state;                       // the prepare kernel makes N too (see chunk_state)
  int vec_in;                           // q, k, v (and a) rows and heads start on boundaries of four elements
  float* N;                             // [d, dv] per (chunk, head): see the kernels that use it
  float* state; const int* slots; float* out;
};

// chunk index -> (sequence, first token, tokens in the chunk); false for a surplus block
__device__ __forceinline__ bool locate_chunk(const int* __restrict__ cu, int n_seq, int chunk, int* seq, int* t0, int* n) {
  int base = 0;
  for (int s = 0; s < n_seq; ++s) {
    const int len = cu[s + 1] - cu[s];
    const int nc = (len + kChunk - 1) / kChunk;
    if (chunk < base + nc) {
      const int local = chunk - base;
      *seq = s;
      *t0 = cu[s] + local * kChunk;
      *n = min(kChunk, len - local * kChunk);
      return true;
    }
    base += nc;
  }
  return false;
}

// ----------------------------------------------------------------------------------------------
// Four neighbouring elements of a row in the storage type (`vec`: the row starts on a boundary of four elements).
template <typename S>
__device__ __forceinline__ float4 load4(const S* p, bool vec) {
  if (!vec) return make_float4(ldf(p), ldf(p + 1), ldf(p + 2), ldf(p + 3));
  return ldf4(p);
}

// ----------------------------------------------------------------------------------------------
// Two floats in one register pair: one instruction for two multiply-adds, each rounded as by itself.
using Pair = unsigned long long;
__device__ __forceinline__ Pair pair(float x, float y) {
  Pair r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float2 halves(Pair v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ Pair fma2(Pair a, Pair b, Pair c) {
  Pair r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
struct Quad { Pair lo, hi; };
__device__ __forceinline__ Quad quad(const float* p) {  // sixteen bytes
  const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
  return {v.x, v.y};
}

// ----------------------------------------------------------------------------------------------
// The delta rule's operands W, Uv, B, Q * exp L, K * exp(L_end - L), exp L_end of one (chunk, head) per block.
//
// Sums of logarithms (to base 2) start anew every 8 tokens, and products across boundaries use two factors, each at most
// one: with r the last row before i's half, exp(L_i - L_j) = exp(L_i - L_r) exp(L_r - L_j).  So only the pairs within 8
// tokens take an exponential per channel; then q_i, k_i (weakened from their half's start) and k_j (weakened to its half's
// end) lie in place as three matrices, pairs across halves of 8, 16 and 32 tokens are plain products in 4 x 4 tiles of A
// and B at once, and between two levels the rows are weakened by one more half's total.  What is left at the end is
// Q * exp L, K * exp L and K * exp(L_end - L).
// The triangular solve takes a thread per column of [W | Uv], 16 rows at a time in registers: what the rows solved before
// take off is summed first, then each row that becomes known enters the sums of those below, with A read as broadcast rows of
// its transpose, which lies where q was (its entries wait in registers until q is done).  A row is its sum taken off in one
// subtraction: a subtraction a term rounds the whole row up to 63 times (error of the states against float64 after 600
// tokens of weak decays 1.9e-7 at d = 64 to 244, so 1.5e-7, at the same speed).
// A chunk of n tokens makes rows up to the next multiple of 16 (chunk_rows), those from n on as zeros; the chain takes as many.
// All 64 rows of every chunk cost a step of one portion of 512 tokens beside 63 lone ones, 4 heads of 244 x 244, 703 us where
// 587 us are enough.
//
// Bound by latency on few warps: 256 threads and 109 KB at d = 128 put two blocks on an SM, 3.4 warps a scheduler, which issue in
// 43 % of the cycles (a warp waits about alike for global reads, shared-memory reads and its own arithmetic; DRAM 3 %).  One
// block's barriers and reads are the other's turn, and the 256 blocks of 2,048 tokens and 8 heads are one wave.
// That size, 128 x 128, inside a step: first form (rows scaled per sub-block of 16 into copies, scalar shared-memory reads, a column
// walking A in shared memory, 157 KB) 160 us, 4 x 4 tiles with the solve's whole column in registers (unrolled past the
// instruction cache, one block an SM) 96 us, this form 59 us (68 alone with cold caches).
constexpr float kLogDecayMin = -1e4f;  // a token's logarithm to base 2: the power is zero long before, and sums stay finite
constexpr int kPrepRows = kChunk / 8;  // halves of 8 tokens

// Rows of the operands that a chunk of n tokens fills: the solve's and the chain's steps are whole sixteens.
__device__ __forceinline__ int chunk_rows(int n) { return (n + 15) & ~15; }

inline size_t delta_prepare_smem(int d) {
  const size_t row = static_cast<size_t>(d) + 4;
  const size_t q = kChunk * row > kChunk * kChunk ? kChunk * row : kChunk * kChunk;
  return sizeof(float) * (q + 2 * kChunk * row + 14 * static_cast<size_t>(d));
}

// v[32] summed over LANES neighbouring lanes; lane l keeps sums (l % LANES) * 32 / LANES .. in v[0 .. 32 / LANES - 1]
template <int LANES>
__device__ __forceinline__ void sum_scatter(float (&v)[32], int lane) {
  int count = 32;
#pragma unroll
  for (int off = LANES / 2; off >= 1; off >>= 1) {
    count >>= 1;
    const bool up = (lane & off) != 0;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      if (i < count) {
        const float send = up ? v[i] : v[i + count], keep = up ? v[i + count] : v[i];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
      }
    }
  }
}

// A and B of the pairs (i, j), i in the odd and j in the even half of HALF tokens of every span of 2 HALF tokens, in 4 x 4
// tiles whose channels are shared by kSlices lanes.  B goes out, A stays with the threads: `keep` entry e is entry
// slice * kKeep + e of its tile where that is below 16.
template <int HALF>
struct CrossPairs {
  static constexpr int kSide = HALF / 4, kTiles = (kChunk / (2 * HALF)) * kSide * kSide;  // 16, 32 and 64 tiles
  static constexpr int kSlices = kPrepThreads / kTiles, kKeep = 32 / kSlices;             // 16, 8 and 4 lanes
  int slice, i0, j0;
  float keep[kKeep];
  __device__ __forceinline__ void run(const float* __restrict__ sQ, const float* __restrict__ sK, const float* __restrict__ sKd,
                                      float* __restrict__ oB, int ds, int d4, int n, int rows, int tid) {
    const int tile = tid / kSlices, g = tile / (kSide * kSide), in = tile % (kSide * kSide);
    slice = tid % kSlices;
    i0 = 2 * HALF * g + HALF + 4 * (in / kSide);
    j0 = 2 * HALF * g + 4 * (in % kSide);
    Pair acc[32];
#pragma unroll
    for (int e = 0; e < 32; ++e) acc[e] = 0;
    const int c_end = i0 < rows ? d4 : 0;  // (a tile behind the last row: zeros, its lanes stay for the sums)
    for (int c4 = slice; c4 < c_end; c4 += kSlices) {
      Quad kd[4];
#pragma unroll
      for (int s = 0; s < 4; ++s) kd[s] = quad(sKd + (j0 + s) * ds + 4 * c4);
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const Quad k = quad(sK + (i0 + r) * ds + 4 * c4), q = quad(sQ + (i0 + r) * ds + 4 * c4);
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          acc[4 * r + s] = fma2(k.hi, kd[s].hi, fma2(k.lo, kd[s].lo, acc[4 * r + s]));
          acc[16 + 4 * r + s] = fma2(q.hi, kd[s].hi, fma2(q.lo, kd[s].lo, acc[16 + 4 * r + s]));
        }
      }
    }
    float v[32];
#pragma unroll
    for (int e = 0; e < 32; ++e) {
      const float2 two = halves(acc[e]);
      v[e] = two.x + two.y;
    }
    sum_scatter<kSlices>(v, slice);
#pragma unroll
    for (int e = 0; e < kKeep; ++e) {
      const int at = slice * kKeep + e, i = i0 + (at % 16) / 4;
      keep[e] = v[e];
      if (at >= 16 && i < n) oB[i * kChunk + j0 + at % 4] = v[e];
    }
  }
  __device__ __forceinline__ void leave(float* __restrict__ sAt) const {
#pragma unroll
    for (int e = 0; e < kKeep; ++e) {
      const int at = slice * kKeep + e;
      if (at < 16) sAt[(j0 + at % 4) * kChunk + i0 + at / 4] = keep[e];
    }
  }
};

template <typename S>
__global__ void __launch_bounds__(kPrepThreads, 2)
    delta_prepare_kernel(ChunkArgs p) {
  extern __shared__ __align__(16) float sm[];
  const int d = p.d, d4 = d / 4, dv = p.dv, ds = d + 4;  // rows of stride d + 4: neighbouring rows' 16-byte reads fall into different banks
  float* sQ = sm;                               // [C][ds]  q, then weakened from its half's start
  float* sAt = sm;                              // [C][C]   A transposed: row j, entries i > j (once q is done)
  float* sK = sQ + max(kChunk * ds, kChunk * kChunk);  // [C][ds]  k, then weakened from its half's start, then W
  float* sL = sK + kChunk * ds;                 // [C][ds]  sums of logarithms, then k weakened to its half's end, then columns of Uv
  float* sT = sL + kChunk * ds;                 // [8 + 4 + 2][d]  totals of 8 tokens, then powers of the totals of 8, 16 and 32
  __shared__ float s_beta[kChunk];
  pdl_launch_dependents();
  pdl_wait();
  const int chunk = blockIdx.x, h = blockIdx.y;
  int seq, t0, n;
  if (!locate_chunk(p.cu, p.n_seq, chunk, &seq, &t0, &n)) return;
  const int hk = h / (p.H / p.Hk);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr int kWarps = kPrepThreads / 32;
  const size_t ch = static_cast<size_t>(chunk) * p.H + h;
  const int rows = chunk_rows(n);
  float* oB = p.B + ch * kChunk * kChunk;
  const bool vec = p.vec_in != 0;
  constexpr float kLog2E = 1.4426950408889634f;

  // ---- unit-length q and k and the decays' logarithms: a warp per token
  const float a_neg = -expf(p.a_log[h]) * kLog2E;
#pragma unroll 2
  for (int i = warp; i < rows; i += kWarps) {
    float *rq = sQ + i * ds, *rk = sK + i * ds, *rl = sL + i * ds;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i >= n) {
      for (int c4 = lane; c4 < d4; c4 += 32) {
        *reinterpret_cast<float4*>(rq + 4 * c4) = zero;
        *reinterpret_cast<float4*>(rk + 4 * c4) = zero;
        *reinterpret_cast<float4*>(rl + 4 * c4) = zero;
      }
      continue;
    }
    const long long t = t0 + i;
    float sq = 0.f, sk = 0.f;
    for (int c4 = lane; c4 < d4; c4 += 32) {
      const int c = 4 * c4;
      const float4 q = load4(static_cast<const S*>(p.q) + t * p.ld_q + hk * d + c, vec);
      const float4 k = load4(static_cast<const S*>(p.k) + t * p.ld_k + hk * d + c, vec);
      const float4 a = load4(static_cast<const S*>(p.a) + t * p.ld_a + h * d + c, vec);
      const float* b = p.dt_bias + h * d + c;
      auto decay = [a_neg](float z) {
        const float l = a_neg * softplus_f(z);
        return l < kLogDecayMin ? kLogDecayMin : l;  // (NaN stays)
      };
      sq += q.x * q.x + q.y * q.y + q.z * q.z + q.w * q.w;
      sk += k.x * k.x + k.y * k.y + k.z * k.z + k.w * k.w;
      *reinterpret_cast<float4*>(rq + c) = q;
      *reinterpret_cast<float4*>(rk + c) = k;
      *reinterpret_cast<float4*>(rl + c) = make_float4(decay(a.x + b[0]), decay(a.y + b[1]), decay(a.z + b[2]), decay(a.w + b[3]));
    }
    const float fq = p.q_scale / sqrtf(warp_sum(sq) + p.unit_eps), fk = 1.f / sqrtf(warp_sum(sk) + p.unit_eps);
    for (int c4 = lane; c4 < d4; c4 += 32) {
      float4 q = *reinterpret_cast<float4*>(rq + 4 * c4), k = *reinterpret_cast<float4*>(rk + 4 * c4);
      *reinterpret_cast<float4*>(rq + 4 * c4) = make_float4(q.x * fq, q.y * fq, q.z * fq, q.w * fq);
      *reinterpret_cast<float4*>(rk + 4 * c4) = make_float4(k.x * fk, k.y * fk, k.z * fk, k.w * fk);
    }
  }
  if (tid < kChunk)
    s_beta[tid] = tid < n ? sigmoid_c(ldf(static_cast<const S*>(p.beta) + static_cast<long long>(t0 + tid) * p.ld_beta + h)) : 0.f;
  __syncthreads();
  for (int blk = warp; blk < kPrepRows; blk += kWarps) {  // running sums within 8 tokens
    for (int c = lane; c < d; c += 32) {
      float run = 0.f;
      if (8 * blk < rows) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          run += sL[(8 * blk + i) * ds + c];
          sL[(8 * blk + i) * ds + c] = run;
        }
      }
      sT[blk * d + c] = run;
    }
  }
  __syncthreads();

  // ---- pairs within 8 tokens: a thread per pair, the exponential per channel
  float own_a[kChunk * 8 / kPrepThreads];
#pragma unroll
  for (int u = 0; u < kChunk * 8 / kPrepThreads; ++u) {
    const int e = tid + kPrepThreads * u, i = e >> 3, j = (i & ~7) + (e & 7);
    own_a[u] = 0.f;
    if (j <= i && i < rows) {
      const float *qi = sQ + i * ds, *ki = sK + i * ds, *li = sL + i * ds, *kj = sK + j * ds, *lj = sL + j * ds;
      Pair accA = 0, accB = 0;
#pragma unroll 2
      for (int c = 0; c < d; c += 4) {
        const Quad q = quad(qi + c), k = quad(ki + c);
        const float4 o = *reinterpret_cast<const float4*>(kj + c), l = *reinterpret_cast<const float4*>(li + c), m = *reinterpret_cast<const float4*>(lj + c);
        const Pair lo = pair(o.x * exp2f(l.x - m.x), o.y * exp2f(l.y - m.y)), hi = pair(o.z * exp2f(l.z - m.z), o.w * exp2f(l.w - m.w));
        accA = fma2(k.hi, hi, fma2(k.lo, lo, accA));
        accB = fma2(q.hi, hi, fma2(q.lo, lo, accB));
      }
      const float2 two_a = halves(accA), two_b = halves(accB);
      own_a[u] = two_a.x + two_a.y;
      if (i < n) oB[i * kChunk + j] = two_b.x + two_b.y;
    }
  }
  __syncthreads();
  auto times = [](float* at, const float4& f) {
    float4 v = *reinterpret_cast<float4*>(at);
    *reinterpret_cast<float4*>(at) = make_float4(v.x * f.x, v.y * f.y, v.z * f.z, v.w * f.w);
  };
  auto power = [](const float4& l) { return make_float4(exp2f(l.x), exp2f(l.y), exp2f(l.z), exp2f(l.w)); };
  for (int i = warp; i < rows; i += kWarps) {
    for (int c = 4 * lane; c < d; c += 128) {
      const float4 l = *reinterpret_cast<const float4*>(sL + i * ds + c), t = *reinterpret_cast<const float4*>(sT + (i >> 3) * d + c);
      const float4 k = *reinterpret_cast<const float4*>(sK + i * ds + c);
      const float4 up = power(l), down = power(make_float4(t.x - l.x, t.y - l.y, t.z - l.z, t.w - l.w));
      *reinterpret_cast<float4*>(sL + i * ds + c) = make_float4(k.x * down.x, k.y * down.y, k.z * down.z, k.w * down.w);
      *reinterpret_cast<float4*>(sK + i * ds + c) = make_float4(k.x * up.x, k.y * up.y, k.z * up.z, k.w * up.w);
      times(sQ + i * ds + c, up);
    }
  }
  __syncthreads();
  for (int c = tid; c < d; c += kPrepThreads) {  // the totals' powers, from the sums
    float t[8];
#pragma unroll
    for (int b = 0; b < 8; ++b) t[b] = sT[b * d + c];
#pragma unroll
    for (int b = 0; b < 8; ++b) sT[b * d + c] = exp2f(t[b]);
#pragma unroll
    for (int b = 0; b < 4; ++b) sT[(8 + b) * d + c] = exp2f(t[2 * b] + t[2 * b + 1]);
#pragma unroll
    for (int b = 0; b < 2; ++b) sT[(12 + b) * d + c] = exp2f((t[4 * b] + t[4 * b + 1]) + (t[4 * b + 2] + t[4 * b + 3]));
    p.Eg[ch * d + c] = exp2f(((t[0] + t[1]) + (t[2] + t[3])) + ((t[4] + t[5]) + (t[6] + t[7])));
  }
  // ---- pairs across halves of 8, 16 and 32 tokens; after each, rows reach through the neighbouring half
  auto widen = [&](int half, int first_total) {
    __syncthreads();
    for (int i = warp; i < rows; i += kWarps) {
      const int b = i / half;
      for (int c = 4 * lane; c < d; c += 128) {
        const float4 f = *reinterpret_cast<const float4*>(sT + (first_total + (b ^ 1)) * d + c);
        if (b & 1) {
          times(sQ + i * ds + c, f);
          times(sK + i * ds + c, f);
        } else {
          times(sL + i * ds + c, f);
        }
      }
    }
    __syncthreads();
  };
  CrossPairs<8> by8;
  by8.run(sQ, sK, sL, oB, ds, d4, n, rows, tid);
  widen(8, 0);
  CrossPairs<16> by16;
  CrossPairs<32> by32;
  if (rows > 16) {  // (behind the last row the totals are zero, their powers one)
    by16.run(sQ, sK, sL, oB, ds, d4, n, rows, tid);
    widen(16, 8);
  }
  if (rows > 32) {
    by32.run(sQ, sK, sL, oB, ds, d4, n, rows, tid);
    widen(32, 12);
  }

  // ---- what the other launches read; V takes the place of K * exp(L_end - L), A that of q
  float* oQg = p.Qg + ch * kChunk * d;
  float* oKe = p.Ke + ch * kChunk * d;
  for (int i = warp; i < rows; i += kWarps) {
    for (int c = 4 * lane; c < d; c += 128) {
      *reinterpret_cast<float4*>(oQg + i * d + c) = *reinterpret_cast<const float4*>(sQ + i * ds + c);
      *reinterpret_cast<float4*>(oKe + i * d + c) = *reinterpret_cast<const float4*>(sL + i * ds + c);
    }
  }
  __syncthreads();
  by8.leave(sAt);
  if (rows > 16) by16.leave(sAt);
  if (rows > 32) by32.leave(sAt);
#pragma unroll
  for (int u = 0; u < kChunk * 8 / kPrepThreads; ++u) {
    const int e = tid + kPrepThreads * u, i = e >> 3, j = (i & ~7) + (e & 7);
    if (j <= i && i < rows) sAt[j * kChunk + i] = own_a[u];  // (the diagonal's is not read for a result)
  }

  // ---- T X = diag(beta) [K * exp L | V] by forward substitution, V's columns d at a time
  const S* gv = static_cast<const S*>(p.v) + static_cast<long long>(t0) * p.ld_v + h * dv;
  for (int v0 = 0; v0 < dv; v0 += d) {
    const int vw = min(d, dv - v0);
    for (int i = warp; i < rows; i += kWarps)
      for (int c = lane; c < vw; c += 32) sL[i * ds + c] = i < n ? ldf(gv + static_cast<long long>(i) * p.ld_v + v0 + c) : 0.f;
    __syncthreads();
    const int n_w = v0 == 0 ? d : 0;  // the first pass also solves for W
    for (int col = tid; col < n_w + vw; col += kPrepThreads) {
      const bool is_w = col < n_w;
      const int c = is_w ? col : col - n_w;
      float* x = (is_w ? sK : sL) + c;
      float* to = is_w ? p.W + ch * kChunk * d + c : p.Uv + ch * kChunk * dv + v0 + c;
      const int ld = is_w ? d : dv;
#pragma unroll 1
      for (int b0 = 0; b0 < rows; b0 += 16) {
        float in[16];
        Pair r[8];   // what the rows solved before add up to, taken off in one subtraction
#pragma unroll
        for (int u = 0; u < 16; ++u) in[u] = x[(b0 + u) * ds];
#pragma unroll
        for (int u = 0; u < 8; ++u) r[u] = 0ull;
        const float* at = sAt + b0;
#pragma unroll 4
        for (int m = 0; m < b0; ++m) {
          const float xm = x[m * ds];
          const Pair xx = pair(xm, xm);
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const Quad a = quad(at + m * kChunk + 4 * u);
            r[2 * u] = fma2(a.lo, xx, r[2 * u]);
            r[2 * u + 1] = fma2(a.hi, xx, r[2 * u + 1]);
          }
        }
        at += b0 * kChunk;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const float2 two = halves(r[j / 2]);
          const float xj = (in[j] - ((j & 1) ? two.y : two.x)) * s_beta[b0 + j];
          x[(b0 + j) * ds] = xj;
          to[(b0 + j) * ld] = xj;
          const Pair xx = pair(xj, xj);
#pragma unroll
          for (int u = (j + 1) / 4; u < 4; ++u) {  // (a pair of rows that is not all below row j: what its done half becomes is not read)
            const Quad a = quad(at + j * kChunk + 4 * u);
            if (4 * u + 1 > j) r[2 * u] = fma2(a.lo, xx, r[2 * u]);
            r[2 * u + 1] = fma2(a.hi, xx, r[2 * u + 1]);
          }
        }
      }
    }
    __syncthreads();  // the next pass loads further columns of V over these
  }
}

// The values of the chunk's tokens as floats (silu of them for kRuleDecay), eight or four bytes at a time where they lie so
template <typename S, bool SILU>
__device__ __forceinline__ void widen_values(const ChunkArgs& p, float* __restrict__ oUv, float* __restrict__ sV, int h, int t0, int n, int tid, int n_threads) {
  const int dv = p.dv;
  const S* gv = static_cast<const S*>(p.v) + static_cast<long long>(t0) * p.ld_v + h * dv;
  if (dv % 4 == 0) {
#pragma unroll 4
    for (int e = tid; e < n * (dv / 4); e += n_threads) {
      const int i = e / (dv / 4), c = 4 * (e - i * (dv / 4));
      float4 v = load4(gv + static_cast<long long>(i) * p.ld_v + c, p.vec_in != 0);
      if (SILU) v = make_float4(silu_f(v.x), silu_f(v.y), silu_f(v.z), silu_f(v.w));
      *reinterpret_cast<float4*>(oUv + static_cast<size_t>(i) * dv + c) = v;
      if (sV) *reinterpret_cast<float4*>(sV + i * dv + c) = v;  // (asked for with dv a multiple of 8 only)
    }
    return;
  }
  for (int e = tid; e < n * dv; e += n_threads) {
    const int i = e / dv, c = e - i * dv;
    const float v = ldf(gv + static_cast<long long>(i) * p.ld_v + c);
    oUv[e] = SILU ? silu_f(v) : v;
  }
}

// N [d, dv] = Ke^T V of a chunk whose weakened keys and values lie in shared memory: 8 x (4 or 8) results a thread, two
// multiply-adds an instruction, every sum in the order of the tokens.  d and dv are multiples of 8.  The prepare kernels end with it where their
// blocks still share an SM: a launch, the keys' way out to memory and back and eight (instead of twelve or sixteen) sixteen-byte reads
// for every 128 multiply-adds less.  Us inside a step, prepare and state: the decayed sum at 2,048 tokens, 8 heads, 128 x 128 20 + 16 -> 25, retention
// at 1,501, 8 heads, 64 x 128 26 + 15 -> 23, time mixing at 1,501, 16 heads, 64 x 64 33 + 15 -> 39.
template <int COLS>
__device__ __forceinline__ void chunk_state(float* __restrict__ gN, const float* __restrict__ sKe, int ds, const float* __restrict__ sV,
                                            int d, int dv, int n, int tid, int n_threads) {
  constexpr int P = COLS / 2;   // pairs of columns: four neighbours, and with 8 columns four more half a row further
  const int per_row = dv / COLS, tiles = (d / 8) * per_row;
  for (int tile = tid; tile < tiles; tile += n_threads) {
    const int c = 4 * (tile % per_row), k0 = 8 * (tile / per_row);
    Pair acc[8][P];
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
      for (int q = 0; q < P; ++q) acc[r][q] = 0ull;
#pragma unroll 2
    for (int j = 0; j < n; ++j) {
      const float4 a0 = *reinterpret_cast<const float4*>(sKe + j * ds + k0), a1 = *reinterpret_cast<const float4*>(sKe + j * ds + k0 + 4);
      const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
      Pair b[P];
#pragma unroll
      for (int q = 0; q < P; q += 2) {
        const Quad v = quad(sV + j * dv + c + (q ? dv / 2 : 0));
        b[q] = v.lo;
        b[q + 1] = v.hi;
      }
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const Pair a2 = pair(a[r], a[r]);
#pragma unroll
        for (int q = 0; q < P; ++q) acc[r][q] = fma2(a2, b[q], acc[r][q]);
      }
    }
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
      for (int q = 0; q < P; q += 2) {
        const float2 lo = halves(acc[r][q]), hi = halves(acc[r][q + 1]);
        *reinterpret_cast<float4*>(gN + static_cast<size_t>(k0 + r) * dv + c + (q ? dv / 2 : 0)) = make_float4(lo.x, lo.y, hi.x, hi.y);
      }
  }
}

// The operands of the decayed sum (kRuleDecay, kRuleRetention): B_ij = (q_i . k_j) a^(i-j), Q * a^(i+1), K * a^(n-1-i), a^n.
// Rows of stride d + 4: sixteen-byte reads of neighbouring rows fall into different banks.  A thread makes the entries of B of
// four neighbouring rows and of every sixteenth column (16 threads read 16 neighbouring rows of k; with four
// neighbouring columns a thread their reads fell into the same banks four by four).
constexpr int kDecayPrepThreads = 256;

inline size_t decay_prepare_smem(int d) { return sizeof(float) * (static_cast<size_t>(2 * kChunk) * (d + 4)); }

template <typename S, int RULE>
__global__ void __launch_bounds__(kDecayPrepThreads)
    decay_prepare_kernel(ChunkArgs p) {
  extern __shared__ __align__(16) float sm[];
  constexpr bool SILU = RULE == kRuleDecay;
  const int d = p.d, d4 = d / 4, ds = d + 4;
  float* sK = sm;                  // [C][ds]
  float* sQ = sK + kChunk * ds;    // [C][ds]
  __shared__ float s_pow[kChunk + 1];  // a^0 .. a^C
  pdl_launch_dependents();
  pdl_wait();
  const int chunk = blockIdx.x, h = blockIdx.y;
  int seq, t0, n;
  if (!locate_chunk(p.cu, p.n_seq, chunk, &seq, &t0, &n)) return;
  const int tid = threadIdx.x;
  const size_t ch = static_cast<size_t>(chunk) * p.H + h;
  if (tid <= kChunk) s_pow[tid] = expf(logf(fmaxf(p.decay[h], 1e-38f)) * static_cast<float>(tid));
#pragma unroll 4
  for (int e = tid; e < n * d4; e += kDecayPrepThreads) {
    const int i = e / d4, c = 4 * (e - i * d4);
    const long long t = t0 + i;
    float4 q = load4(static_cast<const S*>(p.q) + t * p.ld_q + h * d + c, p.vec_in != 0);
    float4 k = load4(static_cast<const S*>(p.k) + t * p.ld_k + h * d + c, p.vec_in != 0);
    if (SILU) {
      q = make_float4(silu_f(q.x), silu_f(q.y), silu_f(q.z), silu_f(q.w));
      k = make_float4(silu_f(k.x), silu_f(k.y), silu_f(k.z), silu_f(k.w));
    } else {
      k = make_float4(k.x * p.k_scale, k.y * p.k_scale, k.z * p.k_scale, k.w * p.k_scale);
    }
    *reinterpret_cast<float4*>(sQ + i * ds + c) = q;
    *reinterpret_cast<float4*>(sK + i * ds + c) = k;
  }
  float* sV = p.with_state ? sQ + kChunk * ds : nullptr;  // [C][dv]
  widen_values<S, SILU>(p, p.Uv + ch * kChunk * p.dv, sV, h, t0, n, tid, kDecayPrepThreads);
  __syncthreads();
  if (RULE == kRuleRetention && p.rot.rot_dims > 0) {
    rotate_rows(sQ, sK, ds, n, t0, p.rot, tid, kDecayPrepThreads);
    __syncthreads();
  }
  float* oB = p.B + ch * kChunk * kChunk;
  // (rows at and beyond n hold stale values whose results are not stored)
  const int i0 = 4 * (tid / 16), j0 = tid % 16, spans = i0 / 16;  // columns j0, j0 + 16 .. up to the rows' own sixteen
  if (i0 < n) {
    float acc[4][4] = {};
    for (int c = 0; c < d; c += 4) {
      float4 q[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) q[r] = *reinterpret_cast<const float4*>(sQ + (i0 + r) * ds + c);
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        if (s > spans) break;
        const float4 k = *reinterpret_cast<const float4*>(sK + (j0 + 16 * s) * ds + c);
#pragma unroll
        for (int r = 0; r < 4; ++r) acc[r][s] += q[r].x * k.x + q[r].y * k.y + q[r].z * k.z + q[r].w * k.w;
      }
    }
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        const int i = i0 + r, j = j0 + 16 * s;
        if (i < n && j <= i) oB[i * kChunk + j] = acc[r][s] * s_pow[i - j];
      }
  }
  if (p.with_state) __syncthreads();  // the keys are weakened in place
  float* oQg = p.Qg + ch * kChunk * d;
  float* oKe = p.Ke + ch * kChunk * d;
  for (int e = tid; e < n * d4; e += kDecayPrepThreads) {
    const int i = e / d4, c = 4 * (e - i * d4);
    const float up = s_pow[i + 1], down = s_pow[n - 1 - i];
    const float4 q = *reinterpret_cast<const float4*>(sQ + i * ds + c), k = *reinterpret_cast<const float4*>(sK + i * ds + c);
    *reinterpret_cast<float4*>(oQg + i * d + c) = make_float4(q.x * up, q.y * up, q.z * up, q.w * up);
    *reinterpret_cast<float4*>(p.with_state ? sK + i * ds + c : oKe + i * d + c) = make_float4(k.x * down, k.y * down, k.z * down, k.w * down);
  }
  for (int c = tid; c < d; c += kDecayPrepThreads) p.Eg[ch * d + c] = s_pow[n];
  if (p.with_state) {
    __syncthreads();
    chunk_state<8>(p.N + ch * static_cast<size_t>(d) * p.dv, sK, ds, sV, d, p.dv, n, tid, kDecayPrepThreads);
  }
}

// ----------------------------------------------------------------------------------------------
// The same operands for time mixing.  Sums of logarithms are kept within sub-blocks of 16 tokens only (sL: up to and
// including the token; sT: a sub-block's total), so that strong decays do not drown the weak ones behind them, and a
// token's logarithm is bounded at -40 (4e-18: below the rounding of anything it could stand beside).  Rows of stride
// d + 4: sixteen-byte reads of neighbouring rows fall into different banks.
//   pairs within a sub-block:  B_ij = sum_c q_i[c] k_j[c] exp(L_(i-1) - L_j),  B_ii with the bonus;
//   then in place  q_i <- q_i exp(L_(i-1) of its sub-block),  k_j <- k_j exp(T - L_j)  (weakened to its sub-block's end);
//   sub-block by sub-block, all rows of k before it are weakened to its start: pairs across are dot products.
// Logarithms are to base 2 (one instruction less for every exponential).
// What is left of q and k at the end is, up to whole sub-blocks' totals, Q * exp L and K * exp(L_end - L).
constexpr float kLogDecayFloor = -40.f;
constexpr float kLog2E = 1.4426950408889634f;

constexpr int kWkvThreads = 256;

inline size_t wkv_prepare_smem(int d) { return sizeof(float) * (static_cast<size_t>(3 * kChunk) * (d + 4) + 4 * static_cast<size_t>(d)); }

template <typename S>
__global__ void __launch_bounds__(kWkvThreads)
    wkv_prepare_kernel(ChunkArgs p) {
  extern __shared__ __align__(16) float sm[];
  const int d = p.d, d4 = d / 4, dv = p.dv, ds = d + 4;
  float* sK = sm;                  // [C][ds]
  float* sQ = sK + kChunk * ds;    // [C][ds]
  float* sL = sQ + kChunk * ds;    // [C][ds]
  float* sT = sL + kChunk * ds;    // [4][d]
  pdl_launch_dependents();
  pdl_wait();
  const int chunk = blockIdx.x, h = blockIdx.y;
  int seq, t0, n;
  if (!locate_chunk(p.cu, p.n_seq, chunk, &seq, &t0, &n)) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const size_t ch = static_cast<size_t>(chunk) * p.H + h;
  float* oB = p.B + ch * kChunk * kChunk;
  float* oQg = p.Qg + ch * kChunk * d;
  float* oKe = p.Ke + ch * kChunk * d;
  float* oUv = p.Uv + ch * kChunk * dv;
  const int nb = (n + 15) >> 4;

  const bool vec = p.vec_in != 0;
#pragma unroll 4
  for (int e = tid; e < n * d4; e += kWkvThreads) {
    const int i = e / d4, c = 4 * (e - i * d4);
    const long long t = t0 + i;
    const float4 q = load4(static_cast<const S*>(p.q) + t * p.ld_q + h * d + c, vec);
    const float4 k = load4(static_cast<const S*>(p.k) + t * p.ld_k + h * d + c, vec);
    const float4 a = load4(static_cast<const float*>(p.a) + t * p.ld_a + h * d + c, vec);
    const float4 b = load4(p.dt_bias + h * d + c, vec);
    auto decay = [](float z) { return fmaxf(-expf(z), kLogDecayFloor) * kLog2E; };
    *reinterpret_cast<float4*>(sQ + i * ds + c) = q;
    *reinterpret_cast<float4*>(sK + i * ds + c) = k;
    *reinterpret_cast<float4*>(sL + i * ds + c) = make_float4(decay(a.x + b.x), decay(a.y + b.y), decay(a.z + b.z), decay(a.w + b.w));
  }
  float* sV = p.with_state ? sT + 4 * d : nullptr;  // [C][dv]
  widen_values<S, false>(p, oUv, sV, h, t0, n, tid, kWkvThreads);
  __syncthreads();
  for (int e = tid; e < nb * d; e += kWkvThreads) {
    const int blk = e / d, c = e - blk * d;
    float run = 0.f;
    for (int i = 16 * blk; i < min(16 * blk + 16, n); ++i) {
      run += sL[i * ds + c];
      sL[i * ds + c] = run;
    }
    sT[blk * d + c] = run;
  }
  __syncthreads();

  // ---- pairs within a sub-block: a warp takes two rows, 16 lanes each, a lane one column of the row's sub-block
  for (int i2 = 2 * warp; i2 < n; i2 += 2 * (kWkvThreads / 32)) {
    const int i = i2 + (lane >> 4), j = (i & ~15) + (lane & 15);
    if (i < n && j <= i) {
      const float *qi = sQ + i * ds, *kj = sK + j * ds, *lj = sL + j * ds, *li = sL + (i > 0 ? i - 1 : 0) * ds;  // (i > j: row i - 1 is in the sub-block)
      const float* u = p.bonus + h * d;
      float acc = 0.f;
      for (int c = 0; c < d; c += 4) {
        const float4 q4 = *reinterpret_cast<const float4*>(qi + c), k4 = *reinterpret_cast<const float4*>(kj + c);
        if (i == j) {
          acc += q4.x * u[c] * k4.x + q4.y * u[c + 1] * k4.y + q4.z * u[c + 2] * k4.z + q4.w * u[c + 3] * k4.w;
        } else {
          const float4 a4 = *reinterpret_cast<const float4*>(li + c), b4 = *reinterpret_cast<const float4*>(lj + c);
          acc += q4.x * k4.x * exp2f(a4.x - b4.x) + q4.y * k4.y * exp2f(a4.y - b4.y) + q4.z * k4.z * exp2f(a4.z - b4.z) +
                 q4.w * k4.w * exp2f(a4.w - b4.w);
        }
      }
      oB[i * kChunk + j] = acc;
    }
  }
  __syncthreads();
  auto weaken = [](float* row, float4 l) {
    float4 v = *reinterpret_cast<float4*>(row);
    *reinterpret_cast<float4*>(row) = make_float4(v.x * exp2f(l.x), v.y * exp2f(l.y), v.z * exp2f(l.z), v.w * exp2f(l.w));
  };
  for (int e = tid; e < n * d4; e += kWkvThreads) {
    const int i = e / d4, c = 4 * (e - i * d4);
    if (i & 15) weaken(sQ + i * ds + c, *reinterpret_cast<const float4*>(sL + (i - 1) * ds + c));
    const float4 t = *reinterpret_cast<const float4*>(sT + (i >> 4) * d + c), l = *reinterpret_cast<const float4*>(sL + i * ds + c);
    weaken(sK + i * ds + c, make_float4(t.x - l.x, t.y - l.y, t.z - l.z, t.w - l.w));
  }
  // ---- pairs across: four rows of the sub-block and 32 columns a warp
  for (int blk = 1; blk < nb; ++blk) {
    __syncthreads();
    if (blk > 1) {  // rows before the last sub-block reach this one through its total
      for (int e = tid; e < 16 * (blk - 1) * d4; e += kWkvThreads) {
        const int j = e / d4, c = 4 * (e - j * d4);
        weaken(sK + j * ds + c, *reinterpret_cast<const float4*>(sT + (blk - 1) * d + c));
      }
      __syncthreads();
    }
    const int rg = warp & 3, j = (warp >> 2) * 32 + lane;
    const int i0 = 16 * blk + 4 * rg;
    if (j < 16 * blk && i0 < n) {
      const float* kj = sK + j * ds;
      const float* q0 = sQ + i0 * ds;   // (rows at and beyond n hold stale values that are not stored)
      float acc[4] = {0.f, 0.f, 0.f, 0.f};
      for (int c = 0; c < d; c += 4) {
        const float4 k4 = *reinterpret_cast<const float4*>(kj + c);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const float4 q4 = *reinterpret_cast<const float4*>(q0 + r * ds + c);
          acc[r] += q4.x * k4.x + q4.y * k4.y + q4.z * k4.z + q4.w * k4.w;
        }
      }
#pragma unroll
      for (int r = 0; r < 4; ++r)
        if (i0 + r < n) oB[(i0 + r) * kChunk + j] = acc[r];
    }
  }
  __syncthreads();
  // ---- what the other launches read: q weakened from the chunk's start, k to its end, the whole chunk's decay
  for (int e = tid; e < n * d4; e += kWkvThreads) {
    const int i = e / d4, c = 4 * (e - i * d4), blk = i >> 4;
    float4 l = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int b = 0; b < blk; ++b) {
      const float4 t = *reinterpret_cast<const float4*>(sT + b * d + c);
      l = make_float4(l.x + t.x, l.y + t.y, l.z + t.z, l.w + t.w);
    }
    const float4 q = *reinterpret_cast<const float4*>(sQ + i * ds + c);
    *reinterpret_cast<float4*>(oQg + i * d + c) = make_float4(q.x * exp2f(l.x), q.y * exp2f(l.y), q.z * exp2f(l.z), q.w * exp2f(l.w));
    if (blk < nb - 1) weaken(sK + i * ds + c, *reinterpret_cast<const float4*>(sT + (nb - 1) * d + c));
    if (!p.with_state) *reinterpret_cast<float4*>(oKe + i * d + c) = *reinterpret_cast<const float4*>(sK + i * ds + c);
  }
  float* oEg = p.Eg + ch * d;
  for (int c = tid; c < d; c += kWkvThreads) {
    float all = 0.f;
    for (int b = 0; b < nb; ++b) all += sT[b * d + c];
    oEg[c] = exp2f(all);
  }
  if (p.with_state) {
    __syncthreads();
    chunk_state<4>(p.N + ch * static_cast<size_t>(d) * dv, sK, ds, sV, d, dv, n, tid, kWkvThreads);
  }
}

__device__ __forceinline__ void cp_async16(float* smem_dst, const float* gmem_src) {
  const unsigned dst = static_cast<unsigned>(__cvta_generic_to_shared(smem_dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// ----------------------------------------------------------------------------------------------
// The decayed sum has no product with the state inside its chain: S_end = a^n S_0 + N with
// N = (K * a^(n-1-j))^T V, so the chain over a sequence's chunks is element-wise.  Three steps after
// the operands', all but the middle one parallel over chunks: (1) N of every chunk (in the operands' launch where
// `launch_chunked` finds that better, else in its own); (2) a running
// pass per state element that leaves every chunk's starting state where its N was; (3) the rows
// o_i = (q_i a^(i+1))^T S_0 + sum_{j<=i} B_ij v_j of every chunk.
constexpr int kDecayTile = 64;      // state columns per block in (1) and (3)
constexpr int kDecayThreads = 256;

// ---- small products on shared-memory operands, 4 x 4 results a thread (16 multiply-adds per two
// 16-byte loads).  Tiles are 64 columns wide; thread t of 256 owns columns 4 (t % 16) .. + 3.
__device__ __forceinline__ void fma4x4(float (&acc)[4][4], const float4& a, const float4& b) {
  const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[r][c] += av[r] * bv[c];
}

// acc[r][c] = sum_{j < n} A[j][k0 + r] * R[j][c0 + c]   (A rows of stride lda, R rows of stride 64)
__device__ __forceinline__ void product_tn(float (&acc)[4][4], const float* __restrict__ A, int lda, int k0,
                                           const float* __restrict__ R, int c0, int n) {
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[r][c] = 0.f;
  for (int j = 0; j < n; ++j)
    fma4x4(acc, *reinterpret_cast<const float4*>(A + j * lda + k0), *reinterpret_cast<const float4*>(R + j * kDecayTile + c0));
}

// `count` floats (a multiple of 4, 16-byte aligned at both ends) by asynchronous copies
__device__ __forceinline__ void copy_rows(float* __restrict__ dst, const float* __restrict__ src, int count, int tid) {
  for (int e = 4 * tid; e < count; e += 4 * kDecayThreads) cp_async16(dst + e, src + e);
}

// Columns c0 .. c0 + 63 of `rows` rows of a [rows, dv] matrix, zeros beyond dv
template <int THREADS = kDecayThreads>
__device__ __forceinline__ void copy_tile(float* __restrict__ dst, const float* __restrict__ src, int rows, int dv, int c0, int tid) {
  if (dv % 4 == 0 && reinterpret_cast<uintptr_t>(src) % 16 == 0) {
    for (int e = tid; e < rows * (kDecayTile / 4); e += THREADS) {
      const int j = e / (kDecayTile / 4), c = 4 * (e % (kDecayTile / 4));
      float* to = dst + j * kDecayTile + c;
      if (c0 + c < dv) cp_async16(to, src + static_cast<size_t>(j) * dv + c0 + c);
      else *reinterpret_cast<float4*>(to) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    return;
  }
  for (int e = tid; e < rows * kDecayTile; e += THREADS) {
    const int j = e / kDecayTile, c = e % kDecayTile;
    dst[e] = (c0 + c < dv) ? src[static_cast<size_t>(j) * dv + c0 + c] : 0.f;
  }
}

// N [d, dv] per (chunk, head), chunk-major
__global__ void __launch_bounds__(kDecayThreads)
    decay_chunk_state_kernel(ChunkArgs p) {
  extern __shared__ __align__(16) float sm[];
  const int d = p.d, dv = p.dv;
  float* sKe = sm;                    // [C][d]
  float* sV = sKe + kChunk * d;       // [C][tile]
  pdl_launch_dependents();
  pdl_wait();
  const int chunk = blockIdx.x, h = blockIdx.y, c0 = (p.tile0 + blockIdx.z) * kDecayTile;
  int seq, t0, n;
  if (!locate_chunk(p.cu, p.n_seq, chunk, &seq, &t0, &n)) return;
  const int tid = threadIdx.x;
  const size_t ch = static_cast<size_t>(chunk) * p.H + h;
  const float* gKe = p.Ke + ch * kChunk * d;
  const float* gV = p.Uv + ch * kChunk * dv;
  copy_rows(sKe, gKe, n * d, tid);
  copy_tile(sV, gV, n, dv, c0, tid);
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  float* gN = p.N + ch * static_cast<size_t>(d) * dv;
  const int cc = 4 * (tid % 16);
  for (int k0 = 4 * (tid / 16); k0 < d; k0 += 4 * (kDecayThreads / 16)) {
    float acc[4][4];
    product_tn(acc, sKe, d, k0, sV, cc, n);
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c)
        if (c0 + cc + c < dv) gN[static_cast<size_t>(k0 + r) * dv + c0 + cc + c] = acc[r][c];
  }
}

// per state element: S_0 of every chunk replaces its N; the request's state moves to the end of the portion
__global__ void __launch_bounds__(kDecayThreads)
    decay_chunk_scan_kernel(ChunkArgs p) {
  pdl_launch_dependents();
  pdl_wait();
  const int seq = blockIdx.z, h = blockIdx.y;
  const int d = p.d, dv = p.dv;
  const int e = blockIdx.x * kDecayThreads + threadIdx.x;
  if (e >= d * dv) return;
  const int first = p.cu[seq], len = p.cu[seq + 1] - first;
  if (len <= 0) return;
  int chunk = 0;
  for (int s = 0; s < seq; ++s) chunk += (p.cu[s + 1] - p.cu[s] + kChunk - 1) / kChunk;
  const int k = e / dv;
  float* st = p.state + (static_cast<size_t>(p.slots[seq]) * p.H + h) * d * dv + e;
  float s = *st;
  const int n_chunks = (len + kChunk - 1) / kChunk;
  constexpr int kAhead = 8;  // the chain is one multiply-add a chunk: the loads are what takes time, so 8 fly at once
  for (int c0 = 0; c0 < n_chunks; c0 += kAhead) {
    float add[kAhead], eg[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      if (c0 + u < n_chunks) {
        const size_t ch = static_cast<size_t>(chunk + c0 + u) * p.H + h;
        add[u] = p.N[ch * static_cast<size_t>(d) * dv + e];
        eg[u] = p.Eg[ch * d + k];
      }
    }
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      if (c0 + u < n_chunks) {
        const size_t ch = static_cast<size_t>(chunk + c0 + u) * p.H + h;
        p.N[ch * static_cast<size_t>(d) * dv + e] = s;
        s = eg[u] * s + add[u];
      }
    }
  }
  *st = s;
}

// The rows of every chunk: [Q * a^(i+1) | B] times [S_0; V], one product whose inner index runs over the d state rows and then
// the chunk's tokens up to the row's own, 64 rows x 64 columns a block.
// Bound by the float units and the latency in front of them: a thread makes ROWS x 4 results, with ROWS = 8 twelve sixteen-byte
// reads for four inner indices and 128 multiply-adds (4: eight for 64), two multiply-adds an instruction, every sum in the
// order of the inner index.  The operands come in slices of 32 through a ring of three, 48 KB a block.  Eight rows a thread, four
// blocks of four warps on an SM, make the 512 blocks of 2,048 tokens, 8 heads and 128 x 128 states one wave (inside a step 30 -> 27
// us against whole operands of 80 KB); a grid that leaves an SM fewer than four wants the warps: four rows a thread, up to
// three blocks of eight warps (kOutWave).  The decayed sum with 8 heads of 64 x 128, us with 8 / 4 rows a thread: 37 tokens
// 21.3 / 20.7, 512 42.7 / 36.5, 1,500 48.8 / 45.3, 2,048 52.3 / 53.5; with 4 heads of 244 x 244 300 tokens 89.8 / 72.5.
// FOURS: four inner indices are summed by themselves before they enter a result, a quarter more instructions and a quarter
// of the long sum's roundings (the rows' error against float64 at d = 244 behind a given state 2.8e-7 -> 1.7e-7); chosen for the
// delta rule's keys from kFoursFrom entries on, which were always summed so.
constexpr int kOutK = 32, kOutStages = 3, kFoursFrom = 224, kOutWave = 3 * 148;
constexpr int kOutStage = kChunk * kOutK + kOutK * kDecayTile;  // floats

template <bool FOURS, int ROWS>
__global__ void __launch_bounds__(1024 / ROWS)
    decay_chunk_output_kernel(ChunkArgs p) {
  constexpr int kOutThreads = 1024 / ROWS;  // 64 rows x 64 columns
  extern __shared__ __align__(16) float sm[];
  const int d = p.d, dv = p.dv;
  pdl_launch_dependents();
  pdl_wait();
  const int chunk = blockIdx.x, h = blockIdx.y, c0 = (p.tile0 + blockIdx.z) * kDecayTile;
  int seq, t0, n;
  if (!locate_chunk(p.cu, p.n_seq, chunk, &seq, &t0, &n)) return;
  const int tid = threadIdx.x;
  const size_t ch = static_cast<size_t>(chunk) * p.H + h;
  const float* gQg = p.Qg + ch * kChunk * d;
  const float* gB = p.B + ch * kChunk * kChunk;
  const float* gS = p.N + ch * static_cast<size_t>(d) * dv;
  const float* gV = p.Uv + ch * kChunk * dv;
  const int n_state = (d + kOutK - 1) / kOutK, n_slices = n_state + (n + kOutK - 1) / kOutK;

  auto stage = [&](int s) {
    if (s < n_slices) {
      float* sA = sm + (s % kOutStages) * kOutStage;  // [C][32]
      float* sR = sA + kChunk * kOutK;                // [32][64]
      const bool own = s >= n_state;
      const int k0 = (own ? s - n_state : s) * kOutK, kn = min(kOutK, (own ? n : d) - k0);
      const float* a = own ? gB + k0 : gQg + k0;
      const int lda = own ? kChunk : d, ka = own ? kOutK : kn;  // (B's rows are whole: entries past the diagonal are not read)
      for (int e = tid; e < n * (kOutK / 4); e += kOutThreads) {
        const int i = e / (kOutK / 4), c = 4 * (e % (kOutK / 4));
        if (c < ka) cp_async16(sA + i * kOutK + c, a + static_cast<size_t>(i) * lda + c);
      }
      copy_tile<kOutThreads>(sR, (own ? gV : gS) + static_cast<size_t>(k0) * dv, kn, dv, c0, tid);
    }
    cp_async_commit();
  };

  // thread: rows i0 .. i0 + ROWS - 1, columns cc .. cc + 3 (rows at and beyond n hold stale values that are not stored)
  const int cc = 4 * (tid % 16), i0 = ROWS * (tid / 16);
  Pair acc[ROWS][2];
#pragma unroll
  for (int r = 0; r < ROWS; ++r) acc[r][0] = acc[r][1] = 0ull;
  // four inner indices from `k` of the slice; with `last`, only those up to last + r enter row r
  auto four = [&](const float* sA, const float* sR, int k, bool whole, int last) {
    float4 a[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) a[r] = *reinterpret_cast<const float4*>(sA + (i0 + r) * kOutK + k);
    if constexpr (FOURS) {
      if (whole) {
        Quad b[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) b[q] = quad(sR + (k + q) * kDecayTile + cc);
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
          const float av[4] = {a[r].x, a[r].y, a[r].z, a[r].w};
          Pair lo = 0ull, hi = 0ull;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const Pair a2 = pair(av[q], av[q]);
            lo = fma2(a2, b[q].lo, lo);
            hi = fma2(a2, b[q].hi, hi);
          }
          acc[r][0] = fma2(pair(1.f, 1.f), lo, acc[r][0]);
          acc[r][1] = fma2(pair(1.f, 1.f), hi, acc[r][1]);
        }
        return;
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const Quad b = quad(sR + (k + q) * kDecayTile + cc);
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        if (!whole && k + q > last + r) continue;
        const float av = q == 0 ? a[r].x : q == 1 ? a[r].y : q == 2 ? a[r].z : a[r].w;
        const Pair a2 = pair(av, av);
        acc[r][0] = fma2(a2, b.lo, acc[r][0]);
        acc[r][1] = fma2(a2, b.hi, acc[r][1]);
      }
    }
  };
  for (int s = 0; s < kOutStages - 1; ++s) stage(s);
  for (int s = 0; s < n_slices; ++s) {
    cp_async_wait<kOutStages - 2>();
    __syncthreads();  // slice s has landed for every thread, and slice s - 1's buffer is free
    stage(s + kOutStages - 1);
    const float* sA = sm + (s % kOutStages) * kOutStage;
    const float* sR = sA + kChunk * kOutK;
    if (i0 >= n) continue;
    if (s < n_state) {
      const int kn = min(kOutK, d - s * kOutK);
      for (int k = 0; k < kn; k += 4) four(sA, sR, k, true, 0);
    } else {
      const int last = i0 - (s - n_state) * kOutK;  // of the slice's tokens, the row i0's own
      int k = 0;
      for (; k + 3 <= last && k < kOutK; k += 4) four(sA, sR, k, true, 0);
      for (; k <= last + ROWS - 1 && k < kOutK; k += 4) four(sA, sR, k, false, last);
    }
  }
  if (i0 >= n) return;
  const bool pieces = dv % 4 == 0 && reinterpret_cast<uintptr_t>(p.out) % 16 == 0;
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    if (i0 + r >= n) break;
    float* o = p.out + static_cast<size_t>(t0 + i0 + r) * (p.H * dv) + h * dv + c0 + cc;
    const float2 lo = halves(acc[r][0]), hi = halves(acc[r][1]);
    if (pieces) {
      if (c0 + cc < dv) *reinterpret_cast<float4*>(o) = make_float4(lo.x, lo.y, hi.x, hi.y);
    } else {
      const float v[4] = {lo.x, lo.y, hi.x, hi.y};
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (c0 + cc + e < dv) o[e] = v[e];
    }
  }
}

// ----------------------------------------------------------------------------------------------
// The delta rule's link from chunk to chunk:  U = Uv - W S_0,  S_end = diag(exp L_end) S_0 + Ke^T U  with
// Ke = K * exp(L_end - L).  A block owns 8 columns of one head's state for one sequence and walks the sequence's chunks;
// U goes where Uv was and every chunk's starting state to N, so that the read-out o_i = (q_i * exp L_i)^T S_0 +
// sum_{j<=i} B_ij u_j of all chunks at once is the decayed sum's (decay_chunk_output_kernel with U as its values).
// Both products are made in 4 x 4 tiles with the summed index shared by 8 (4) lanes, two multiply-adds an instruction;
// the next chunk's W and Ke come by asynchronous copies meanwhile.  Bound by the latency of a link (barriers, reads, sums
// over lanes) on two warps a scheduler (37 % of issue slots, a warp every 5.5 cycles).  2,048 tokens and 8 heads of 128 x 128 (32
// links) inside a step: 70 us (72 alone with cold caches); with
// the summed index shared by 16 (8) lanes of 512 threads 95 us, in 2 x 2 (4 x 2) tiles shared by two lanes 99 us.
// (The form S_end = M S_0 + N with M = diag(exp L_end) - Ke^T W reads as many bytes a link, needs a launch of its own for M
// and N and leaves W S_0 to the read-out: its three launches took 50, 130 and 74 us behind the operands'.)
constexpr int kChainCols = 8;
constexpr int kChainThreads = 256;

inline size_t delta_chain_smem(int d, int n_buf) {
  return sizeof(float) * (static_cast<size_t>(n_buf) * 2 * kChunk * d + static_cast<size_t>(d + 4) * kChainCols + 2 * kChunk * kChainCols);
}

// D: the key size where it is known when compiling (the loops unroll and their addresses are constants), 0: p.d.
template <int D>
__global__ void __launch_bounds__(kChainThreads)
    delta_chunk_chain_kernel(ChunkArgs p, int n_buf) {
  extern __shared__ __align__(16) float sm[];
  constexpr int KT = D == 0 ? 2 : 1;      // 4-row tiles of S per thread (128 rows a pass; d <= 244)
  const int d = D ? D : p.d, dv = p.dv, d4 = d / 4;
  float* sIn = sm;                                                  // [n_buf][W: C x d | Ke: C x d]
  float* sS = sIn + static_cast<size_t>(n_buf) * 2 * kChunk * d;    // [8][ss]: the columns of S
  const int ss = d + 4;                                             // (a stride at which 4 slices of 2 columns fall into different banks)
  float* sU = sS + kChainCols * ss;                                 // [C][8][2]: every entry twice, as a pair
  pdl_launch_dependents();
  pdl_wait();
  const int seq = blockIdx.z, h = blockIdx.y, j0 = blockIdx.x * kChainCols;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int first = p.cu[seq], len = p.cu[seq + 1] - first;
  if (len <= 0) return;
  int chunk0 = 0;
  for (int s = 0; s < seq; ++s) chunk0 += (p.cu[s + 1] - p.cu[s] + kChunk - 1) / kChunk;
  const int n_chunks = (len + kChunk - 1) / kChunk;
  float* st = p.state + ((static_cast<size_t>(p.slots[seq]) * p.H + h) * d) * dv;
  auto unit = [&](int ci) { return static_cast<size_t>(chunk0 + ci) * p.H + h; };
  const int n_full = len / kChunk, last_rows = chunk_rows(len - n_full * kChunk);
  auto fetch = [&](int ci) {
    const float *gW = p.W + unit(ci) * kChunk * d, *gKe = p.Ke + unit(ci) * kChunk * d;
    float* dst = sIn + static_cast<size_t>(ci % n_buf) * 2 * kChunk * d;
    auto copy = [&](int e) {
      cp_async16(dst + 4 * e, gW + 4 * e);
      cp_async16(dst + kChunk * d + 4 * e, gKe + 4 * e);
    };
    if (ci < n_full) {
#pragma unroll 4
      for (int e = tid; e < kChunk * d4; e += kChainThreads) copy(e);
    } else {
      for (int e = tid; e < last_rows * d4; e += kChainThreads) copy(e);
    }
    cp_async_commit();
  };
  fetch(0);
  // product with W: rows u_row .., columns u_col .., the state's rows 4 m .. with m = slice mod 8; this thread keeps the
  // sums of row u_at, columns u_c and the next
  const int u_col = 4 * (lane & 1), u_slice = (lane >> 1) & 7, u_row = 4 * (2 * warp + (lane >> 4));
  const int u_at = u_row + (u_slice >> 1), u_c = u_col + 2 * (u_slice & 1);
  // state update: rows 4 s_tile .., columns s_col .., the chunk's rows j = slice mod 4; kept: row s_slice
  const int s_col = 4 * (warp & 1), s_slice = lane >> 3, s_tile = (warp >> 1) * 8 + (lane & 7);
  for (int e = tid; e < d * kChainCols; e += kChainThreads) {
    const int r = e / kChainCols, c = e % kChainCols;
    sS[c * ss + r] = (j0 + c < dv) ? st[static_cast<size_t>(r) * dv + j0 + c] : 0.f;
  }
  float uv[2] = {0.f, 0.f}, eg[KT];
  const bool col0 = j0 + u_c < dv, col1 = j0 + u_c + 1 < dv;
  auto read_ahead = [&](int ci) {   // the small operands of a chunk, a link ahead of their use
    const float* gU = p.Uv + unit(ci) * kChunk * dv + static_cast<size_t>(u_at) * dv + j0 + u_c;
    if (col0) uv[0] = gU[0];
    if (col1) uv[1] = gU[1];
#pragma unroll
    for (int t = 0; t < KT; ++t) {
      const int k = 4 * (s_tile + 32 * t) + s_slice;
      eg[t] = k < d ? p.Eg[unit(ci) * d + k] : 0.f;
    }
  };
  read_ahead(0);
  // (a sequence's last chunk may hold fewer rows; with their count known when compiling the others' links are 4 % shorter)
  auto link = [&](int ci, auto full) {
    constexpr bool FULL = decltype(full)::value;
    const int rows = FULL ? kChunk : last_rows;
    cp_async_wait<0>();
    __syncthreads();        // W and Ke of this chunk and everyone's rows of S are there; everyone is done with the chunk before
    if (n_buf > 1 && ci + 1 < n_chunks) fetch(ci + 1);
    const float* W = sIn + static_cast<size_t>(ci % n_buf) * 2 * kChunk * d;
    const float* Ke = W + kChunk * d;
    if (FULL || 8 * warp < rows) {
      Pair acc[4][4];
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[r][c] = 0;
#pragma unroll 4
      for (int m = u_slice; m < d4; m += 8) {
        Quad w[4], s[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) w[r] = quad(W + (u_row + r) * d + 4 * m);
#pragma unroll
        for (int c = 0; c < 4; ++c) s[c] = quad(sS + (u_col + c) * ss + 4 * m);
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
          for (int c = 0; c < 4; ++c) acc[r][c] = fma2(w[r].lo, s[c].lo, acc[r][c]);
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
          for (int c = 0; c < 4; ++c) acc[r][c] = fma2(w[r].hi, s[c].hi, acc[r][c]);
      }
      float v[4][4];
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const float2 two = halves(acc[r][c]);
          v[r][c] = two.x + two.y;
        }
      // summed over the 8 slices (lane bits 1 to 3); a lane keeps row slice >> 1, columns 2 (slice & 1) and the next
      float x[8], y[4], z[2];
      const bool b3 = lane & 8, b2 = lane & 4, b1 = lane & 2;
#pragma unroll
      for (int e = 0; e < 8; ++e)
        x[e] = (b3 ? v[2 + e / 4][e % 4] : v[e / 4][e % 4]) + __shfl_xor_sync(0xffffffffu, b3 ? v[e / 4][e % 4] : v[2 + e / 4][e % 4], 8);
#pragma unroll
      for (int e = 0; e < 4; ++e) y[e] = (b2 ? x[4 + e] : x[e]) + __shfl_xor_sync(0xffffffffu, b2 ? x[e] : x[4 + e], 4);
#pragma unroll
      for (int e = 0; e < 2; ++e) z[e] = (b1 ? y[2 + e] : y[e]) + __shfl_xor_sync(0xffffffffu, b1 ? y[e] : y[2 + e], 2);
      const float u0 = uv[0] - z[0], u1 = uv[1] - z[1];
      *reinterpret_cast<float4*>(sU + 2 * (u_at * kChainCols + u_c)) = make_float4(u0, u0, u1, u1);
      float* gU = p.Uv + unit(ci) * kChunk * dv + static_cast<size_t>(u_at) * dv + j0 + u_c;
      if (col0) gU[0] = u0;
      if (col1) gU[1] = u1;
    }
    float eg_now[KT];
#pragma unroll
    for (int t = 0; t < KT; ++t) eg_now[t] = eg[t];
    __syncthreads();        // U is whole; everyone has read S
    if (ci + 1 < n_chunks) read_ahead(ci + 1);
    float* gN = p.N + unit(ci) * static_cast<size_t>(d) * dv;
#pragma unroll
    for (int t = 0; t < KT; ++t) {
      const int m = s_tile + 32 * t;
      const bool mine = D == 128 || m < d4;
      Pair acc[2][4];   // rows 4 m, 4 m + 1 and 4 m + 2, 4 m + 3
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[0][c] = acc[1][c] = 0;
      if (mine) {
        auto add_row = [&](int j) {
          const Quad k = quad(Ke + j * d + 4 * m);
          const float* u = sU + 2 * (j * kChainCols + s_col);
          const Quad u01 = quad(u), u23 = quad(u + 4);
          const Pair uu[4] = {u01.lo, u01.hi, u23.lo, u23.hi};
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            acc[0][c] = fma2(k.lo, uu[c], acc[0][c]);
            acc[1][c] = fma2(k.hi, uu[c], acc[1][c]);
          }
        };
        if constexpr (FULL) {
#pragma unroll 8
          for (int j = s_slice; j < kChunk; j += 4) add_row(j);
        } else {
#pragma unroll 4
          for (int j = s_slice; j < rows; j += 4) add_row(j);
        }
      }
      float v[4][4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float2 top = halves(acc[0][c]), low = halves(acc[1][c]);
        v[0][c] = top.x;
        v[1][c] = top.y;
        v[2][c] = low.x;
        v[3][c] = low.y;
      }
      // summed over the 4 slices (lane bits 3 and 4); a lane keeps row 4 m + slice
      float x[8], y[4];
      const bool b4 = lane & 16, b3 = lane & 8;
#pragma unroll
      for (int e = 0; e < 8; ++e)
        x[e] = (b4 ? v[2 + e / 4][e % 4] : v[e / 4][e % 4]) + __shfl_xor_sync(0xffffffffu, b4 ? v[e / 4][e % 4] : v[2 + e / 4][e % 4], 16);
#pragma unroll
      for (int e = 0; e < 4; ++e) y[e] = (b3 ? x[4 + e] : x[e]) + __shfl_xor_sync(0xffffffffu, b3 ? x[e] : x[4 + e], 8);
      if (mine) {
        float* at = sS + s_col * ss + 4 * m + s_slice;
        const float4 old = make_float4(at[0], at[ss], at[2 * ss], at[3 * ss]);
        at[0] = eg_now[t] * old.x + y[0];
        at[ss] = eg_now[t] * old.y + y[1];
        at[2 * ss] = eg_now[t] * old.z + y[2];
        at[3 * ss] = eg_now[t] * old.w + y[3];
        float* to = gN + static_cast<size_t>(4 * m + s_slice) * dv + j0 + s_col;  // the chunk's starting state
        if (dv % 4 == 0) {
          if (j0 + s_col < dv) *reinterpret_cast<float4*>(to) = old;
        } else {
          const float o[4] = {old.x, old.y, old.z, old.w};
#pragma unroll
          for (int c = 0; c < 4; ++c)
            if (j0 + s_col + c < dv) to[c] = o[c];
        }
      }
    }
    if (n_buf == 1 && ci + 1 < n_chunks) {
      __syncthreads();      // everyone is done with the one buffer
      fetch(ci + 1);
    }
  };
  for (int ci = 0; ci < n_full; ++ci) link(ci, std::true_type{});
  if (n_full < n_chunks) link(n_full, std::false_type{});
  __syncthreads();
  for (int e = tid; e < d * kChainCols; e += kChainThreads) {
    const int r = e / kChainCols, c = e % kChainCols;
    if (j0 + c < dv) st[static_cast<size_t>(r) * dv + j0 + c] = sS[c * ss + r];
  }
}

constexpr int kMostSmem = 220 * 1024;

// Largest key sizes: what the blocks that hold a chunk's operands take of shared memory (200 KB and more).
inline int largest_key(int rule) { return rule == kRuleDelta ? 244 : rule == kRuleWkv ? 280 : 352; }

inline size_t prepare_smem(int d, int rule) {
  return rule == kRuleWkv ? wkv_prepare_smem(d) : rule == kRuleDelta ? delta_prepare_smem(d) : decay_prepare_smem(d);
}

template <typename S, int RULE>
int launch_chunked(ChunkArgs a, int n_chunks, cudaStream_t stream) {
  constexpr bool DELTA = RULE == kRuleDelta;
  const int d = a.d, tiles = (a.dv + kDecayTile - 1) / kDecayTile;
  void (*prep)(ChunkArgs) = nullptr;
  if constexpr (RULE == kRuleWkv) prep = wkv_prepare_kernel<S>;
  else if constexpr (DELTA) prep = delta_prepare_kernel<S>;
  else prep = decay_prepare_kernel<S, RULE>;
  const size_t unit = 4 * sizeof(S);
  auto whole = [&](const void* ptr, long long ld) { return reinterpret_cast<uintptr_t>(ptr) % unit == 0 && ld % 4 == 0; };
  a.vec_in = whole(a.q, a.ld_q) && whole(a.k, a.ld_k) && whole(a.v, a.ld_v) && (!DELTA || whole(a.a, a.ld_a)) &&
             (RULE != kRuleWkv || (reinterpret_cast<uintptr_t>(a.a) % 16 == 0 && a.ld_a % 4 == 0 && reinterpret_cast<uintptr_t>(a.dt_bias) % 16 == 0));
  // (One limit for all calls: were it the call's own, a thread with smaller values could lower it between another thread's
  // asking and its launch, which would then be refused.)
  auto allow = [](auto kernel, size_t bytes) {
    return bytes <= 48 * 1024 ? cudaSuccess : cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMostSmem);
  };
  size_t sp = prepare_smem(d, RULE);
  const size_t with_v = sp + sizeof(float) * kChunk * static_cast<size_t>(a.dv);
  // The prepare kernel makes the state's part too where at least two of its blocks share an SM with the values beside the
  // keys and there are blocks for more than half of the SMs; larger sizes and shorter portions keep the launch of its own,
  // whose blocks split the columns (8 heads of 64 x 128, us so and in the prepare launch: 64 tokens 25 / 36, 300 37 / 37, 800 46 / 40;
  // time mixing, 16 heads of 64 x 64: 128 tokens 37 / 49, 300 43 / 35).  States of up to 64 x 64 of the decayed sums are too little
  // work for a launch however few the blocks (4 heads of it, 512 tokens: 33 / 25).
  const bool blocks_enough = static_cast<long long>(n_chunks) * a.H >= 80 || (RULE != kRuleWkv && d * a.dv <= 64 * 64);
  a.with_state = !DELTA && d % 8 == 0 && a.dv % 8 == 0 && with_v <= 110 * 1024 && blocks_enough;
  if (a.with_state) sp = with_v;
  const size_t s1 = sizeof(float) * kChunk * (static_cast<size_t>(d) + kDecayTile);
  const size_t s3 = sizeof(float) * kOutStages * kOutStage;
  const int n_buf = delta_chain_smem(d, 2) <= 200 * 1024 ? 2 : 1;
  const size_t s2 = delta_chain_smem(d, n_buf);
  const bool one_wave = static_cast<long long>(n_chunks) * a.H * tiles <= kOutWave;
  const int out_threads = one_wave ? 1024 / 4 : 1024 / 8;
  auto output = DELTA && d >= kFoursFrom ? (one_wave ? decay_chunk_output_kernel<true, 4> : decay_chunk_output_kernel<true, 8>)
                                         : (one_wave ? decay_chunk_output_kernel<false, 4> : decay_chunk_output_kernel<false, 8>);
  auto chain = d == 128 ? delta_chunk_chain_kernel<128> : d == 64 ? delta_chunk_chain_kernel<64> : delta_chunk_chain_kernel<0>;
  cudaError_t e = allow(prep, sp);
  if (e == cudaSuccess) e = DELTA ? allow(chain, s2) : allow(decay_chunk_state_kernel, s1);
  if (e == cudaSuccess) e = allow(output, s3);
  if (e != cudaSuccess) return static_cast<int>(e);
  auto for_tiles = [&](auto launch) {
    for (a.tile0 = 0; a.tile0 < tiles; a.tile0 += 65535) launch(std::min(tiles - a.tile0, 65535));
  };
  launch_pdl(prep, dim3(n_chunks, a.H), dim3(DELTA ? kPrepThreads : RULE == kRuleWkv ? kWkvThreads : kDecayPrepThreads), sp, stream, a);
  if (DELTA) {
    launch_pdl(chain, dim3((a.dv + kChainCols - 1) / kChainCols, a.H, a.n_seq), dim3(kChainThreads), s2, stream, a, n_buf);
  } else {
    if (!a.with_state)
      for_tiles([&](int n) { launch_pdl(decay_chunk_state_kernel, dim3(n_chunks, a.H, n), dim3(kDecayThreads), s1, stream, a); });
    launch_pdl(decay_chunk_scan_kernel, dim3((d * a.dv + kDecayThreads - 1) / kDecayThreads, a.H, a.n_seq),
               dim3(kDecayThreads), 0, stream, a);
  }
  for_tiles([&](int n) { launch_pdl(output, dim3(n_chunks, a.H, n), dim3(out_threads), s3, stream, a); });
  return launch_status();
}

}  // namespace pmm

// Whether the chunked kernels take this key size (whole float4 rows, operands of a chunk in one block's
// shared memory).
// rule: kRuleDecay .. kRuleWkv (0: the decayed sum, 1: the delta rule, 2: retention, 3: time mixing).
PMM_EXPORT int pmm_recurrent_chunked_supported(int d, int rule) {
  return d > 0 && d % 4 == 0 && d <= pmm::largest_key(rule) ? 1 : 0;
}

// Floats of scratch per (chunk, head).
PMM_EXPORT long long pmm_recurrent_chunked_scratch(int d, int dv, int rule) {
  // Ke, Qg, Uv, B, Eg; N (then every chunk's starting state); for the delta rule also W
  const long long w = rule == pmm::kRuleDelta ? static_cast<long long>(pmm::kChunk) * d : 0;
  return static_cast<long long>(pmm::kChunk) * (2 * d + dv + pmm::kChunk) + static_cast<long long>(d) * dv + w + d;
}

namespace pmm {
// The arrays of the scratch.  Every one starts on a 16-byte boundary, as the 16-byte copies and stores of the kernels need (of N
// too, whose rows are read in 16 bytes where dv is a multiple of 4): d is a multiple of 4, so every array before another holds a
// multiple of four floats.
inline void place_scratch(ChunkArgs& p, float* s, size_t ch, bool delta) {
  const int d = p.d, dv = p.dv;
  p.Ke = s; s += ch * kChunk * d;
  p.Qg = s; s += ch * kChunk * d;
  p.B = s; s += ch * kChunk * kChunk;
  p.N = s; s += ch * static_cast<size_t>(d) * dv;
  if (delta) {
    p.W = s; s += ch * kChunk * d;
  }
  p.Uv = s; s += ch * kChunk * dv;
  p.Eg = s;
}
}  // namespace pmm

// n_chunks = sum over sequences of ceil(tokens / 64) (an upper bound is fine: surplus blocks leave).
// scratch: n_chunks * H * pmm_recurrent_chunked_scratch(...) floats, 16-byte aligned.  Other arguments as
// pmm_delta_scan / pmm_decay_scan (decay != nullptr selects the decayed sum).
PMM_EXPORT int pmm_recurrent_chunked(const void* q, long long ld_q, const void* k, long long ld_k, const void* v,
                                     long long ld_v, const void* beta, long long ld_beta, const void* a,
                                     long long ld_a, const float* dt_bias, const float* a_log, const float* decay,
                                     float* state, const int* cu, const int* slots, float* out, float* scratch,
                                     int n_seq, int n_chunks, int H, int Hk, int d, int dv, float unit_eps,
                                     float q_scale, int dtype, cudaStream_t stream) {
  if (n_seq <= 0 || n_chunks <= 0) return 0;
  const bool delta = decay == nullptr;
  if (H <= 0 || Hk <= 0 || H % Hk || dv <= 0 || H > 65535 || n_seq > 65535 || !scratch ||
      reinterpret_cast<uintptr_t>(scratch) % 16 || !pmm_recurrent_chunked_supported(d, delta ? pmm::kRuleDelta : pmm::kRuleDecay))
    return PMM_ERR_BAD_ARGUMENT;
  pmm::ChunkArgs p{};
  p.q = q; p.ld_q = ld_q; p.k = k; p.ld_k = ld_k; p.v = v; p.ld_v = ld_v;
  p.beta = beta; p.ld_beta = ld_beta; p.a = a; p.ld_a = ld_a;
  p.dt_bias = dt_bias; p.a_log = a_log; p.decay = decay;
  p.cu = cu; p.n_seq = n_seq; p.H = H; p.Hk = Hk; p.d = d; p.dv = dv;
  p.unit_eps = unit_eps; p.q_scale = q_scale;
  const size_t ch = static_cast<size_t>(n_chunks) * H;
  pmm::place_scratch(p, scratch, ch, delta);
  p.state = state; p.slots = slots; p.out = out;
  PMM_DISPATCH_DTYPE(dtype, S, {
    return delta ? pmm::launch_chunked<S, pmm::kRuleDelta>(p, n_chunks, stream) : pmm::launch_chunked<S, pmm::kRuleDecay>(p, n_chunks, stream);
  });
  return 0;
}

// kRuleRetention (decay given) and kRuleWkv in chunks: arguments as pmm_recurrence, n_chunks and scratch as above.
PMM_EXPORT int pmm_recurrence_chunked(const void* q, long long ld_q, const void* k, long long ld_k, const void* v, long long ld_v,
                                      const float* decay, float k_scale, const int* positions, const float* inv_freq,
                                      int rot_dims, int half_layout, const float* a, long long ld_a, const float* a_bias,
                                      const float* bonus, float* state, const int* cu, const int* slots, float* out,
                                      float* scratch, int n_seq, int n_chunks, int H, int d, int dv, int dtype,
                                      cudaStream_t stream) {
  if (n_seq <= 0 || n_chunks <= 0) return 0;
  if (H <= 0 || dv <= 0 || H > 65535 || n_seq > 65535 || !scratch || reinterpret_cast<uintptr_t>(scratch) % 16 ||
      !pmm_recurrent_chunked_supported(d, decay ? pmm::kRuleRetention : pmm::kRuleWkv) || rot_dims < 0 || rot_dims > d ||
      rot_dims % 2 || (rot_dims > 0 && (!positions || !inv_freq)) || (!decay && (!a || !a_bias || !bonus)))
    return PMM_ERR_BAD_ARGUMENT;
  pmm::ChunkArgs p{};
  p.q = q; p.ld_q = ld_q; p.k = k; p.ld_k = ld_k; p.v = v; p.ld_v = ld_v;
  p.a = a; p.ld_a = ld_a; p.dt_bias = a_bias; p.decay = decay; p.bonus = bonus; p.k_scale = k_scale;
  p.rot = {positions, inv_freq, rot_dims, half_layout};
  p.cu = cu; p.n_seq = n_seq; p.H = H; p.Hk = H; p.d = d; p.dv = dv;
  pmm::place_scratch(p, scratch, static_cast<size_t>(n_chunks) * H, false);
  p.state = state; p.slots = slots; p.out = out;
  PMM_DISPATCH_DTYPE(dtype, S, {
    return decay ? pmm::launch_chunked<S, pmm::kRuleRetention>(p, n_chunks, stream)
                 : pmm::launch_chunked<S, pmm::kRuleWkv>(p, n_chunks, stream);
  });
  return 0;
}
