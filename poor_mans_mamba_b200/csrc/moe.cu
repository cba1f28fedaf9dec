// Routed feed-forward (mixture of experts): router with top-k choice, the plan that sorts the
// (token, choice) pairs by expert, grouped products over the sorted rows, and the weighted sum.
//
//   z = x Wr^T + br (float; Wr, br float);  the `top` largest z are chosen (the lower index wins a tie),
//   p = softmax over the chosen z only;
//   pairs (t, j) are sorted by expert: offsets[e] .. offsets[e+1] are expert e's rows of `perm`,
//   perm[i] = t * top + j;
//   act[i]  = glu(x[perm[i] / top] Wgu_e^T)        [gate | up] rows of expert e, clamped gated activation
//   y[perm[i]] = act[i] Wd_e^T                     storage type
//   out[t] = sum_j p[t, j] y[t * top + j] (+ shared[t])
//
// Everything stays on the device: the grouped products are launched for an upper bound of row
// tiles, sum_e ceil(n_e / TM) <= floor(A / TM) + min(E, A) with A = T * top, and a block beyond the
// last tile leaves.  A row's result does not depend on which other rows share its tile.
#include "common.cuh"
#include "mma_helpers.cuh"
#include "moe_tile.cuh"
#include <cmath>

namespace pmm {

// A block routes TOK tokens: their rows wait in shared memory as floats, every warp takes one expert (one token) or two
// (several tokens) at a time and reads a router row once (16 bytes a lane and access) for all TOK dot
// products; then a warp per token picks the `top` largest logits and norms their exponentials.
// A chain of reads and reductions, bound by their latency: a warp's first router rows are read before the wait for the
// kernel before this one (they are weights), and up to 32 experts are ranked by one lane each against all others at once
// (`ranked`) where picking them one after the other takes ten exchanges between lanes apiece.  16 experts, 4 chosen in 2
// of 4 groups, width 1,024, inside a step: 8 tokens 11 -> 4.5 us.  Of many tokens' 19,000 clocks 3,900 went to rows read one
// piece after the other behind an integer division, 5,000 to 80 exchanges a warp for its 16 sums and 4,000 to the ranking's
// chain: a row's pieces are read together, sums over lanes are halved as they are exchanged (`warp_sums`, the same
// order), the ranking's reads go out eight at a time.  Alone, us: 2,048 tokens 10.4 -> 8.0, 4,096 20.2 -> 15.5, 512 6.5 -> 5.7; 8,192
// of width 2,048, 32 experts 97 -> 83.  What is left most is the products' reads of the rows from shared memory.
constexpr int kRouteAhead = 8;   // sixteen-byte pieces of a router row a lane holds before the wait (128 columns each)

// This lane's place (0: the largest; the lower index wins a tie) among values v[0 .. n - 1], n <= 32, none of them NaN.
__device__ __forceinline__ int ranked(const float* v, int n, int lane) {
  const float mine = lane < n ? v[lane] : -INFINITY;
  int rank = 0;
  for (int e0 = 0; e0 < n; e0 += 8) {  // eight reads in flight
    float o[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) o[k] = v[min(e0 + k, n - 1)];
#pragma unroll
    for (int k = 0; k < 8; ++k) rank += (e0 + k < n && (o[k] > mine || (o[k] == mine && e0 + k < lane))) ? 1 : 0;
  }
  return rank;
}
// v[0] + v[1] + ... + v[n - 1] in this order, eight reads in flight.
__device__ __forceinline__ float sum_in_order(const float* v, int n) {
  float sum = 0.f;
  for (int j0 = 0; j0 < n; j0 += 8) {
    float o[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) o[k] = v[min(j0 + k, n - 1)];
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (j0 + k < n) sum += o[k];
  }
  return sum;
}
// The sums over a warp's lanes of N values each (a power of two, up to 32): lane l gets that of value l / (32 / N), added in
// warp_sum's order, for N + log2(32 / N) exchanges instead of 5 N.
template <int N>
__device__ __forceinline__ float warp_sums(const float (&v)[N], int lane, int o = 16) {
  if constexpr (N == 1) {
    float sum = v[0];
    for (; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    return sum;
  } else {
    const bool high = lane & o;
    float half[N / 2];
#pragma unroll
    for (int i = 0; i < N / 2; ++i)
      half[i] = (high ? v[N / 2 + i] : v[i]) + __shfl_xor_sync(0xffffffffu, high ? v[i] : v[N / 2 + i], o);
    return warp_sums(half, lane, o >> 1);
  }
}
// Whether one lane an expert can rank them: the picks of a row with NaN or infinite entries are left to the serial form.
__device__ __forceinline__ bool all_finite(const float* v, int n, int lane) {
  return n <= 32 && __all_sync(0xffffffffu, lane >= n || fabsf(v[lane]) < INFINITY);
}

template <typename S, int TOK, int WARPS>
__global__ void __launch_bounds__(WARPS * 32)
    moe_route_kernel(const S* __restrict__ x, long long ld_x, const float* __restrict__ w,
                     const float* __restrict__ bias, int* __restrict__ ids, float* __restrict__ weights, int T, int D,
                     int E, int top, int scored, const float* __restrict__ correction, int groups, int keep,
                     float scale, const float* __restrict__ gate_w, float* __restrict__ gate_out) {
  extern __shared__ __align__(16) float route_smem[];  // rows [TOK][Dpad] | logits [TOK][E] (scored: | scores, group scores [TOK][2E])
  const int Dpad = (D + 3) & ~3;
  float* rows = route_smem;
  float* logits = route_smem + TOK * Dpad;
  pdl_launch_dependents();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int t0 = blockIdx.x * TOK;
  const int nt = min(TOK, T - t0);
  const bool vec = (D & 3) == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0 && (reinterpret_cast<uintptr_t>(gate_w) & 15) == 0;
  // (gate_w: one more row, whose product goes through a sigmoid into gate_out[t]: a gate per token that reads the
  // router's input, such as a shared expert's)
  const int n_rows = E + (gate_w ? 1 : 0);
  constexpr int kPer = TOK == 1 ? 1 : 2;  // experts a warp makes at a time: several tokens' rows are read once for both
  constexpr int kRouteWarps = WARPS;
  auto router_row = [&](int e) { return e < E ? w + static_cast<size_t>(e) * D : gate_w; };
  float4 ahead[kPer][kRouteAhead];
  if (vec) {
#pragma unroll
    for (int q = 0; q < kPer; ++q)
#pragma unroll
      for (int k = 0; k < kRouteAhead; ++k)
        if (warp * kPer + q < n_rows && lane * 4 + 128 * k < D)
          ahead[q][k] = *reinterpret_cast<const float4*>(router_row(warp * kPer + q) + lane * 4 + 128 * k);
  }
  // (weights and divisions of the ranking, ahead of the wait as well)
  const float correction0 = scored && correction && lane < E ? correction[lane] : 0.f;
  const int per = scored && groups > 1 ? E / groups : 1, lane_group = scored && groups > 1 ? lane / per : 0;
  pdl_wait();
  pdl_written(x);
  if ((D & 3) == 0 && ld_x % 4 == 0 && reinterpret_cast<uintptr_t>(x) % (4 * sizeof(S)) == 0) {
    constexpr int kParts = WARPS / TOK;  // warps a row
    const int r = warp / kParts, part = warp % kParts;
    const S* from = x + static_cast<long long>(t0 + min(r, nt - 1)) * ld_x;
#pragma unroll 8
    for (int c = 4 * (part * 32 + lane); c < D; c += 128 * kParts)
      *reinterpret_cast<float4*>(rows + r * Dpad + c) = r < nt ? ldf4(from + c) : make_float4(0.f, 0.f, 0.f, 0.f);
  } else {
    for (int r = 0; r < TOK; ++r)
      for (int i = threadIdx.x; i < Dpad; i += blockDim.x)
        rows[r * Dpad + i] = (r < nt && i < D) ? ldf(x + static_cast<long long>(t0 + r) * ld_x + i) : 0.f;
  }
  __syncthreads();
  for (int e0 = warp * kPer; e0 < n_rows; e0 += kRouteWarps * kPer) {
    const int n_here = min(kPer, n_rows - e0);
    float acc[kPer][TOK];
#pragma unroll
    for (int q = 0; q < kPer; ++q)
#pragma unroll
      for (int r = 0; r < TOK; ++r) acc[q][r] = 0.f;
    if (vec) {
      auto piece = [&](int i, const float4 (&wv)[kPer]) {
#pragma unroll
        for (int r = 0; r < TOK; ++r) {
          const float4 xv = *reinterpret_cast<const float4*>(rows + r * Dpad + i);
#pragma unroll
          for (int q = 0; q < kPer; ++q) acc[q][r] += xv.x * wv[q].x + xv.y * wv[q].y + xv.z * wv[q].z + xv.w * wv[q].w;
        }
      };
      int done = lane * 4;
      if (e0 == warp * kPer) {
#pragma unroll
        for (int k = 0; k < kRouteAhead; ++k)
          if (lane * 4 + 128 * k < D) {
            float4 wv[kPer];
#pragma unroll
            for (int q = 0; q < kPer; ++q) wv[q] = q < n_here ? ahead[q][k] : make_float4(0.f, 0.f, 0.f, 0.f);
            piece(lane * 4 + 128 * k, wv);
          }
        done += 128 * kRouteAhead;
      }
#pragma unroll 4
      for (int i = done; i < D; i += 128) {
        float4 wv[kPer];
#pragma unroll
        for (int q = 0; q < kPer; ++q)
          wv[q] = q < n_here ? *reinterpret_cast<const float4*>(router_row(e0 + q) + i) : make_float4(0.f, 0.f, 0.f, 0.f);
        piece(i, wv);
      }
    } else {
      for (int i = lane; i < D; i += 32) {
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
          const float wv = q < n_here ? router_row(e0 + q)[i] : 0.f;
#pragma unroll
          for (int r = 0; r < TOK; ++r) acc[q][r] += rows[r * Dpad + i] * wv;
        }
      }
    }
    float of_lane[kPer * TOK];
#pragma unroll
    for (int q = 0; q < kPer; ++q)
#pragma unroll
      for (int r = 0; r < TOK; ++r) of_lane[q * TOK + r] = acc[q][r];
    const float sum = warp_sums(of_lane, lane);
    constexpr int kLanes = 32 / (kPer * TOK);  // that hold the same sum
    const int q = lane / kLanes / TOK, r = lane / kLanes % TOK, e = e0 + q;
    if (lane % kLanes == 0 && q < n_here) {
      if (e < E) logits[r * E + e] = sum + (bias ? bias[e] : 0.f);
      else if (r < nt) gate_out[t0 + r] = 1.f / (1.f + expf(-sum));
    }
  }
  __syncthreads();
  if (scored) {
    // Scores s = sigmoid(z) (scored == 2: s = softmax(z) over all experts, a group's score is its largest choice
    // score, and the weights are the chosen s times scale, not divided by their sum; scored == 3: sigmoids whose
    // weights are not divided by their sum either).  The choice runs on s + correction, among the experts of the `keep` groups (of `groups`
    // equal groups of neighbours) whose two largest choice scores sum highest; every other expert's choice score is
    // -inf.  The weights are the chosen s over their sum (+ 1e-20), times scale.  The lower index wins a tie.
    float* extra = logits + TOK * E;
    for (int r = warp; r < nt; r += kRouteWarps) {
      float* z = logits + r * E;         // becomes the choice scores
      float* sc = extra + r * 2 * E;     // s
      float* gs = sc + E;                // group scores
      if (scored == 2) {
        // scores: the softmax of z over all experts
        float zmax = -INFINITY;
        for (int e = lane; e < E; e += 32) zmax = fmaxf(zmax, z[e]);
        zmax = warp_max(zmax);
        float zsum = 0.f;
        for (int e = lane; e < E; e += 32) {
          const float ev = expf(z[e] - zmax);
          sc[e] = ev;
          zsum += ev;
        }
        const float zinv = 1.f / warp_sum(zsum);
        for (int e = lane; e < E; e += 32) {
          const float sv = sc[e] * zinv;
          sc[e] = sv;
          z[e] = sv + (e < 32 ? correction0 : correction ? correction[e] : 0.f);
        }
      } else {
        for (int e = lane; e < E; e += 32) {
          const float sv = 1.f / (1.f + expf(-z[e]));
          sc[e] = sv;
          z[e] = sv + (e < 32 ? correction0 : correction ? correction[e] : 0.f);
        }
      }
      __syncwarp();
      const bool at_once = all_finite(z, E, lane);
      if (groups > 1) {
        for (int g = lane; g < groups; g += 32) {
          float a = -INFINITY, b = -INFINITY;  // the largest and the second largest
          for (int e0 = 0; e0 < per; e0 += 8) {  // eight reads in flight
            float o[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) o[k] = z[g * per + min(e0 + k, per - 1)];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              const float v = o[k];
              if (e0 + k < per) {
                if (v > a) { b = a; a = v; } else if (v > b) { b = v; }
              }
            }
          }
          gs[g] = (per > 1 && scored != 2) ? a + b : a;
        }
        __syncwarp();
        // the `keep` best groups are marked by +inf in gs; then the others' experts drop out
        const bool groups_at_once = at_once && all_finite(gs, groups, lane);
        if (groups_at_once) {
          const bool kept = ranked(gs, groups, lane) < keep;
          __syncwarp();
          if (lane < groups && kept) gs[lane] = INFINITY;
          __syncwarp();
        }
        for (int j = groups_at_once ? keep : 0; j < keep; ++j) {
          float best = -INFINITY;
          int arg = 0x7fffffff;
          for (int g = lane; g < groups; g += 32) {
            const float v = gs[g];
            if (v != INFINITY && (v > best || (v == best && g < arg) || arg == 0x7fffffff)) { best = v; arg = g; }
          }
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) {
            const float ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int oa = __shfl_xor_sync(0xffffffffu, arg, o);
            if (oa != 0x7fffffff && (arg == 0x7fffffff || ob > best || (ob == best && oa < arg))) { best = ob; arg = oa; }
          }
          if (lane == 0 && arg < groups) gs[arg] = INFINITY;
          __syncwarp();
        }
        for (int e = lane; e < E; e += 32)
          if (gs[e < 32 ? lane_group : e / per] != INFINITY) z[e] = -INFINITY;
        __syncwarp();
      }
      if (at_once) {
        const int place = ranked(z, E, lane);
        const bool chosen = lane < E && place < top;
        __syncwarp();
        if (chosen) z[place] = sc[lane];  // the chosen scores in their order
        __syncwarp();
        const float denom = sum_in_order(z, top);
        const float inv = scored >= 2 ? scale : scale / (denom + 1e-20f);
        if (chosen) {
          ids[static_cast<size_t>(t0 + r) * top + place] = lane;
          weights[static_cast<size_t>(t0 + r) * top + place] = sc[lane] * inv;
        }
        continue;
      }
      float denom = 0.f;
      for (int j = 0; j < top; ++j) {
        float best = -INFINITY;
        int arg = 0x7fffffff;
        for (int e = lane; e < E; e += 32) {
          const float v = z[e];
          if (v > best || (v == best && e < arg)) { best = v; arg = e; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const float ob = __shfl_xor_sync(0xffffffffu, best, o);
          const int oa = __shfl_xor_sync(0xffffffffu, arg, o);
          if (ob > best || (ob == best && oa < arg)) { best = ob; arg = oa; }
        }
        if (arg >= E) arg = j;  // nothing left to choose from: keep the indices valid
        const float p = sc[arg];
        denom += p;
        if (lane == 0) {
          ids[static_cast<size_t>(t0 + r) * top + j] = arg;
          weights[static_cast<size_t>(t0 + r) * top + j] = p;
          z[arg] = -INFINITY;
        }
        __syncwarp();
      }
      const float inv = scored >= 2 ? scale : scale / (denom + 1e-20f);
      for (int j = lane; j < top; j += 32) weights[static_cast<size_t>(t0 + r) * top + j] *= inv;
    }
    return;
  }
  for (int r = warp; r < nt; r += kRouteWarps) {
    float* z = logits + r * E;
    if (all_finite(z, E, lane)) {
      const int place = ranked(z, E, lane);
      const float mine = lane < E ? z[lane] : -INFINITY;
      const unsigned top_lane = __ballot_sync(0xffffffffu, lane < E && place == 0);
      const float p = expf(mine - z[__ffs(top_lane) - 1]);
      const bool chosen = lane < E && place < top;
      __syncwarp();
      if (chosen) z[place] = p;
      __syncwarp();
      const float denom = sum_in_order(z, top);
      const float inv = 1.f / denom;
      if (chosen) {
        ids[static_cast<size_t>(t0 + r) * top + place] = lane;
        weights[static_cast<size_t>(t0 + r) * top + place] = p * inv;
      }
      continue;
    }
    float first = 0.f, denom = 0.f;
    for (int j = 0; j < top; ++j) {
      float best = -INFINITY;
      int arg = 0x7fffffff;
      for (int e = lane; e < E; e += 32) {
        const float v = z[e];
        if (v > best || (v == best && e < arg)) { best = v; arg = e; }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oa = __shfl_xor_sync(0xffffffffu, arg, o);
        if (ob > best || (ob == best && oa < arg)) { best = ob; arg = oa; }
      }
      if (arg >= E) arg = j;  // every logit left is NaN or -inf: keep the indices valid
      if (j == 0) first = best;
      const float p = expf(best - first);
      denom += p;
      if (lane == 0) {
        ids[static_cast<size_t>(t0 + r) * top + j] = arg;
        weights[static_cast<size_t>(t0 + r) * top + j] = p;
        z[arg] = -INFINITY;
      }
      __syncwarp();
    }
    const float inv = 1.f / denom;
    for (int j = lane; j < top; j += 32) weights[static_cast<size_t>(t0 + r) * top + j] *= inv;
  }
}

// One block: rows per expert, their exclusive sums, and the exclusive sums of the row tiles.
__global__ void __launch_bounds__(1024)
    moe_plan_kernel(const int* __restrict__ ids, int A, int E, int tile_rows, int* __restrict__ offsets,
                    int* __restrict__ tile_start) {
  extern __shared__ int plan_counts[];  // [E]
  pdl_launch_dependents();
  for (int e = threadIdx.x; e < E; e += blockDim.x) plan_counts[e] = 0;
  pdl_wait();
  pdl_written(ids);
  __syncthreads();
  for (int i = threadIdx.x; i < A; i += blockDim.x) {
    const int e = ids[i];
    if (e >= 0 && e < E) atomicAdd(&plan_counts[e], 1);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int rows = 0, tiles = 0;
    for (int e = 0; e < E; ++e) {
      offsets[e] = rows;
      tile_start[e] = tiles;
      rows += plan_counts[e];
      tiles += (plan_counts[e] + tile_rows - 1) / tile_rows;
    }
    offsets[E] = rows;
    tile_start[E] = tiles;
  }
}

// One block per expert: its pairs in the order of their index (stable, so the plan is the same every time).
// A thread owns a run of consecutive pairs: it counts its matches, the block sums the counts before each
// thread, and the thread writes its matches from there.
__global__ void __launch_bounds__(1024)
    moe_fill_kernel(const int* __restrict__ ids, int A, const int* __restrict__ offsets, int* __restrict__ perm) {
  __shared__ int warp_total[32];
  pdl_launch_dependents();
  pdl_wait();
  const int e = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int base = offsets[e];
  if (offsets[e + 1] == base) return;
  const int run = (A + blockDim.x - 1) / blockDim.x;
  const int i0 = min(A, static_cast<int>(threadIdx.x) * run), i1 = min(A, i0 + run);
  int mine = 0;
  for (int i = i0; i < i1; ++i) mine += ids[i] == e;
  int incl = mine;  // inclusive sum over the warp
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) warp_total[warp] = incl;
  __syncthreads();
  int before = base + incl - mine;
  for (int w2 = 0; w2 < warp; ++w2) before += warp_total[w2];
  for (int i = i0; i < i1; ++i)
    if (ids[i] == e) perm[before++] = i;
}

// Plan and fill in one launch for up to kPlanExperts experts: a block per expert counts all pairs (a histogram a warp, so that
// few threads meet on a counter), sums the experts before its own, and writes its pairs in their order; block 0 writes the
// offsets.  At 8,192 pairs of 16 experts, inside a step: 4.8 us, the two launches 8.
constexpr int kPlanExperts = 128;

__global__ void __launch_bounds__(1024)
    moe_plan_fill_kernel(const int* __restrict__ ids, int A, int E, int tile_rows, int* __restrict__ offsets,
                         int* __restrict__ tile_start, int* __restrict__ perm) {
  extern __shared__ int plan_hist[];  // [32 warps][E] | counts [E]
  __shared__ int warp_total[32];
  int* counts = plan_hist + 32 * E;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  pdl_launch_dependents();
  for (int i = threadIdx.x; i < 32 * E; i += blockDim.x) plan_hist[i] = 0;
  __syncthreads();
  pdl_wait();
  pdl_written(ids);
  const int e = blockIdx.x;
  const int run = (A + 1023) / 1024;  // a thread owns a run of consecutive pairs
  const int i0 = min(A, static_cast<int>(threadIdx.x) * run), i1 = min(A, i0 + run);
  int mine = 0;
  for (int i = i0; i < i1; ++i) {
    const int id = ids[i];
    if (id >= 0 && id < E) atomicAdd(&plan_hist[warp * E + id], 1);
    mine += id == e;
  }
  int incl = mine;  // inclusive sum over the warp
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) warp_total[warp] = incl;
  __syncthreads();
  for (int i = threadIdx.x; i < E; i += blockDim.x) {
    int c = 0;
#pragma unroll 8
    for (int w = 0; w < 32; ++w) c += plan_hist[w * E + i];
    counts[i] = c;
  }
  __syncthreads();
  if (e == 0)
    for (int i = threadIdx.x; i <= E; i += blockDim.x) {
      int rows = 0, tiles = 0;
      for (int o = 0; o < i; ++o) {
        rows += counts[o];
        tiles += (counts[o] + tile_rows - 1) / tile_rows;
      }
      offsets[i] = rows;
      tile_start[i] = tiles;
    }
  if (counts[e] == 0) return;
  int before = incl - mine;
  for (int o = 0; o < e; ++o) before += counts[o];
  for (int w = 0; w < warp; ++w) before += warp_total[w];
  for (int i = i0; i < i1; ++i)
    if (ids[i] == e) perm[before++] = i;
}

// The whole plan of a step with few pairs (a decode step) in one block and one launch: a thread per expert
// counts its pairs, one thread sums, then every expert's thread writes its pairs in their order.
constexpr int kPlanSmallPairs = 512;

__global__ void __launch_bounds__(256)
    moe_plan_small_kernel(const int* __restrict__ ids, int A, int E, int tile_rows, int* __restrict__ offsets,
                          int* __restrict__ tile_start, int* __restrict__ perm) {
  extern __shared__ int plan_small[];  // ids [A] | counts, then starts [E]
  int* ids_s = plan_small;
  int* cnt = plan_small + A;
  pdl_launch_dependents();
  pdl_wait();
  for (int i = threadIdx.x; i < A; i += blockDim.x) ids_s[i] = ids[i];
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    int c = 0;
    for (int i = 0; i < A; ++i) c += ids_s[i] == e;
    cnt[e] = c;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int rows = 0, tiles = 0;
    for (int e = 0; e < E; ++e) {
      const int c = cnt[e];
      offsets[e] = rows;
      tile_start[e] = tiles;
      cnt[e] = rows;
      rows += c;
      tiles += (c + tile_rows - 1) / tile_rows;
    }
    offsets[E] = rows;
    tile_start[E] = tiles;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    int pos = cnt[e];
    for (int i = 0; i < A; ++i)
      if (ids_s[i] == e) perm[pos++] = i;
  }
}

__device__ __forceinline__ float clamped_glu(float g, float u, float limit, float alpha, float shift) {
  g = fminf(g, limit);
  u = fminf(fmaxf(u, -limit), limit);
  return g / (1.f + expf(-alpha * g)) * (u + shift);
}

// The ungated experts' activation: max(z, 0)^2.
__device__ __forceinline__ float relu_squared(float z) {
  z = fmaxf(z, 0.f);
  return z * z;
}

// The grouped product in float arithmetic on the CUDA cores, for any sizes and both storage types.
// UP (the [gate | up] product with the activation): a = x [T, K], row i reads x[perm[i] / top]; w [E, 2N, K];
// out = act [A, N] in the storage type.  Otherwise (the down product): a = act [A, K]; w [E, N, K];
// out = y [A, N] in the storage type, row perm[i].
constexpr int kGenRows = 32, kGenCols = 32, kGenK = 32;

template <typename S, bool UP>
__global__ void __launch_bounds__(256)
    moe_gemm_generic_kernel(const S* __restrict__ a, long long ld_a, const S* __restrict__ w,
                            const int* __restrict__ perm, const int* __restrict__ offsets,
                            const int* __restrict__ tile_start, int E, int top, int K, int N, float limit, float alpha,
                            float shift, int ungated, const float* __restrict__ row_w, void* __restrict__ out) {
  __shared__ float As[kGenRows][kGenK + 1];
  __shared__ float Bs[UP ? 2 : 1][kGenCols][kGenK + 1];
  __shared__ int src_row[kGenRows];
  pdl_launch_dependents();
  pdl_wait();
  int e, row0, row1;
  if (!moe_tile(blockIdx.y, offsets, tile_start, E, kGenRows, e, row0, row1)) return;
  const int n0 = blockIdx.x * kGenCols;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  if (threadIdx.x < kGenRows) {
    const int i = row0 + threadIdx.x;
    src_row[threadIdx.x] = i < row1 ? ((UP || ungated) ? perm[i] / top : i) : -1;
  }
  __syncthreads();
  const S* we = w + static_cast<size_t>(e) * (UP ? 2 : 1) * N * K;
  float acc[UP ? 2 : 1][4];
#pragma unroll
  for (int m = 0; m < (UP ? 2 : 1); ++m)
#pragma unroll
    for (int r = 0; r < 4; ++r) acc[m][r] = 0.f;
  for (int k0 = 0; k0 < K; k0 += kGenK) {
    for (int idx = threadIdx.x; idx < kGenRows * kGenK; idx += 256) {
      const int r = idx / kGenK, k = idx - r * kGenK;
      const int src = src_row[r];
      As[r][k] = (src >= 0 && k0 + k < K) ? ldf(a + static_cast<long long>(src) * ld_a + k0 + k) : 0.f;
    }
    for (int idx = threadIdx.x; idx < kGenCols * kGenK; idx += 256) {
      const int c = idx / kGenK, k = idx - c * kGenK;
      const bool ok = n0 + c < N && k0 + k < K;
      Bs[0][c][k] = ok ? ldf(we + static_cast<size_t>(n0 + c) * K + k0 + k) : 0.f;
      if (UP) Bs[UP ? 1 : 0][c][k] = ok ? ldf(we + static_cast<size_t>(N + n0 + c) * K + k0 + k) : 0.f;
    }
    __syncthreads();
#pragma unroll 8
    for (int k = 0; k < kGenK; ++k) {
      const float b0 = Bs[0][tx][k];
      const float b1 = UP ? Bs[UP ? 1 : 0][tx][k] : 0.f;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const float av = As[ty * 4 + r][k];
        acc[0][r] += av * b0;
        if (UP) acc[UP ? 1 : 0][r] += av * b1;
      }
    }
    __syncthreads();
  }
  if (n0 + tx >= N) return;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int i = row0 + ty * 4 + r;
    if (i >= row1) continue;
    if (UP) {
      const float rw = row_w ? row_w[perm[i]] : 1.f;
      stf(static_cast<S*>(out) + static_cast<size_t>(i) * N + n0 + tx,
          clamped_glu(rw * acc[0][r], rw * acc[UP ? 1 : 0][r], limit, alpha, shift));
    } else {
      // (ungated: the activation's rows stay in the order of the sorted pairs, like the gated form's)
      stf(static_cast<S*>(out) + static_cast<size_t>(ungated ? i : perm[i]) * N + n0 + tx,
          ungated ? relu_squared(acc[0][r]) : acc[0][r]);
    }
  }
}

// The grouped product on the tensor cores (mma.sync m16n8k16, bfloat16 operands, float accumulation):
// tiles of 64 rows x 64 columns (UP: 64 gate and 64 up columns), K in slices of 32 through a
// two-stage ring of 16-byte asynchronous copies.  Needs K % 8 == 0 and 16-byte aligned rows.
constexpr int kMmaRows = 64, kMmaCols = 64, kMmaK = 32, kMmaPad = 8;

template <bool UP>
__global__ void __launch_bounds__(128)
    moe_gemm_mma_kernel(const bf16* __restrict__ a, long long ld_a, const bf16* __restrict__ w,
                        const int* __restrict__ perm, const int* __restrict__ offsets,
                        const int* __restrict__ tile_start, int E, int top, int K, int N, float limit, float alpha,
                        float shift, int ungated, const float* __restrict__ row_w, void* __restrict__ out) {
  constexpr int BROWS = UP ? 2 * kMmaCols : kMmaCols;
  constexpr int LD = kMmaK + kMmaPad;  // 40 elements = 80 bytes: ldmatrix rows fall into different banks
  __shared__ __align__(16) bf16 As[2][kMmaRows][LD];
  __shared__ __align__(16) bf16 Bs[2][BROWS][LD];
  __shared__ int src_row[kMmaRows];
  __shared__ int dst_row[kMmaRows];
  pdl_launch_dependents();
  pdl_wait();
  int e, row0, row1;
  if (!moe_tile(blockIdx.y, offsets, tile_start, E, kMmaRows, e, row0, row1)) return;
  const int n0 = blockIdx.x * kMmaCols;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x < kMmaRows) {
    const int i = row0 + threadIdx.x;
    const int p = i < row1 ? perm[i] : -1;
    src_row[threadIdx.x] = i < row1 ? ((UP || ungated) ? p / top : i) : -1;
    dst_row[threadIdx.x] = p;
  }
  __syncthreads();
  const bf16* we = w + static_cast<size_t>(e) * (UP ? 2 : 1) * N * K;

  auto stage = [&](int buf, int k0) {
    // 64 rows x 4 pieces of 8 elements for A; BROWS x 4 for B
    for (int idx = threadIdx.x; idx < kMmaRows * 4; idx += 128) {
      const int r = idx >> 2, c = (idx & 3) * 8;
      const int src = src_row[r];
      const bool ok = src >= 0 && k0 + c < K;
      cp_async16(&As[buf][r][c], ok ? a + static_cast<long long>(src) * ld_a + k0 + c : a, ok);
    }
    for (int idx = threadIdx.x; idx < BROWS * 4; idx += 128) {
      const int r = idx >> 2, c = (idx & 3) * 8;
      const int col = UP ? (r < kMmaCols ? n0 + r : N + n0 + (r - kMmaCols)) : n0 + r;
      const bool ok = (UP ? (r < kMmaCols ? n0 + r : n0 + r - kMmaCols) : n0 + r) < N && k0 + c < K;
      cp_async16(&Bs[buf][r][c], ok ? we + static_cast<size_t>(col) * K + k0 + c : we, ok);
    }
    cp_async_commit();
  };

  float acc[BROWS / 8][4];
#pragma unroll
  for (int j = 0; j < BROWS / 8; ++j)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[j][q] = 0.f;

  const int n_slices = (K + kMmaK - 1) / kMmaK;
  stage(0, 0);
  for (int s = 0; s < n_slices; ++s) {
    if (s + 1 < n_slices) {
      stage((s + 1) & 1, (s + 1) * kMmaK);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    const int buf = s & 1;
#pragma unroll
    for (int kk = 0; kk < kMmaK; kk += 16) {
      unsigned af[4];
      // the warp's 16 rows: matrices (rows 0-7, k 0-7), (rows 8-15, k 0-7), (rows 0-7, k 8-15), (rows 8-15, k 8-15)
      ldmatrix_x4(af[0], af[1], af[2], af[3], &As[buf][warp * 16 + (lane & 15)][kk + ((lane >> 4) << 3)]);
#pragma unroll
      for (int j = 0; j < BROWS / 16; ++j) {
        unsigned b0, b1, b2, b3;
        // 16 weight rows (two groups of 8 columns of the result) x 16 k
        ldmatrix_x4(b0, b1, b2, b3, &Bs[buf][j * 16 + (lane & 7) + ((lane >> 4) << 3)][kk + (((lane >> 3) & 1) << 3)]);
        mma_bf16(acc[2 * j], af, b0, b1);
        mma_bf16(acc[2 * j + 1], af, b2, b3);
      }
    }
    __syncthreads();
  }

  // accumulator layout: acc[j][0..1] row lane/4, columns j*8 + (lane%4)*2 + {0,1}; acc[j][2..3] row lane/4 + 8
  const int r_lo = warp * 16 + (lane >> 2), c_in = (lane & 3) * 2;
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const int r = r_lo + half * 8;
    const int i = row0 + r;
    if (i >= row1) continue;
    const float rw = (UP && row_w) ? row_w[dst_row[r]] : 1.f;
#pragma unroll
    for (int j = 0; j < kMmaCols / 8; ++j) {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int col = n0 + j * 8 + c_in + q;
        if (col >= N) continue;
        if (UP) {
          const float g = rw * acc[j][half * 2 + q], u = rw * acc[UP ? j + kMmaCols / 8 : j][half * 2 + q];
          static_cast<bf16*>(out)[static_cast<size_t>(i) * N + col] = __float2bfloat16_rn(clamped_glu(g, u, limit, alpha, shift));
        } else {
          const float val = acc[j][half * 2 + q];
          static_cast<bf16*>(out)[static_cast<size_t>(ungated ? i : dst_row[r]) * N + col] =
              __float2bfloat16_rn(ungated ? relu_squared(val) : val);
        }
      }
    }
  }
}

// The same product for steps of few pairs (decode steps), where an expert has a handful of rows and the
// launch is a read of the chosen experts' matrices: tiles of 16 rows, the four warps share the
// columns, K in slices through a four-stage ring, so that a block keeps three slices in flight.  What it takes is a block's
// walk along K, times the waves of blocks (two on an SM).  64 columns and slices of 64 for the down product, whose K is an
// expert's width.  The up product, whose K is the model's width, has two forms: NARROW, 32 gate and 32 up columns and slices
// of 128, walks twice the blocks in 0.4 to 0.6 of the time each (8 tokens, 4 of 16 experts of 256, width 1,024, inside a step: 14.5
// against 10 us), which loses where a wave becomes two (4 tokens, 6 of 64 experts of 512: 17.0 against 19.0 us; 32
// tokens 32.5 against 39.7); `few_narrow` decides.
constexpr int kFewRows = 16, kFewStages = 4;
template <bool UP, bool NARROW>
struct FewTile {
  static constexpr int kCols = NARROW ? 32 : 64, kK = NARROW ? 128 : 64, kLd = kK + 8, kBRows = UP ? 2 * kCols : kCols;
  static constexpr int kStageElems = (kFewRows + kBRows) * kLd;
};

// Whether the up product of A pairs takes its narrow tiles: waves of blocks, times 5/8 for a narrow one, with the tiles that
// evenly chosen experts have (the experts met by A draws, and past 8 rows an expert the second tiles of some).
inline bool few_narrow(int A, int E, int N) {
  const double met = E * (1.0 - std::pow(1.0 - 1.0 / E, A)) + (A > 8 * E ? A / 32.0 : 0.0);
  constexpr int kSlots = 2 * 148;
  auto waves = [&](int cols) { return static_cast<int>(std::ceil(met * ((N + cols - 1) / cols) / kSlots)); };
  return 5 * waves(32) <= 8 * waves(64);
}

template <bool UP, bool NARROW>
__global__ void __launch_bounds__(128)
    moe_gemm_few_kernel(const bf16* __restrict__ a, long long ld_a, const bf16* __restrict__ w,
                        const int* __restrict__ perm, const int* __restrict__ offsets,
                        const int* __restrict__ tile_start, int E, int top, int K, int N, float limit, float alpha,
                        float shift, int ungated, const float* __restrict__ row_w, bf16* __restrict__ out) {
  using Tile = FewTile<UP, NARROW>;
  constexpr int kCols = Tile::kCols, kK = Tile::kK, kLd = Tile::kLd, BROWS = Tile::kBRows, kStageElems = Tile::kStageElems;
  constexpr int NJ = kCols / 32;  // groups of 8 columns a warp (of the gate's and as many of the up matrix's)
  extern __shared__ __align__(16) unsigned char few_smem[];
  bf16* ring = reinterpret_cast<bf16*>(few_smem);
  __shared__ int src_row[kFewRows];
  __shared__ int dst_row[kFewRows];
  pdl_launch_dependents();
  pdl_wait();
  int e, row0, row1;
  if (!moe_tile(blockIdx.y, offsets, tile_start, E, kFewRows, e, row0, row1)) return;
  const int n0 = blockIdx.x * kCols;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x < kFewRows) {
    const int i = row0 + threadIdx.x;
    const int p = i < row1 ? perm[i] : -1;
    src_row[threadIdx.x] = i < row1 ? ((UP || ungated) ? p / top : i) : -1;
    dst_row[threadIdx.x] = p;
  }
  __syncthreads();
  const bf16* we = w + static_cast<size_t>(e) * (UP ? 2 : 1) * N * K;

  auto stage = [&](int buf, int k0) {
    bf16* As = ring + static_cast<size_t>(buf) * kStageElems;
    bf16* Bs = As + kFewRows * kLd;
    constexpr int kPieces = kK / 8;  // of 8 elements in a row of the slice
    for (int idx = threadIdx.x; idx < kFewRows * kPieces; idx += 128) {
      const int r = idx / kPieces, c = (idx % kPieces) * 8;
      const int src = src_row[r];
      const bool ok = src >= 0 && k0 + c < K;
      cp_async16(As + r * kLd + c, ok ? a + static_cast<long long>(src) * ld_a + k0 + c : a, ok);
    }
#pragma unroll
    for (int idx = threadIdx.x; idx < BROWS * kPieces; idx += 128) {
      const int r = idx / kPieces, c = (idx % kPieces) * 8;
      const int col = UP ? (r < kCols ? n0 + r : n0 + r - kCols) : n0 + r;
      const bool ok = col < N && k0 + c < K;
      const size_t wrow = UP && r >= kCols ? static_cast<size_t>(N) + col : col;
      cp_async16(Bs + r * kLd + c, ok ? we + wrow * K + k0 + c : we, ok);
    }
    cp_async_commit();
  };

  float acc[UP ? 2 * NJ : NJ][4];   // UP: the gate's columns, then the up matrix's
#pragma unroll
  for (int j = 0; j < (UP ? 2 * NJ : NJ); ++j)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[j][q] = 0.f;

  const int n_slices = (K + kK - 1) / kK;
#pragma unroll
  for (int s = 0; s < kFewStages - 1; ++s) {
    if (s < n_slices) stage(s, s * kK);
    else cp_async_commit();
  }
  for (int s = 0; s < n_slices; ++s) {
    cp_async_wait<kFewStages - 2>();  // slice s has landed
    __syncthreads();                  // ... for every thread, and slice s - 1's buffer is free
    if (s + kFewStages - 1 < n_slices) stage((s + kFewStages - 1) % kFewStages, (s + kFewStages - 1) * kK);
    else cp_async_commit();
    const bf16* As = ring + static_cast<size_t>(s % kFewStages) * kStageElems;
    const bf16* Bs = As + kFewRows * kLd;
#pragma unroll
    for (int kk = 0; kk < kK; kk += NARROW ? 32 : 16) {
      unsigned af[4], b0, b1, b2, b3;
      ldmatrix_x4(af[0], af[1], af[2], af[3], As + (lane & 15) * kLd + kk + ((lane >> 4) << 3));
      if (NARROW) {
        // 8 rows of the gate's (the up) matrix x 32 k, in two steps of 16
        unsigned ag[4];
        ldmatrix_x4(ag[0], ag[1], ag[2], ag[3], As + (lane & 15) * kLd + kk + 16 + ((lane >> 4) << 3));
#pragma unroll
        for (int part = 0; part < (UP ? 2 : 1); ++part) {
          ldmatrix_x4(b0, b1, b2, b3, Bs + (part * kCols + warp * 8 + (lane & 7)) * kLd + kk + ((lane >> 3) << 3));
          mma_bf16(acc[part], af, b0, b1);
          mma_bf16(acc[part], ag, b2, b3);
        }
      } else {
#pragma unroll
        for (int part = 0; part < (UP ? 2 : 1); ++part) {
          ldmatrix_x4(b0, b1, b2, b3, Bs + (part * kCols + warp * 16 + (lane & 7) + ((lane >> 4) << 3)) * kLd + kk + (((lane >> 3) & 1) << 3));
          mma_bf16(acc[part * NJ], af, b0, b1);
          mma_bf16(acc[part * NJ + NJ - 1], af, b2, b3);
        }
      }
    }
  }

  const int c_in = (lane & 3) * 2;
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const int r = (lane >> 2) + half * 8;
    const int i = row0 + r;
    if (i >= row1) continue;
    const float rw = (UP && row_w) ? row_w[dst_row[r]] : 1.f;
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int col = n0 + (warp * NJ + j) * 8 + c_in + q;
        if (col >= N) continue;
        if (UP) {
          out[static_cast<size_t>(i) * N + col] =
              __float2bfloat16_rn(clamped_glu(rw * acc[j][half * 2 + q], rw * acc[UP ? NJ + j : j][half * 2 + q], limit, alpha, shift));
        } else {
          const float val = acc[j][half * 2 + q];
          out[static_cast<size_t>(ungated ? i : dst_row[r]) * N + col] = __float2bfloat16_rn(ungated ? relu_squared(val) : val);
        }
      }
    }
  }
}

// out[t] = sum_j p[t, j] y[t * top + j] (weights null: every p is 1) (+ shared[t], times shared_gate[t] where there is one); y, shared and out in the storage type, the sum in float.
template <typename S>
__global__ void __launch_bounds__(256)
    moe_combine_kernel(const S* __restrict__ y, const float* __restrict__ weights, const S* __restrict__ shared,
                       const float* __restrict__ shared_gate, S* __restrict__ out, int D, int top) {
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x;
  for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < D; i += gridDim.y * blockDim.x) {
    float acc = 0.f;
    for (int j = 0; j < top; ++j)
      acc += (weights ? weights[static_cast<size_t>(t) * top + j] : 1.f) * ldf(y + (static_cast<size_t>(t) * top + j) * D + i);
    if (shared) acc += (shared_gate ? shared_gate[t] : 1.f) * ldf(shared + static_cast<size_t>(t) * D + i);
    stf(out + static_cast<size_t>(t) * D + i, acc);
  }
}

// The same sums for rows of whole sixteen-byte pieces: a thread makes one piece (8 values in bfloat16, 4 in float) of one
// token, so that all of its reads are in flight together.  2,048 tokens of 4 experts, width 1,024, inside a step: 4.4 us,
// a value a thread and read 8.2.
template <typename S>
__global__ void __launch_bounds__(256)
    moe_combine_vec_kernel(const S* __restrict__ y, const float* __restrict__ weights, const S* __restrict__ shared,
                           const float* __restrict__ shared_gate, S* __restrict__ out, int T, int D, int top) {
  constexpr int V = 16 / sizeof(S);
  pdl_launch_dependents();
  pdl_wait();
  const unsigned per_row = D / V;
  const unsigned at = blockIdx.x * blockDim.x + threadIdx.x;   // (below 2^32: the launch sees to it)
  const int t = static_cast<int>(at / per_row), c = static_cast<int>(at - t * per_row) * V;
  if (t >= T) return;
  float acc[V];
#pragma unroll
  for (int v = 0; v < V; ++v) acc[v] = 0.f;
  auto add = [&](const S* row, float p) {
    float x[V];
#pragma unroll
    for (int v = 0; v < V; v += 4) {
      const float4 q = ldf4(row + v);
      x[v] = q.x, x[v + 1] = q.y, x[v + 2] = q.z, x[v + 3] = q.w;
    }
#pragma unroll
    for (int v = 0; v < V; ++v) acc[v] += p * x[v];
  };
#pragma unroll 4
  for (int j = 0; j < top; ++j)
    add(y + (static_cast<size_t>(t) * top + j) * D + c, weights ? weights[static_cast<size_t>(t) * top + j] : 1.f);
  if (shared) add(shared + static_cast<size_t>(t) * D + c, shared_gate ? shared_gate[t] : 1.f);
#pragma unroll
  for (int v = 0; v < V; v += 4) stf4(out + static_cast<size_t>(t) * D + c + v, make_float4(acc[v], acc[v + 1], acc[v + 2], acc[v + 3]));
}

}  // namespace pmm

namespace pmm {
template <typename S, int TOK, int WARPS = 8>
int launch_route(const void* x, long long ld_x, const float* w, const float* bias, int* ids, float* weights, int T, int D,
                 int E, int top, int scored, const float* correction, int groups, int keep, float scale,
                 const float* gate_w, float* gate_out, cudaStream_t stream) {
  const size_t smem = (static_cast<size_t>(TOK) * ((D + 3) & ~3) + static_cast<size_t>(TOK) * E * (scored ? 3 : 1)) * sizeof(float);
  if (smem > 200 * 1024) return PMM_ERR_BAD_ARGUMENT;
  auto kern = moe_route_kernel<S, TOK, WARPS>;
  if (smem > 48 * 1024) {
    cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (err != cudaSuccess) return static_cast<int>(err);
  }
  launch_pdl(kern, dim3((T + TOK - 1) / TOK), dim3(WARPS * 32), smem, stream, static_cast<const S*>(x), ld_x, w, bias,
             ids, weights, T, D, E, top, scored, correction, groups, keep, scale, gate_w, gate_out);
  return launch_status();
}
}  // namespace pmm

// scored == 0: the `top` largest logits, weights their softmax.  scored != 0: scores sigmoid(z); the choice runs on
// score + correction (may be null) within the `keep` best of `groups` groups of neighbours; weights are the chosen
// scores over their sum, times scale (scored == 3: the chosen scores times scale).  scored == 2: scores softmax(z) over all experts; groups are ranked by their
// largest choice score; weights are the chosen scores times scale.
PMM_EXPORT int pmm_moe_route(const void* x, long long ld_x, const float* w, const float* bias, int* ids, float* weights,
                             int T, int D, int E, int top, int scored, const float* correction, int groups, int keep,
                             float scale, const float* gate_w, float* gate_out, int dtype, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (D <= 0 || E <= 0 || top <= 0 || top > E || (gate_w && !gate_out)) return PMM_ERR_BAD_ARGUMENT;
  if (scored && (groups <= 0 || E % groups || keep <= 0 || keep > groups || top > keep * (E / groups)))
    return PMM_ERR_BAD_ARGUMENT;
  // Few tokens: a block each, of 16 warps while two such blocks an SM are one wave (296 tokens; past it they are two: 300 tokens of
  // width 2,048, 64 experts 31.7 us), of 8 warps while three are (444; 21.1 us).  More: four or eight tokens a block, which
  // read the router a quarter or an eighth as often (the same at 511 tokens, a block of 16 warps a token 32.9, four tokens a
  // block 26.5 us).
  // Rows too long for that keep a block of 8 warps a token.
  constexpr int kSms = 148;
  auto room = [&](int tok) { return (static_cast<size_t>(tok) * (((D + 3) & ~3) + 3 * E)) * sizeof(float) <= 96 * 1024; };
  PMM_DISPATCH_DTYPE(dtype, S, {
    if (T >= 1024 && room(8))
      return pmm::launch_route<S, 8>(x, ld_x, w, bias, ids, weights, T, D, E, top, scored, correction, groups, keep, scale,
                                     gate_w, gate_out, stream);
    if (T > 3 * kSms && room(4))
      return pmm::launch_route<S, 4>(x, ld_x, w, bias, ids, weights, T, D, E, top, scored, correction, groups, keep, scale,
                                     gate_w, gate_out, stream);
    if (T <= 2 * kSms)
      return pmm::launch_route<S, 1, 16>(x, ld_x, w, bias, ids, weights, T, D, E, top, scored, correction, groups, keep, scale,
                                         gate_w, gate_out, stream);
    return pmm::launch_route<S, 1>(x, ld_x, w, bias, ids, weights, T, D, E, top, scored, correction, groups, keep, scale,
                                   gate_w, gate_out, stream);
  });
  return 0;
}

// ids [A] -> offsets [E + 1], tile_start [E + 1] (row tiles of `tile_rows`), perm [A].  One launch for up to
// kPlanSmallPairs pairs or kPlanExperts experts, else two.
PMM_EXPORT int pmm_moe_plan(const int* ids, int A, int E, int tile_rows, int* offsets, int* tile_start, int* perm,
                            cudaStream_t stream) {
  if (A <= 0) return 0;
  if (E <= 0 || E > 4096 || tile_rows <= 0) return PMM_ERR_BAD_ARGUMENT;
  if (A <= pmm::kPlanSmallPairs) {
    pmm::launch_pdl(pmm::moe_plan_small_kernel, dim3(1), dim3(256), static_cast<size_t>(A + E) * sizeof(int), stream, ids,
                    A, E, tile_rows, offsets, tile_start, perm);
    return pmm::launch_status();
  }
  if (E <= pmm::kPlanExperts) {
    pmm::launch_pdl(pmm::moe_plan_fill_kernel, dim3(E), dim3(1024), static_cast<size_t>(33) * E * sizeof(int), stream, ids, A, E,
                    tile_rows, offsets, tile_start, perm);
    return pmm::launch_status();
  }
  pmm::launch_pdl(pmm::moe_plan_kernel, dim3(1), dim3(1024), static_cast<size_t>(E) * sizeof(int), stream, ids, A, E,
                  tile_rows, offsets, tile_start);
  int rc = pmm::launch_status();
  if (rc != 0) return rc;
  pmm::launch_pdl(pmm::moe_fill_kernel, dim3(E), dim3(1024), 0, stream, ids, A, static_cast<const int*>(offsets), perm);
  return pmm::launch_status();
}

// 0: float products on the CUDA cores, 1: mma.sync tiles, 2: mma.sync tiles for few pairs
PMM_EXPORT int pmm_moe_tile_rows(int tensor_cores) {
  return tensor_cores == 2 ? pmm::kFewRows : tensor_cores ? pmm::kMmaRows : pmm::kGenRows;
}

// up == 1: a = x [T, K] (ld_a), w [E, 2N, K], out act [A, N] (storage type).  up == 0: a = act [A, K], w [E, N, K],
// out y [A, N] in the storage type.  up == 2 (ungated experts): a = x [T, K], w [E, N, K], out act [A, N] = max(x W^T, 0)^2
// in the order of the sorted pairs.  row_w [A] (up == 1, or null): pair i's input is row_w[perm[i]] * x, applied to its
// gate and up sums before the activation.  tensor_cores != 0 needs bfloat16, K % 8 == 0, ld_a % 8 == 0 and 16-byte aligned a, w; the
// plan must have been made with pmm_moe_tile_rows(tensor_cores) rows a tile.
PMM_EXPORT int pmm_moe_gemm(const void* a, long long ld_a, const void* w, const int* perm, const int* offsets,
                            const int* tile_start, int A, int E, int top, int K, int N, int up, float limit, float alpha,
                            float shift, const float* row_w, void* out, int tensor_cores, int dtype, cudaStream_t stream) {
  if (A <= 0) return 0;
  if (row_w && up != 1) return PMM_ERR_BAD_ARGUMENT;
  if (E <= 0 || top <= 0 || K <= 0 || N <= 0 || up < 0 || up > 2) return PMM_ERR_BAD_ARGUMENT;
  const int ungated = up == 2 ? 1 : 0;
  if (ungated) up = 0;
  const int tile_rows = pmm_moe_tile_rows(tensor_cores);
  const int row_tiles = A / tile_rows + (E < A ? E : A);
  if (row_tiles > 65535) return PMM_ERR_BAD_ARGUMENT;
  if (tensor_cores) {
    if (dtype != PMM_DTYPE_BF16 || K % 8 || ld_a % 8 || reinterpret_cast<uintptr_t>(a) % 16 ||
        reinterpret_cast<uintptr_t>(w) % 16)
      return PMM_ERR_BAD_ARGUMENT;
    if (tensor_cores == 2) {
      auto few = [&](auto kern, int cols, int stage_elems) {
        const size_t smem = static_cast<size_t>(pmm::kFewStages) * sizeof(pmm::bf16) * stage_elems;
        const cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
        if (err != cudaSuccess) return static_cast<int>(err);
        pmm::launch_pdl(kern, dim3((N + cols - 1) / cols, row_tiles), dim3(128), smem, stream, static_cast<const pmm::bf16*>(a), ld_a,
                        static_cast<const pmm::bf16*>(w), perm, offsets, tile_start, E, top, K, N, limit, alpha, shift,
                        ungated, row_w, static_cast<pmm::bf16*>(out));
        return pmm::launch_status();
      };
      using Down = pmm::FewTile<false, false>;
      using Narrow = pmm::FewTile<true, true>;
      using Wide = pmm::FewTile<true, false>;
      if (!up) return few(pmm::moe_gemm_few_kernel<false, false>, Down::kCols, Down::kStageElems);
      if (pmm::few_narrow(A, E, N)) return few(pmm::moe_gemm_few_kernel<true, true>, Narrow::kCols, Narrow::kStageElems);
      return few(pmm::moe_gemm_few_kernel<true, false>, Wide::kCols, Wide::kStageElems);
    }
    const dim3 grid((N + pmm::kMmaCols - 1) / pmm::kMmaCols, row_tiles);
    if (up)
      pmm::launch_pdl(pmm::moe_gemm_mma_kernel<true>, grid, dim3(128), 0, stream, static_cast<const pmm::bf16*>(a), ld_a,
                      static_cast<const pmm::bf16*>(w), perm, offsets, tile_start, E, top, K, N, limit, alpha, shift, ungated, row_w, out);
    else
      pmm::launch_pdl(pmm::moe_gemm_mma_kernel<false>, grid, dim3(128), 0, stream, static_cast<const pmm::bf16*>(a), ld_a,
                      static_cast<const pmm::bf16*>(w), perm, offsets, tile_start, E, top, K, N, limit, alpha, shift, ungated, row_w, out);
    return pmm::launch_status();
  }
  const dim3 grid((N + pmm::kGenCols - 1) / pmm::kGenCols, row_tiles);
  PMM_DISPATCH_DTYPE(dtype, S, {
    if (up)
      pmm::launch_pdl(pmm::moe_gemm_generic_kernel<S, true>, grid, dim3(256), 0, stream, static_cast<const S*>(a), ld_a,
                      static_cast<const S*>(w), perm, offsets, tile_start, E, top, K, N, limit, alpha, shift, ungated, row_w, out);
    else
      pmm::launch_pdl(pmm::moe_gemm_generic_kernel<S, false>, grid, dim3(256), 0, stream, static_cast<const S*>(a), ld_a,
                      static_cast<const S*>(w), perm, offsets, tile_start, E, top, K, N, limit, alpha, shift, ungated, row_w, out);
  });
  return pmm::launch_status();
}

PMM_EXPORT int pmm_moe_combine(const void* y, const float* weights, const void* shared, const float* shared_gate, void* out,
                               int T, int D, int top, int dtype, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (D <= 0 || top <= 0) return PMM_ERR_BAD_ARGUMENT;
  const int v = dtype == PMM_DTYPE_BF16 ? 8 : 4;
  auto whole = [](const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
  // A thread a piece for rows of more than one value a thread of the other form, and for steps of many short rows; few short rows
  // are latency alone, of which a value a thread has less (64 tokens of 2 experts, width 128: 1.24 against 1.45 us, of 8
  // 1.76 against 2.37; 2,048 of 2, width 128: 2.68 against 1.59; one token of 2, width 512: 1.24 against 1.14).
  const long long blocks = (static_cast<long long>(T) * (D / v) + 255) / 256;
  const bool wide = D > 256 || static_cast<long long>(T) * D >= (1 << 18);
  if (wide && D % v == 0 && blocks < (1 << 24) && whole(y) && whole(out) && (!shared || whole(shared))) {
    PMM_DISPATCH_DTYPE(dtype, S, pmm::launch_pdl(pmm::moe_combine_vec_kernel<S>, dim3(static_cast<unsigned>(blocks)), dim3(256), 0,
                                                 stream, static_cast<const S*>(y), weights, static_cast<const S*>(shared),
                                                 shared_gate, static_cast<S*>(out), T, D, top));
    return pmm::launch_status();
  }
  int ytiles = (D + 1023) / 1024;
  if (ytiles > 64) ytiles = 64;
  PMM_DISPATCH_DTYPE(dtype, S, pmm::launch_pdl(pmm::moe_combine_kernel<S>, dim3(T, ytiles), dim3(256), 0, stream,
                                               static_cast<const S*>(y), weights, static_cast<const S*>(shared), shared_gate,
                                               static_cast<S*>(out), D, top));
  return pmm::launch_status();
}
