// Chunked Mamba2 SSD scan for prompt portions on the fifth-generation tensor cores
// (tcgen05.mma, accumulators in tensor memory; bfloat16 activations, float state).
//
// The recurrence  s_t = s_{t-1} exp(a_t) + delta_t B_t x_t^T ,  y_t = C_t . s_t + D x_t ,
// a_t = delta_t A  (reference src/ops/gpu/mamba2_scan.cu:11-50 walks it token by token) is
// evaluated per chunk of 128 tokens of one sequence portion.  With cs_i = a_0 + ... + a_i inside
// the chunk and S the state at the chunk's start:
//   y_i   = sum_{j<=i} (C_i.B_j) exp(cs_i-cs_j) delta_j x_j  +  exp(cs_i) (C_i . S)  +  D x_i
//   S_end = exp(cs_last) S  +  sum_j exp(cs_last-cs_j) delta_j x_j B_j^T
// Three launches, or two (1 and 2 as one walk, ssd_tc_walk_kernel, where the caller asks for it):
//   1. ssd_tc_state:   one block per (chunk, 128 channels of x): the local term of S_end as ONE
//                      product  D[channel, n] = sum_j (w_j x_j[channel]) B_j[n].  Both operands are
//                      the chunk's rows as they lie in memory (tokens = the K dimension, so both
//                      are MN-major; x is scaled by w_j in shared memory after it arrives); a thread
//                      reads its channel's row of the accumulator from tensor memory and the rows
//                      go out as float.
//   2. the state pass of ssd_chunked.cu walks the chunks of a sequence in float and hands the
//      state at every chunk's start on as bfloat16.
//   3. ssd_tc_output:  one block per chunk and run of units (a unit = a head's slab of up to 64
//                      channels), four threads per token: G = C B^T (128 x 128, tensor memory) once
//                      a block; per unit Y2 = C S^T, every thread reads its row of G, applies the
//                      decay, the causal mask and delta_j and writes the row of M as a bfloat16
//                      operand into the shared memory that held B, Y1 = M x follows (x as it lies in
//                      memory, MN-major); y = Y1 + exp(cs_i) Y2 + D x, the gate y silu(z) fused.
// Tiles come in the 128-byte swizzled layout that the tensor core reads, by 16-byte asynchronous
// copies (rows beyond a short chunk zero-filled, so they change nothing: their delta is zero) or,
// in phase 3, by TMA where they are whole tiles of 64 columns.  Any head size that is a multiple of 16 up to 128 and any state
// size that is a multiple of 16 up to 256 is taken.  All differences of cs are <= 0: no exponential overflows;
// delta, cs and every accumulator are float.  Every mbarrier wait is bounded (status codes
// 31..33 in *status; the block then skips its output, frees its tensor memory and returns).
#include "tcgen05.cuh"

namespace pmm {

using bf16 = __nv_bfloat16;

constexpr int kTQ = 128;        // tokens per chunk
constexpr int kTSub = 16384;    // bytes of a sub-tile of 128 rows x 128 bytes
constexpr float kLog2e = 1.4426950408889634f;

// Launches the state pass of ssd_chunked.cu for chunks of `q` tokens.
int launch_ssd_state_pass(const float* chunk_state, const float* chunk_decay, bf16* start_state, float* state,
                          const int* cu, const int* slots, int n_seq, int H, int PN, int q, int skip_single, int n_multi,
                          cudaStream_t stream);

__device__ __forceinline__ int tq_swz(int row, int chunk) {
  return (row >> 3) * 1024 + (row & 7) * 128 + ((chunk ^ (row & 7)) << 4);
}
__device__ __forceinline__ void tq_cp16(void* smem, const void* gmem, bool pred) {
  const unsigned s = smem_u32(smem);
  const int sz = pred ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(sz));
}
__device__ __forceinline__ void tq_cp_wait() { asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory"); }
__device__ __forceinline__ float tq_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ unsigned tq_pack(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const unsigned*>(&v);
}
__device__ __forceinline__ void tmem_ld16(unsigned taddr, unsigned* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}

// Which (first token, length) chunk `c` is; chunk ids run over the sequences in order.  Called by
// all threads of the block (a multiple of 32, at most 1,024); `sh` is shared memory for 36 ints.
// Every thread takes sequences tid, tid + blockDim, ...: the loads of the sequence bounds go out
// together instead of one after the other (a step may hold hundreds of sequences).
__device__ __forceinline__ bool tq_locate(const int* __restrict__ cu, int n_seq, int c, int& t0, int& len, int& seq_tokens,
                                          int* sh) {
  if (n_seq <= 4) {  // few sequences: every thread walks them itself
    int acc = 0;
    for (int seq = 0; seq < n_seq; ++seq) {
      const int lo = cu[seq], hi = cu[seq + 1];
      const int nc = (hi - lo + kTQ - 1) / kTQ;
      if (c < acc + nc) {
        t0 = lo + (c - acc) * kTQ;
        len = min(kTQ, hi - t0);
        seq_tokens = hi - lo;
        return true;
      }
      acc += nc;
    }
    return false;
  }
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n_warps = blockDim.x >> 5;
  if (tid == 0) sh[34] = -1;
  int base = 0;  // chunks of the sequences before this round
  for (int s0 = 0; s0 < n_seq; s0 += blockDim.x) {
    const int s = s0 + tid;
    int lo = 0, hi = 0;
    if (s < n_seq) lo = cu[s], hi = cu[s + 1];
    const int nc = (hi - lo + kTQ - 1) / kTQ;
    int incl = nc;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += up;
    }
    if (lane == 31) sh[warp] = incl;
    __syncthreads();
    int before = base;
    for (int w = 0; w < warp; ++w) before += sh[w];
    const int first = before + incl - nc;
    if (s < n_seq && c >= first && c < first + nc) {
      sh[34] = lo + (c - first) * kTQ;
      sh[35] = hi;
      sh[33] = hi - lo;
    }
    for (int w = 0; w < n_warps; ++w) base += sh[w];
    __syncthreads();
    if (sh[34] >= 0 || base > c) break;  // the same decision in every thread
  }
  if (sh[34] < 0) return false;
  t0 = sh[34];
  len = min(kTQ, sh[35] - t0);
  seq_tokens = sh[33];
  return true;
}

// 128 consecutive threads (four warps, `t` = 0..127 the thread's token): delta_t and cs_t (inclusive
// sum of delta * A over the chunk's tokens).  Tokens >= len get delta 0.  `totals` is shared memory
// for four floats; the caller synchronises the block before anybody reads what is derived from it.
struct TqDelta {
  float delta, incl;  // of this token; incl is the sum within the thread's warp only
};
__device__ __forceinline__ TqDelta tq_delta_warp(const bf16* __restrict__ dt_raw, long long ld_dt, float dt_scale,
                                                 float shift, float A, int t0, int len, int h, int t, float* totals) {
  TqDelta r;
  r.delta = t < len ? softplus_f(__bfloat162float(dt_raw[static_cast<long long>(t0 + t) * ld_dt + h]) * dt_scale + shift) : 0.f;
  float incl = r.delta * A;
  const int lane = t & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float up = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += up;
  }
  if (lane == 31) totals[t >> 5] = incl;
  r.incl = incl;
  return r;
}
// cs of token t once `totals` is visible: the warp's inclusive sum plus the warps before it.
__device__ __forceinline__ float tq_cs(const TqDelta& d, int t, const float* totals) {
  float cs = d.incl;
  for (int w = 0; w < (t >> 5); ++w) cs += totals[w];
  return cs;
}

__device__ __forceinline__ unsigned tq_idesc(int n, bool b_mn_major) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (b_mn_major ? (1u << 16) : 0u) | (static_cast<unsigned>(n >> 3) << 17) |
         (static_cast<unsigned>(kTQ >> 4) << 24);
}

// Descriptor of an MN-major operand of more than 64 rows: atoms of 64 (MN) x 8 (K) elements with
// the 128-byte swizzle, 1,024 bytes from one group of 8 K-rows to the next (stride byte offset),
// `atom_stride` bytes from one atom of 64 MN elements to the next (leading byte offset).
__device__ __forceinline__ unsigned long long umma_desc_mn(const void* tile, unsigned atom_stride) {
  const unsigned addr = smem_u32(tile);
  const unsigned lo = ((addr & 0x3FFFFu) >> 4) | ((atom_stride >> 4) << 16);
  const unsigned hi = (1024u >> 4) | (1u << 14) | (2u << 29);
  return (static_cast<unsigned long long>(hi) << 32) | lo;
}

__device__ __forceinline__ unsigned tq_tmem_alloc(unsigned* slot, int cols, int warp) {
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(slot)), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  return *slot;
}
__device__ __forceinline__ void tq_tmem_free(unsigned base, int cols, int warp) {
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(base), "r"(cols) : "memory");
  }
}

// ----------------------------------------------------------------------------- phase 1
// grid (chunks, groups * slabs_per_group); a slab is 128 consecutive channels of x inside one
// group (all its heads read the same B).  512 threads: the sixteen warps share the copies and the
// scaling; warps w, w+4, w+8, w+12 read the tensor-memory lanes 32 (w % 4) .. +31 (= channels)
// and split the columns.  The block in which a head begins also writes the head's exp(cs_last)
// and, for phase 3, delta_j and cs_j log2(e) of the chunk's tokens.
constexpr int kTState = 512;

__host__ __device__ constexpr size_t tq_state_smem(int nb) { return 1024 + 2 * kTSub + static_cast<size_t>(nb + (nb & 1)) * kTSub; }

__global__ void __launch_bounds__(kTState)
    ssd_tc_state_kernel(const bf16* __restrict__ xbc, int ld_xbc, const bf16* __restrict__ dt_raw, long long ld_dt,
                        float dt_scale, const float* __restrict__ dt_shift, const float* __restrict__ a_log,
                        const int* __restrict__ cu, int n_seq, float* __restrict__ chunk_state,
                        float* __restrict__ chunk_decay, float* __restrict__ chunk_dt, int H, int P, int N, int G,
                        int slabs_per_group, int tmem_cols, int skip_single, int* __restrict__ status) {
  pdl_launch_dependents();
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) unsigned long long bar;
  __shared__ unsigned s_tmem;
  __shared__ int s_abort;
  __shared__ float s_w[8][kTQ];      // per head of the slab: exp(cs_last - cs_j) * delta_j
  __shared__ float s_tot[8][4];      // per head: the four warps' sums of delta * A

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int c = blockIdx.x;
  int t0, len;
  __shared__ int s_loc[36];
  int seq_tokens;
  if (!tq_locate(cu, n_seq, c, t0, len, seq_tokens, s_loc)) return;
  if (skip_single && seq_tokens == 1) return;  // lone tokens of a mixed step are the token-serial kernel's
  pdl_wait();  // (the sequences' bounds are inputs of the step)
  pdl_written(xbc, dt_raw);
  unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* sA = tiles;                 // [128 tokens][128 channels]: two atoms of 64 channels
  unsigned char* sB = tiles + 2 * kTSub;     // [128 tokens][N]: one atom per 64 state columns
  const int I = H * P;
  const int g = blockIdx.y / slabs_per_group, slab = blockIdx.y % slabs_per_group;
  const int ch_per_group = (H / G) * P;
  const int ch0 = g * ch_per_group + slab * kTQ;
  const int n_ch = min(kTQ, ch_per_group - slab * kTQ);
  const int head0 = ch0 / P;
  const int n_heads = (ch0 + n_ch - 1) / P - head0 + 1;  // <= 8: a head has at least 16 channels

  if (len == 1) {
    // A lone token (a decoding request in a mixed step): S_local[ch][n] = delta x[ch] B[n], no product
    // worth a tensor core.  Thread = (channel, quarter of the state columns).
    if (tid < n_heads) {
      const int h = head0 + tid;
      const float d = softplus_f(__bfloat162float(dt_raw[static_cast<long long>(t0) * ld_dt + h]) * dt_scale + dt_shift[h]);
      const float a = -expf(a_log[h]) * d;
      s_w[tid][0] = d;
      if (h * P >= ch0) {
        float* dtp = chunk_dt + (static_cast<size_t>(c) * H + h) * (2 * kTQ);
        dtp[0] = d;
        dtp[kTQ] = a * kLog2e;
        chunk_decay[static_cast<size_t>(c) * H + h] = expf(a);
      }
    }
    __syncthreads();
    const int ch = tid & (kTQ - 1), quarter = tid >> 7;
    if (ch < n_ch) {
      const bf16* rowp = xbc + static_cast<size_t>(t0) * ld_xbc;
      const float xv = __bfloat162float(rowp[ch0 + ch]) * s_w[(ch0 + ch) / P - head0][0];
      const bf16* bp = rowp + I + g * N;
      float* dst = chunk_state + (static_cast<size_t>(c) * I + ch0 + ch) * N;
      for (int n = quarter * (N / 4); n < (quarter + 1) * (N / 4); n += 4) {
        const uint2 braw = *reinterpret_cast<const uint2*>(bp + n);
        const float2 b01 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&braw.x));
        const float2 b23 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&braw.y));
        *reinterpret_cast<float4*>(dst + n) = make_float4(xv * b01.x, xv * b01.y, xv * b23.x, xv * b23.y);
      }
    }
    return;
  }

  if (tid == 0) {
    mbar_init(&bar, 1);
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  // B rows of the chunk and x of the slab's channels, as they lie in memory (rows = tokens): both
  // operands are MN-major.  x is scaled by w_j in place below.
  {
    const int cpr = N / 8;  // 16-byte pieces per row of B
    int j = tid / cpr, ck = tid % cpr;
    const int dj = kTState / cpr, dck = kTState % cpr;
    while (j < kTQ) {
      const bool ok = j < len;
      tq_cp16(sB + (ck >> 3) * kTSub + tq_swz(j, ck & 7),
              xbc + (ok ? static_cast<size_t>(t0 + j) * ld_xbc + I + g * N + ck * 8 : 0), ok);
      j += dj, ck += dck;
      if (ck >= cpr) ck -= cpr, ++j;
    }
  }
  for (int i = tid; i < kTQ * 16; i += kTState) {
    const int j = i >> 4, ck = i & 15;
    const bool ok = j < len && ck * 8 < n_ch;
    tq_cp16(sA + (ck >> 3) * kTSub + tq_swz(j, ck & 7),
            xbc + (ok ? static_cast<size_t>(t0 + j) * ld_xbc + ch0 + ck * 8 : 0), ok);
  }
  // delta and cs of every head of the slab: head hh by the 128 threads of quarter hh % 4, a token each
  const int quarter = tid >> 7, tok = tid & (kTQ - 1);
  TqDelta dl[2];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int hh = quarter + 4 * r;
    if (hh < n_heads) {
      const int h = head0 + hh;
      dl[r] = tq_delta_warp(dt_raw, ld_dt, dt_scale, dt_shift[h], -expf(a_log[h]), t0, len, h, tok, s_tot[hh]);
    }
  }
  const unsigned tmem_base = tq_tmem_alloc(&s_tmem, tmem_cols, warp);  // includes a __syncthreads: s_tot is visible
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int hh = quarter + 4 * r;
    if (hh < n_heads) {
      const int h = head0 + hh;
      const float cs = tq_cs(dl[r], tok, s_tot[hh]);
      const float last = (s_tot[hh][0] + s_tot[hh][1]) + (s_tot[hh][2] + s_tot[hh][3]);
      s_w[hh][tok] = expf(last - cs) * dl[r].delta;
      if (h * P >= ch0) {  // the head begins in this slab
        float* dtp = chunk_dt + (static_cast<size_t>(c) * H + h) * (2 * kTQ);
        dtp[tok] = dl[r].delta;
        dtp[kTQ + tok] = cs * kLog2e;
        if (tok == 0) chunk_decay[static_cast<size_t>(c) * H + h] = expf(last);
      }
    }
  }
  tq_cp_wait();
  __syncthreads();  // s_w
  // every thread scales the pieces of x that it copied itself
#pragma unroll 4
  for (int i = tid; i < kTQ * 16; i += kTState) {
    const int j = i >> 4, ck = i & 15;
    if (j < len && ck * 8 < n_ch) {
      uint4* cell = reinterpret_cast<uint4*>(sA + (ck >> 3) * kTSub + tq_swz(j, ck & 7));
      const uint4 raw = *cell;
      const float w = s_w[(ch0 + ck * 8) / P - head0][j];
      const unsigned rw[4] = {raw.x, raw.y, raw.z, raw.w};
      unsigned o[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&rw[e]));
        o[e] = tq_pack(f.x * w, f.y * w);
      }
      *cell = make_uint4(o[0], o[1], o[2], o[3]);
    }
  }
  fence_proxy_async();
  __syncthreads();

  if (tid == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const unsigned long long a_desc = umma_desc_mn(sA, kTSub);
    for (int s = 0; s * 128 < N; ++s) {  // up to 128 state columns (two atoms) an instruction
      const int ncols = min(128, N - 128 * s);
      const unsigned idesc = tq_idesc(ncols, true) | (1u << 15);  // A and B both MN-major
      const unsigned long long b_desc = umma_desc_mn(sB + 2 * s * kTSub, kTSub);
#pragma unroll
      for (int k = 0; k < kTQ / 16; ++k)  // 16 tokens further = 16 rows of 128 bytes in both operands
        umma_f16(tmem_base + 128 * s, a_desc + ((k * 16 * 128) >> 4), b_desc + ((k * 16 * 128) >> 4), idesc, k > 0 ? 1u : 0u);
    }
    umma_commit(&bar);
  }
  volatile int* abort_flag = &s_abort;
  bool ok = mbar_wait(&bar, 0, abort_flag);
  ok = __all_sync(0xffffffffu, ok);
  if (!ok && lane == 0) {
    if (!*abort_flag) atomicExch(status, 31);
    s_abort = 1;
  }
  if (ok) {
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const int rw = warp & 3, part = warp >> 2;
    const unsigned lane_base = tmem_base + (static_cast<unsigned>(rw * 32) << 16);
    // A lane holds a channel's row; rows go out 16 columns at a time through shared memory (the
    // operand tiles are no longer read), so that a store covers whole 64-byte pieces of 8 rows.
    float* stage = reinterpret_cast<float*>(tiles) + warp * (32 * 20);  // 32 rows of 16 + 4 floats
    float* dst = chunk_state + (static_cast<size_t>(c) * I + ch0 + rw * 32) * N;
    for (int c16 = part; c16 < N / 16; c16 += 4) {
      unsigned v[16];
      tmem_ld16(lane_base + c16 * 16, v);
      asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
      for (int q4 = 0; q4 < 4; ++q4)
        *reinterpret_cast<float4*>(stage + lane * 20 + q4 * 4) =
            make_float4(__uint_as_float(v[q4 * 4]), __uint_as_float(v[q4 * 4 + 1]), __uint_as_float(v[q4 * 4 + 2]),
                        __uint_as_float(v[q4 * 4 + 3]));
      __syncwarp();
#pragma unroll
      for (int pass = 0; pass < 4; ++pass) {
        const int r = pass * 8 + (lane >> 2);
        if (rw * 32 + r < n_ch)
          *reinterpret_cast<float4*>(dst + static_cast<size_t>(r) * N + c16 * 16 + (lane & 3) * 4) =
              *reinterpret_cast<const float4*>(stage + r * 20 + (lane & 3) * 4);
      }
      __syncwarp();
    }
  }
  tq_tmem_free(tmem_base, tmem_cols, warp);
}

// ----------------------------------------------------------------------------- phases 1 and 2 in one walk
// grid (slabs of 128 channels * blocks of NB state columns, sequences): a block walks the chunks of one sequence with its part
// of the state in registers.  Per chunk: the local term as in phase 1 (x scaled by w_j in shared memory, one product with K =
// the tokens), the state before the chunk out as bfloat16, S <- exp(cs_last) S + local as in the state pass: the same sums
// in the same order, without the local terms (float, written and read once) and the second launch between them.
// 512 threads scale and fold: warps w, w + 4, w + 8, w + 12 share the tensor-memory lanes (= channels) 32 (w % 4) ... and split the
// NB columns; warp 16 asks for the tiles (TMA), issues the products (two accumulators) and sends the start states off, so
// that the product of a chunk runs while the chunk behind it is scaled.  The decays of up to 16 (chunk, head)s are made
// at a time by all warps.
constexpr int kTWalk = 512;
constexpr int kTWalkAll = kTWalk + 32;
constexpr int kTWalkDecays = 16;  // (chunk, head)s whose decays lie in shared memory
__host__ __device__ constexpr int tq_walk_stages(int NB) { return NB == 64 ? 3 : 2; }
__host__ __device__ constexpr int tq_walk_stage(int NB) { return 2 * kTSub + NB * 256; }  // x, then 128 rows of NB columns of B
__host__ __device__ constexpr size_t tq_walk_smem(int NB) {  // ..., two tiles of start states [128 channels][NB], the decays
  return 1024 + static_cast<size_t>(tq_walk_stages(NB)) * tq_walk_stage(NB) + 2 * NB * 256 + 2 * kTWalkDecays * kTQ * sizeof(float);
}

template <int NB>
__global__ void __launch_bounds__(kTWalkAll, 1)
    ssd_tc_walk_kernel(const __grid_constant__ CUtensorMap map_xbc, const __grid_constant__ CUtensorMap map_out,
                       const bf16* __restrict__ xbc, int ld_xbc, const bf16* __restrict__ dt_raw, long long ld_dt, float dt_scale,
                       const float* __restrict__ dt_shift, const float* __restrict__ a_log, const int* __restrict__ cu,
                       const int* __restrict__ slots, float* __restrict__ state, float* __restrict__ chunk_dt,
                       bf16* __restrict__ start_state, int H, int P, int N, int G, int slabs_per_group, int skip_single,
                       int* __restrict__ status) {
  constexpr int kCols = NB / 4;        // state columns a thread
  constexpr int kBSub = NB / 64;       // sub-tiles of B, and of a tile of start states
  constexpr int kStages = tq_walk_stages(NB);
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) unsigned long long bar_in[kStages], bar_scaled[2], bar_mma[2], bar_out[2];
  __shared__ unsigned s_tmem;
  __shared__ int s_abort, s_first[kTWalkAll / 32];
  __shared__ float s_tot[kTWalkDecays][4];  // per (chunk, head): the sums of delta * A of four groups of 32 tokens
  __shared__ float s_decay[kTWalkDecays];

  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int seq = blockIdx.y;
  // the sequence and its chunks (inputs of the step, read before the wait)
  const int t_begin = cu[seq], n_tok = cu[seq + 1] - t_begin;
  if (n_tok <= 0 || (skip_single && n_tok == 1)) return;
  const int nc = (n_tok + kTQ - 1) / kTQ;
  int mine = 0;
  for (int q = tid; q < seq; q += kTWalkAll) mine += (cu[q + 1] - cu[q] + kTQ - 1) / kTQ;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, o);
  if (lane == 0) s_first[warp] = mine;
  const int col_blocks = N / NB;
  const int slab_id = blockIdx.x / col_blocks, n0 = (blockIdx.x % col_blocks) * NB;
  const int I = H * P, g = slab_id / slabs_per_group, slab = slab_id % slabs_per_group;
  const int ch_per_group = (H / G) * P;
  const int ch0 = g * ch_per_group + slab * kTQ;
  const int n_ch = min(kTQ, ch_per_group - slab * kTQ);
  const int head0 = ch0 / P;
  const int n_heads = (ch0 + n_ch - 1) / P - head0 + 1;  // <= 8: a head has at least 16 channels
  const int span = kTWalkDecays / n_heads;               // chunks whose decays are made at a time
  unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  auto stage = [&](int k) { return tiles + (k % kStages) * tq_walk_stage(NB); };
  unsigned char* sOut = tiles + kStages * tq_walk_stage(NB);
  float* s_w = reinterpret_cast<float*>(sOut + 2 * NB * 256);  // [(chunk, head)][token]: exp(cs_last - cs_j) * delta_j
  float* s_delta = s_w + kTWalkDecays * kTQ;
  if (tid == 0) {
#pragma unroll
    for (int i = 0; i < kStages; ++i) mbar_init(&bar_in[i], 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bar_scaled[i], kTWalk / 32);
      mbar_init(&bar_mma[i], 1);
      mbar_init(&bar_out[i], kTWalk / 32);
    }
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  pdl_wait();
  pdl_written(xbc, dt_raw);
  const unsigned tmem_base = tq_tmem_alloc(&s_tmem, 2 * NB, warp);  // includes a __syncthreads
  volatile int* abort_flag = &s_abort;
  auto wait_all = [&](unsigned long long* bar, unsigned parity) {  // the same answer in a warp
    if (__all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag))) return true;
    if (lane == 0) {
      if (!*abort_flag) atomicExch(status, 31);
      s_abort = 1;
    }
    return false;
  };
  int first = 0;  // chunks of the sequences before this one
  for (int w = 0; w < kTWalkAll / 32; ++w) first += s_first[w];
  const bool whole = n_ch == kTQ;  // the slab's start states go out as one tile (else a thread writes its own)

  if (warp == kTWalk / 32) {
    // ---------------------------------------------------------------- tiles and products
    auto request = [&](int k) {
      unsigned char* dst = stage(k);
      unsigned long long* bar = &bar_in[k % kStages];
      const int t0 = t_begin + k * kTQ;
      mbar_expect_tx(bar, tq_walk_stage(NB));
      tma_load_2d(dst, &map_xbc, ch0, t0, bar);
      tma_load_2d(dst + kTSub, &map_xbc, ch0 + 64, t0, bar);  // (columns behind the slab's channels: rows of the product nobody reads)
#pragma unroll
      for (int b = 0; b < kBSub; ++b) tma_load_2d(dst + (2 + b) * kTSub, &map_xbc, I + g * N + n0 + b * 64, t0, bar);
    };
    if (lane < min(kStages, nc)) request(lane);
    __syncwarp();
    auto send = [&](int k) {  // the states before chunk k
      if (!wait_all(&bar_out[k & 1], (k >> 1) & 1)) return false;
      if (lane == 0) {
#pragma unroll
        for (int b = 0; b < kBSub; ++b)
          asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];\n" ::"l"(
                           reinterpret_cast<unsigned long long>(&map_out)),
                       "r"(smem_u32(sOut + (k & 1) * (NB * 256) + b * kTSub)), "r"(n0 + b * 64), "r"((first + k) * I + ch0)
                       : "memory");
        asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
      }
      __syncwarp();
      return true;
    };
    const unsigned lead = lane == 0 ? 1u : 0u;
    constexpr unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | (static_cast<unsigned>(NB >> 3) << 17) |
                               (static_cast<unsigned>(kTQ >> 4) << 24);  // A and B both MN-major
    bool ok = true;
    for (int k = 0; k < nc && ok; ++k) {
      if (!wait_all(&bar_scaled[k & 1], (k >> 1) & 1)) break;
      // (the states before chunk k - 2 have left their tile: who waits for this product may write it)
      if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");
      __syncwarp();
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      const unsigned long long a_desc = umma_desc_mn(stage(k), kTSub), b_desc = umma_desc_mn(stage(k) + 2 * kTSub, kTSub);
#pragma unroll
      for (int i = 0; i < kTQ / 16; ++i)  // 16 tokens further = 16 rows of 128 bytes in both operands
        umma_f16_lead(tmem_base + (k & 1) * NB, a_desc + ((i * 16 * 128) >> 4), b_desc + ((i * 16 * 128) >> 4), idesc, i > 0 ? 1u : 0u, lead);
      umma_commit_lead(&bar_mma[k & 1], lead);
      // a stage takes its next chunk once its product has finished: of three stages the one of chunk k - 1, of two this one
      const int done = kStages == 3 ? k - 1 : k;
      if (done >= 0 && done + kStages < nc) {
        ok = wait_all(&bar_mma[done & 1], (done >> 1) & 1);
        if (ok && lane == 0) request(done + kStages);
        __syncwarp();
      }
      if (k > 0 && whole) ok = ok && send(k - 1);
    }
    if (whole && ok) send(nc - 1);
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory");
  } else {
    // ---------------------------------------------------------------- scaling and folding
    const int rw = warp & 3, part = warp >> 2, row = rw * 32 + lane;
    const unsigned lane_base = tmem_base + (static_cast<unsigned>(rw * 32) << 16);
    const bool row_ok = row < n_ch;
    const int my_head = row_ok ? (ch0 + row) / P - head0 : 0;
    const int col = n0 + part * kCols;
    float* sp = state + (static_cast<size_t>(slots[seq]) * I + ch0 + row) * N + col;
    float S[kCols];
#pragma unroll
    for (int i = 0; i < kCols; i += 4) {
      const float4 v = row_ok ? *reinterpret_cast<const float4*>(sp + i) : make_float4(0.f, 0.f, 0.f, 0.f);
      S[i] = v.x, S[i + 1] = v.y, S[i + 2] = v.z, S[i + 3] = v.w;
    }
    auto sync_workers = [&]() { asm volatile("bar.sync 1, 512;\n" ::: "memory"); };
    // delta, cs and w of chunks k0 .. k0 + span - 1, every head of the slab: a warp per 32 tokens of a (chunk, head), four at a time
    auto make_decays = [&](int k0) {
      const int tasks = min(span, nc - k0) * n_heads * 4;
      sync_workers();  // (what lay there has been used)
#pragma unroll 1
      for (int base = warp; base < tasks; base += 4 * (kTWalk / 32)) {
        float delta[4], incl[4], raw[4], shift[4], al[4];
        bool in[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {  // (the loads of all four before anything waits for one)
          const int task = min(base + u * (kTWalk / 32), tasks - 1), item = task >> 2, tok = (task & 3) * 32 + lane;
          const int kk = item / n_heads, t = (k0 + kk) * kTQ + tok, h = head0 + (item - kk * n_heads);
          in[u] = t < n_tok;
          raw[u] = __bfloat162float(dt_raw[static_cast<long long>(t_begin + min(t, n_tok - 1)) * ld_dt + h]);
          shift[u] = dt_shift[h];
          al[u] = a_log[h];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          delta[u] = in[u] ? softplus_f(raw[u] * dt_scale + shift[u]) : 0.f;
          incl[u] = delta[u] * -expf(al[u]);
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const float up = __shfl_up_sync(0xffffffffu, incl[u], o);
            if (lane >= o) incl[u] += up;
          }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int task = base + u * (kTWalk / 32), item = task >> 2, tok = (task & 3) * 32 + lane;
          if (task < tasks) {
            s_delta[item * kTQ + tok] = delta[u];
            s_w[item * kTQ + tok] = incl[u];
            if (lane == 31) s_tot[item][task & 3] = incl[u];
          }
        }
      }
      sync_workers();
#pragma unroll 1
      for (int base = warp; base < tasks; base += 4 * (kTWalk / 32))
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int task = base + u * (kTWalk / 32), item = task >> 2, tok = (task & 3) * 32 + lane;
          if (task < tasks) {
            const int kk = item / n_heads, k = k0 + kk, h = head0 + (item - kk * n_heads);
            const float* tot = s_tot[item];
            const float delta = s_delta[item * kTQ + tok];
            float cs = s_w[item * kTQ + tok];
            for (int w = 0; w < (task & 3); ++w) cs += tot[w];
            const float last = (tot[0] + tot[1]) + (tot[2] + tot[3]);
            s_w[item * kTQ + tok] = expf(last - cs) * delta;
            if (tok == 0) s_decay[item] = expf(last);
            if (n0 == 0 && h * P >= ch0) {  // the head begins in this slab
              float* dtp = chunk_dt + (static_cast<size_t>(first + k) * H + h) * (2 * kTQ);
              dtp[tok] = delta;
              dtp[kTQ + tok] = cs * kLog2e;
            }
          }
        }
      sync_workers();
    };
    float decay = 0.f, lone_w = 0.f;  // of the chunk that is folded in next
    auto fold = [&](int k) {  // chunk k: the state before it out, its local term in
      const int c = first + k, len = min(kTQ, n_tok - k * kTQ);
      unsigned char* out = sOut + (k & 1) * (NB * 256);
      bf16* dst = start_state + (static_cast<size_t>(c) * I + ch0 + row) * N + col;
      wait_all(&bar_mma[k & 1], (k >> 1) & 1);
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      unsigned v[16];
      tmem_ld16(lane_base + (k & 1) * NB + part * kCols, v);
#pragma unroll
      for (int i = 0; i < kCols; i += 8) {
        const uint4 p = make_uint4(tq_pack(S[i], S[i + 1]), tq_pack(S[i + 2], S[i + 3]), tq_pack(S[i + 4], S[i + 5]), tq_pack(S[i + 6], S[i + 7]));
        const int ck = (part * kCols + i) >> 3;
        if (whole)
          *reinterpret_cast<uint4*>(out + (ck >> 3) * kTSub + tq_swz(row, ck & 7)) = p;
        else if (row_ok)
          *reinterpret_cast<uint4*>(dst + i) = p;
      }
      if (whole) {
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar_out[k & 1]);
      }
#pragma unroll
      for (int i = 0; i < kCols; i += 16) {
        if (i > 0) tmem_ld16(lane_base + (k & 1) * NB + part * kCols + i, v);
        asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
        if (len > 1) {
#pragma unroll
          for (int e = 0; e < 16; ++e) S[i + e] = fmaf(S[i + e], decay, __uint_as_float(v[e]));
        }
      }
      if (len == 1) {  // one token: S_local[ch][n] = delta x[ch] B[n], not through bfloat16 operands
        const bf16* rowp = xbc + static_cast<size_t>(t_begin + k * kTQ) * ld_xbc;
        const float xv = row_ok ? __bfloat162float(rowp[ch0 + row]) * lone_w : 0.f;
#pragma unroll
        for (int i = 0; i < kCols; ++i) S[i] = fmaf(S[i], decay, __fmul_rn(xv, __bfloat162float(rowp[I + g * N + col + i])));
      }
      asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    };
    // this thread's pieces of x: 16 bytes (8 channels of one head) of every 32nd token
    const int ck = tid & 15, j0 = tid >> 4;
    const bool piece_ok = ck * 8 < n_ch;
    const int piece_head = piece_ok ? (ch0 + ck * 8) / P - head0 : 0;
    const int piece_off = (ck >> 3) * kTSub + tq_swz(j0, ck & 7);  // (32 tokens further: 4,096 bytes)
    // (a wait that gave up does not leave the loop: the warps meet at named barriers, and the waits behind it end at once)
    int at = span;  // the chunk's place among those whose decays lie there
    for (int k = 0; k < nc; ++k) {
      const int len = min(kTQ, n_tok - k * kTQ);
      if (at == span) {
        make_decays(k);
        at = 0;
      }
      const float* w_row = s_w + (at * n_heads + piece_head) * kTQ + j0;
      const float next_decay = s_decay[at * n_heads + my_head], next_w = s_w[(at * n_heads + my_head) * kTQ];
      ++at;
      wait_all(&bar_in[k % kStages], (k / kStages) & 1);
      unsigned char* sA = stage(k);
      if (piece_ok) {
        uint4 in[4];
        float w[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          in[r] = *reinterpret_cast<const uint4*>(sA + piece_off + r * 4096);
          w[r] = w_row[32 * r];
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const unsigned rw4[4] = {in[r].x, in[r].y, in[r].z, in[r].w};
          unsigned o[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&rw4[e]));
            o[e] = j0 + 32 * r < len ? tq_pack(f.x * w[r], f.y * w[r]) : 0u;  // (rows beyond the chunk belong to others: zero, whatever they hold)
          }
          *reinterpret_cast<uint4*>(sA + piece_off + r * 4096) = make_uint4(o[0], o[1], o[2], o[3]);
        }
      }
      if (len < kTQ)
        for (int i = tid; i < (kTQ - len) * kBSub * 8; i += kTWalk) {
          const int j = len + i / (kBSub * 8), cb = i % (kBSub * 8);
          *reinterpret_cast<uint4*>(sA + (2 + (cb >> 3)) * kTSub + tq_swz(j, cb & 7)) = make_uint4(0u, 0u, 0u, 0u);
        }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_scaled[k & 1]);
      // The launch behind this one is let go with the last chunk: behind the wait, so that it may read what came before this
      // one, and late, so that its blocks do not hold the SMs that other streams' launches could use.
      if (k == nc - 1) pdl_launch_dependents();
      if (k > 0) fold(k - 1);
      decay = next_decay, lone_w = next_w;
    }
    fold(nc - 1);
    if (row_ok && !*abort_flag) {
#pragma unroll
      for (int i = 0; i < kCols; i += 4) *reinterpret_cast<float4*>(sp + i) = make_float4(S[i], S[i + 1], S[i + 2], S[i + 3]);
    }
  }
  if (s_abort && tid == kTWalk) {
    // copies that were asked for still write into this block's shared memory: a bounded time for them to land
    for (unsigned i = 0; i < kSpinLimit / 4; ++i) __nanosleep(32);
  }
  tq_tmem_free(tmem_base, 2 * NB, warp);
}

// ----------------------------------------------------------------------------- phase 3
// grid (chunks, groups * blocks a group); a block takes `per_block` units of one chunk and one group, a unit being a head's
// slab of PB channels.  C and B of the chunk are brought once and G = C B^T is made once; then unit by unit the start state's
// rows, x and the gate's input arrive while the unit before is worked on: Y2 = C S^T is issued, M made from G for the unit's
// head (slabs of one head share it), Y1 = M x issued, and the rows y go out.  512 threads: threads t, t + 128, t + 256 and
// t + 384 share token t of the chunk (= tensor-memory lane t) and split its columns; warp 16 issues the products.  Tensor
// memory: G columns 0..127, Y2 columns 128..128+PB, Y1 columns 192..192+PB.
// C, B, x and the gate's input were finished before the launch before this one (which lets this one go behind its own wait):
// they are brought and G is made before this launch's wait.  The start states and the tokens' steps and decays (chunk_dt) are not:
// the walk, directly before this launch, writes both, so they are read behind the wait only.
// What bounds it: a unit is a chain of two products, an exponential per entry of M's lower half and two per output, about
// 2,400 clocks.  One block a unit (two blocks an SM, C and B brought and G made for every head) took 19.5 us at 24 heads of
// 64 x 128 and 2,048 tokens and 56 us at 48 heads of 128 x 256 and 1,024 tokens.
constexpr int kTOut = 512;
constexpr int kTOutAll = kTOut + 32;

__host__ __device__ constexpr int tq_state_bytes(int nb, int PB) { return nb * PB * 128; }
// The second stage of the start states lies behind M in B's place where it fits there.
__host__ __device__ constexpr bool tq_second_in_b(int nb, int PB) { return (nb - 2) * kTSub >= tq_state_bytes(nb, PB); }
__host__ __device__ constexpr size_t tq_output_smem(int nb, int PB) {
  return 1024 + static_cast<size_t>(nb + (nb > 2 ? nb : 2)) * kTSub + tq_state_bytes(nb, PB) * (tq_second_in_b(nb, PB) ? 1 : 2) + 3 * kTSub;
}

// Calls f(row, piece) for the 16-byte pieces tid, tid + 512, ... of `rows` rows of `cpr` pieces.
template <typename F>
__device__ __forceinline__ void tq_pieces(int tid, int rows, int cpr, F f) {
  int j = tid / cpr, ck = tid % cpr;
  const int dj = kTOut / cpr, dck = kTOut % cpr;
  while (j < rows) {
    f(j, ck);
    j += dj, ck += dck;
    if (ck >= cpr) ck -= cpr, ++j;
  }
}

// A lone token (a decoding request in a mixed step): y[p] = (C.B) delta x[p] + exp(cs_0) C.S[p] + D x[p] for the channels
// col0 .. col0 + PB - 1 of head h, a warp per channel.
__device__ __forceinline__ void tq_lone_output(const bf16* __restrict__ xbc, int ld_xbc, const float* __restrict__ dtp, float Dh1, int t0,
                                               const bf16* __restrict__ start, bf16* __restrict__ y, int I, int g, int G, int N,
                                               size_t col0, int PB, const bf16* __restrict__ z_raw, long long ld_z, float z_scale,
                                               const float* __restrict__ z_bias, int warp, int lane) {
  const float d0 = dtp[0], e0 = tq_ex2(dtp[kTQ]);
  const bf16* rowp = xbc + static_cast<size_t>(t0) * ld_xbc;
  const bf16* bp = rowp + I + g * N;
  const bf16* cp = bp + G * N;
  float cb = 0.f;
  float cv[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (lane * 8 < N) {
    const uint4 cq = *reinterpret_cast<const uint4*>(cp + lane * 8), bq = *reinterpret_cast<const uint4*>(bp + lane * 8);
    const unsigned cw[4] = {cq.x, cq.y, cq.z, cq.w}, bw[4] = {bq.x, bq.y, bq.z, bq.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 cf = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&cw[e]));
      const float2 bf = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&bw[e]));
      cv[2 * e] = cf.x, cv[2 * e + 1] = cf.y;
      cb += cf.x * bf.x + cf.y * bf.y;
    }
  }
  cb = warp_sum(cb);
  constexpr int kW = kTOut / 32;
  for (int pbase = warp; pbase < PB; pbase += 4 * kW) {  // four channels of this warp at a time: their loads go out together
    uint4 sq[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int p = pbase + u * kW;
      sq[u] = make_uint4(0u, 0u, 0u, 0u);
      if (p < PB && lane * 8 < N) sq[u] = *reinterpret_cast<const uint4*>(start + static_cast<size_t>(p) * N + lane * 8);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int p = pbase + u * kW;
      if (p >= PB) break;  // the same in every lane
      const unsigned sw[4] = {sq[u].x, sq[u].y, sq[u].z, sq[u].w};
      float acc = 0.f;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 sf = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&sw[e]));
        acc += cv[2 * e] * sf.x + cv[2 * e + 1] * sf.y;
      }
      acc = warp_sum(acc);
      if (lane == 0) {
        const float xv = __bfloat162float(rowp[col0 + p]);
        float v = cb * d0 * xv + e0 * acc + Dh1 * xv;
        if (z_raw) {
          const float zv = __bfloat162float(z_raw[static_cast<long long>(t0) * ld_z + col0 + p]);
          v *= silu_fast(zv * z_scale + (z_bias ? z_bias[col0 + p] : 0.f));
        }
        y[static_cast<size_t>(t0) * I + col0 + p] = __float2bfloat16_rn(v);
      }
    }
  }
}

template <bool kTma>
__global__ void __launch_bounds__(kTOutAll, 1)
    ssd_tc_output_kernel(const __grid_constant__ CUtensorMap map_xbc, const __grid_constant__ CUtensorMap map_start,
                         const __grid_constant__ CUtensorMap map_z, const bf16* __restrict__ xbc, int ld_xbc, const float* __restrict__ chunk_dt,
                         const float* __restrict__ d_skip, const int* __restrict__ cu, int n_seq,
                         const bf16* __restrict__ start_state, bf16* __restrict__ y, int H, int P, int N, int G, int PB_any,
                         int per_block, const bf16* __restrict__ z_raw, long long ld_z, float z_scale,
                         const float* __restrict__ z_bias, int z_vec, int skip_single, int* __restrict__ status) {
  pdl_launch_dependents();
  const int PB = kTma ? 64 : PB_any;
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) unsigned long long bar_g, bar_y, bar_cb, bar_x[2], bar_s[2], bar_z;
  __shared__ unsigned s_tmem;
  __shared__ int s_abort;
  __shared__ __align__(16) float s_dt[2][2 * kTQ];  // per stage: delta_j, then cs_j * log2(e)

  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int row = tid & (kTQ - 1), part = tid >> 7, rw = warp & 3;
  const bool worker = tid < kTOut;  // (warp 16 issues the products)
  const int c = blockIdx.x;
  int t0, len;
  __shared__ int s_loc[36];
  int seq_tokens;
  if (!tq_locate(cu, n_seq, c, t0, len, seq_tokens, s_loc)) return;
  if (skip_single && seq_tokens == 1) return;  // lone tokens of a mixed step are the token-serial kernel's
  const int slabs = P / PB, heads = H / G, group_units = heads * slabs;
  const int group_blocks = (group_units + per_block - 1) / per_block;
  const int g = blockIdx.y / group_blocks;
  const int unit0 = static_cast<int>(blockIdx.y % group_blocks) * per_block, n_units = min(per_block, group_units - unit0);
  const int I = H * P;
  auto head_of = [&](int k) { return g * heads + (unit0 + k) / slabs; };
  auto col_of = [&](int k) { return static_cast<size_t>(g * heads * P) + static_cast<size_t>(unit0 + k) * PB; };

  if (len == 1) {
    pdl_wait();
    pdl_written(chunk_dt, start_state);
    if (worker)
      for (int k = 0; k < n_units; ++k) {
        const int h = head_of(k);
        tq_lone_output(xbc, ld_xbc, chunk_dt + (static_cast<size_t>(c) * H + h) * (2 * kTQ), d_skip[h], t0,
                       start_state + (static_cast<size_t>(c) * I + col_of(k)) * N, y, I, g, G, N, col_of(k), PB, z_raw, ld_z, z_scale,
                       z_bias, warp, lane);
      }
    return;
  }

  const int nb = (N + 63) / 64;
  const int s_sub = PB * 128;  // bytes of one 64-column block of the start state's rows
  unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* sC = tiles;                                // [128 tokens][N], K-major
  unsigned char* sB = sC + nb * kTSub;                      // [128 tokens][N], K-major; later M [128][128]
  unsigned char* sX = sB + (nb > 2 ? nb : 2) * kTSub;       // two stages of [128 tokens][PB], MN-major; later y, in place
  unsigned char* sZ = sX + 2 * kTSub;                       // [128 tokens][PB]
  unsigned char* sS0 = sZ + kTSub;                          // [PB channels][N], K-major
  unsigned char* sS1 = tq_second_in_b(nb, PB) ? sB + 2 * kTSub : sS0 + tq_state_bytes(nb, PB);

  if (tid == 0) {
    mbar_init(&bar_g, 1);
    mbar_init(&bar_y, 1);
    mbar_init(&bar_cb, 1);
    mbar_init(&bar_x[0], 1);
    mbar_init(&bar_x[1], 1);
    mbar_init(&bar_s[0], 1);
    mbar_init(&bar_s[1], 1);
    mbar_init(&bar_z, 1);
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  auto copy_x = [&](int k) {  // x of unit k into its stage
    unsigned char* dst = sX + (k & 1) * kTSub;
    const size_t col = col_of(k);
    tq_pieces(tid, kTQ, PB / 8, [&](int j, int ck) {
      const bool ok = j < len;
      tq_cp16(dst + tq_swz(j, ck), xbc + (ok ? static_cast<size_t>(t0 + j) * ld_xbc + col + ck * 8 : 0), ok);
    });
  };
  auto copy_s = [&](int k) {  // its start states, steps and decays (results of the launch before: behind the wait)
    unsigned char* dst = (k & 1) ? sS1 : sS0;
    const bf16* src = start_state + (static_cast<size_t>(c) * I + col_of(k)) * N;
    tq_pieces(tid, PB, N / 8, [&](int p, int ck) {
      tq_cp16(dst + (ck >> 3) * s_sub + tq_swz(p, ck & 7), src + static_cast<size_t>(p) * N + ck * 8, true);
    });
    if (tid < kTQ / 2)
      tq_cp16(&s_dt[k & 1][tid * 4], chunk_dt + (static_cast<size_t>(c) * H + head_of(k)) * (2 * kTQ) + tid * 4, true);
  };
  auto commit = [&]() { asm volatile("cp.async.commit_group;\n" ::: "memory"); };
  // (whole tiles of 64 columns) one lane of warp 16 asks for them; rows beyond the chunk bring what lies there: a row of C reaches
  // only its own output, a row of B only entries of M that are set to zero, and x's rows are zeroed below
  const unsigned dt_bytes = 2 * kTQ * sizeof(float);
  auto tma_x = [&](int k) {
    unsigned long long* bar = &bar_x[k & 1];
    mbar_expect_tx(bar, kTSub);
    tma_load_2d(sX + (k & 1) * kTSub, &map_xbc, static_cast<int>(col_of(k)), t0, bar);
  };
  auto tma_s = [&](int k) {  // the start state's rows and the decays
    unsigned long long* bar = &bar_s[k & 1];
    unsigned char* dst = (k & 1) ? sS1 : sS0;
    mbar_expect_tx(bar, tq_state_bytes(nb, 64) + dt_bytes);
    for (int b = 0; b < nb; ++b) tma_load_2d(dst + b * s_sub, &map_start, b * 64, c * I + static_cast<int>(col_of(k)), bar);
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(smem_u32(s_dt[k & 1])),
                 "l"(chunk_dt + (static_cast<size_t>(c) * H + head_of(k)) * (2 * kTQ)), "r"(dt_bytes), "r"(smem_u32(bar))
                 : "memory");
  };
  auto tma_z = [&](int k) {
    mbar_expect_tx(&bar_z, kTSub);
    tma_load_2d(sZ, &map_z, static_cast<int>(col_of(k)), t0, &bar_z);
  };
  const bool gate_tile = z_raw && z_vec;
  if (kTma) {
    __syncthreads();  // the barriers
    if (tid == kTOut) {
      mbar_expect_tx(&bar_cb, 2 * nb * kTSub);
      for (int b = 0; b < nb; ++b) {
        tma_load_2d(sB + b * kTSub, &map_xbc, I + g * N + b * 64, t0, &bar_cb);
        tma_load_2d(sC + b * kTSub, &map_xbc, I + (G + g) * N + b * 64, t0, &bar_cb);
      }
      tma_x(0);
      if (gate_tile) tma_z(0);
    }
  } else if (worker) {
    tq_pieces(tid, kTQ, N / 8, [&](int j, int ck) {
      const bool ok = j < len;
      const size_t src = ok ? static_cast<size_t>(t0 + j) * ld_xbc + I + g * N + ck * 8 : 0;
      tq_cp16(sB + (ck >> 3) * kTSub + tq_swz(j, ck & 7), xbc + src, ok);
      tq_cp16(sC + (ck >> 3) * kTSub + tq_swz(j, ck & 7), xbc + src + (ok ? G * N : 0), ok);
    });
    commit();
    copy_x(0);
    commit();
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    fence_proxy_async();
  }
  const unsigned tmem_base = tq_tmem_alloc(&s_tmem, 256, warp);  // includes the __syncthreads after the copies
  volatile int* abort_flag = &s_abort;
  bool ok = true;
  auto wait_all = [&](unsigned long long* bar, unsigned parity, int code) {  // the same answer in a warp
    if (!__all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag))) {
      if (lane == 0) {
        if (!*abort_flag) atomicExch(status, code);
        s_abort = 1;
      }
      ok = false;
    }
    return ok;
  };
  const unsigned lead = lane == 0 ? 1u : 0u;
  const unsigned long long c_desc = umma_desc(sC), b_desc = umma_desc(sB);
  if (warp == kTOut / 32 && (!kTma || wait_all(&bar_cb, 0, 32))) {
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    for (int k = 0; k < N / 16; ++k)  // G = C B^T, K = the state columns
      umma_f16_lead(tmem_base, c_desc + (k >> 2) * (kTSub >> 4) + 2 * (k & 3), b_desc + (k >> 2) * (kTSub >> 4) + 2 * (k & 3),
                    tq_idesc(kTQ, false), k > 0 ? 1u : 0u, lead);
    umma_commit_lead(&bar_g, lead);
  }
  pdl_wait();  // the start states come from the launch before this one
  pdl_written(chunk_dt, start_state);
  if (kTma) {
    if (tid == kTOut) tma_s(0);
  } else if (worker) {
    copy_s(0);
    commit();
  }
  wait_all(&bar_g, 0, 32);
  const unsigned lane_base = tmem_base + (static_cast<unsigned>(rw * 32) << 16);
  unsigned char* sM = sB;
  int made = -1;  // the head whose M lies there
  for (int k = 0; k < n_units; ++k) {
    const int st = k & 1, h = head_of(k);
    const size_t col0 = col_of(k);
    const float Dh = d_skip[h];
    if (kTma) {
      wait_all(&bar_x[st], (k >> 1) & 1, 33);
      if (len < kTQ) {  // x's rows beyond the chunk belong to others: zero times what they hold is not always zero
        if (worker)
          for (int i = tid; i < (kTQ - len) * 8; i += kTOut)
            *reinterpret_cast<uint4*>(sX + st * kTSub + tq_swz(len + (i >> 3), i & 7)) = make_uint4(0u, 0u, 0u, 0u);
        fence_proxy_async();
      }
      wait_all(&bar_s[st], (k >> 1) & 1, 33);
    } else if (worker) {
      if (z_raw && z_vec)
        tq_pieces(tid, kTQ, PB / 8, [&](int j, int ck) {
          const bool in = j < len;
          tq_cp16(sZ + tq_swz(j, ck), z_raw + (in ? static_cast<long long>(t0 + j) * ld_z + col0 + ck * 8 : 0), in);
        });
      commit();
      asm volatile("cp.async.wait_group 1;\n" ::: "memory");  // the unit's state rows, x and decays
      fence_proxy_async();
    }
    if (!kTma) __syncthreads();
    if (warp == kTOut / 32) {
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      const unsigned long long s_desc = umma_desc(st ? sS1 : sS0);
      for (int i = 0; i < N / 16; ++i)  // Y2 = C S^T
        umma_f16_lead(tmem_base + 128, c_desc + (i >> 2) * (kTSub >> 4) + 2 * (i & 3), s_desc + (i >> 2) * (s_sub >> 4) + 2 * (i & 3),
                      tq_idesc(PB, false), i > 0 ? 1u : 0u, lead);
    }
    const float* s_delta = s_dt[st];
    const float* s_csl = s_dt[st] + kTQ;
    const float csl_i = s_csl[row];
    if (worker) {
      if (!kTma) {
        if (k + 1 < n_units) {  // the next unit's, while this one is worked on
          copy_s(k + 1);
          copy_x(k + 1);
        }
        commit();
      }
      // M[i][j] = G[i][j] exp(cs_i - cs_j) delta_j for j <= i, as the A operand of Y1 = M x, in B's place; this thread's 32 columns
      if (h != made) {
        const int jc = part;
        if (jc <= rw) {  // the warp's rows reach this block of 32 columns
          asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
          unsigned v[32];
          tmem_ld32(lane_base + jc * 32, v);
          asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
          for (int c8 = 0; c8 < 4; ++c8) {
            float m[8];
#pragma unroll
            for (int e = 0; e < 8; e += 4) {
              const int j = jc * 32 + c8 * 8 + e;
              const float4 cs4 = *reinterpret_cast<const float4*>(s_csl + j), de4 = *reinterpret_cast<const float4*>(s_delta + j);
              const float cs[4] = {cs4.x, cs4.y, cs4.z, cs4.w}, de[4] = {de4.x, de4.y, de4.z, de4.w};
#pragma unroll
              for (int q = 0; q < 4; ++q)
                m[e + q] = j + q <= row ? __uint_as_float(v[c8 * 8 + e + q]) * tq_ex2(csl_i - cs[q]) * de[q] : 0.f;
            }
            uint4 pk;
            pk.x = tq_pack(m[0], m[1]);
            pk.y = tq_pack(m[2], m[3]);
            pk.z = tq_pack(m[4], m[5]);
            pk.w = tq_pack(m[6], m[7]);
            const int ck = jc * 4 + c8;
            *reinterpret_cast<uint4*>(sM + (ck >> 3) * kTSub + tq_swz(row, ck & 7)) = pk;
          }
        } else if (made < 0) {  // (zeros stay)
#pragma unroll
          for (int c8 = 0; c8 < 4; ++c8) {
            const int ck = jc * 4 + c8;
            *reinterpret_cast<uint4*>(sM + (ck >> 3) * kTSub + tq_swz(row, ck & 7)) = make_uint4(0u, 0u, 0u, 0u);
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
        fence_proxy_async();
      }
      if (!kTma) asm volatile("cp.async.wait_group 1;\n" ::: "memory");  // the gate's inputs
    }
    made = h;
    __syncthreads();
    if (s_abort) break;  // (the same in every thread: the waits that raise it lie between the barriers of a round)
    if (warp == kTOut / 32) {
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      const unsigned long long m_desc = umma_desc(sM), x_desc = umma_desc(sX + st * kTSub);
#pragma unroll
      for (int i = 0; i < kTQ / 16; ++i)
        umma_f16_lead(tmem_base + 192, m_desc + (i >> 2) * (kTSub >> 4) + 2 * (i & 3), x_desc + ((i * 16 * 128) >> 4), tq_idesc(PB, true),
                      i > 0 ? 1u : 0u, lead);
      umma_commit_lead(&bar_y, lead);
      if (kTma && k + 1 < n_units && lane == 0) {  // the next unit's (the rows of the unit before have left that stage)
        tma_s(k + 1);
        tma_x(k + 1);
      }
      __syncwarp();
    }
    wait_all(&bar_y, k & 1, 33);
    if (kTma && gate_tile && worker) wait_all(&bar_z, k & 1, 33);
    unsigned char* xt = sX + st * kTSub;
    if (ok && worker) {
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      const float e_i = tq_ex2(csl_i);
      const bool row_ok = row < len;
      for (int pc = part; pc < PB / 16; pc += 4) {
        unsigned y1[16], y2[16];
        tmem_ld16(lane_base + 192 + pc * 16, y1);
        tmem_ld16(lane_base + 128 + pc * 16, y2);
        asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          const int ck = pc * 2 + hf;
          uint4* cell = reinterpret_cast<uint4*>(xt + tq_swz(row, ck));  // x in, y out: the product has read x
          const uint4 xq = *cell;
          const unsigned xw[4] = {xq.x, xq.y, xq.z, xq.w};
          unsigned zw[4] = {0u, 0u, 0u, 0u};
          if (z_raw) {
            if (z_vec) {
              const uint4 zq = *reinterpret_cast<const uint4*>(sZ + tq_swz(row, ck));
              zw[0] = zq.x, zw[1] = zq.y, zw[2] = zq.z, zw[3] = zq.w;
            } else if (row_ok) {  // rows of z that do not start on 16-byte boundaries
              const bf16* zp = z_raw + static_cast<long long>(t0 + row) * ld_z + col0 + ck * 8;
#pragma unroll
              for (int e2 = 0; e2 < 4; ++e2)
                zw[e2] = static_cast<unsigned>(__bfloat16_as_ushort(zp[2 * e2])) |
                         (static_cast<unsigned>(__bfloat16_as_ushort(zp[2 * e2 + 1])) << 16);
            }
          }
          unsigned out[4];
#pragma unroll
          for (int e2 = 0; e2 < 4; ++e2) {
            const float2 xv = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&xw[e2]));
            const int e = hf * 8 + e2 * 2;
            float v0 = __uint_as_float(y1[e]) + e_i * __uint_as_float(y2[e]) + Dh * xv.x;
            float v1 = __uint_as_float(y1[e + 1]) + e_i * __uint_as_float(y2[e + 1]) + Dh * xv.y;
            if (z_raw) {  // gate fused: y * silu(z), z = z_raw * z_scale + z_bias
              const float2 zv = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&zw[e2]));
              const size_t ch = col0 + ck * 8 + e2 * 2;
              v0 *= silu_fast(zv.x * z_scale + (z_bias ? z_bias[ch] : 0.f));
              v1 *= silu_fast(zv.y * z_scale + (z_bias ? z_bias[ch + 1] : 0.f));
            }
            out[e2] = tq_pack(v0, v1);
          }
          *cell = make_uint4(out[0], out[1], out[2], out[3]);
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    }
    if (kTma) fence_proxy_async();  // (a copy may take the place of what was read and written here)
    __syncthreads();
    if (s_abort) break;
    if (kTma && gate_tile && k + 1 < n_units && tid == kTOut) tma_z(k + 1);
    if (worker) {  // the finished rows go out in whole lines
      tq_pieces(tid, len, PB / 8, [&](int j, int ck) {
        *reinterpret_cast<uint4*>(y + static_cast<size_t>(t0 + j) * I + col0 + ck * 8) =
            *reinterpret_cast<const uint4*>(xt + tq_swz(j, ck));
      });
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  if (kTma && s_abort && tid == kTOut) {
    // copies that were asked for still write into this block's shared memory: a bounded time for them to land
    for (unsigned i = 0; i < kSpinLimit / 4; ++i) __nanosleep(32);
  }
  tq_tmem_free(tmem_base, 256, warp);
}

}  // namespace pmm

// Head sizes and state sizes the tcgen05 scan takes: multiples of 16, up to 128 and up to 256.
PMM_EXPORT int pmm_ssd_tc_supported(int P, int N) {
  return (P >= 16 && P <= 128 && P % 16 == 0 && N >= 16 && N <= 256 && N % 16 == 0) ? 1 : 0;
}

// xbc [T, ld_xbc] = [x | B | C] after the convolution; dt_raw [T, ld_dt]; state [slots, H, P, N]
// float.  Scratch: chunk_state n_chunks*H*P*N floats, chunk_decay n_chunks*H floats, chunk_dt
// n_chunks*H*256 floats, start_state n_chunks*H*P*N bfloat16 (16-byte aligned); n_chunks = sum over
// sequences of ceil(new tokens / 128).
// z_raw (or nullptr): the gate's input [T, ld_z], y <- y * silu(z_raw * z_scale + z_bias).
// n_tokens: rows of xbc (and z_raw).  walk_cols: 0 for phases 1 and 2 as two launches, 64 or 128 for the walk with blocks of so
// many state columns (N a multiple of them).
// skip_single: sequences that bring exactly one token are left alone (state and y): in a mixed step
// the token-serial kernel takes them (pmm_ssm_scan_seq with one_token = 2); n_multi is then the
// number of sequences that bring more than one token (0: not known).
// status: one int in device memory that stays 0 unless a bounded wait gave up.
PMM_EXPORT int pmm_ssd_tc(const void* xbc, int ld_xbc, const void* dt_raw, long long ld_dt, float dt_scale,
                          const float* dt_shift, const float* a_log, const float* d_skip, float* state, const int* cu,
                          const int* slots, void* y, float* chunk_state, float* chunk_decay, float* chunk_dt,
                          void* start_state, int n_seq, int n_tokens, int walk_cols, int n_chunks, int H, int P, int N, int G, const void* z_raw,
                          long long ld_z, float z_scale, const float* z_bias, int skip_single, int n_multi, int* status,
                          cudaStream_t stream) {
  using namespace pmm;
  if (n_seq <= 0 || n_chunks <= 0) return 0;
  if (!pmm_ssd_tc_supported(P, N) || H <= 0 || G <= 0 || H % G || n_seq > 65535 || !chunk_state || !chunk_decay ||
      !chunk_dt || !start_state || reinterpret_cast<uintptr_t>(start_state) % 16 || !status || ld_xbc % 8 ||
      reinterpret_cast<uintptr_t>(xbc) % 16 || reinterpret_cast<uintptr_t>(y) % 16)
    return PMM_ERR_BAD_ARGUMENT;
  const int z_vec = (z_raw && ld_z % 8 == 0 && reinterpret_cast<uintptr_t>(z_raw) % 16 == 0) ? 1 : 0;
  const int PB = P <= 64 ? P : (P % 64 == 0 ? 64 : (P % 48 == 0 ? 48 : (P % 32 == 0 ? 32 : 16)));
  const int nb = (N + 63) / 64;
  const int ch_per_group = (H / G) * P;
  const int slabs_per_group = (ch_per_group + kTQ - 1) / kTQ;
  if (static_cast<long long>(G) * slabs_per_group > 65535 || static_cast<long long>(H) * (P / PB) > 65535)
    return PMM_ERR_BAD_ARGUMENT;
  int tmem_cols = 32;
  while (tmem_cols < N) tmem_cols *= 2;
  const size_t smem1 = tq_state_smem(nb);
  const size_t smem3 = tq_output_smem(nb, PB);
  const int sms = 148;
  // Phase 3: as many units a block as keep the blocks within one an SM
  const int group_units = (H / G) * (P / PB);
  const int per_block = min(group_units, static_cast<int>((static_cast<long long>(n_chunks) * G * group_units + sms - 1) / sms));
  const int group_blocks = (group_units + per_block - 1) / per_block;
  // Whole tiles of 64 columns come by TMA: a unit's copies took its 512 threads 2,800 clocks of issue, of about 7,500.
  const bool tiles64 = N % 64 == 0 && n_tokens > 0, tma = PB == 64 && tiles64;
  const int NB = walk_cols;
  const bool walk = NB > 0;
  if (walk && ((NB != 64 && NB != 128) || !tiles64 || N % NB)) return PMM_ERR_BAD_ARGUMENT;
  CUtensorMap map_xbc{}, map_start{}, map_z{}, map_out{};
  if (tma || walk) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) return PMM_ERR_BAD_ARGUMENT;
    auto tiles_of = [&](CUtensorMap* map, const void* base, long long cols, long long rows, long long ld, unsigned box_rows) {
      const cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
      const cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld) * 2};
      const cuuint32_t box[2] = {64, box_rows}, elem[2] = {1, 1};
      return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    };
    const long long I = static_cast<long long>(H) * P;
    if (!tiles_of(&map_xbc, xbc, I + 2LL * G * N, n_tokens, ld_xbc, kTQ) || (tma && !tiles_of(&map_start, start_state, N, n_chunks * I, N, 64)) ||
        (walk && !tiles_of(&map_out, start_state, N, n_chunks * I, N, kTQ)) ||
        (tma && z_vec && !tiles_of(&map_z, z_raw, I, n_tokens, ld_z, kTQ)))
      return PMM_ERR_BAD_ARGUMENT;
  }
  // the opt-in to large shared memory holds for the current device: asked for at every call, always for the largest shape, so
  // that a call on another device or thread never finds less than it needs
  auto opt_in = [](const void* kern, size_t most) {
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(most));
  };
  auto output = tma ? ssd_tc_output_kernel<true> : ssd_tc_output_kernel<false>;
  cudaError_t e = opt_in(reinterpret_cast<const void*>(output), tq_output_smem(4, 64));
  if (e == cudaSuccess && !walk) e = opt_in(reinterpret_cast<const void*>(ssd_tc_state_kernel), tq_state_smem(4));
  if (e != cudaSuccess) return static_cast<int>(e);
  const bf16* xb = static_cast<const bf16*>(xbc);
  const bf16* dtb = static_cast<const bf16*>(dt_raw);
  if (walk) {
    auto kern = NB == 64 ? ssd_tc_walk_kernel<64> : ssd_tc_walk_kernel<128>;
    const size_t smem2 = tq_walk_smem(NB);
    e = opt_in(reinterpret_cast<const void*>(kern), smem2);
    if (e != cudaSuccess) return static_cast<int>(e);
    launch_pdl(kern, dim3(G * slabs_per_group * (N / NB), n_seq), dim3(kTWalkAll), smem2, stream, map_xbc, map_out, xb, ld_xbc, dtb, ld_dt, dt_scale,
               dt_shift, a_log, cu, slots, state, chunk_dt, static_cast<bf16*>(start_state), H, P, N, G, slabs_per_group, skip_single, status);
  } else {
    launch_pdl(ssd_tc_state_kernel, dim3(n_chunks, G * slabs_per_group), dim3(kTState), smem1, stream, xb, ld_xbc, dtb, ld_dt,
               dt_scale, dt_shift, a_log, cu, n_seq, chunk_state, chunk_decay, chunk_dt, H, P, N, G, slabs_per_group, tmem_cols,
               skip_single, status);
    int rc = launch_ssd_state_pass(chunk_state, chunk_decay, static_cast<bf16*>(start_state), state, cu, slots, n_seq, H,
                                   P * N, kTQ, skip_single, n_multi, stream);
    if (rc != 0) return rc;
  }
  launch_pdl(output, dim3(n_chunks, G * group_blocks), dim3(kTOutAll), smem3, stream, map_xbc, map_start, map_z, xb, ld_xbc,
             static_cast<const float*>(chunk_dt), d_skip, cu, n_seq, static_cast<const bf16*>(start_state),
             static_cast<bf16*>(y), H, P, N, G, PB, per_block, static_cast<const bf16*>(z_raw), ld_z, z_scale, z_bias, z_vec, skip_single, status);
  return launch_status();
}
