// Paged grouped-query attention for prompt portions on the fifth-generation tensor cores
// (bfloat16 storage, float accumulate, head size 64 or 128, page sizes that are multiples of 64).
//
// One block = 64 or 128 query rows of ONE sequence and ONE key/value head (a row is a (token, query
// head of the group) pair, as in the mma.sync kernel) and one key split.  It walks its keys in
// tiles of 128:
//   S  = Q K^T     tcgen05.mma, both operands in shared memory: Q written there by the block's
//                  threads (128-byte swizzle by hand), the K tile brought by TMA straight from the
//                  cache pages (two boxes of 64 keys, each inside one page); S (rows x 128 float)
//                  lands in tensor memory;
//   P  = softmax   a warp per 16 rows, FOUR THREADS PER ROW: tcgen05.ld in the 16x128b shape gives
//                  thread k of a quad the columns 4 i + k of two rows, so the row's sum in four
//                  interleaved partial sums needs no order of its own and the maximum two shuffles;
//                  P goes to shared memory as bfloat16 (a shuffle pairs neighbouring columns; the
//                  32 stores of a thread are free of bank conflicts), swizzled as an mma operand,
//                  and is handed over with fence.proxy.async + mbarrier;
//   O += P V       tcgen05.mma with the V tile as an MN-major operand (rows = keys, as the cache
//                  stores them), accumulated in a second tensor-memory range over all tiles.  The
//                  running maximum that the exponentials are taken against is only raised when a
//                  row's true maximum exceeds it by more than 8 (a factor 256, harmless in
//                  bfloat16 and float); only then the accumulated O and sum are rescaled (a
//                  tensor-memory load, multiply and store by the row's threads).  The result is
//                  exact: P, the sum and O always refer to the same maximum.
// Warp roles: 0 = TMA producer (a ring of three tiles in the order of the products, K_0 K_1 V_0 K_2
// V_1 ...), 1 = tensor-memory owner and MMA issuer (S of the next tile is issued as soon as the
// softmax threads have taken the current S into registers, so the tensor core works while they
// compute; the whole warp walks and one lane issues by predicate, 50 clocks a product instead of 90
// inside a branch), the others softmax and output.  Head size 64: 72 KB (64 rows) or 96 KB (128
// rows) of shared memory and 128 or 256 columns of tensor memory a block, two blocks per SM.  Head
// size 128: every tile is two sub-tiles of 64 head-size columns, one block per SM.
// What bounds it: a tile is a serial chain of load, maximum, exponentials and hand-over in each
// warp, 1,900 clocks at 64 rows, of them 1,000 for the exponentials where two blocks share an SM's
// special-function units (512 alone).  One thread per row (four warps, 128 values each) took 3,100
// clocks a tile and 6 us around the tiles (divisions, uncoalesced output) where this takes 3.  At 8
// query and 2 key/value heads of 64 (us, that form / this): 2,048 tokens 32.0 / 21.3, behind a
// window of 1,024 23.1 / 16.1, 300 tokens 11.2 / 6.7; 12 and 2 heads of 128, 1,024 tokens 22.9 /
// 17.8.  Both forms give the same bits.
// With several key splits the block writes (max, sum, unnormalised output) and the last block of
// a row tile merges them, as in the mma.sync kernel.  Every mbarrier wait is bounded (status
// codes 11..15 in *status, the block then leaves its loops, waits for its copies in flight and
// frees its tensor memory).  No cluster multicast.
//   sc[s] = (q.K[s]) * scale;  p = exp(sc - max);  o = sum p V / sum p
// (reference src/ops/gpu/attention.cu:44-105), keys lo..pos per token, lo from the window.
#include "tcgen05.cuh"
#include <math_constants.h>

namespace pmm {

using bf16 = __nv_bfloat16;

constexpr int kAtKeys = 128;    // keys per tile
constexpr int kAtBox = 64;      // keys per TMA box (inside one page)
constexpr int kAtDhBlock = 64;  // head-size columns per sub-tile (128 bytes of bfloat16)
constexpr float kAtLazy = 8.f;  // how far (log2) a row's maximum may run ahead of the one in use
constexpr int kAtBoxCap = 512;  // boxes of the block's key range whose rows of the pool are kept in shared memory
constexpr int kAtKvSub = kAtKeys * kAtDhBlock * 2;  // 16 KB: 128 keys x 64 head-size columns
constexpr int kAtRing = 3;                          // K and V tiles in flight
__host__ __device__ constexpr int at_q_sub(int rows) { return rows * kAtDhBlock * 2; }      // a sub-tile of Q (64 head-size columns) or of P (64 keys)
__host__ __device__ constexpr int at_threads(int rows) { return 64 + 2 * rows; }            // producer, issuer, a warp per 16 rows
__host__ __device__ constexpr size_t at_smem(int dh, int rows) {  // Q, the ring (each head size / 64 sub-tiles), P
  return static_cast<size_t>(dh / kAtDhBlock) * (at_q_sub(rows) + kAtRing * kAtKvSub) + 2 * at_q_sub(rows) + 1024 /*alignment*/;
}
// Tensor memory.  128 rows: S in columns 0..127, O behind it.  64 rows: a product leaves row i in lane 32 (i / 16) + i % 16,
// so S takes the lower 16 lanes of every warp's 32 and O the upper 16 of the same columns.
__host__ __device__ constexpr int at_tmem_cols(int rows) { return rows == 64 ? 128 : 256; }
__host__ __device__ constexpr unsigned at_o_offset(int rows) { return rows == 64 ? (16u << 16) : static_cast<unsigned>(kAtKeys); }

// kind::f16 instruction descriptors: float accumulate, bfloat16 operands, A K-major.
__host__ __device__ constexpr unsigned at_idesc_s(int rows) {  // B = K tile, K-major
  return (1u << 4) | (1u << 7) | (1u << 10) | ((kAtKeys >> 3) << 17) | (static_cast<unsigned>(rows >> 4) << 24);
}
__host__ __device__ constexpr unsigned at_idesc_o(int rows) {  // B = 64 columns of the V tile, MN-major
  return (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((kAtDhBlock >> 3) << 17) | (static_cast<unsigned>(rows >> 4) << 24);
}

__device__ __forceinline__ float at_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ unsigned at_pack(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const unsigned*>(&v);
}
// Byte offset of 16-byte chunk `chunk` (0..7) of row `row` in a [rows][64] bfloat16 tile with the
// 128-byte swizzle that TMA and the tensor core use (8-row groups of 1024 bytes).
__device__ __forceinline__ int at_swizzled(int row, int chunk) {
  return (row >> 3) * 1024 + (row & 7) * 128 + ((chunk ^ (row & 7)) << 4);
}

// 16 lanes of tensor memory x 64 columns: lane l of the warp gets columns 4 i + l % 4 of rows l / 4 (r[2 i]) and l / 4 + 8 (r[2 i + 1]).
__device__ __forceinline__ void at_tmem_ld(unsigned taddr, unsigned* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x128b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
// The same for 32 columns, and its store.
__device__ __forceinline__ void at_tmem_ld32(unsigned taddr, unsigned* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x128b.x8.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void at_tmem_st32(unsigned taddr, const unsigned* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.16x128b.x8.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};\n"
      :
      : "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
// Two columns' values of one row, k = column % 4 of this lane: columns 4 i + k (x0) and 4 i + 4 + k (x1), i even, become the
// word (two neighbouring bfloat16) of the row's 16-byte piece i / 2 that this lane owns, word 2 (k & 1) + (k >> 1).
__device__ __forceinline__ unsigned at_pair(float x0, float x1, unsigned sel) {
  const unsigned own = at_pack(x0, x1);
  return __byte_perm(own, __shfl_xor_sync(0xffffffffu, own, 1), sel);
}
__device__ __forceinline__ float at_max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;\n" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// Place of a tile among the copies: K_0, K_1, V_0, K_2, V_1, ..., K_{n-1}, V_{n-2}, V_{n-1}, the order of the products.
__device__ __forceinline__ int at_k_item(int j) { return j == 0 ? 0 : 2 * j - 1; }
__device__ __forceinline__ int at_v_item(int j, int n) { return j + 1 < n ? 2 * j + 2 : 2 * j + 1; }

template <int DH, int M>
__global__ void __launch_bounds__(at_threads(M), DH == 64 ? 2 : 1)
    attention_tc_kernel(const bf16* __restrict__ q, const __grid_constant__ CUtensorMap map_kv,
                        const int* __restrict__ block_table, int max_blocks, const int* __restrict__ positions,
                        const int* __restrict__ cu, bf16* __restrict__ out, float* __restrict__ part_o,
                        float* __restrict__ part_ml, float scale_log2, int window, int split_len, int n_splits,
                        int page_size, int n_seq, int Hq, int Hkv, int* __restrict__ split_counter,
                        int* __restrict__ status, const float* __restrict__ sink, float* __restrict__ lse) {
  pdl_launch_dependents();
  constexpr int NSUB = DH / kAtDhBlock;            // sub-tiles of 64 head-size columns
  constexpr int kThreads = at_threads(M);
  constexpr int kWarps = M / 16;                   // softmax warps
  constexpr int kQSub = at_q_sub(M);
  constexpr int kSlot = NSUB * kAtKvSub;           // a K or V tile
  constexpr unsigned kOff = at_o_offset(M);
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) unsigned long long bar_q, bar_full[kAtRing], bar_empty[kAtRing], bar_s, bar_sfree, bar_p, bar_pv;
  __shared__ unsigned s_tmem_base;
  __shared__ int s_abort, s_last;
  __shared__ int s_row[kAtBoxCap];

  unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* sQ = tiles;
  unsigned char* sRing = sQ + NSUB * kQSub;
  unsigned char* sP = sRing + kAtRing * kSlot;

  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // (known to be the same in the whole warp)
  const int G = Hq / Hkv;
  const int tpt = M / G;  // tokens per tile; rows beyond tpt * G stay empty when G does not divide M
  // heavy tiles first (as in the mma.sync kernel), those of all key/value heads together
  const int n_row_tiles = static_cast<int>(gridDim.x) / Hkv;
  const int hk = static_cast<int>(blockIdx.x) % Hkv, z = blockIdx.y;
  const int tile_id = n_row_tiles - 1 - static_cast<int>(blockIdx.x) / Hkv;

  // Sequence bounds, positions and block tables are inputs of the step, written before its first kernel: they are read
  // before the wait for the kernel before this one.
  // Which sequence and which of its tokens this tile covers:
  int seq = 0, acc = 0;
  for (; seq < n_seq; ++seq) {
    const int n = cu[seq + 1] - cu[seq];
    const int nt = (n + tpt - 1) / tpt;
    if (tile_id < acc + nt) break;
    acc += nt;
  }
  if (seq >= n_seq) return;
  const int tok0 = cu[seq] + (tile_id - acc) * tpt;
  const int n_tok = min(cu[seq + 1], tok0 + tpt) - tok0;
  const int n_rows = n_tok * G;
  const int* bt = block_table + static_cast<size_t>(seq) * max_blocks;
  const int pos_min = positions[tok0], pos_max = positions[tok0 + n_tok - 1];
  // (64-row tiles, groups that divide 64: the keys are cut into tiles as for the 128 rows that hold this tile's, so that a row's
  // sums do not depend on the tile's height)
  const int lo_tok = M == 64 && tpt * G == M && ((tile_id - acc) & 1) ? tok0 - tpt : tok0;
  const int lo_all = first_visible(lo_tok == tok0 ? pos_min : positions[lo_tok], window);
  const int k_begin = max(lo_all, z * split_len);
  const int k_end = min(pos_max + 1, (z + 1) * split_len);
  const int first = (k_begin / kAtBox) * kAtBox;  // boxes start on multiples of 64 keys: inside one page
  const int n_tiles = k_end > k_begin ? (k_end - first + kAtKeys - 1) / kAtKeys : 0;
  // The row of the pool at which the keys of box b (keys first + 64 b ...) begin.  A box that starts beyond the keys of this
  // block is read from the tile's first page instead (any real page: its scores are masked, its values multiplied by zero).
  auto box_row = [&](int b) {
    int key = first + b * kAtBox;
    if (key >= k_end) key -= kAtBox;
    const int idx = key / page_size;
    return bt[idx] * 2 * page_size + (key - idx * page_size);
  };

  if (tid == 0) {
    mbar_init(&bar_q, kWarps);
#pragma unroll
    for (int i = 0; i < kAtRing; ++i) {
      mbar_init(&bar_full[i], 1);
      mbar_init(&bar_empty[i], 1);
    }
    mbar_init(&bar_s, 1);
    mbar_init(&bar_sfree, kWarps);
    mbar_init(&bar_p, kWarps);
    mbar_init(&bar_pv, 1);
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    asm volatile("prefetch.tensormap [%0];\n" ::"l"(reinterpret_cast<unsigned long long>(&map_kv)) : "memory");
  }
  for (int b = tid; b < min(2 * n_tiles, kAtBoxCap); b += kThreads) s_row[b] = box_row(b);
  // the softmax threads' places: a warp takes 16 rows; 128 rows: which 16 of the 32 tensor-memory lanes that a warp may read
  const int half = (warp - 2) >> 2;
  const int base_row = M == 64 ? (warp & 3) * 16 : (warp & 3) * 32 + half * 16;
  int piece_off[DH / 16];  // 16-byte pieces of the warp's query rows and output rows, a lane each: offset from token tok0, -1: no row
  int my_pos[2] = {-1, -1};
  if (warp > 1) {
#pragma unroll
    for (int i = 0; i < DH / 16; ++i) {
      const int piece = lane + 32 * i;
      const int rr = base_row + piece / (DH / 8), c = piece % (DH / 8);
      const int tk = rr / G;
      piece_off[i] = rr < n_rows ? (tk * Hq + hk * G + (rr - tk * G)) * DH + c * 8 : -1;
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int row = base_row + (lane >> 2) + 8 * r;
      if (row < n_rows) my_pos[r] = positions[tok0 + row / G];
    }
  }
  const size_t q_base = static_cast<size_t>(tok0) * Hq * DH;
  pdl_wait();
  pdl_written(q);
  uint4 q_piece[DH / 16];
  if (warp > 1) {
#pragma unroll
    for (int i = 0; i < DH / 16; ++i)
      q_piece[i] = piece_off[i] >= 0 ? *reinterpret_cast<const uint4*>(q + q_base + piece_off[i]) : make_uint4(0u, 0u, 0u, 0u);
  }
  // (tensor memory only behind the wait: the kernel before this one may need it to finish)
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&s_tmem_base)), "r"(at_tmem_cols(M)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const unsigned tmem_base = s_tmem_base;
  volatile int* abort_flag = &s_abort;
  auto give_up = [&](int code) {
    if (!*abort_flag) atomicExch(status, code);
    s_abort = 1;
  };

  if (warp == 0) {
    // ---------------------------------------------------------------- TMA producer
    if (n_tiles > 0) {
      const int items = 2 * n_tiles;
      int issued = 0;
      auto request = [&](int it) {  // one lane: the copy of item `it` into its slot
        const int slot = it % kAtRing;
        // which tile: K at odd places (and the first), V at even ones (and the last)
        const bool is_v = it == items - 1 || (it > 0 && it % 2 == 0);
        const int j = is_v ? (it == items - 1 ? n_tiles - 1 : it / 2 - 1) : (it + 1) / 2;
        const int plane = is_v ? page_size : 0;
        const int r0 = (2 * j < kAtBoxCap ? s_row[2 * j] : box_row(2 * j)) + plane;
        const int r1 = (2 * j + 1 < kAtBoxCap ? s_row[2 * j + 1] : box_row(2 * j + 1)) + plane;
        unsigned char* dst = sRing + slot * kSlot;
        mbar_expect_tx(&bar_full[slot], kSlot);
#pragma unroll
        for (int d = 0; d < NSUB; ++d) {  // a sub-tile = 64 head-size columns of 128 keys: two boxes of 64 keys
          tma_load_2d(dst + d * kAtKvSub, &map_kv, hk * DH + d * kAtDhBlock, r0, &bar_full[slot]);
          tma_load_2d(dst + d * kAtKvSub + kAtKvSub / 2, &map_kv, hk * DH + d * kAtDhBlock, r1, &bar_full[slot]);
        }
      };
      if (lane < min(kAtRing, items)) request(lane);  // the first filling: a lane a slot
      issued = min(kAtRing, items);
      __syncwarp();
      bool ok = true;
      for (int it = kAtRing; it < items && ok; ++it) {
        if (lane == 0) {
          ok = mbar_wait(&bar_empty[it % kAtRing], (it / kAtRing - 1) & 1, abort_flag);  // the product that read the slot has finished
          if (ok) {
            request(it);
            issued = it + 1;
          } else {
            give_up(12);
          }
        }
      }
      if (lane == 0 && s_abort) {
        // copies already requested still write into this block's shared memory: wait for them
        for (int it = max(0, issued - kAtRing); it < issued; ++it)
          for (unsigned i = 0; i < kSpinLimit && !mbar_try_wait(&bar_full[it % kAtRing], (it / kAtRing) & 1); ++i) {
          }
      }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issuer (the whole warp walks, one lane issues)
    if (n_tiles > 0) {
      const int items = 2 * n_tiles;
      const unsigned lead = lane == 0 ? 1u : 0u;
      const unsigned long long q_desc = umma_desc(sQ), p_desc = umma_desc(sP), ring_desc = umma_desc(sRing);
      auto wait = [&](unsigned long long* bar, unsigned parity) {
        const bool got = mbar_wait(bar, parity, abort_flag);
        __syncwarp();  // (no lane may fall a phase behind)
        return got;
      };
      auto full = [&](int it) { return wait(&bar_full[it % kAtRing], (it / kAtRing) & 1); };
      auto issue_s = [&](int j) {  // S_j = Q K_j^T
        const int slot = at_k_item(j) % kAtRing;
        const unsigned long long k_desc = ring_desc + static_cast<unsigned>(slot * (kSlot >> 4));
#pragma unroll
        for (int k = 0; k < DH / 16; ++k)  // 16 head-size columns a step, four steps a sub-tile
          umma_f16_lead(tmem_base, q_desc + (k >> 2) * (kQSub >> 4) + 2 * (k & 3), k_desc + (k >> 2) * (kAtKvSub >> 4) + 2 * (k & 3),
                  at_idesc_s(M), k > 0 ? 1u : 0u, lead);
        umma_commit_lead(&bar_s, lead);
        if (at_k_item(j) + kAtRing < items) umma_commit_lead(&bar_empty[slot], lead);  // (nobody waits for the last copies' slots)
      };
      int code = 0;
      if (wait(&bar_q, 0) && full(0)) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        issue_s(0);
      } else {
        code = 13;
      }
      for (int j = 0; j < n_tiles && code == 0; ++j) {
        if (j + 1 < n_tiles) {
          // the softmax threads hold S_j in registers: the next S may overwrite it, and the
          // tensor core works on it while they compute
          if (!full(at_k_item(j + 1)) || !wait(&bar_sfree, j & 1)) {
            code = 13;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
          issue_s(j + 1);
        }
        const int v_item = at_v_item(j, n_tiles);
        if (!full(v_item) || !wait(&bar_p, j & 1)) {
          code = 14;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        // O += P V_j: A = P (two sub-tiles of 64 keys), B = V rows as they lie in the cache
        // (MN-major): 16 keys further = 16 rows of 128 bytes
        const int slot = v_item % kAtRing;
        const unsigned long long v_desc = ring_desc + static_cast<unsigned>(slot * (kSlot >> 4));
#pragma unroll
        for (int d = 0; d < NSUB; ++d)  // 64 head-size columns of O an instruction
#pragma unroll
          for (int k = 0; k < kAtKeys / 16; ++k)
            umma_f16_lead(tmem_base + kOff + d * kAtDhBlock, p_desc + (k / 4) * (kQSub >> 4) + 2 * (k % 4),
                    v_desc + d * (kAtKvSub >> 4) + ((k * 16 * 128) >> 4), at_idesc_o(M), (j > 0 || k > 0) ? 1u : 0u, lead);
        umma_commit_lead(&bar_pv, lead);
        if (v_item + kAtRing < items) umma_commit_lead(&bar_empty[slot], lead);
      }
      if (code != 0) give_up(code);
    }
  } else {
    // ---------------------------------------------------------------- softmax and output (a warp per 16 rows)
    const unsigned lane_base = tmem_base + (static_cast<unsigned>((warp & 3) * 32 + half * 16) << 16);
    if (n_tiles > 0) {
      // the warp's query rows -> shared memory, swizzled (rows beyond the tile are zero)
#pragma unroll
      for (int i = 0; i < DH / 16; ++i) {
        const int piece = lane + 32 * i;
        const int rr = base_row + piece / (DH / 8), c = piece % (DH / 8);
        *reinterpret_cast<uint4*>(sQ + (c >> 3) * kQSub + at_swizzled(rr, c & 7)) = q_piece[i];
      }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_q);
    }
    const int k4 = lane & 3;                              // this thread's columns: 4 i + k4
    const unsigned sel = (k4 & 1) ? 0x3276u : 0x5410u;    // see at_pair
    unsigned char* p_row = sP + ((k4 & 1) * 2 + (k4 >> 1)) * 4;  // this thread's word of a piece
    int my_lo[2];
    float m_run[2], l_run[2];  // the maximum in use (exponent's unit) and the sum against it
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      my_lo[r] = max(first_visible(my_pos[r], window), k_begin);
      m_run[r] = -CUDART_INF_F;
      l_run[r] = 0.f;
    }
    const int row0 = base_row + (lane >> 2);  // (row0 + 8 has the same swizzle: 1,024 bytes further)
    const int full_lo = max(k_begin, first_visible(pos_max, window)), full_hi = min(k_end, pos_min + 1);
    bool alive = true;
    float sum[2] = {0.f, 0.f}, alpha[2] = {1.f, 1.f};
    // a row's sum over a tile in the order of four interleaved partial sums (a thread's columns are one of them)
    auto take_sums = [&]() {
      float t0 = sum[0] + __shfl_xor_sync(0xffffffffu, sum[0], 1), t1 = sum[1] + __shfl_xor_sync(0xffffffffu, sum[1], 1);
      t0 += __shfl_xor_sync(0xffffffffu, t0, 2);
      t1 += __shfl_xor_sync(0xffffffffu, t1, 2);
      l_run[0] = l_run[0] * alpha[0] + t0;
      l_run[1] = l_run[1] * alpha[1] + t1;
    };
    for (int j = 0; j < n_tiles; ++j) {
      const int base = first + j * kAtKeys;
      bool ok = mbar_wait(&bar_s, j & 1, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) {
        if (lane == 0) give_up(15);
        alive = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      // this thread's quarter of two rows of S into registers, then the tensor memory is free for the next S
      unsigned v[kAtKeys / 2];
      at_tmem_ld(lane_base, v);
      at_tmem_ld(lane_base + 64, v + 32);
      if (j > 0) take_sums();  // (of the tile before, while these travel)
      asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_sfree);
      // a tile that every row of the block may read in full needs no mask
      if (base < full_lo || base + kAtKeys > full_hi) {
#pragma unroll
        for (int i = 0; i < kAtKeys / 4; ++i) {
          const int key = base + 4 * i + k4;
#pragma unroll
          for (int r = 0; r < 2; ++r)
            if (!(key <= my_pos[r] && key >= my_lo[r] && key < k_end)) v[2 * i + r] = __float_as_uint(-CUDART_INF_F);
        }
      }
      float mx[2][2];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        mx[r][0] = fmaxf(__uint_as_float(v[r]), __uint_as_float(v[2 + r]));
        mx[r][1] = fmaxf(__uint_as_float(v[4 + r]), __uint_as_float(v[6 + r]));
      }
#pragma unroll
      for (int i = 4; i < kAtKeys / 4; i += 4)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          mx[r][0] = at_max3(mx[r][0], __uint_as_float(v[2 * i + r]), __uint_as_float(v[2 * i + 2 + r]));
          mx[r][1] = at_max3(mx[r][1], __uint_as_float(v[2 * i + 4 + r]), __uint_as_float(v[2 * i + 6 + r]));
        }
      mx[0][0] = fmaxf(mx[0][0], mx[0][1]);
      mx[1][0] = fmaxf(mx[1][0], mx[1][1]);
#pragma unroll
      for (int o = 1; o <= 2; ++o) {
        const float o0 = __shfl_xor_sync(0xffffffffu, mx[0][0], o), o1 = __shfl_xor_sync(0xffffffffu, mx[1][0], o);
        mx[0][0] = fmaxf(mx[0][0], o0);
        mx[1][0] = fmaxf(mx[1][0], o1);
      }
      float mu[2];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const float m = mx[r][0] * scale_log2;  // scale > 0
        // raise the maximum in use only when the row's maximum has run ahead of it by more than kAtLazy
        const bool raise = (m > m_run[r] + kAtLazy || m_run[r] == -CUDART_INF_F) && m != -CUDART_INF_F;
        alpha[r] = raise ? at_ex2(m_run[r] - m) : 1.f;  // 0 for the first visible tile
        m_run[r] = raise ? m : m_run[r];
        mu[r] = (m_run[r] == -CUDART_INF_F) ? 0.f : m_run[r];
      }
      if (j > 0) {
        // P V_{j-1} must have finished: it read the P tile that is written below, and it wrote O
        ok = mbar_wait(&bar_pv, (j - 1) & 1, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) {
          if (lane == 0) give_up(15);
          alive = false;
          break;
        }
        if (__any_sync(0xffffffffu, alpha[0] != 1.f || alpha[1] != 1.f)) {
          asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll
          for (int c = 0; c < DH / 32; ++c) {
            unsigned ov[16];
            at_tmem_ld32(lane_base + kOff + c * 32, ov);
            asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
            for (int e = 0; e < 16; ++e) ov[e] = __float_as_uint(__uint_as_float(ov[e]) * alpha[e & 1]);
            at_tmem_st32(lane_base + kOff + c * 32, ov);
          }
          asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
        }
      }
      // P: four columns of both rows at a time, the exponentials of one group ahead of the packing of the one before
      sum[0] = sum[1] = 0.f;
      float p[2][4];
      auto exps = [&](int g, float* dst) {  // columns 8 g + k4 and 8 g + 4 + k4 of both rows
#pragma unroll
        for (int e = 0; e < 4; ++e) dst[e] = at_ex2(fmaf(__uint_as_float(v[4 * g + e]), scale_log2, -mu[e & 1]));  // masked: ex2(-inf) = 0
      };
      exps(0, p[0]);
#pragma unroll
      for (int g = 0; g < kAtKeys / 8; ++g) {
        float* cur = p[g & 1];
        if (g + 1 < kAtKeys / 8) exps(g + 1, p[(g + 1) & 1]);
        unsigned char* dst = p_row + (g >> 3) * kQSub + at_swizzled(row0, g & 7);
        sum[0] += cur[0];
        sum[1] += cur[1];
        sum[0] += cur[2];
        sum[1] += cur[3];
        *reinterpret_cast<unsigned*>(dst) = at_pair(cur[0], cur[2], sel);
        *reinterpret_cast<unsigned*>(dst + 1024) = at_pair(cur[1], cur[3], sel);
      }
      asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_p);
    }
    if (alive && n_tiles > 0) take_sums();

    // ---- this block's result: O from tensor memory once the last product has finished
    constexpr float kLn2 = 0.6931471805599453f;
    const bool row_ok[2] = {row0 < n_rows, row0 + 8 < n_rows};
    size_t out_row[2] = {0, 0};  // (token, query head) of this thread's rows, where it is asked for
    float corr[2] = {1.f, 1.f};
    if (sink != nullptr || lse != nullptr || n_splits > 1) {
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int row = row0 + 8 * r, tk = row / G, hq = hk * G + (row - tk * G);
        out_row[r] = static_cast<size_t>(tok0 + tk) * Hq + hq;
        if (sink != nullptr && z == 0 && row_ok[r]) {
          // a score without key or value that counts once: it joins the first key range (which may
          // hold no key); maxima are kept in units of log 2
          const float sk = sink[hq] * 1.4426950408889634f;
          const float m_new = fmaxf(m_run[r], sk);
          corr[r] = exp2f(m_run[r] - m_new);
          l_run[r] = l_run[r] * corr[r] + exp2f(sk - m_new);
          m_run[r] = m_new;
        }
      }
    }
    const float inv[2] = {l_run[0] > 0.f ? 1.f / l_run[0] : 0.f, l_run[1] > 0.f ? 1.f / l_run[1] : 0.f};
    if (alive && n_tiles > 0) {
      const bool ok = mbar_wait(&bar_pv, (n_tiles - 1) & 1, abort_flag);
      if (!ok && lane == 0) give_up(15);
      alive = ok;
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    }
    if (__all_sync(0xffffffffu, alive && !*abort_flag)) {
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        // (for a later merge with keys outside this launch's range: the row's maximum in natural-log units and sum)
        if (k4 == 0 && row_ok[r]) {
          if (n_splits > 1)
            *reinterpret_cast<float2*>(part_ml + (out_row[r] * n_splits + z) * 2) = make_float2(m_run[r] * kLn2, l_run[r]);
          else if (lse != nullptr)
            *reinterpret_cast<float2*>(lse + out_row[r] * 2) = make_float2(m_run[r] * kLn2, l_run[r]);
        }
      }
#pragma unroll
      for (int c = 0; c < NSUB; ++c) {
        unsigned o[32];
#pragma unroll
        for (int e = 0; e < 32; ++e) o[e] = 0u;
        if (n_tiles > 0) {
          at_tmem_ld(lane_base + kOff + c * 64, o);
          asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
        }
        if (n_splits == 1) {  // the rows go out in whole pieces, through this warp's rows of P's tiles
#pragma unroll
          for (int g = 0; g < 8; ++g) {
            unsigned char* dst = p_row + c * kQSub + at_swizzled(row0, g);
#pragma unroll
            for (int r = 0; r < 2; ++r)
              *reinterpret_cast<unsigned*>(dst + 1024 * r) = at_pair(__uint_as_float(o[4 * g + r]) * corr[r] * inv[r],
                                                                    __uint_as_float(o[4 * g + 2 + r]) * corr[r] * inv[r], sel);
          }
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) {
#pragma unroll
            for (int r = 0; r < 2; ++r)
              if (row_ok[r])
                part_o[(out_row[r] * n_splits + z) * DH + c * 64 + 4 * i + k4] = __uint_as_float(o[2 * i + r]) * corr[r];
          }
        }
      }
      if (n_splits == 1) {
        __syncwarp();
#pragma unroll
        for (int i = 0; i < DH / 16; ++i) {
          const int piece = lane + 32 * i;
          const int rr = base_row + piece / (DH / 8), c = piece % (DH / 8);
          if (piece_off[i] >= 0)
            *reinterpret_cast<uint4*>(out + q_base + piece_off[i]) =
                *reinterpret_cast<const uint4*>(sP + (c >> 3) * kQSub + at_swizzled(rr, c & 7));
        }
      }
    }
  }

  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(at_tmem_cols(M)) : "memory");
  }

  // The block that finishes a row tile's last key split merges all of them (the counter returns
  // to zero for the next use).
  if (n_splits > 1) {
    __threadfence();
    __syncthreads();
    int* counter = split_counter + static_cast<size_t>(tile_id) * Hkv + hk;
    if (tid == 0) s_last = (atomicAdd(counter, 1) == n_splits - 1);
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    if (tid == 0) *counter = 0;
    constexpr int C4 = DH / 4;
    constexpr int kBatch = 8;
    for (int i = tid; i < n_rows * C4; i += kThreads) {
      const int r = i / C4, d = (i % C4) * 4;
      const int t = tok0 + r / G, hq = hk * G + r % G;
      const size_t orow = static_cast<size_t>(t) * Hq + hq;
      const float2* ml = reinterpret_cast<const float2*>(part_ml + orow * n_splits * 2);
      const float* po = part_o + orow * n_splits * DH + d;
      float mx = -CUDART_INF_F, tot = 0.f;
      float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int z0 = 0; z0 < n_splits; z0 += kBatch) {
        float2 v[kBatch];
        float4 x[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
          const int zz = min(z0 + u, n_splits - 1);
          v[u] = __ldcg(ml + zz);
          x[u] = __ldcg(reinterpret_cast<const float4*>(po + static_cast<size_t>(zz) * DH));
        }
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
          if (z0 + u < n_splits && v[u].y > 0.f) {
            const float mn = fmaxf(mx, v[u].x);
            const float keep = expf(mx - mn), w = expf(v[u].x - mn);  // mx = -inf: keep = 0
            a.x = a.x * keep + w * x[u].x;
            a.y = a.y * keep + w * x[u].y;
            a.z = a.z * keep + w * x[u].z;
            a.w = a.w * keep + w * x[u].w;
            tot = tot * keep + w * v[u].y;
            mx = mn;
          }
        }
      }
      const float inv = tot > 0.f ? 1.f / tot : 0.f;
      uint2 packed;
      packed.x = at_pack(a.x * inv, a.y * inv);
      packed.y = at_pack(a.z * inv, a.w * inv);
      *reinterpret_cast<uint2*>(out + orow * DH + d) = packed;
    }
  }
}

}  // namespace pmm

// Whether the tcgen05 attention takes this shape: head size 64 or 128, up to 64 query heads per
// key/value head (a tile of `rows` rows, 64 or 128, holds floor(rows / group) tokens; with a group
// size that does not divide them its last rows stay empty), pages that hold whole boxes of 64 keys.
PMM_EXPORT int pmm_attention_tc_supported(int Hq, int Hkv, int Dh, int page_size) {
  if (Hkv <= 0 || Hq % Hkv) return 0;
  const int G = Hq / Hkv;
  return ((Dh == 64 || Dh == 128) && G <= 64 && page_size > 0 && page_size % pmm::kAtBox == 0) ? 1 : 0;
}

// q [T, Hq*Dh] rotated queries; pool [n_pages + spare, 2, page_size, Hkv*Dh]; rows: 64 or 128 (token,
// query head of a group) rows a block; n_tiles = sum over sequences of ceil(new tokens / floor(rows /
// G)), or more (surplus blocks leave).  Several key splits need part_o / part_ml and split_counter
// (n_tiles * Hkv ints, zero between calls; at most 64 splits, split_len a multiple of 64).  positions,
// cu and block_table are read ahead of the wait: see launch_pdl.  status: one int, stays 0 unless a
// bounded wait gave up.
PMM_EXPORT int pmm_attention_tc(const void* q, const void* pool, long long pool_pages, const int* block_table,
                                int max_blocks, const int* positions, const int* cu, void* out, float* part_o,
                                float* part_ml, float scale, int window, int split_len, int n_splits, int page_size,
                                int n_seq, int n_tiles, int rows, int Hq, int Hkv, int Dh, int* split_counter, int* status,
                                const float* sink, float* lse, cudaStream_t stream) {
  if (n_seq <= 0 || n_tiles <= 0) return 0;
  if (lse && n_splits != 1) return PMM_ERR_BAD_ARGUMENT;
  if (rows != 64 && rows != 128) return PMM_ERR_BAD_ARGUMENT;
  if (!pmm_attention_tc_supported(Hq, Hkv, Dh, page_size) || !status || !(scale > 0.f) || n_splits < 1 ||
      n_splits > 64 || Hkv > 65535 || pool_pages <= 0 || reinterpret_cast<uintptr_t>(pool) % 16 ||
      reinterpret_cast<uintptr_t>(q) % 16 || reinterpret_cast<uintptr_t>(out) % 16)
    return PMM_ERR_BAD_ARGUMENT;
  if (n_splits > 1 && (!part_o || !part_ml || !split_counter || split_len <= 0 || split_len % pmm::kAtBox))
    return PMM_ERR_BAD_ARGUMENT;
  if (n_splits == 1) split_len = 0x40000000;
  // the whole pool as a matrix [pages * 2 * page_size, Hkv * head size]; a box is 64 rows x 64 columns
  pmm::EncodeTiledFn fn = pmm::encode_tiled_fn();
  if (!fn) return PMM_ERR_BAD_ARGUMENT;
  CUtensorMap map;
  const long long kv_dim = static_cast<long long>(Hkv) * Dh;
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(kv_dim), static_cast<cuuint64_t>(pool_pages * 2 * page_size)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(kv_dim) * 2};
  const cuuint32_t box[2] = {pmm::kAtDhBlock, pmm::kAtBox};
  const cuuint32_t elem[2] = {1, 1};
  if (fn(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(pool), dims, strides, box, elem,
         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return PMM_ERR_BAD_ARGUMENT;
  auto kern = rows == 64 ? (Dh == 64 ? pmm::attention_tc_kernel<64, 64> : pmm::attention_tc_kernel<128, 64>)
                         : (Dh == 64 ? pmm::attention_tc_kernel<64, 128> : pmm::attention_tc_kernel<128, 128>);
  const size_t smem = pmm::at_smem(Dh, rows);
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
  if (e != cudaSuccess) return static_cast<int>(e);
  if (static_cast<long long>(n_tiles) * Hkv > 0x7fffffff) return PMM_ERR_BAD_ARGUMENT;
  dim3 grid(n_tiles * Hkv, n_splits);
  pmm::launch_pdl(kern, grid, dim3(pmm::at_threads(rows)), smem, stream,
      static_cast<const pmm::bf16*>(q), map, block_table, max_blocks, positions, cu, static_cast<pmm::bf16*>(out), part_o,
      part_ml, scale * 1.4426950408889634f, window, split_len, n_splits, page_size, n_seq, Hq, Hkv, split_counter, status,
      sink, lse);
  return pmm::launch_status();
}
