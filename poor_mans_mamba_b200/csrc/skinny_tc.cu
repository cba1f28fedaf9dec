// Weight-streaming matrix product for steps of 33..64 tokens (it takes 1..64) on the fifth-generation
// tensor cores:
//   y[T, N] = x[T, K] W[N, K]^T, bfloat16 operands, float accumulation,
// with the same epilogues as the mma.sync form for fewer tokens (skinny_gemm.cu): STORE (bfloat16; with gelu on it),
// SWIGLU (W = [gate rows; up rows], act = silu(gate * mult) * up) and RESIDUAL (h += scale * y with
// float atomics; two products may share a launch).
//
// At these sizes the product is one read of W and its time is the chain behind the kernel before it: x arrives, the
// products run, the sums leave.  So a block holds one piece of W alone, 128 rows x at most 256 columns, requested in
// one go before the wait for that kernel (the weights depend on nothing it writes), and after the wait brings in only the
// same columns of x (32 KB; a block that took all of K would fetch all of x, 128 KB, on every SM: more than W itself).
// W's rows are the M side of the instruction (128), the tokens (rounded up to 16) its N side, so that a block issues 16
// instructions at most.  The blocks along K of a tile are one thread-block cluster: each leaves its partial sums [token][row]
// in its shared memory and, behind one cluster barrier, block r adds up the r-th part of the tokens from all of them in
// the order of K (float) and runs the epilogue, four columns of a row a thread.  RESIDUAL products longer than a cluster's
// 1,024 columns, and two products in one launch, meet in more than one atomic add an element, whose order is not fixed.  97 KB of shared memory a block: two fit an SM, so the
// next product's weights are on their way while this one runs.  Clusters of 8 blocks of 128 columns were slower inside a
// decode step of 64 requests (602 against 543 us).
// Inside a prompt step of 37 tokens, layers of 1,024 -> 4,120, 1,536 + 512 -> 1,024, 1,024 -> 2 x 2,048 -> 1,024, us from
// the end of the kernel before: 5.5, 7.8, 5.6, 4.9; with the tokens as the M side and all of K in a block 7.7, 7.8, 8.0, 5.9.
// Warps: 0 = copies and products, 1 = tensor-memory owner, all four = epilogue (tensor-memory lane = row of W).
// Every mbarrier wait is bounded: on a time-out the waiter writes a code (22: operands, 24: products) to *status, the
// block's other waits end too, the copies in flight are waited for (bounded), the cluster barriers are passed and the tensor
// memory is freed.  No cluster multicast.
// (reference: linear layers are cublasSgemm calls, src/ops/gpu/linear.cu:3-21.)
#include "tcgen05.cuh"

namespace pmm {

using bf16 = __nv_bfloat16;

constexpr int kStTok = 64;      // tokens at most
constexpr int kStRows = 128;    // rows of W per block
constexpr int kStKB = 64;       // columns per box: one 128-byte swizzle row
constexpr int kStMaxKB = 4;     // boxes per block at most
constexpr int kStCluster = 4;   // blocks along K of a tile that add up their sums
constexpr int kStThreads = 128;
constexpr int kStTmemCols = 64;
constexpr int kStWBox = kStRows * kStKB * 2;   // 16 KB

enum { kStStore = 0, kStSwiglu = 1, kStResidual = 2, kStGelu = 3 };  // GELU: STORE with y = gelu(x W^T), the erf form

struct SkinnyTcArgs {
  int T, N;          // tokens, output columns (SWIGLU: F)
  int t_pad;         // T rounded up to a multiple of 16
  int K[2];
  int groups[2];     // clusters along K of each product
  float scale[2];    // RESIDUAL: factor on y; SWIGLU: gate multiplier
  bf16* y;           // STORE / SWIGLU output
  long long ldy;
  float* h_out;      // RESIDUAL target [T, N]
  int* status;
};

__device__ __forceinline__ void st_red4(float* p, float4 v) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};\n" ::"l"(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
// Four floats of shared memory address `addr` of block `rank` of the cluster.
__device__ __forceinline__ float4 st_peer4(unsigned addr, unsigned rank) {
  unsigned a;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(a) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}

template <int MODE>
__global__ void __launch_bounds__(kStThreads)
    skinny_tc_kernel(const __grid_constant__ CUtensorMap map_x0, const __grid_constant__ CUtensorMap map_w0,
                     const __grid_constant__ CUtensorMap map_x1, const __grid_constant__ CUtensorMap map_w1,
                     const SkinnyTcArgs args) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) unsigned long long bar_w, bar_x, bar_acc;
  __shared__ unsigned s_tmem_base;
  __shared__ int s_abort;
  pdl_launch_dependents();

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = blockIdx.x % kStCluster;   // of this block in its cluster
  const int prob = static_cast<int>(blockIdx.x) >= kStCluster * args.groups[0] ? 1 : 0;
  const CUtensorMap* map_x = prob == 0 ? &map_x0 : &map_x1;
  const CUtensorMap* map_w = prob == 0 ? &map_w0 : &map_w1;
  // this block's boxes of K: an even share (none, where K has fewer boxes than the clusters blocks)
  const int boxes = (args.K[prob] + kStKB - 1) / kStKB, shares = kStCluster * args.groups[prob];
  const int share = static_cast<int>(blockIdx.x) - prob * kStCluster * args.groups[0];
  const int kb0 = boxes * share / shares, n_kb = boxes * (share + 1) / shares - kb0;
  constexpr int kTileCols = MODE == kStSwiglu ? kStRows / 2 : kStRows;  // output columns of a block
  const long long tile = static_cast<long long>(blockIdx.z) * gridDim.y + blockIdx.y;
  const int n0 = static_cast<int>(tile) * kTileCols;
  const int x_box = args.t_pad * kStKB * 2;

  unsigned char* sW = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* sX = sW + kStMaxKB * kStWBox;   // [max_kb] boxes of t_pad rows
  float* part = reinterpret_cast<float*>(sW);       // [t_pad][128] partial sums, once the products have read W

  if (tile * kTileCols >= args.N) return;   // (the last z holds fewer tiles; the whole cluster leaves)

  if (threadIdx.x == 0) {
    mbar_init(&bar_w, 1);
    mbar_init(&bar_x, 1);
    mbar_init(&bar_acc, 1);
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    // the weights: this warp's own copies, before anything else in the block is ready
    if (n_kb > 0) mbar_expect_tx(&bar_w, n_kb * kStWBox);
  }
  __syncwarp();
  if (warp == 0) {
    if (MODE == kStSwiglu) {
      if (lane < 2 * n_kb) {  // 64 gate rows and their 64 up rows of box lane / 2
        const int b = lane >> 1, up = lane & 1;
        tma_load_2d(sW + b * kStWBox + up * (kStWBox / 2), map_w, (kb0 + b) * kStKB, up * args.N + n0, &bar_w);
      }
    } else if (lane < n_kb) {
      tma_load_2d(sW + lane * kStWBox, map_w, (kb0 + lane) * kStKB, n0, &bar_w);
    }
    if (lane == 31) asm volatile("prefetch.tensormap [%0];\n" ::"l"(reinterpret_cast<unsigned long long>(map_x)) : "memory");
  } else if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&s_tmem_base)), "r"(kStTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const unsigned tmem_base = s_tmem_base;
  volatile int* abort_flag = &s_abort;
  auto give_up = [&](int code) {
    if (!*abort_flag) atomicExch(args.status, code);
    s_abort = 1;
  };

  pdl_wait();
  if (warp == 0 && n_kb > 0) {
    if (lane == 0) mbar_expect_tx(&bar_x, n_kb * x_box);
    __syncwarp();
    if (lane < n_kb) tma_load_2d(sX + lane * x_box, map_x, (kb0 + lane) * kStKB, 0, &bar_x);
    if (lane == 0) {
      if (mbar_wait(&bar_w, 0, abort_flag) && mbar_wait(&bar_x, 0, abort_flag)) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        // kind::f16 instruction: float accumulate, bfloat16 A and B, both K-major, M = 128, N = t_pad
        const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<unsigned>(args.t_pad >> 3) << 17) | ((128u >> 4) << 24);
        for (int b = 0; b < n_kb; ++b) {
          const unsigned long long a_desc = umma_desc(sW + b * kStWBox);
          const unsigned long long b_desc = umma_desc(sX + b * x_box);
#pragma unroll
          for (int k = 0; k < kStKB / 16; ++k)  // 16 columns further inside the swizzled row: 32 bytes = 2 units
            umma_f16(tmem_base, a_desc + 2 * k, b_desc + 2 * k, idesc, (b > 0 || k > 0) ? 1u : 0u);
        }
        umma_commit(&bar_acc);
      } else {
        give_up(22);
        // copies already requested still write into this block's shared memory: wait for them
        for (unsigned n = 0; n < kSpinLimit && !mbar_try_wait(&bar_w, 0); ++n) {
        }
        for (unsigned n = 0; n < kSpinLimit && !mbar_try_wait(&bar_x, 0); ++n) {
        }
      }
    }
    __syncwarp();
  }

  // ---------------------------------------------------------------- the block's partial sums
  bool made = n_kb > 0;
  if (made && !mbar_wait(&bar_acc, 0, abort_flag)) {
    give_up(24);
    made = false;
  }
  made = __all_sync(0xffffffffu, made);
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const int row = threadIdx.x;  // of the tile = tensor-memory lane
  const unsigned lane_base = tmem_base + (static_cast<unsigned>(warp * 32) << 16);
  for (int t = 0; t < args.t_pad; t += 32) {
    unsigned v[32];
    if (made) {
      tmem_ld32(lane_base + t, v);
      asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
    } else {
#pragma unroll
      for (int e = 0; e < 32; ++e) v[e] = 0u;
    }
#pragma unroll
    for (int e = 0; e < 32; ++e)
      if (t + e < args.t_pad) part[(t + e) * kStRows + row] = __uint_as_float(v[e]);
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(kStTmemCols) : "memory");
  }

  // ---------------------------------------------------------------- block `rank` finishes its part of the tokens
  const int per = args.t_pad / kStCluster;
  constexpr int kPieces = kTileCols / 4;  // of four columns in a row of the tile
  const unsigned part_at = smem_u32(part);
  const float scale = args.scale[prob];
  for (int i = threadIdx.x; i < per * kPieces; i += kStThreads) {
    const int m = rank * per + i / kPieces, c = (i % kPieces) * 4;
    if (m >= args.T || n0 + c >= args.N) continue;
    const unsigned at = part_at + static_cast<unsigned>(m * kStRows + c) * 4;
    float4 p[kStCluster], q[MODE == kStSwiglu ? kStCluster : 1];
#pragma unroll
    for (int r = 0; r < kStCluster; ++r) {
      p[r] = st_peer4(at, r);
      if (MODE == kStSwiglu) q[r] = st_peer4(at + kTileCols * 4, r);
    }
#pragma unroll
    for (int r = 1; r < kStCluster; ++r) {
      p[0].x += p[r].x, p[0].y += p[r].y, p[0].z += p[r].z, p[0].w += p[r].w;
      if (MODE == kStSwiglu) q[0].x += q[r].x, q[0].y += q[r].y, q[0].z += q[r].z, q[0].w += q[r].w;
    }
    float4 v = p[0];
    if (MODE == kStSwiglu)
      v = make_float4(silu_fast(v.x * scale) * q[0].x, silu_fast(v.y * scale) * q[0].y, silu_fast(v.z * scale) * q[0].z,
                      silu_fast(v.w * scale) * q[0].w);
    if (MODE == kStGelu) v = make_float4(gelu_erf_fast(v.x), gelu_erf_fast(v.y), gelu_erf_fast(v.z), gelu_erf_fast(v.w));
    const bool whole = n0 + c + 4 <= args.N;
    const float e[4] = {v.x, v.y, v.z, v.w};
    if (MODE == kStResidual) {
      float* dst = args.h_out + static_cast<long long>(m) * args.N + n0 + c;
      if (whole && (args.N & 3) == 0) {
        st_red4(dst, make_float4(scale * v.x, scale * v.y, scale * v.z, scale * v.w));
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (n0 + c + k < args.N) atomicAdd(dst + k, scale * e[k]);
      }
    } else {
      bf16* dst = args.y + static_cast<long long>(m) * args.ldy + n0 + c;
      if (whole) {
        stf4(dst, v);
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (n0 + c + k < args.N) dst[k] = __float2bfloat16_rn(e[k]);
      }
    }
  }
  // the others may still read this block's sums
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

// bfloat16 matrix [rows, cols] with row stride ld (elements); box = 64 columns x box_rows rows.
static bool st_make_map(CUtensorMap* map, const void* base, long long rows, long long cols, long long ld, int box_rows) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return false;
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld) * 2};
  const cuuint32_t box[2] = {kStKB, static_cast<cuuint32_t>(box_rows)};
  const cuuint32_t elem[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int MODE>
int launch_skinny_tc(const CUtensorMap* maps, const SkinnyTcArgs& a, cudaStream_t stream) {
  auto kern = skinny_tc_kernel<MODE>;
  const size_t smem = 1024 /*alignment*/ + kStMaxKB * (kStWBox + a.t_pad * kStKB * 2);
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 1024 + kStMaxKB * (kStWBox + kStTok * kStKB * 2));
  if (e != cudaSuccess) return static_cast<int>(e);
  constexpr int kTileCols = MODE == kStSwiglu ? kStRows / 2 : kStRows;
  cudaLaunchConfig_t cfg{};
  const int tiles = (a.N - 1) / kTileCols + 1, deep = (tiles + 65534) / 65535;
  cfg.gridDim = dim3(kStCluster * (a.groups[0] + a.groups[1]), (tiles + deep - 1) / deep, deep);
  cfg.blockDim = dim3(kStThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attrs[2];
  attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attrs[0].val.programmaticStreamSerializationAllowed = 1;
  attrs[1].id = cudaLaunchAttributeClusterDimension;
  attrs[1].val.clusterDim.x = kStCluster;
  attrs[1].val.clusterDim.y = 1;
  attrs[1].val.clusterDim.z = 1;
  cfg.attrs = attrs;
  cfg.numAttrs = 2;
  cudaLaunchKernelEx(&cfg, kern, maps[0], maps[1], maps[2], maps[3], a);
  return launch_status();
}

}  // namespace pmm

// Whether pmm_skinny_tc takes these sizes: 1..64 tokens, K a multiple of 8 (rows of 16-byte
// multiples); STORE and SWIGLU end within a cluster: at most 1,024 columns; outputs with
// 16-byte aligned rows.
PMM_EXPORT int pmm_skinny_tc_supported(int mode, int T, int N, int K0, int K1, long long ldx0, long long ldx1, long long ldy) {
  if (T < 1 || T > pmm::kStTok || N < 1 || K0 < 8 || K0 % 8 || ldx0 % 8) return 0;
  if (K1 && (K1 < 8 || K1 % 8 || ldx1 % 8)) return 0;
  if (mode == pmm::kStResidual) return 1;
  if (mode != pmm::kStStore && mode != pmm::kStSwiglu && mode != pmm::kStGelu) return 0;
  return (K1 == 0 && K0 <= pmm::kStCluster * pmm::kStMaxKB * pmm::kStKB && ldy % 8 == 0) ? 1 : 0;
}

// mode 0 STORE (y bfloat16 [T, ldy]), 1 SWIGLU (w0 = [gate; up] rows, N = F, scale0 = gate multiplier),
// 2 RESIDUAL (h_out[T, N] += scale * y; one or two products; K cut into slices over clusters), 3 GELU
// (STORE with y = gelu(x W^T)).
// status: one int in device memory that stays 0 unless a bounded wait gave up.
PMM_EXPORT int pmm_skinny_tc(int mode, int T, int N, const void* x0, long long ldx0, const void* w0, int K0, float scale0,
                             const void* x1, long long ldx1, const void* w1, int K1, float scale1, void* y,
                             long long ldy, float* h_out, int* status, cudaStream_t stream) {
  if (T <= 0 || N <= 0) return 0;
  if (!x0 || !w0 || !status || !pmm_skinny_tc_supported(mode, T, N, K0, w1 ? K1 : 0, ldx0, w1 ? ldx1 : 0, ldy))
    return PMM_ERR_BAD_ARGUMENT;
  auto aligned16 = [](const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
  if (!aligned16(x0) || !aligned16(w0) || (w1 && (!x1 || !aligned16(x1) || !aligned16(w1)))) return PMM_ERR_BAD_ARGUMENT;
  if (mode == pmm::kStResidual ? !h_out : (!y || !aligned16(y) || w1)) return PMM_ERR_BAD_ARGUMENT;
  pmm::SkinnyTcArgs a{};
  a.T = T;
  a.N = N;
  a.K[0] = K0;
  a.K[1] = w1 ? K1 : 0;
  a.scale[0] = scale0;
  a.scale[1] = scale1;
  a.y = static_cast<pmm::bf16*>(y);
  a.ldy = ldy;
  a.h_out = h_out;
  a.status = status;
  a.t_pad = (T + 15) / 16 * 16;
  for (int p = 0; p < (w1 ? 2 : 1); ++p) {
    const int boxes = (a.K[p] + pmm::kStKB - 1) / pmm::kStKB, held = pmm::kStCluster * pmm::kStMaxKB;
    a.groups[p] = (boxes + held - 1) / held;
  }
  const int w_box_rows = mode == pmm::kStSwiglu ? pmm::kStRows / 2 : pmm::kStRows;
  const long long w_rows = mode == pmm::kStSwiglu ? 2LL * N : N;
  CUtensorMap maps[4];
  if (!pmm::st_make_map(&maps[0], x0, T, K0, ldx0, a.t_pad) || !pmm::st_make_map(&maps[1], w0, w_rows, K0, K0, w_box_rows))
    return PMM_ERR_BAD_ARGUMENT;
  if (w1) {
    if (!pmm::st_make_map(&maps[2], x1, T, K1, ldx1, a.t_pad) || !pmm::st_make_map(&maps[3], w1, w_rows, K1, K1, w_box_rows))
      return PMM_ERR_BAD_ARGUMENT;
  } else {
    maps[2] = maps[0];
    maps[3] = maps[1];
  }
  switch (mode) {
    case pmm::kStStore: return pmm::launch_skinny_tc<pmm::kStStore>(maps, a, stream);
    case pmm::kStSwiglu: return pmm::launch_skinny_tc<pmm::kStSwiglu>(maps, a, stream);
    case pmm::kStGelu: return pmm::launch_skinny_tc<pmm::kStGelu>(maps, a, stream);
    default: return pmm::launch_skinny_tc<pmm::kStResidual>(maps, a, stream);
  }
}
