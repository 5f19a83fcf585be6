// 16x16-block weight quantizer for weights in whole 128 x 128 tiles (sm_100a): W and W^T, codes and scales, from one
// read of W (bf16 or FP32).
//
// HBM-bound in principle (3.125 bytes per bf16 value); what a direct kernel is bound by is L1: a lane owns a row of a
// block, so the 32 lanes of every load and store are on 32 rows.  Here TMA does the walking: tiles of 128 rows (N) x
// KT columns (K) arrive in a two-stage ring as 128-byte-swizzled boxes, from which 16 lanes on 16 rows read without bank
// conflicts, and the codes leave through staging tiles that TMA stores as whole boxes: W as [128, KT/2] bytes, W^T as
// [KT, 64] bytes.  A half-warp owns a 16-row strip of the tile and half its columns: the block maximum takes four
// shuffles, the transposed codes the four butterfly steps of NibbleTranspose.  Two CTAs per SM, so that one loads while
// the other computes; 256 threads, all of them quantize, thread 0 also issues the copies.  KT = 128 for bf16, 64 for
// FP32: 32 KB a stage either way.  [11264, 2048] bf16: 18.7 us, 3.9 TB/s (direct kernels, lanes of a warp spread over a
// block or over 32 rows: 28 us).
// Every mbarrier wait is bounded: on expiry the CTA raises its abort flag, stores a role code in the quantizer status
// word, lets copies in flight land and returns.
#include "tma.cuh"

namespace nvfp4 {

constexpr int kWRows = 128;
constexpr int kWStages = 2;
constexpr int kWStageBytes = 32768;
constexpr int kWBoxBytes = kWRows * 128;                 // one 128-byte-wide box
constexpr int kWStaging = 16384 + 2048;                  // codes of W and of W^T (at most 8 KB each), scales (1 KB each)
constexpr int kWSmem = kWStages * kWStageBytes + kWStaging + 1024 /*alignment slack*/;

__device__ int g_quant_w2d_status;     // 0, or 1 once a wait has expired

struct W2dParams {
  unsigned char *s, *st;               // scales of W and of W^T; null: that output is not wanted
  const float* amax;
  float* gs_out;
  int N, K, layout;
};

__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, u32 src, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];"
               ::"l"(map), "r"(x), "r"(y), "r"(src) : "memory");
}

// 16-byte unit `u` of row `r` in a staging tile with rows of ROW bytes: the 64-byte TMA swizzle (bits 4..5 ^= bits 7..8
// of the offset) for 64-byte rows, plain for 32-byte rows
template <int ROW>
__device__ __forceinline__ u32 staged(u32 r, u32 byte) {
  const u32 off = r * ROW + byte;
  return ROW == 64 ? off ^ ((off >> 3) & 0x30u) : off;
}

template <typename T>
__global__ void __launch_bounds__(256, 2) quant_w2d_tile_kernel(const __grid_constant__ CUtensorMap map_w,
                                                                const __grid_constant__ CUtensorMap map_q,
                                                                const __grid_constant__ CUtensorMap map_qt, const W2dParams p) {
  constexpr int KT = sizeof(T) == 2 ? 128 : 64;          // columns of a tile
  constexpr int KB = KT / 16;                            // blocks along K
  constexpr int WK = KB / 2;                             // of which a half-warp has half
  constexpr int kBoxCols = 128 / sizeof(T);
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) float lut[kLutFloats];
  __shared__ __align__(8) u64 full_bar[kWStages];
  __shared__ int abort_word;
  volatile int* abort_flag = &abort_word;

  pdl_trigger();
  const u32 tiles0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const u32 out_w = tiles0 + kWStages * kWStageBytes, out_t = out_w + 8192, sc_w = out_t + 8192, sc_t = sc_w + 1024;
  const u32 full0 = smem_u32(full_bar);
  const int nkt = p.K / KT, ntiles = (p.N / kWRows) * nkt;
  if (threadIdx.x == 0) {
    abort_word = 0;
    for (int s = 0; s < kWStages; s++) mbar_init(full0 + 8 * s, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  auto load_tile = [&](int tile, int stage) {            // thread 0
    const u32 bar = full0 + 8 * stage, dst = tiles0 + stage * kWStageBytes;
    const int y = tile / nkt * kWRows, x = tile % nkt * KT;
    mbar_arrive_expect_tx(bar, kWStageBytes);
    tma_load_2d(dst, &map_w, x, y, bar);
    tma_load_2d(dst + kWBoxBytes, &map_w, x + kBoxCols, y, bar);
  };
  pdl_wait();
  if (threadIdx.x == 0)
    for (int s = 0; s < kWStages; s++)
      if ((int)blockIdx.x + s * (int)gridDim.x < ntiles) load_tile(blockIdx.x + s * gridDim.x, s);
  const TensorScale ts = make_tensor_scale<NVFP4_ROUND_NEAREST>(ld_cg_f32(p.amax), 1.f, lut,
                                                               (blockIdx.x == 0 && threadIdx.x == 0) ? p.gs_out : nullptr);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, i = lane & 15;
  const int kb0 = (lane >> 4) * WK;                      // first block column of this half-warp in the tile
  const u32 row = warp * 16 + i;                         // this lane's row of the tile; its block row is the warp
  const NibbleTranspose transpose(lane);
  u32 t = 0;
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x, t++) {
    const u32 stage = t & 1u, src = tiles0 + stage * kWStageBytes;
    if (!mbar_wait(full0 + 8 * stage, (t >> 1) & 1u, abort_flag)) atomicCAS(&g_quant_w2d_status, 0, 1);
    uint2 wq[WK], wt[WK];
    u32 sbs = 0u;
#pragma unroll
    for (int c = 0; c < WK; c++) {
      u64 P[8];
      if constexpr (sizeof(T) == 2) {
        // 16 values = two 16-byte units of the row; unit u sits at u ^ (row & 7)
        const u32 u = (u32)((kb0 + c) & 3) * 2u, box = src + (u32)((kb0 + c) >> 2) * kWBoxBytes + row * 128u;
        u32 w[8];
        asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "r"(box + ((u ^ (row & 7u)) << 4)));
        asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7]) : "r"(box + (((u + 1u) ^ (row & 7u)) << 4)));
#pragma unroll
        for (int k = 0; k < 8; k++) P[k] = f2_from_bf16x2(w[k]);
      } else {
        const u32 u = (u32)((kb0 + c) & 1) * 4u, box = src + (u32)((kb0 + c) >> 1) * kWBoxBytes + row * 128u;
#pragma unroll
        for (int k = 0; k < 4; k++) {
          u32 w[4];
          asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "r"(box + (((u + k) ^ (row & 7u)) << 4)));
          P[2 * k] = (u64)w[0] | ((u64)w[1] << 32); P[2 * k + 1] = (u64)w[2] | ((u64)w[3] << 32);
        }
      }
      float m = absmax16(P);
#pragma unroll
      for (int o = 8; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
      const u32 sb = block_scale_byte(m, ts);
      wq[c] = quant_block16<NVFP4_ROUND_NEAREST>(P, sb, ts, 0u, 0u, 0u);
      wt[c] = transpose(wq[c]);
      sbs |= sb << (8 * c);
    }
    // the staging tiles are free once the previous tile's stores have read them
    if (threadIdx.x == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    __syncthreads();
    if (*abort_flag) break;                              // read by all threads between two barriers: uniform
    if (p.s) {
#pragma unroll
      for (int c = 0; c < WK; c += 2)
        asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(out_w + staged<KT / 2>(row, (kb0 + c) * 8)), "r"(wq[c].x),
                     "r"(wq[c].y), "r"(wq[c + 1].x), "r"(wq[c + 1].y) : "memory");
      // scale bytes in the order of the swizzled layout: 512 bytes per four block columns
#pragma unroll
      for (int c = 0; c < WK; c++)
        asm volatile("st.shared.u8 [%0], %1;" ::"r"(sc_w + (u32)((kb0 + c) >> 2) * 512u + (row & 31u) * 16u + (row >> 5) * 4u + ((kb0 + c) & 3)),
                     "r"((sbs >> (8 * c)) & 0xFFu) : "memory");
    }
    if (p.st) {
#pragma unroll
      for (int c = 0; c < WK; c++) {
        const u32 krow = (u32)(kb0 + c) * 16u + i;       // row of W^T
        asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(out_t + staged<64>(krow, warp * 8)), "r"(wt[c].x), "r"(wt[c].y) : "memory");
        asm volatile("st.shared.u8 [%0], %1;" ::"r"(sc_t + (u32)(warp >> 2) * 512u + (krow & 31u) * 16u + (krow >> 5) * 4u + (warp & 3)),
                     "r"((sbs >> (8 * c)) & 0xFFu) : "memory");
      }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();                                     // staged; and nobody reads this tile any more
    const int rb = tile / nkt, ct = tile % nkt;
    if (threadIdx.x == 0) {
      if (p.s) tma_store_2d(&map_q, out_w, ct * (KT / 2), rb * kWRows);
      if (p.st) tma_store_2d(&map_qt, out_t, rb * 64, ct * KT);
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      const int ahead = tile + kWStages * (int)gridDim.x;
      if (ahead < ntiles) load_tile(ahead, stage);
    }
    // scale bytes: thread -> one word of W's (128 rows x KB bytes) and one of W^T's (KT rows x 8 bytes)
    const int nb = p.N >> 4, kb = p.K >> 4;
    const u32 h = threadIdx.x >> 7, r = ((threadIdx.x & 3u) << 5) | ((threadIdx.x & 127u) >> 2);   // word h of row r: consecutive threads, consecutive words
    if (p.s && h < KB / 4) {
      u32 v;
      asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(sc_w + 4u * threadIdx.x));
      const long long lin = (long long)(rb * kWRows + r) * kb + ct * KB + 4 * h;
      if (p.layout != NVFP4_SCALES_SWIZZLED) *reinterpret_cast<u32*>(p.s + lin) = v;
      if (p.layout != NVFP4_SCALES_LINEAR)
        *reinterpret_cast<u32*>(p.s + (p.layout == NVFP4_SCALES_BOTH ? (long long)p.N * kb : 0) + ((long long)rb * (kb >> 2) + ct * (KB / 4) + h) * 512 + 4 * (threadIdx.x & 127u)) = v;
    }
    // W^T: KT = 64 tiles own half of the 128 rows of a 512-byte scale tile (its words with (row >> 5) & 2 == that half)
    if (p.st && (r < KT)) {
      u32 v;
      asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(sc_t + 4u * threadIdx.x));
      const long long krow = (long long)ct * KT + r;
      const long long lin = krow * nb + rb * 8 + 4 * h;
      if (p.layout != NVFP4_SCALES_SWIZZLED) *reinterpret_cast<u32*>(p.st + lin) = v;
      if (p.layout != NVFP4_SCALES_LINEAR)
        *reinterpret_cast<u32*>(p.st + (p.layout == NVFP4_SCALES_BOTH ? (long long)p.K * nb : 0) + sw_off(krow, rb * 8 + 4 * h, nb >> 2)) = v;
    }
  }
  // the stores are complete before the kernel is
  if (threadIdx.x == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  if (*abort_flag) {
    const u64 t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
}

// rows x cols tensor of `elt` bytes, box box_cols x box_rows
static bool make_w_map(CUtensorMap* map, CUtensorMapDataType type, int elt, const void* base, long long rows, long long cols,
                       int box_cols, int box_rows, CUtensorMapSwizzle swizzle) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)(cols * elt)};
  const cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1, 1};
  return fn(map, type, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <typename T>
static int launch_w2d(const void* w, void* q, void* qt, const W2dParams& p, cudaStream_t st) {
  constexpr bool bf16 = sizeof(T) == 2;
  constexpr int KT = bf16 ? 128 : 64;
  CUtensorMap mw, mq = {}, mt = {};
  if (!make_w_map(&mw, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, sizeof(T), w, p.N, p.K,
                  128 / (int)sizeof(T), kWRows, CU_TENSOR_MAP_SWIZZLE_128B))
    return NVFP4_ERR_CUDA;
  if (q && !make_w_map(&mq, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, q, p.N, p.K / 2, KT / 2, kWRows,
                       bf16 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_NONE))
    return NVFP4_ERR_CUDA;
  if (qt && !make_w_map(&mt, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, qt, p.K, p.N / 2, 64, KT, CU_TENSOR_MAP_SWIZZLE_64B)) return NVFP4_ERR_CUDA;
  static bool configured[64] = {false};
  static int sms[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return NVFP4_ERR_CUDA;
  if (!configured[dev]) {
    if (cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaFuncSetAttribute(quant_w2d_tile_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, kWSmem) != cudaSuccess)
      return NVFP4_ERR_CUDA;
    configured[dev] = true;
  }
  const long long ntiles = (long long)(p.N / kWRows) * (p.K / KT);
  const unsigned grid = (unsigned)(ntiles < 2 * sms[dev] ? ntiles : 2 * sms[dev]);
  if (nvfp4_launch_kernel(quant_w2d_tile_kernel<T>, nvfp4_brief((long long)p.N * p.K * (long long)sizeof(T)), dim3(grid), dim3(256), kWSmem, st, mw, mq, mt, p) != cudaSuccess) {
    (void)cudaGetLastError();
    return NVFP4_ERR_CUDA;
  }
  return NVFP4_OK;
}

}  // namespace nvfp4

using namespace nvfp4;

// Whether the tile kernel takes this call: whole tiles, and the alignment TMA and the word stores of scales need.
bool nvfp4_quant_w2d_tile_accepts(const void* w, int N, int K, const void* q, const void* s, const void* qt, const void* st) {
  auto off = [](const void* p, unsigned mask) { return (reinterpret_cast<uintptr_t>(p) & mask) != 0; };
  return N > 0 && K > 0 && N % 128 == 0 && K % 128 == 0 && !off(w, 15u) && !off(q, 15u) && !off(qt, 15u) && !(q && off(s, 3u)) && !(qt && off(st, 3u));
}

// Arguments as nvfp4_quant_w2d, already validated by it.
int nvfp4_quant_w2d_tile_launch(const void* w, int w_dtype, int N, int K, void* q, void* s, void* qt, void* st, int scale_layout,
                                const float* amax, float* gs_out, void* stream) {
  W2dParams p;
  p.s = q ? static_cast<unsigned char*>(s) : nullptr; p.st = qt ? static_cast<unsigned char*>(st) : nullptr;
  p.amax = amax; p.gs_out = gs_out; p.N = N; p.K = K; p.layout = scale_layout;
  cudaStream_t stm = static_cast<cudaStream_t>(stream);
  return w_dtype == NVFP4_DTYPE_BF16 ? launch_w2d<__nv_bfloat16>(w, q, qt, p, stm) : launch_w2d<float>(w, q, qt, p, stm);
}

int nvfp4_quant_w2d_status(int* out, int reset) {
  if (cudaMemcpyFromSymbol(out, g_quant_w2d_status, sizeof(int)) != cudaSuccess) return NVFP4_ERR_CUDA;
  if (reset) {
    const int zero = 0;
    if (cudaMemcpyToSymbol(g_quant_w2d_status, &zero, sizeof(int)) != cudaSuccess) return NVFP4_ERR_CUDA;
  }
  return NVFP4_OK;
}
