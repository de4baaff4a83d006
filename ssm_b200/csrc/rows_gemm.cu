// Products of a few activation rows (up to 256 sequences, one token each) with up to five weight matrices, sm_100a.
//
// Out^T = W X^T: the weight rows are the M of the MMA (128 per CTA, one TMEM lane each), the token rows its N, so a step of any
// batch streams every weight once and no tile is padded in the large dimension.  Operands arrive by TMA in the 128-byte swizzle, 64
// columns of K per stage, from one lane; another issues tcgen05.mma into one TMEM accumulator; all eight warps read it back, lane =
// weight row, and write 32 neighbouring outputs of a token per warp.
//
// Where the row tiles cannot fill the GPU the columns are split over a cluster of up to eight CTAs, whose partial sums meet through
// distributed shared memory: no workspace, no second launch, and the order of the sum is fixed.  Unsplit, the outputs are the library's bit for bit; a
// split sums in another order (up to 0.4 % of the 16-bit outputs round the other way) and is as near to 64 bits: 1.648e-3 to 1.741e-3 relative over
// forty products of 20 to 256 rows, in none of them further off than the library's.
#include <cooperative_groups.h>

#include <atomic>

#include "decode_parts.h"
#include "ssd_common.cuh"

namespace ssmb {

constexpr int kGemmRows = 128, kGemmK = 64, kGemmThreads = 256, kGemmMaxStages = 8;
constexpr int kGemmWBytes = kGemmRows * kGemmK * 2;
constexpr size_t kGemmSmem = 200 * 1024;

struct GemmMaps {
  CUtensorMap x, w[SSMB_GEMM_MATS];
};
struct GemmShape {
  int mats, batch, n, nkb, stages, splits, status_code, weights_ahead;
  int rows[SSMB_GEMM_MATS], tiles_end[SSMB_GEMM_MATS];
  void* out[SSMB_GEMM_MATS];
  int64_t ldo[SSMB_GEMM_MATS];
  int32_t* status;
};

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const void* tmap, uint32_t mbar, int c0, int c1) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n" ::"r"(dst), "l"(tmap), "r"(mbar),
               "r"(c0), "r"(c1)
               : "memory");
}

template <typename T>
__global__ void __launch_bounds__(kGemmThreads, 1) rows_gemm_kernel(const __grid_constant__ GemmMaps maps, const __grid_constant__ GemmShape g) {
  extern __shared__ unsigned char gemm_raw[];
  __shared__ __align__(8) uint64_t bars[2 * kGemmMaxStages + 1];
  __shared__ uint32_t tmem_slot;
  __shared__ int gave_up;  // a stage did not arrive in time
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(gemm_raw) + 1023) & ~(uintptr_t)1023);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = blockIdx.x % g.splits, tile = blockIdx.x / g.splits;
  int seg = 0, first = 0;
#pragma unroll
  for (int s = 0; s < SSMB_GEMM_MATS - 1; ++s)
    if (s < g.mats - 1 && tile >= g.tiles_end[s]) seg = s + 1, first = g.tiles_end[s];
  const int row0 = (tile - first) * kGemmRows, tok0 = blockIdx.y * g.n, batch = min(g.batch - tok0, g.n);
  const int kb0 = g.nkb * rank / g.splits, kb1 = g.nkb * (rank + 1) / g.splits;
  const int xbytes = g.n * kGemmK * 2, stage_bytes = kGemmWBytes + xbytes;
  const uint32_t full = tc::smem_u32(bars), empty = full + 8 * kGemmMaxStages, done = full + 16 * kGemmMaxStages;
  int cols = 32;
  while (cols < g.n) cols *= 2;

  if (tid == 0) {
    for (int s = 0; s < g.stages; ++s) tc::mbar_init(full + 8 * s, 1), tc::mbar_init(empty + 8 * s, 1);
    tc::mbar_init(done, 1);
    gave_up = 0;
  }
  if (warp == 2) tc::tmem_alloc(tc::smem_u32(&tmem_slot), cols);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tmem_slot;

  auto ran_out = [&]() {
    if (g.status) *reinterpret_cast<volatile int32_t*>(g.status) = g.status_code;
  };
  int issued = 0;  // stages that this thread has filled
  if (warp == 0) {
    if (tc::elect_one()) {
      // the first stages' weights go out ahead of the wait for the kernel before this one
      const int ahead = g.weights_ahead ? min(g.stages, kb1 - kb0) : 0;
      for (int i = 0; i < ahead; ++i) {
        tc::mbar_expect_tx(full + 8 * i, stage_bytes);
        tma_load_2d(tc::smem_u32(base + (size_t)i * stage_bytes), &maps.w[seg], full + 8 * i, (kb0 + i) * kGemmK, row0);
      }
      pdl_wait();
      const uint32_t stage0 = tc::smem_u32(base);
      int st = 0, parity = 1, kc = kb0 * kGemmK;
      for (int i = 0; i < kb1 - kb0; ++i, kc += kGemmK) {
        const uint32_t at = stage0 + st * stage_bytes, bar = full + 8 * st;
        if (i >= ahead) {
          if (i >= g.stages && !tc::mbar_wait(empty + 8 * st, parity)) {
            ran_out();
            break;
          }
          tc::mbar_expect_tx(bar, stage_bytes);
          tma_load_2d(at, &maps.w[seg], bar, kc, row0);
        }
        tma_load_2d(at + kGemmWBytes, &maps.x, bar, kc, tok0);
        if (++st == g.stages) st = 0, parity ^= 1;
        issued = i + 1;
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (tc::elect_one()) {
      const uint32_t idesc = tc::instr_desc(kGemmRows, g.n, std::is_same<T, __nv_bfloat16>::value ? 1 : 0, 0, 0);
      const uint32_t stage0 = tc::smem_u32(base);
      int st = 0, parity = 0;
      for (int i = 0; i < kb1 - kb0; ++i) {
        if (!tc::mbar_wait(full + 8 * st, parity)) {
          ran_out();
          gave_up = 1;
          break;
        }
        tc::fence_after_sync();
        const uint32_t at = stage0 + st * stage_bytes;
        const uint64_t dw = tc::smem_desc_sw128(at, 16, 1024), dx = tc::smem_desc_sw128(at + kGemmWBytes, 16, 1024);
#pragma unroll
        for (int kk = 0; kk < kGemmK / 16; ++kk) tc::mma_ss(tmem, dw + 2 * kk, dx + 2 * kk, idesc, i > 0 || kk > 0);
        tc::commit(empty + 8 * st);
        if (++st == g.stages) st = 0, parity ^= 1;
      }
      tc::commit(done);
    }
    __syncwarp();
  }
  pdl_wait();  // the outputs may still be read by the kernel before
  pdl_trigger();
  const bool ok = tc::mbar_wait(done, 0);
  if (!ok && lane == 0) ran_out();
  tc::fence_after_sync();

  // accumulator -> shared memory as [token][128 weight rows], over the stages, which every MMA has read.  Where the columns were split,
  // token t goes to CTA t % splits of the cluster, which adds the partial sums of all ranks in their order.
  float* part = reinterpret_cast<float*>(base);
  const uint32_t tw = tmem + ((uint32_t)(warp & 3) << 21);  // this warp's 32 TMEM lanes
  const int at = (warp & 3) * 32 + lane, slots = g.n / g.splits;  // tokens of a CTA (n is a multiple of 16)
  namespace cg = cooperative_groups;
  if (g.splits > 1) cg::this_cluster().sync();  // every rank's stages are free
  for (int c = (warp >> 2) * 16; c < g.n; c += 32) {
    float v[16];
    tc::tmem_ld16(tw + c, v);
    if (g.splits == 1) {
#pragma unroll
      for (int j = 0; j < 16; ++j) part[(c + j) * kGemmRows + at] = v[j];
    } else {
      const int log = g.splits == 2 ? 1 : g.splits == 4 ? 2 : 3;
#pragma unroll
      for (int j = 0; j < 16; ++j) cg::this_cluster().map_shared_rank(part, j & (g.splits - 1))[(rank * slots + ((c + j) >> log)) * kGemmRows + at] = v[j];
    }
  }
  if (g.splits == 1) __syncthreads();
  else cg::this_cluster().sync();
  // a warp per token, four rows per lane
  const int64_t ldo = g.ldo[seg];
  T* __restrict__ out = reinterpret_cast<T*>(g.out[seg]) + tok0 * ldo + row0 + lane * 4;
  const int left = ok ? g.rows[seg] - row0 - lane * 4 : 0;  // rows from this lane's first to the matrix's end
  const bool wide = left >= 4 && (reinterpret_cast<uintptr_t>(out) & 7) == 0 && ldo % 4 == 0;
#pragma unroll 4
  for (int q = warp; q < slots; q += 8) {
    const int t = q * g.splits + rank;
    if (t >= batch) break;
    float4 v = *reinterpret_cast<const float4*>(part + q * kGemmRows + lane * 4);
    for (int p = 1; p < g.splits; ++p) {
      const float4 w = *reinterpret_cast<const float4*>(part + (p * slots + q) * kGemmRows + lane * 4);
      v.x += w.x, v.y += w.y, v.z += w.z, v.w += w.w;
    }
    const T e[4] = {from_f<T>(v.x), from_f<T>(v.y), from_f<T>(v.z), from_f<T>(v.w)};
    T* to = out + (int64_t)t * ldo;
    if (wide) {
      *reinterpret_cast<uint2*>(to) = *reinterpret_cast<const uint2*>(e);
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (k < left) to[k] = e[k];
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 2) tc::tmem_dealloc(tmem, cols);
  // Where every stage was multiplied, no copy is under way by now.  Otherwise (a filling thread that gave up leaves the multiplying one without its next
  // stage, too) the block ends once its copies have landed.
  if (gave_up) {
    for (int i = max(0, issued - g.stages); i < issued; ++i) tc::mbar_wait(full + 8 * (i % g.stages), (i / g.stages) & 1);
  }
}

// (rows, k) matrix of 16-bit elements with `ld` elements from row to row; box = 64 columns x `box_rows` rows
static int encode_matrix(CUtensorMap* m, const void* base, int64_t rows, int64_t k, int64_t ld, int box_rows, int io_dtype) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return fail(SSM_ERR_DEVICE, "rows_gemm: cuTensorMapEncodeTiled is not available from this driver");
  const cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)ld * 2};
  const cuuint32_t box[2] = {kGemmK, (cuuint32_t)box_rows}, estr[2] = {1, 1};
  const CUtensorMapDataType dt = io_dtype == SSM_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  const CUresult rc = fn(m, dt, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return rc == CUDA_SUCCESS ? SSM_OK : fail(SSM_ERR_DEVICE, "rows_gemm: cuTensorMapEncodeTiled rejected the matrix");
}

template <typename T>
static int gemm_launch(const GemmMaps& maps, const GemmShape& g, dim3 grid, size_t smem, cudaStream_t st) {
  auto kern = rows_gemm_kernel<T>;
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = g.splits, attr[1].val.clusterDim.y = 1, attr[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid, cfg.blockDim = dim3(kGemmThreads), cfg.dynamicSmemBytes = smem, cfg.stream = st, cfg.attrs = attr, cfg.numAttrs = 2;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, maps, g);
  if (e != cudaSuccess) {
    cudaGetLastError();
    set_error("rows_gemm_kernel: %s", cudaGetErrorString(e));
    return (int)e;
  }
  return launch_status("rows_gemm_kernel");
}

// Clusters of the kernel that run at once.  A cluster lies within one GPC: 74 of two, 33 of four, 15 of eight CTAs on 148 SMs.
static int gemm_clusters(int dev, int sms, int splits) {
  static std::atomic<int> known[64][4];
  if (dev < 0 || dev >= 64) return sms / splits;
  std::atomic<int>& n = known[dev][splits == 2 ? 1 : splits == 4 ? 2 : 3];
  if (n == 0) {
    auto kern = rows_gemm_kernel<__nv_bfloat16>;
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGemmSmem);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = splits, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(splits), cfg.blockDim = dim3(kGemmThreads), cfg.dynamicSmemBytes = kGemmSmem, cfg.attrs = attr, cfg.numAttrs = 1;
    int fit = 0;
    if (cudaOccupancyMaxActiveClusters(&fit, kern, &cfg) != cudaSuccess || fit < 1) cudaGetLastError(), fit = sms / splits;
    n = fit;
  }
  return n;
}

// Token rows of a CTA and CTAs that share its columns: the least estimated time.  Operands at what one SM and all of them together read (from
// the L2: token tiles share the weights), the accumulator's way out per token row, and the exchange of partial sums.  Clusters that do not
// run at once take a second round that is as long as the first (2048 rows of 4096 columns, 17 to 128 sequences: 10.8 to 14.4 us in 16 clusters
// of eight, 6.6 to 8.5 in clusters of four) and are not considered.  Against all plans of 203 products of 17 to 256 rows with 320 to 10576 weight rows
// and 48 to 5120 columns: median 0.2 % above the best, nine in ten within 7 %, the worst 16 % (64 rows, 320 x 640: 4.0 us against 3.4).
struct GemmPlan {
  int n, splits;
};
constexpr double kSmRate = 115e3, kAllRate = 11e6;                               // bytes per us
constexpr double kReadOut = 0.008, kExchange = 0.6, kExchangePerRow = 0.011;  // us
static GemmPlan gemm_plan(int tiles, int batch, int nkb, int sms) {
  GemmPlan best{16, 1};
  double least = 1e300;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) dev = -1;
  for (int s = 1; s <= 8 && s <= nkb; s *= 2) {
    const int clusters = s > 1 ? gemm_clusters(dev, sms, s) : 0, steps = (nkb + s - 1) / s;
    for (int p = 1; p <= 8; p *= 2) {
      const int n = ((batch + p - 1) / p + 15) / 16 * 16, toks = (batch + n - 1) / n, ctas = tiles * toks * s;
      if (s > 1 && tiles * toks > clusters) continue;
      const double bytes = (double)steps * (kGemmWBytes + n * kGemmK * 2.0), rounds = (ctas + sms - 1) / sms;
      double t = bytes / kSmRate;
      if (t < ctas * bytes / kAllRate) t = ctas * bytes / kAllRate;
      t += (rounds - 1) * bytes / kSmRate + n * kReadOut + (s > 1 ? kExchange + n * kExchangePerRow : 0.0);
      if (t < least) least = t, best = GemmPlan{n, s};
    }
  }
  return best;
}

}  // namespace ssmb

using namespace ssmb;

extern "C" int ssmb_rows_gemm_supported(int32_t batch, int32_t k, int64_t ldx, int32_t io_dtype) {
  return batch >= 1 && batch <= SSMB_GEMM_MAX_ROWS && k >= 8 && k % 8 == 0 && ldx % 8 == 0 && ldx >= k && (io_dtype == SSM_BF16 || io_dtype == SSM_F16);
}

extern "C" int ssmb_rows_gemm(const ssmb_rows_gemm_args* a, void* stream) {
  SSM_REQUIRE(a != nullptr && a->x, SSM_ERR_NULL, "rows_gemm: missing tensor");
  SSM_REQUIRE(ssmb_rows_gemm_supported(a->batch, a->k, a->ldx, a->io_dtype) && a->mats >= 1 && a->mats <= SSMB_GEMM_MATS, SSM_ERR_UNSUPPORTED, "rows_gemm: unsupported shape");
  SSM_REQUIRE(aligned_to(a->x, 16), SSM_ERR_ALIGN, "rows_gemm: tensors must be 16-byte aligned");
  GemmMaps maps;
  GemmShape g{};
  g.mats = a->mats, g.batch = a->batch, g.nkb = (a->k + kGemmK - 1) / kGemmK, g.status = a->status, g.status_code = 64, g.weights_ahead = a->weights_ahead;
  int tiles = 0;
  for (int i = 0; i < a->mats; ++i) {
    SSM_REQUIRE(a->w[i] && a->out[i] && a->rows[i] >= 1, SSM_ERR_NULL, "rows_gemm: missing tensor");
    SSM_REQUIRE(aligned_to(a->w[i], 16), SSM_ERR_ALIGN, "rows_gemm: tensors must be 16-byte aligned");
    if (int rc = encode_matrix(&maps.w[i], a->w[i], a->rows[i], a->k, a->k, kGemmRows, a->io_dtype)) return rc;
    tiles += (a->rows[i] + kGemmRows - 1) / kGemmRows;
    g.rows[i] = a->rows[i], g.tiles_end[i] = tiles, g.out[i] = a->out[i], g.ldo[i] = a->ldo[i];
  }
  const int sms = sm_count();
  GemmPlan plan;
  if (a->plan_rows) {
    plan = GemmPlan{a->plan_rows, a->plan_splits};
    SSM_REQUIRE(plan.n >= 16 && plan.n <= SSMB_GEMM_MAX_ROWS && plan.n % 16 == 0 && (plan.splits == 1 || plan.splits == 2 || plan.splits == 4 || plan.splits == 8) &&
                    plan.splits <= g.nkb, SSM_ERR_UNSUPPORTED, "rows_gemm: unsupported plan");
  } else {
    plan = gemm_plan(tiles, a->batch, g.nkb, sms);
  }
  g.n = plan.n, g.splits = plan.splits;
  const int tok_tiles = (a->batch + g.n - 1) / g.n;
  if (int rc = encode_matrix(&maps.x, a->x, a->batch, a->k, a->ldx, g.n, a->io_dtype)) return rc;
  const size_t stage = kGemmWBytes + (size_t)g.n * kGemmK * 2, part = (size_t)g.n * kGemmRows * 4;
  const int steps = (g.nkb + g.splits - 1) / g.splits;
  // more CTAs than SMs: half the ring, so that two of them share an SM, where the accumulator tile that lies over the ring leaves room for it (up to
  // 208 token rows; 3 KB per CTA for the alignment, the barriers and the system)
  const bool two = tiles * tok_tiles * g.splits > sms && 2 * ((part > kGemmSmem / 2 ? part : kGemmSmem / 2) + 3 * 1024) <= 228 * 1024;
  g.stages = (int)((two ? kGemmSmem / 2 : kGemmSmem) / stage);
  g.stages = g.stages > kGemmMaxStages ? kGemmMaxStages : g.stages < 2 ? 2 : g.stages;
  g.stages = g.stages > steps ? steps : g.stages;
  size_t smem = g.stages * stage;
  smem = (smem > part ? smem : part) + 1024;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  return a->io_dtype == SSM_BF16 ? gemm_launch<__nv_bfloat16>(maps, g, dim3(tiles * g.splits, tok_tiles), smem, st) : gemm_launch<__half>(maps, g, dim3(tiles * g.splits, tok_tiles), smem, st);
}
