// Gradients of B and C of the state-space-dual scan, for sm_100a.
//
//   dC_i = sum_h exp2(c_i) S_h dy_i          + sum_{j <= i} W_ij B_j        S_h: the state before the chunk
//   dB_j = sum_h exp2(off - c'_j) G_h x_j    + sum_{i >= j} W_ij C_i        G_h: the adjoint that enters it from the right
//   W_ij = sum_h exp2(c_i - c'_j) (dy_i . x_j)                              sums over the heads of a B / C group
//
// (c, c' = c - log2 delta: running decay exponents of the chunk; off: the decay of the chunk and of the step after it.)  The
// 256 x 256 products dy x^T are the only per-head work of that size: masked by the decay they add up over the heads in
// registers, so the products with B and C happen once per CTA and not once per head, and nothing per head is written out.
// The terms with S and G accumulate over the heads in tensor memory.  (Before, dB and dC were two more runs of the scan
// kernels with the head and state axes exchanged, 0.57 ms of 1.46 at (2, 4001, 48 heads); see the figures at the launch.)
//
// One CTA (512 threads) per (batch, chunk, 128-row block m of i, part of a group's heads).  Thread = row i x every fourth
// 32-step column chunk, as in the scan kernel: its part of W stays in registers.  Per head: dy rows of the block, x rows up to
// its last step, S, G and the exponents by TMA, one head ahead; T = dy x^T [128 x 128 (m + 1), K 64] into TMEM; meanwhile dy
// and x rows of block m are scaled into operand tiles of their own; their products with S and G are issued; then T is read back
// and added into W.  At the end W goes to shared memory once, where it is the K-major operand of W B and the MN-major one of W^T C.
// Sums over CTAs (row blocks, parts) by fp32 additions to zero-filled dB and dC.
// TMEM columns: T [0, 256), dC [256, 384), dB of block m [384, 512); dB of block 0 in a CTA of block 1 takes T's place.
#include "ssd_common.cuh"

namespace ssmb {

struct BcMaps {
  CUtensorMap x0, x1, dy, b, c;
};

struct BcSmem {
  static constexpr int X = kQ * kP * 2;      // x rows, 32 KB (x2); at the end: B rows (two blocks of 64 states), 64 KB
  static constexpr int Y = kBlk * kP * 2;    // dy rows of the block, 16 KB (x2); at the end: C rows, 32 KB
  static constexpr int S = kP * kN * 2;      // S and G, 16 KB each (x2); at the end: W, 64 KB
  static constexpr int V = 2 * kQ * 4;       // c and c' (x2)
  static constexpr int SCALED = 2 * Y;       // scaled dy and x rows
  static constexpr int W = 16 * 64 * 4;      // column factors, per warp
  static constexpr int TOTAL = 2 * (X + Y + 2 * S + V) + SCALED + W;
  static constexpr int ALLOC = TOTAL + 1024;
};

constexpr int kBcThreads = 512;

__device__ __forceinline__ void red_add4(float* p, float a, float b, float c, float d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

template <typename T, int MB>
__device__ __forceinline__ void ssd_bc_body(const ssm_ssd_bc_args& a, const BcMaps& maps, int nchunks, int hpc, int nparts, unsigned char* sm, uint64_t* mbar,
                                            uint32_t* tmem_slot) {
  using M = BcSmem;
  constexpr int KJ = (MB + 1) * kBlk, NCH = KJ / 128;  // columns, and 32-step column chunks per thread
  constexpr int fmt = std::is_same<T, __nv_bfloat16>::value ? 1 : 0;
  unsigned char* sX = sm;
  unsigned char* sY = sX + 2 * M::X;
  unsigned char* sS = sY + 2 * M::Y;  // per buffer S, then G
  unsigned char* sYs = sS + 4 * M::S;
  unsigned char* sXs = sYs + M::Y;
  float* sVec = reinterpret_cast<float*>(sXs + M::Y);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, wg = tid >> 7;
  float* sW = sVec + 2 * (M::V / 4) + warp * 64;
  // mbar: 0 / 1 operands of buffer 0 / 1 landed; 2 T complete; 3 the products with S and G complete; 4 B and C landed; 5 the last products complete
  auto bar = [&](int i) { return tc::smem_u32(&mbar[i]); };
  const int half = gridDim.x >> 1, rem = (int)blockIdx.x % half;
  const int part = rem % nparts, bc = rem / nparts;
  const int c = bc % nchunks, b = bc / nchunks;
  const int h0 = part * hpc, g = h0 / (a.heads / a.groups);
  const int t0 = c * kQ;
  if (MB && t0 + kBlk >= a.len) return;  // the whole CTA: no rows, nothing has been issued
  const int i_loc = (warp & 3) * 32 + lane, i_chunk = MB * kBlk + i_loc, rc = MB * 4 + (warp & 3);
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;

  auto load_head = [&](int h, int buf) {
    const uint32_t full = bar(buf);
    tc::mbar_expect_tx(full, KJ * kP * 2 + M::Y + 2 * M::S + M::V);
    tc::tma_load_4d(tc::smem_u32(sX + buf * M::X), MB ? &maps.x1 : &maps.x0, full, 0, h, t0, b);
    tc::tma_load_4d(tc::smem_u32(sY + buf * M::Y), &maps.dy, full, 0, h, t0 + MB * kBlk, b);
    const int64_t tile = (((int64_t)b * nchunks + c) * a.heads + h) * (int64_t)(kP * kN);
    tc::bulk_load(tc::smem_u32(sS + buf * 2 * M::S), reinterpret_cast<const T*>(a.state_in) + tile, M::S, full);
    tc::bulk_load(tc::smem_u32(sS + buf * 2 * M::S + M::S), reinterpret_cast<const T*>(a.adjoint_in) + tile, M::S, full);
    const int64_t v = (((int64_t)b * a.heads + h) * nchunks + c) * kQ;
    float* dv = sVec + buf * (2 * kQ);
    tc::bulk_load(tc::smem_u32(dv), a.ws_cum + v, kQ * 4, full);
    tc::bulk_load(tc::smem_u32(dv + kQ), a.ws_dt + v, kQ * 4, full);
  };
  if (tid == 0) load_head(h0, 0);

  float W[NCH][32];
#pragma unroll
  for (int k = 0; k < NCH; ++k)
#pragma unroll
    for (int e = 0; e < 32; ++e) W[k][e] = 0.f;

  bool ok = true;
#pragma unroll 1
  for (int hi = 0; hi < hpc; ++hi) {
    const int h = h0 + hi, buf = hi & 1;
    ok = ok && tc::mbar_wait(bar(buf), (hi >> 1) & 1);
    if (hi > 0) ok = ok && tc::mbar_wait(bar(3), (hi - 1) & 1);  // the products of the head before: their operand tiles and the other buffer are free
    tc::fence_before_sync();
    ok = __syncthreads_and(ok);  // also: every warp has read the T of the head before
    tc::fence_after_sync();
    if (!ok) break;
    if (warp == 0 && tc::elect_one()) {
      const uint64_t dy0 = tc::smem_desc_sw128(tc::smem_u32(sY + buf * M::Y), 16, 1024), dx0 = tc::smem_desc_sw128(tc::smem_u32(sX + buf * M::X), 16, 1024);
      constexpr uint32_t id = tc::instr_desc(kBlk, KJ, fmt, 0, 0);
#pragma unroll
      for (int kk = 0; kk < kP / 16; ++kk) tc::mma_ss(tmem, dy0 + (uint64_t)(kk * 2), dx0 + (uint64_t)(kk * 2), id, kk > 0);
      tc::commit(bar(2));
    }
    if (tid == 32 && hi + 1 < hpc) load_head(h + 1, buf ^ 1);
    const float* vc = sVec + buf * (2 * kQ);
    const float* vcp = vc + kQ;
    const float next = c + 1 < nchunks ? __ldg(a.ws_cum + (((int64_t)b * a.heads + h) * nchunks + c + 1) * kQ) : 0.f;
    const float off = vc[kQ - 1] + next;
    // scaled operand rows: exp2(c_i) dy_i and exp2(off - c'_j) x_j for the rows of block m, at the places of the unscaled ones
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int u = tid + (q & 1) * kBcThreads, row = u >> 3;  // 16-byte unit of a tile of 128 rows
      const bool isx = q >= 2;
      const float w = ex2_approx(isx ? off - vcp[MB * kBlk + row] : vc[MB * kBlk + row]);
      const unsigned char* src = isx ? sX + buf * M::X + MB * kBlk * 128 : sY + buf * M::Y;
      Vec16<T> v;
      v.raw = *reinterpret_cast<const uint4*>(src + (size_t)u * 16);
      float f[8];
      v.unpack(f);
#pragma unroll
      for (int e = 0; e < 8; ++e) f[e] *= w;
      v.pack(f);
      *reinterpret_cast<uint4*>((isx ? sXs : sYs) + (size_t)u * 16) = v.raw;
    }
    // factors of the decay mask, as in the scan kernel
    float arow[NCH];
    bool fast[NCH];
#pragma unroll
    for (int k = 0; k < NCH; ++k) {
      const int cc = wg + 4 * k;
      arow[k] = 0.f, fast[k] = false;
      if (cc <= rc) {
        const float r = vc[cc * 32];
        fast[k] = r - vc[cc * 32 + 31] < 60.f;
        arow[k] = ex2_approx(vc[i_chunk] - r);
        sW[k * 32 + lane] = ex2_approx(r - vcp[cc * 32 + lane]);
      }
    }
    tc::fence_async_smem();
    __syncthreads();
    if (warp == 0 && tc::elect_one()) {
      const uint64_t ay = tc::smem_desc_sw128(tc::smem_u32(sYs), 16, 1024), ax = tc::smem_desc_sw128(tc::smem_u32(sXs), 16, 1024);
      // the state tile [p / 8][n][8] read as a K-major operand: rows n, K = p
      const uint64_t bs = tc::smem_desc(tc::smem_u32(sS + buf * 2 * M::S), kN * 16, 128), bg = tc::smem_desc(tc::smem_u32(sS + buf * 2 * M::S + M::S), kN * 16, 128);
      constexpr uint32_t id = tc::instr_desc(kBlk, kN, fmt, 0, 0);
#pragma unroll
      for (int kk = 0; kk < kP / 16; ++kk) tc::mma_ss(tmem + 256, ay + (uint64_t)(kk * 2), bs + (uint64_t)(kk * (2 * kN * 16 >> 4)), id, hi > 0 || kk > 0);
#pragma unroll
      for (int kk = 0; kk < kP / 16; ++kk) tc::mma_ss(tmem + 384, ax + (uint64_t)(kk * 2), bg + (uint64_t)(kk * (2 * kN * 16 >> 4)), id, hi > 0 || kk > 0);
      tc::commit(bar(3));
    }
    // W += T o L
    ok = __all_sync(0xffffffffu, tc::mbar_wait(bar(2), hi & 1));
    tc::fence_after_sync();
    if (ok) {
#pragma unroll
      for (int k = 0; k < NCH; ++k) {
        const int cc = wg + 4 * k;
        if (cc > rc) continue;
        float t[32];
        tc::tmem_ld32(tmem + lane_base + cc * 32, t);
        const bool diag = cc == rc;
        if (fast[k] && !diag) {
          const float2 a2 = make_float2(arow[k], arow[k]);
#pragma unroll
          for (int e = 0; e < 32; e += 4) {
            const float4 f = *reinterpret_cast<const float4*>(sW + k * 32 + e);
            const float2 w0 = __ffma2_rn(__fmul2_rn(make_float2(t[e], t[e + 1]), make_float2(f.x, f.y)), a2, make_float2(W[k][e], W[k][e + 1]));
            const float2 w1 = __ffma2_rn(__fmul2_rn(make_float2(t[e + 2], t[e + 3]), make_float2(f.z, f.w)), a2, make_float2(W[k][e + 2], W[k][e + 3]));
            W[k][e] = w0.x, W[k][e + 1] = w0.y, W[k][e + 2] = w1.x, W[k][e + 3] = w1.y;
          }
        } else {
#pragma unroll
          for (int e = 0; e < 32; ++e) {
            const float w = fast[k] ? arow[k] * sW[k * 32 + e] : ex2_approx(vc[i_chunk] - vcp[cc * 32 + e]);
            if (!diag || e <= lane) W[k][e] = fmaf(t[e], w, W[k][e]);
          }
        }
      }
    }
  }
  if (ok) ok = tc::mbar_wait(bar(3), (hpc - 1) & 1);
  tc::fence_before_sync();
  ok = __syncthreads_and(ok);
  tc::fence_after_sync();
  if (ok) {
    // ---- B and C rows over the x and dy buffers; W as an operand over the state buffers: [64-column block][row][128 bytes], swizzled
    if (tid == 0) {
      tc::mbar_expect_tx(bar(4), KJ * kN * 2 + kBlk * kN * 2);
#pragma unroll
      for (int nb = 0; nb < 2; ++nb) {
        tc::tma_load_4d(tc::smem_u32(sY + nb * (kBlk * 128)), &maps.c, bar(4), nb * 64, g, t0 + MB * kBlk, b);
#pragma unroll
        for (int jb = 0; jb <= MB; ++jb) tc::tma_load_4d(tc::smem_u32(sX + nb * (KJ * 128) + jb * (kBlk * 128)), &maps.b, bar(4), nb * 64, g, t0 + jb * kBlk, b);
      }
    }
#pragma unroll
    for (int k = 0; k < NCH; ++k) {
      const int cc = wg + 4 * k;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        Vec16<T> v;
        v.pack(*reinterpret_cast<const float(*)[8]>(&W[k][q * 8]));
        const int chunk = (cc & 1) * 4 + q;
        *reinterpret_cast<uint4*>(sS + (cc >> 1) * (kBlk * 128) + (size_t)i_loc * 128 + ((chunk ^ (i_loc & 7)) * 16)) = v.raw;
      }
    }
    tc::fence_async_smem();
    ok = tc::mbar_wait(bar(4), 0);
  }
  ok = __syncthreads_and(ok);
  if (ok) {
    if (warp == 0 && tc::elect_one()) {
      tc::fence_after_sync();
      // dC += W B: A = W, K-major (K = columns j); B = B rows, MN-major (N = states in two blocks of 64)
      const uint64_t aw = tc::smem_desc_sw128(tc::smem_u32(sS), 16, 1024), bb = tc::smem_desc_sw128(tc::smem_u32(sX), KJ * 128, 1024);
      constexpr uint32_t idc = tc::instr_desc(kBlk, kN, fmt, 0, 1), idb = tc::instr_desc(kBlk, kN, fmt, 1, 1);
#pragma unroll
      for (int kk = 0; kk < KJ / 16; ++kk)
        tc::mma_ss(tmem + 256, aw + (uint64_t)(((kk >> 2) * (kBlk * 128) + (kk & 3) * 32) >> 4), bb + (uint64_t)(kk * (2048 >> 4)), idc, true);
      // dB += W^T C: A = W, MN-major (M = columns j in blocks of 64, K = rows i); B = C rows, MN-major
      const uint64_t bcd = tc::smem_desc_sw128(tc::smem_u32(sY), kBlk * 128, 1024);
#pragma unroll
      for (int jb = 0; jb <= MB; ++jb) {
        const uint64_t at = tc::smem_desc_sw128(tc::smem_u32(sS + jb * 2 * (kBlk * 128)), kBlk * 128, 1024);
#pragma unroll
        for (int kk = 0; kk < kBlk / 16; ++kk)
          tc::mma_ss(tmem + (jb == MB ? 384 : 0), at + (uint64_t)(kk * (2048 >> 4)), bcd + (uint64_t)(kk * (2048 >> 4)), idb, jb == MB || kk > 0);
      }
      tc::commit(bar(5));
    }
    ok = __all_sync(0xffffffffu, tc::mbar_wait(bar(5), 0));
    tc::fence_after_sync();
    if (ok) {
      // thread = row, 32 of the 128 states
      auto add_rows = [&](uint32_t col, float* dst, int row_block) {
        float v[32];
        tc::tmem_ld32(tmem + lane_base + col + wg * 32, v);
        const int t = t0 + row_block * kBlk + i_loc;
        if (t < a.len) {
          float* p = dst + (((int64_t)b * a.len + t) * a.groups + g) * kN + wg * 32;
#pragma unroll
          for (int e = 0; e < 32; e += 4) red_add4(p + e, v[e], v[e + 1], v[e + 2], v[e + 3]);
        }
      };
      add_rows(256, a.dC, MB);
      add_rows(384, a.dB, MB);
      if (MB) add_rows(0, a.dB, 0);
    }
  }
  if (!ok && lane == 0 && a.status) *(volatile int32_t*)a.status = 4;
}

template <typename T>
__global__ void __launch_bounds__(kBcThreads, 1) ssd_bc_kernel(const ssm_ssd_bc_args a, const __grid_constant__ BcMaps maps, int nchunks, int hpc, int nparts) {
  extern __shared__ unsigned char smdyn[];
  unsigned char* sm = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smdyn) + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t mbar[6];
  __shared__ uint32_t tmem_slot;
  if (threadIdx.x < 32) tc::tmem_alloc(tc::smem_u32(&tmem_slot), 512);
  if (threadIdx.x == 0)
    for (int i = 0; i < 6; ++i) tc::mbar_init(tc::smem_u32(&mbar[i]), 1);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  if ((int)blockIdx.x < (int)(gridDim.x >> 1)) ssd_bc_body<T, 1>(a, maps, nchunks, hpc, nparts, sm, mbar, &tmem_slot);  // the longer blocks first
  else ssd_bc_body<T, 0>(a, maps, nchunks, hpc, nparts, sm, mbar, &tmem_slot);
  tc::fence_before_sync();
  __syncthreads();
  if (threadIdx.x < 32) tc::tmem_dealloc(tmem_slot, 512);
}

template <typename T>
static int ssd_bc_launch(const ssm_ssd_bc_args& a, cudaStream_t st) {
  const int nchunks = (a.len + kQ - 1) / kQ, hpg = a.heads / a.groups, sms = sm_count();
  // heads per CTA, a divisor of a group's heads: a CTA costs about four heads' worth beside them (the last products, the sums over CTAs)
  int hpc = 1;
  double best = 1e300;
  for (int d = 1; d <= hpg; ++d) {
    if (hpg % d) continue;
    const int64_t ctas = 2ll * a.batch * nchunks * (a.heads / d);
    const double cost = (double)((ctas + sms - 1) / sms) * (4.0 + d);
    if (cost < best) best = cost, hpc = d;
  }
  BcMaps maps;
  if (int rc = encode_rows_map(&maps.x0, a.X, a.batch, a.len, a.heads, kP, kBlk, a.io_dtype)) return rc;
  if (int rc = encode_rows_map(&maps.x1, a.X, a.batch, a.len, a.heads, kP, kQ, a.io_dtype)) return rc;
  if (int rc = encode_rows_map(&maps.dy, a.dy, a.batch, a.len, a.heads, kP, kBlk, a.io_dtype)) return rc;
  if (int rc = encode_rows_map(&maps.b, a.Bm, a.batch, a.len, a.groups, kN, kBlk, a.io_dtype)) return rc;
  if (int rc = encode_rows_map(&maps.c, a.Cm, a.batch, a.len, a.groups, kN, kBlk, a.io_dtype)) return rc;
  cudaFuncSetAttribute(ssd_bc_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, BcSmem::ALLOC);
  const int nparts = a.heads / hpc;
  ssd_bc_kernel<T><<<2u * nparts * a.batch * nchunks, kBcThreads, BcSmem::ALLOC, st>>>(a, maps, nchunks, hpc, nparts);
  return launch_status("ssd_bc_kernel");
}

}  // namespace ssmb

using namespace ssmb;

extern "C" int ssm_ssd_bwd_bc(const ssm_ssd_bc_args* a, ssm_stream_t stream) {
  SSM_REQUIRE(a != nullptr, SSM_ERR_NULL, "ssd_bwd_bc: args is NULL");
  SSM_REQUIRE(a->batch >= 0 && a->len >= 0 && a->heads >= 1 && a->groups >= 1 && a->heads % a->groups == 0, SSM_ERR_SHAPE, "ssd_bwd_bc: bad shape");
  SSM_REQUIRE(a->io_dtype == SSM_BF16 || a->io_dtype == SSM_F16, SSM_ERR_DTYPE, "ssd_bwd_bc: operands must be bf16 or fp16");
  if (a->batch == 0 || a->len == 0) return SSM_OK;
  SSM_REQUIRE(a->X && a->dy && a->Bm && a->Cm && a->ws_dt && a->ws_cum && a->state_in && a->adjoint_in && a->dB && a->dC, SSM_ERR_NULL, "ssd_bwd_bc: missing tensor");
  SSM_REQUIRE(aligned_to(a->X, 16) && aligned_to(a->dy, 16) && aligned_to(a->Bm, 16) && aligned_to(a->Cm, 16) && aligned_to(a->ws_dt, 16) && aligned_to(a->ws_cum, 16) &&
                  aligned_to(a->state_in, 16) && aligned_to(a->adjoint_in, 16) && aligned_to(a->dB, 16) && aligned_to(a->dC, 16),
              SSM_ERR_ALIGN, "ssd_bwd_bc: tensors must be 16-byte aligned");
  const int64_t nchunks = (a->len + kQ - 1) / kQ;
  SSM_REQUIRE((int64_t)a->batch * nchunks * a->heads * 2 < (1ll << 31), SSM_ERR_TOO_LARGE, "ssd_bwd_bc: grid too large");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  return a->io_dtype == SSM_BF16 ? ssd_bc_launch<__nv_bfloat16>(*a, st) : ssd_bc_launch<__half>(*a, st);
}
