// Element-wise passes and step-size bookkeeping of the dual-form backward of the state-space-dual scan.  The contractions run on
// the tensor cores: the forward kernels, their mirror image in time (ssd_scan.cu) and the B / C gradients (ssd_bwd_bc.cu).
//
//   ssd_bwd_gate_kernel    dy = gY * silu(z)
//   ssd_bwd_finish_kernel  dz = gY * (y + D x) * silu'(z);  dX = dx + D dy;  dD = sum dy x
//   ssd_bwd_steps_kernel   ddt, dA, d dt_bias from the per-step dot products of the two scan passes
//
// The first two move 16-byte units of (batch, len, heads * 64) rows, several steps' loads in flight per thread.
#include <type_traits>

#include "ssd_common.cuh"

namespace ssmb {

constexpr int kUnit = 8;  // 16-bit elements per 16-byte unit

// thread = one unit of a row, four units apart by the grid
template <typename T>
__global__ void __launch_bounds__(256) ssd_bwd_gate_kernel(const ssm_ssd_bwd_args a, int64_t units) {
  constexpr int U = 4;
  const uint4* gy = reinterpret_cast<const uint4*>(a.gY);
  const uint4* z = reinterpret_cast<const uint4*>(a.z);
  const int64_t i0 = (int64_t)blockIdx.x * (256 * U) + threadIdx.x;
  uint4 gr[U], zr[U];
#pragma unroll
  for (int k = 0; k < U; ++k) {
    const int64_t i = i0 + k * 256 < units ? i0 + k * 256 : units - 1;
    gr[k] = __ldg(gy + i), zr[k] = __ldg(z + i);
  }
#pragma unroll
  for (int k = 0; k < U; ++k) {
    Vec16<T> g, zz;
    float f[8], zv[8];
    g.raw = gr[k], zz.raw = zr[k];
    g.unpack(f), zz.unpack(zv);
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] *= silu_fast(zv[e]);
    g.pack(f);
    if (i0 + k * 256 < units) reinterpret_cast<uint4*>(a.dy)[i0 + k * 256] = g.raw;
  }
}

// thread = one unit column of the (heads * 64) row, walking steps_per_block steps two at a time; grid.y = slices of the time axis
template <typename T>
__global__ void __launch_bounds__(256) ssd_bwd_finish_kernel(const ssm_ssd_bwd_args a, int steps_per_block) {
  constexpr int U = 2;
  const int units = a.heads * kP / kUnit;
  const int u_raw = blockIdx.x * 256 + threadIdx.x;
  const bool live = u_raw < units;
  const int u = live ? u_raw : units - 1;
  const int b = blockIdx.z;
  const int t_begin = blockIdx.y * steps_per_block, t_end = min(t_begin + steps_per_block, a.len);
  const int64_t row = units;  // in units
  const int h = u / (kP / kUnit), p0 = (u % (kP / kUnit)) * kUnit;
  float Dv[8], acc[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) Dv[e] = !a.D ? 0.f : (a.d_has_p ? __ldg(a.D + h * kP + p0 + e) : __ldg(a.D + h)), acc[e] = 0.f;
  const uint4 *gy = reinterpret_cast<const uint4*>(a.gY), *z = reinterpret_cast<const uint4*>(a.z), *X = reinterpret_cast<const uint4*>(a.X);
  const uint4 *yp = reinterpret_cast<const uint4*>(a.y_plain), *dx = reinterpret_cast<const uint4*>(a.dx);
  uint4 *dX = reinterpret_cast<uint4*>(a.dX), *dz = reinterpret_cast<uint4*>(a.dz);
  auto unpack = [](const uint4& r, float (&f)[8]) {
    Vec16<T> v;
    v.raw = r;
    v.unpack(f);
  };
  for (int t0 = t_begin; t0 < t_end; t0 += U) {
    uint4 xr[U], dr[U], gr[U], zr[U], yr[U];
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const int64_t at = ((int64_t)b * a.len + min(t0 + k, t_end - 1)) * row + u;
      xr[k] = __ldcs(X + at), dr[k] = __ldcs(dx + at), gr[k] = __ldcs(gy + at);
      if (z) zr[k] = __ldcs(z + at), yr[k] = __ldcs(yp + at);
    }
#pragma unroll
    for (int k = 0; k < U; ++k) {
      if (t0 + k >= t_end) break;
      const int64_t at = ((int64_t)b * a.len + t0 + k) * row + u;
      float x[8], g[8], o[8];
      unpack(xr[k], x), unpack(gr[k], g), unpack(dr[k], o);
      Vec16<T> v;
      if (z) {
        float zv[8], y[8], dzo[8];
        unpack(zr[k], zv), unpack(yr[k], y);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float s = sigmoid_fast(zv[e]);
          dzo[e] = g[e] * fmaf(Dv[e], x[e], y[e]) * (s * (1.f + zv[e] * (1.f - s)));
          g[e] *= zv[e] * s;
        }
        v.pack(dzo);
        if (live) __stcs(dz + at, v.raw);
        v.pack(g), v.unpack(g);  // dy as the scan passes read it
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        acc[e] = fmaf(g[e], x[e], acc[e]);
        o[e] = fmaf(Dv[e], g[e], o[e]);
      }
      v.pack(o);
      if (live) __stcs(dX + at, v.raw);
    }
  }
  if (!a.dD) return;
  if (a.d_has_p) {
    if (live) {
#pragma unroll
      for (int e = 0; e < 8; ++e) atomicAdd(a.dD + h * kP + p0 + e, acc[e]);
    }
  } else {  // the eight units of a head are neighbouring lanes
    float s = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) s += acc[e];
    if (!live) s = 0.f;
    s = group_sum<8, 1>(s);
    if (live && u % (kP / kUnit) == 0) atomicAdd(a.dD + h, s);
  }
}

// One CTA per (batch, chunk, four heads).  The per-step values are read as they lie in memory (heads innermost) and transposed through
// shared memory; two warps per head form the product <state, adjoint> at the chunk's left boundary (fp32, 8192 terms; what the kernel
// spends its time on: a warp per head and eight heads per CTA left too few loads in flight, 43 us against 28 for 2 x 4001 steps, 48 heads),
// then one of them the running sum of qd - u over the chunk's 256 steps, eight of them per lane.
constexpr int kStepHeads = 4, kStepLd = kQ + 4;
template <typename T>
__global__ void __launch_bounds__(kQ) ssd_bwd_steps_kernel(const ssm_ssd_steps_args a, int nchunks) {
  __shared__ __align__(16) float sPre[kStepHeads][kStepLd], sQ[kStepHeads][kStepLd], sR[kStepHeads][kStepLd];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int h0 = blockIdx.x * kStepHeads, c = blockIdx.y, b = blockIdx.z, nh = min(kStepHeads, a.heads - h0);
  const int t0 = c * kQ, steps = min(kQ, a.len - t0);
  const T* dt = reinterpret_cast<const T*>(a.dt);
  for (int i = tid; i < kQ * kStepHeads; i += kQ) {
    const int t = i / kStepHeads, hh = i % kStepHeads;
    float pre = 0.f, q = 0.f, r = 0.f;
    if (t < steps && hh < nh) {
      const int64_t at = ((int64_t)b * a.len + t0 + t) * a.heads + h0 + hh;
      pre = to_f<T>(dt[at]) + (a.dt_bias ? __ldg(a.dt_bias + h0 + hh) : 0.f);
      q = __ldg(a.qd + at), r = q - __ldg(a.u + at);
    }
    sPre[hh][t] = pre, sQ[hh][t] = q, sR[hh][t] = r;
  }
  static_assert(kQ / 32 == 2 * kStepHeads, "two warps per head");
  __shared__ float sDot[2 * kStepHeads];
  if (warp % kStepHeads < nh && c > 0) {
    const int h = h0 + warp % kStepHeads, part = warp / kStepHeads * (kP * kN / 8);
    const float4* s = reinterpret_cast<const float4*>(a.state_f32 + (((int64_t)b * nchunks + c) * a.heads + h) * (kP * kN)) + part;
    const float4* g = reinterpret_cast<const float4*>(a.adjoint_f32 + (((int64_t)b * nchunks + c - 1) * a.heads + h) * (kP * kN)) + part;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
    for (int i = lane; i < kP * kN / 8; i += 32) {
      const float4 x = __ldcs(s + i), y = __ldcs(g + i);
      acc.x = fmaf(x.x, y.x, acc.x), acc.y = fmaf(x.y, y.y, acc.y), acc.z = fmaf(x.z, y.z, acc.z), acc.w = fmaf(x.w, y.w, acc.w);
    }
    const float dot = warp_sum((acc.x + acc.y) + (acc.z + acc.w));
    if (lane == 0) sDot[warp] = dot;
  }
  __syncthreads();
  if (warp < nh) {
    const int h = h0 + warp;
    const float Ah = __ldg(a.A + h);
    float start = 0.f;
    if (c > 0) start = (sDot[warp] + sDot[warp + kStepHeads]) * ex2_approx(__ldg(a.ws_cum + (((int64_t)b * a.heads + h) * nchunks + c) * kQ));
    else if (a.start0) start = __ldg(a.start0 + b * a.heads + h);
    float r[8], run = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) r[k] = sR[warp][lane * 8 + k], run += r[k];
    float incl = run;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const float o = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= off) incl += o;
    }
    float da = start + (incl - run), dA = 0.f, db = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int t = lane * 8 + k;
      const float pre = sPre[warp][t], delta = a.dt_softplus ? softplus_f(pre) : pre;
      float d = (delta > 0.f ? sQ[warp][t] / delta : 0.f) + Ah * da;
      if (a.dt_softplus) d *= sigmoid_f(pre);
      if (t < steps) dA = fmaf(delta, da, dA), db += d;
      sR[warp][t] = d;
      da += r[k];
    }
    dA = warp_sum(dA), db = warp_sum(db);
    if (lane == 0) {
      atomicAdd(a.dA + h, dA);
      if (a.ddt_bias) atomicAdd(a.ddt_bias + h, db);
    }
  }
  __syncthreads();
  for (int i = tid; i < steps * kStepHeads; i += kQ) {
    const int t = i / kStepHeads, hh = i % kStepHeads;
    if (hh < nh) reinterpret_cast<T*>(a.ddt)[((int64_t)b * a.len + t0 + t) * a.heads + h0 + hh] = from_f<T>(sR[hh][t]);
  }
}

static int bwd_common_checks(const ssm_ssd_bwd_args* a) {
  SSM_REQUIRE(a != nullptr, SSM_ERR_NULL, "ssd backward: args is NULL");
  SSM_REQUIRE(a->batch >= 0 && a->len >= 0 && a->heads >= 1 && a->headdim == kP, SSM_ERR_SHAPE, "ssd backward: bad shape");
  SSM_REQUIRE(a->io_dtype == SSM_BF16 || a->io_dtype == SSM_F16, SSM_ERR_DTYPE, "ssd backward: operands must be bf16 or fp16");
  SSM_REQUIRE(a->batch <= 65535, SSM_ERR_TOO_LARGE, "ssd backward: batch too large for one launch");
  return SSM_OK;
}

}  // namespace ssmb

using namespace ssmb;

extern "C" int ssm_ssd_bwd_gate(const ssm_ssd_bwd_args* a, ssm_stream_t stream) {
  if (int rc = bwd_common_checks(a)) return rc;
  if (a->batch == 0 || a->len == 0) return SSM_OK;
  SSM_REQUIRE(a->gY && a->z && a->dy, SSM_ERR_NULL, "ssd_bwd_gate: missing tensor");
  SSM_REQUIRE(aligned_to(a->gY, 16) && aligned_to(a->dy, 16) && aligned_to(a->z, 16), SSM_ERR_ALIGN, "ssd_bwd_gate: tensors must be 16-byte aligned");
  const int64_t units = (int64_t)a->batch * a->len * a->heads * kP / kUnit, grid = (units + 1023) / 1024;
  SSM_REQUIRE(grid < (1ll << 31), SSM_ERR_TOO_LARGE, "ssd_bwd_gate: too large for one launch");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (a->io_dtype == SSM_BF16) ssd_bwd_gate_kernel<__nv_bfloat16><<<(unsigned)grid, 256, 0, st>>>(*a, units);
  else ssd_bwd_gate_kernel<__half><<<(unsigned)grid, 256, 0, st>>>(*a, units);
  return launch_status("ssd_bwd_gate_kernel");
}

extern "C" int ssm_ssd_bwd_finish(const ssm_ssd_bwd_args* a, ssm_stream_t stream) {
  if (int rc = bwd_common_checks(a)) return rc;
  if (a->batch == 0 || a->len == 0) return SSM_OK;
  SSM_REQUIRE(a->X && a->gY && a->dx && a->dX && (!a->z || (a->y_plain && a->dz)), SSM_ERR_NULL, "ssd_bwd_finish: missing tensor");
  SSM_REQUIRE(aligned_to(a->X, 16) && aligned_to(a->gY, 16) && aligned_to(a->dx, 16) && aligned_to(a->dX, 16) && aligned_to(a->z, 16) && aligned_to(a->y_plain, 16) &&
                  aligned_to(a->dz, 16),
              SSM_ERR_ALIGN, "ssd_bwd_finish: tensors must be 16-byte aligned");
  // steps per CTA: long enough that dD costs few additions, short enough to fill the GPU a few times
  const int units = a->heads * kP / kUnit, gx = (units + 255) / 256;
  int spb = 64;
  while (spb > 8 && (int64_t)gx * a->batch * ((a->len + spb - 1) / spb) < 4ll * sm_count()) spb /= 2;
  while ((a->len + spb - 1) / spb > 65535) spb *= 2;
  const dim3 grid(gx, (a->len + spb - 1) / spb, a->batch);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (a->io_dtype == SSM_BF16) ssd_bwd_finish_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>(*a, spb);
  else ssd_bwd_finish_kernel<__half><<<grid, 256, 0, st>>>(*a, spb);
  return launch_status("ssd_bwd_finish_kernel");
}

extern "C" int ssm_ssd_bwd_steps(const ssm_ssd_steps_args* a, ssm_stream_t stream) {
  SSM_REQUIRE(a != nullptr, SSM_ERR_NULL, "ssd_bwd_steps: args is NULL");
  SSM_REQUIRE(a->batch >= 0 && a->len >= 0 && a->heads >= 1, SSM_ERR_SHAPE, "ssd_bwd_steps: bad shape");
  SSM_REQUIRE(a->io_dtype == SSM_BF16 || a->io_dtype == SSM_F16, SSM_ERR_DTYPE, "ssd_bwd_steps: dt must be bf16 or fp16");
  if (a->batch == 0 || a->len == 0) return SSM_OK;
  SSM_REQUIRE(a->dt && a->A && a->u && a->qd && a->ws_cum && a->state_f32 && a->adjoint_f32 && a->ddt && a->dA, SSM_ERR_NULL, "ssd_bwd_steps: missing tensor");
  SSM_REQUIRE(aligned_to(a->state_f32, 16) && aligned_to(a->adjoint_f32, 16), SSM_ERR_ALIGN, "ssd_bwd_steps: states must be 16-byte aligned");
  const int64_t nchunks = (a->len + kQ - 1) / kQ;
  SSM_REQUIRE(nchunks <= 65535 && a->batch <= 65535, SSM_ERR_TOO_LARGE, "ssd_bwd_steps: too large for one launch");
  const dim3 grid((a->heads + kStepHeads - 1) / kStepHeads, (unsigned)nchunks, a->batch);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (a->io_dtype == SSM_BF16) ssd_bwd_steps_kernel<__nv_bfloat16><<<grid, kQ, 0, st>>>(*a, (int)nchunks);
  else ssd_bwd_steps_kernel<__half><<<grid, kQ, 0, st>>>(*a, (int)nchunks);
  return launch_status("ssd_bwd_steps_kernel");
}
