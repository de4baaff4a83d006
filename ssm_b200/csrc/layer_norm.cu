// Residual add fused with LayerNorm / RMSNorm, forward and backward, sm_100a.
//
// HBM-bound: each row is read once, the mean and the centred variance are both computed from what was read (the two-pass
// form of the specification, no E[x^2]-mean^2 cancellation), and y / residual_out are written once.  Forward: a row is
// owned by a warp or by 128 or 512 threads and lies in their registers, x and residual as 16-byte vectors.  Backward: a warp, or 64 to 512
// threads, granules of four columns, the next row on its way into shared memory.  The backward kernel is persistent:
// every thread keeps the weight / bias gradient of its own columns in registers across all rows its CTA visits, the CTA
// writes one partial row, and a second small kernel folds the partials -- no atomics, bitwise reproducible.
#include <algorithm>
#include <mutex>
#include <type_traits>

#include "common.cuh"

namespace ssmb {

constexpr int kNormFwdChunks = 4;  // 16-byte chunks of x per thread, forward
constexpr int kNormBwdChunks = 4;  // widest backward configuration: 512 threads x 4 chunks of 16 bytes
constexpr int kNormBwdMaxCtas = 592;  // 4 per SM on a 148-SM part

// fp32 -> V consecutive elements of run-time type
template <int V>
__device__ __forceinline__ void store_dyn_vec(void* base, int64_t i, int dtype, const float (&f)[V]) {
  if (dtype == SSM_F32) {
    float4* p = reinterpret_cast<float4*>(reinterpret_cast<float*>(base) + i);
#pragma unroll
    for (int k = 0; k < V / 4; ++k) __stcs(p + k, make_float4(f[4 * k], f[4 * k + 1], f[4 * k + 2], f[4 * k + 3]));
  } else if constexpr (V == 8) {
    uint4 raw;
    if (dtype == SSM_BF16) {
      __nv_bfloat16* e = reinterpret_cast<__nv_bfloat16*>(&raw);
#pragma unroll
      for (int k = 0; k < 8; ++k) e[k] = __float2bfloat16_rn(f[k]);
    } else {
      __half* e = reinterpret_cast<__half*>(&raw);
#pragma unroll
      for (int k = 0; k < 8; ++k) e[k] = __float2half_rn(f[k]);
    }
    __stcs(reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(base) + i), raw);
  } else {
    uint2 raw;
    if (dtype == SSM_BF16) {
      __nv_bfloat16* e = reinterpret_cast<__nv_bfloat16*>(&raw);
#pragma unroll
      for (int k = 0; k < 4; ++k) e[k] = __float2bfloat16_rn(f[k]);
    } else {
      __half* e = reinterpret_cast<__half*>(&raw);
#pragma unroll
      for (int k = 0; k < 4; ++k) e[k] = __float2half_rn(f[k]);
    }
    __stcs(reinterpret_cast<uint2*>(reinterpret_cast<uint16_t*>(base) + i), raw);
  }
}

// Sum over the G threads of a row group.  G == 32: shuffles only.  G > 32: one row per CTA.
template <int G>
__device__ __forceinline__ float group_allsum(float v, float* scratch) {
  v = warp_sum(v);
  if constexpr (G > 32) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();  // scratch reuse
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < G / 32; ++w) t += scratch[w];
    v = t;
  }
  return v;
}

template <typename T, int G>
struct NormCfg {
  static constexpr int V = 16 / sizeof(T);
  static constexpr int BLOCK = G < 128 ? 128 : G;
  static constexpr int RPC = BLOCK / G;  // rows per CTA pass
};

// A row's pieces of a tensor of run-time element type, in two steps: every load of the row is issued first (the type switch
// sits outside the loop over chunks, so each arm is a straight run of independent loads), the conversions come afterwards.
// With the load, the conversion and the next load of a chunk in one loop body the loads of a row went out one memory
// latency after the other.  Threads beyond the end of the row read its last chunk (a valid address) and drop the value.
template <int V, int G, int MC>
__device__ __forceinline__ void dyn_issue_row(const void* base, int64_t row_off, int gt, int nchunk, int dtype, uint4 (&a)[MC], uint4 (&b)[MC]) {
  if (dtype == SSM_F32) {
#pragma unroll
    for (int c = 0; c < MC; ++c) {
      const int ch = min(c * G + gt, nchunk - 1);
      const uint4* p = reinterpret_cast<const uint4*>(reinterpret_cast<const float*>(base) + row_off + (int64_t)ch * V);
      a[c] = __ldcs(p);
      if constexpr (V == 8) b[c] = __ldcs(p + 1);
    }
  } else if constexpr (V == 8) {
#pragma unroll
    for (int c = 0; c < MC; ++c) {
      const int ch = min(c * G + gt, nchunk - 1);
      a[c] = __ldcs(reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(base) + row_off + (int64_t)ch * V));
    }
  } else {
#pragma unroll
    for (int c = 0; c < MC; ++c) {
      const int ch = min(c * G + gt, nchunk - 1);
      const uint2 t = __ldcs(reinterpret_cast<const uint2*>(reinterpret_cast<const uint16_t*>(base) + row_off + (int64_t)ch * V));
      a[c] = make_uint4(t.x, t.y, 0u, 0u);
    }
  }
}
template <int V>
__device__ __forceinline__ void dyn_convert(int dtype, const uint4& a, const uint4& b, float (&f)[V]) {
  if (dtype == SSM_F32) {
    f[0] = __uint_as_float(a.x), f[1] = __uint_as_float(a.y), f[2] = __uint_as_float(a.z), f[3] = __uint_as_float(a.w);
    if constexpr (V == 8) f[4] = __uint_as_float(b.x), f[5] = __uint_as_float(b.y), f[6] = __uint_as_float(b.z), f[7] = __uint_as_float(b.w);
  } else if (dtype == SSM_BF16) {
    const __nv_bfloat16* e = reinterpret_cast<const __nv_bfloat16*>(&a);
#pragma unroll
    for (int k = 0; k < V; ++k) f[k] = __bfloat162float(e[k]);
  } else {
    const __half* e = reinterpret_cast<const __half*>(&a);
#pragma unroll
    for (int k = 0; k < V; ++k) f[k] = __half2float(e[k]);
  }
}
// the row's pieces of a tensor of the io type
template <typename T, int G, int MC>
__device__ __forceinline__ void io_issue_row(const void* base, int64_t row_off, int gt, int nchunk, uint4 (&a)[MC]) {
  constexpr int V = 16 / sizeof(T);
#pragma unroll
  for (int c = 0; c < MC; ++c) {
    const int ch = min(c * G + gt, nchunk - 1);
    a[c] = __ldcs(reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(base) + row_off + (int64_t)ch * V));
  }
}

// Raw pieces of a row of x and of the residual, in flight.
template <int MC>
struct NormRowRaw {
  uint4 x[MC], ra[MC], rb[MC];
};
template <typename T, int G, int MC, bool RES = true>
__device__ __forceinline__ void norm_issue_row(const ssm_norm_args& a, int64_t row, int gt, int nchunk, NormRowRaw<MC>& raw) {
  constexpr int V = 16 / sizeof(T);
  io_issue_row<T, G, MC>(a.x, row * a.hidden, gt, nchunk, raw.x);
  if (RES && a.residual) dyn_issue_row<V, G, MC>(a.residual, row * a.hidden, gt, nchunk, a.res_dtype, raw.ra, raw.rb);
}
// s = x (+ residual when prenorm), r = residual; zero beyond the end of the row.
template <typename T, int G, int MC, bool RES = true>
__device__ __forceinline__ void norm_convert_row(const ssm_norm_args& a, int gt, int nchunk, const NormRowRaw<MC>& raw, float (&s)[MC][16 / sizeof(T)],
                                                 float (&r)[MC][16 / sizeof(T)]) {
  constexpr int V = 16 / sizeof(T);
#pragma unroll
  for (int c = 0; c < MC; ++c) {
    if (c * G + gt < nchunk) {
      Vec16<T> v;
      v.raw = raw.x[c];
      v.unpack(s[c]);
      if (RES && a.residual) {
        dyn_convert<V>(a.res_dtype, raw.ra[c], raw.rb[c], r[c]);
        if (a.prenorm) {
#pragma unroll
          for (int i = 0; i < V; ++i) s[c][i] += r[c][i];
        }
      }
    } else {
#pragma unroll
      for (int i = 0; i < V; ++i) s[c][i] = 0.f, r[c][i] = 0.f;
    }
  }
}
// Loads the row into registers as s = x (+ residual when prenorm); returns through refs.
template <typename T, int G, int MC, bool RES = true>
__device__ __forceinline__ void norm_load_row(const ssm_norm_args& a, int64_t row, int gt, int nchunk, float (&s)[MC][16 / sizeof(T)],
                                              float (&r)[MC][16 / sizeof(T)]) {
  NormRowRaw<MC> raw;
  norm_issue_row<T, G, MC, RES>(a, row, gt, nchunk, raw);
  norm_convert_row<T, G, MC, RES>(a, gt, nchunk, raw, s, r);
}

template <typename T, int G, int MC>
__device__ __forceinline__ void norm_stats(const ssm_norm_args& a, int gt, int nchunk, const float (&s)[MC][16 / sizeof(T)], float* scratch,
                                           float& mean, float& rstd) {
  constexpr int V = 16 / sizeof(T);
  const float inv = 1.f / (float)a.hidden;
  mean = 0.f;
  if (!a.is_rms) {
    float t = 0.f;
#pragma unroll
    for (int c = 0; c < MC; ++c)
#pragma unroll
      for (int i = 0; i < V; ++i) t += s[c][i];
    mean = group_allsum<G>(t, scratch) * inv;
  }
  float q = 0.f;
#pragma unroll
  for (int c = 0; c < MC; ++c) {
    if (c * G + gt < nchunk) {
#pragma unroll
      for (int i = 0; i < V; ++i) {
        const float d = s[c][i] - mean;
        q = fmaf(d, d, q);
      }
    }
  }
  rstd = rsqrtf(group_allsum<G>(q, scratch) * inv + a.eps);
}

// MC = 16-byte chunks of a row per thread.  Rows of up to 768 chunks stay with 128 threads (several rows in flight per SM keep
// more loads outstanding than one wide CTA per row does); only wider rows take 512 threads.
// RES = false: the call has no residual (its registers are then free, which raises the number of rows in flight).
template <typename T, int G, int MC = kNormFwdChunks, bool RES = true>
__global__ void __launch_bounds__(NormCfg<T, G>::BLOCK) norm_fwd_kernel(const ssm_norm_args a) {
  pdl_wait();
  pdl_trigger();
  using Cfg = NormCfg<T, G>;
  constexpr int V = Cfg::V;
  constexpr int kNormFwdChunks = MC;
  __shared__ float scratch[32];
  const int gt = threadIdx.x % G;
  const int64_t row = (int64_t)blockIdx.x * Cfg::RPC + threadIdx.x / G;
  if (row >= a.rows) return;  // whole groups leave together (G >= 32; G > 32 has one row per CTA)
  const int nchunk = a.hidden / V;
  float s[kNormFwdChunks][V], r[kNormFwdChunks][V];
  norm_load_row<T, G, kNormFwdChunks, RES>(a, row, gt, nchunk, s, r);
  if (a.residual_out) {
#pragma unroll
    for (int c = 0; c < kNormFwdChunks; ++c) {
      const int ch = c * G + gt;
      if (ch < nchunk) {
        float o[V];
#pragma unroll
        for (int i = 0; i < V; ++i) o[i] = (RES && a.residual && !a.prenorm) ? s[c][i] + r[c][i] : s[c][i];
        store_dyn_vec<V>(a.residual_out, row * a.hidden + (int64_t)ch * V, a.resout_dtype, o);
      }
    }
  }
  float mean, rstd;
  norm_stats<T, G, kNormFwdChunks>(a, gt, nchunk, s, scratch, mean, rstd);
#pragma unroll
  for (int c = 0; c < kNormFwdChunks; ++c) {
    const int ch = c * G + gt;
    if (ch < nchunk) {
      float o[V], wv[V], bv[V];
      load_param_vec<V>(a.weight, ch * V, a.param_dtype, wv);
      if (a.bias) {
        load_param_vec<V>(a.bias, ch * V, a.param_dtype, bv);
      } else {
#pragma unroll
        for (int i = 0; i < V; ++i) bv[i] = 0.f;
      }
#pragma unroll
      for (int i = 0; i < V; ++i) {
        float y = fmaf((s[c][i] - mean) * rstd, wv[i], bv[i]);
        if (RES && a.residual && !a.prenorm) y += r[c][i];
        o[i] = y;
      }
      Vec16<T> v;
      v.pack(o);
      v.store_stream(reinterpret_cast<T*>(a.y) + row * a.hidden + (int64_t)ch * V);
    }
  }
}

// Sums of two values over the G threads of a row group.  Wide groups exchange them through one of two scratch rows used in turn,
// so a reduction costs one barrier: whoever writes a row again has passed the barrier of the reduction in between.
template <int G>
__device__ __forceinline__ void group_allsum2(float& a, float& b, float2 (*scratch)[16], int& turn) {
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, off);
    b += __shfl_xor_sync(0xffffffffu, b, off);
  }
  if constexpr (G > 32) {
    const int first = G == 64 ? threadIdx.x >> 6 << 1 : 0;  // two groups of two warps to a CTA, each with a barrier of its own
    if ((threadIdx.x & 31) == 0) scratch[turn][threadIdx.x >> 5] = make_float2(a, b);
    if constexpr (G == 64) asm volatile("bar.sync %0, 64;\n" ::"r"(1 + (first >> 1)) : "memory");
    else __syncthreads();
    a = 0.f, b = 0.f;
#pragma unroll
    for (int w = 0; w < G / 32; ++w) {
      const float2 v = scratch[turn][first + w];
      a += v.x, b += v.y;
    }
    turn ^= 1;
  }
}

// Backward.  A row is split into granules of four elements, MG to a thread: granule k of thread t is k * G + t, so that every access
// of a warp is contiguous in 16-bit and 32-bit tensors alike (8 elements a thread read fp32 rows in half sectors: twice the L2 traffic).
// The time of a row is a chain of latencies (loads, two rounds of sums, stores), so the rows travel through a ring in shared
// memory: each thread copies its own granules of x, dy, the residual and the gradient arriving through the x + residual output
// (asynchronous copies, no barrier) and has its next row under way while it works on this one.  What a row still needs at its end is
// read there again, which leaves the registers to the running weight / bias gradients of the thread's columns.  Packed fp32 arithmetic.
//  * A row of up to 32 * 4 granules is owned by ONE warp (G = 32), four rows to a CTA; wider rows take 64 to 512 threads, four granules
//    each if they can (eight leave no room for what a row keeps in registers: 4096 bf16 columns, fp32 residual, 336 us; four of 256 threads: 173).
//  * Two rounds of sums, two values each: {sum s, sum w dy}, then {sum (s - mean)^2, sum w dy (s - mean)}, from which the standard
//    deviation and both correction terms follow (one round for RMSNorm).
// 16376 rows of 1600 bf16 columns, fp32 residual and its gradient, 471 MB: 104 us with the loads in registers, scalar arithmetic and 16
// bytes of x per access (63 instructions per element), 69 us so (28; 6.3 TB/s).
//  * STREAM: a residual stream of fp32, in and out, known at compile time, and FULL granules that every thread has: with run-time types
//    and every granule guarded the loads of a row could not be put together (54 instructions per element, 104 us).
template <typename T, int G, int MG>
constexpr int norm_bwd_ctas_per_sm() {
  if (G > 128) return G == 256 ? 2 : 1;
  return MG <= 4 ? 4 : (MG <= 6 ? 3 : 2);
}
__host__ __device__ constexpr int dtype_bytes(int dtype) { return dtype == SSM_F32 ? 4 : 2; }
// four elements of a shared-memory slot as fp32 pairs
template <typename T>
__device__ __forceinline__ void granule(const unsigned char* p, float2 (&f)[2]) {
  if constexpr (sizeof(T) == 4) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    f[0] = make_float2(v.x, v.y), f[1] = make_float2(v.z, v.w);
  } else if constexpr (std::is_same<T, __half>::value) {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    f[0] = __half22float2(*reinterpret_cast<const __half2*>(&v.x)), f[1] = __half22float2(*reinterpret_cast<const __half2*>(&v.y));
  } else {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    f[0] = make_float2(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u));
    f[1] = make_float2(__uint_as_float(v.y << 16), __uint_as_float(v.y & 0xffff0000u));
  }
}
__device__ __forceinline__ void granule_dyn(const unsigned char* p, int dtype, float2 (&f)[2]) {
  if (dtype == SSM_F32) granule<float>(p, f);
  else if (dtype == SSM_BF16) granule<__nv_bfloat16>(p, f);
  else granule<__half>(p, f);
}
template <typename T>
__device__ __forceinline__ void granule_store(T* p, const float2 (&f)[2]) {
  if constexpr (sizeof(T) == 4) {
    __stcs(reinterpret_cast<float4*>(p), make_float4(f[0].x, f[0].y, f[1].x, f[1].y));
  } else if constexpr (std::is_same<T, __half>::value) {
    const __half2 a = __float22half2_rn(f[0]), b = __float22half2_rn(f[1]);
    __stcs(reinterpret_cast<uint2*>(p), make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b)));
  } else {
    const __nv_bfloat162 a = __float22bfloat162_rn(f[0]), b = __float22bfloat162_rn(f[1]);
    __stcs(reinterpret_cast<uint2*>(p), make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b)));
  }
}
__device__ __forceinline__ void granule_store_dyn(void* base, int64_t i, int dtype, const float2 (&f)[2]) {
  if (dtype == SSM_F32) granule_store(reinterpret_cast<float*>(base) + i, f);
  else if (dtype == SSM_BF16) granule_store(reinterpret_cast<__nv_bfloat16*>(base) + i, f);
  else granule_store(reinterpret_cast<__half*>(base) + i, f);
}
__device__ __forceinline__ void granule_copy(uint32_t dst, const char* src, bool wide) {
  if (wide) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(dst), "l"(src) : "memory");
}

template <typename T, int G, int MG, int FULL, int ST, bool STREAM>
__global__ void __launch_bounds__(NormCfg<T, G>::BLOCK, norm_bwd_ctas_per_sm<T, G, MG>()) norm_bwd_kernel(const ssm_norm_bwd_args g) {
  pdl_wait();
  pdl_trigger();
  using Cfg = NormCfg<T, G>;
  constexpr int BLOCK = Cfg::BLOCK, RPC = Cfg::RPC, E = 4 * (int)sizeof(T);
  constexpr bool HOLD = MG <= 6;  // w dy stays in registers between the rounds of sums
  constexpr bool HOLD_W = MG <= 4;      // the weights of the thread's columns too
  constexpr int MH = HOLD ? MG : 1, MW = HOLD_W ? MG : 1;
  const ssm_norm_args& a = g.fwd;
  extern __shared__ __align__(16) unsigned char norm_ring[];
  __shared__ float2 scratch[2][16];
  const int tid = threadIdx.x, gt = tid % G, slot = tid / G;
  const int ngran = a.hidden / 4;
  const float inv = 1.f / (float)a.hidden;
  const bool has_r = STREAM || (a.residual && a.prenorm), has_g = STREAM || g.dresidual_out != nullptr;
  const int rtype = STREAM ? SSM_F32 : a.res_dtype, gtype = STREAM ? SSM_F32 : a.resout_dtype;
  const int re = has_r ? 4 * dtype_bytes(rtype) : 0, ge = has_g ? 4 * dtype_bytes(gtype) : 0;  // bytes per granule
  // a stage: x, dy, residual, gradient of the x + residual output, each [granule][thread]
  const int stage_bytes = MG * BLOCK * (2 * E + re + ge);
  unsigned char* const sx = norm_ring + tid * E;
  unsigned char* const sr = norm_ring + 2 * MG * BLOCK * E + tid * re;
  unsigned char* const sg = norm_ring + MG * BLOCK * (2 * E + re) + tid * ge;
  const uint32_t ux = (uint32_t)__cvta_generic_to_shared(sx), ur = (uint32_t)__cvta_generic_to_shared(sr), ug = (uint32_t)__cvta_generic_to_shared(sg);
  const int64_t step = (int64_t)gridDim.x * RPC;
  auto issue = [&](int64_t row, int at) {
    if (row < a.rows) {
      const char* px = reinterpret_cast<const char*>(a.x) + (row * a.hidden + gt * 4) * sizeof(T);
      const char* pd = reinterpret_cast<const char*>(g.dy) + (row * a.hidden + gt * 4) * sizeof(T);
      const char* pr = reinterpret_cast<const char*>(a.residual) + (row * ngran + gt) * re;
      const char* pg = reinterpret_cast<const char*>(g.dresidual_out) + (row * ngran + gt) * ge;
#pragma unroll
      for (int k = 0; k < MG; ++k) {
        if (k < FULL || k * G + gt < ngran) {
          granule_copy(ux + at + k * BLOCK * E, px + k * G * E, E == 16);
          granule_copy(ux + at + (MG + k) * BLOCK * E, pd + k * G * E, E == 16);
          if (has_r) granule_copy(ur + at + k * BLOCK * re, pr + k * G * re, re == 16);
          if (has_g) granule_copy(ug + at + k * BLOCK * ge, pg + k * G * ge, ge == 16);
        }
      }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  const float2 zero = make_float2(0.f, 0.f);
  float2 dw[MG][2], db[MG][2];
#pragma unroll
  for (int k = 0; k < MG; ++k) dw[k][0] = dw[k][1] = db[k][0] = db[k][1] = zero;
  float wh[MW][4];
  if (HOLD_W) {
#pragma unroll
    for (int k = 0; k < MG; ++k) load_param_vec<4>(a.weight, min(k * G + gt, ngran - 1) * 4, a.param_dtype, wh[HOLD_W ? k : 0]);
  }
  auto load_wdy = [&](int k, int at, float2 (&wdy)[2]) {
    float w[4];
    float2 dy[2];
    if (HOLD_W) {
#pragma unroll
      for (int i = 0; i < 4; ++i) w[i] = wh[HOLD_W ? k : 0][i];
    } else {
      load_param_vec<4>(a.weight, (k * G + gt) * 4, a.param_dtype, w);
    }
    granule<T>(sx + at + (MG + k) * BLOCK * E, dy);
    wdy[0] = __fmul2_rn(make_float2(w[0], w[1]), dy[0]), wdy[1] = __fmul2_rn(make_float2(w[2], w[3]), dy[1]);
  };
  int turn = 0, at = 0;
  int64_t row = (int64_t)blockIdx.x * RPC + slot;  // the same for all threads of a group, and a group of more than a warp is the CTA
  if (ST == 2) issue(row, 0);
  for (; row < a.rows; row += step) {
    if (ST == 2) {
      issue(row + step, at ^ stage_bytes);
      asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    } else {
      issue(row, 0);
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    }
    float2 s[MG][2], wdyh[MH][2];
    float2 m2 = zero, e2 = zero;
#pragma unroll
    for (int k = 0; k < MG; ++k) {
      s[k][0] = s[k][1] = zero;
      if (HOLD) wdyh[HOLD ? k : 0][0] = wdyh[HOLD ? k : 0][1] = zero;
      if (k < FULL || k * G + gt < ngran) {
        granule<T>(sx + at + k * BLOCK * E, s[k]);
        if (has_r) {
          float2 r[2];
          granule_dyn(sr + at + k * BLOCK * re, rtype, r);
          s[k][0] = __fadd2_rn(s[k][0], r[0]), s[k][1] = __fadd2_rn(s[k][1], r[1]);
        }
        if (HOLD || !a.is_rms) {
          float2 wdy[2];
          load_wdy(k, at, wdy);
          m2 = __fadd2_rn(m2, __fadd2_rn(s[k][0], s[k][1])), e2 = __fadd2_rn(e2, __fadd2_rn(wdy[0], wdy[1]));
          if (HOLD) wdyh[HOLD ? k : 0][0] = wdy[0], wdyh[HOLD ? k : 0][1] = wdy[1];
        }
      }
    }
    float mean = 0.f, c2 = 0.f;
    if (!a.is_rms) {
      mean = m2.x + m2.y, c2 = e2.x + e2.y;
      group_allsum2<G>(mean, c2, scratch, turn);
      mean *= inv, c2 *= inv;
    }
    const float2 nmean = make_float2(-mean, -mean);
    float2 q2 = zero, d2 = zero;
#pragma unroll
    for (int k = 0; k < MG; ++k) {
      if (k < FULL || k * G + gt < ngran) {
        float2 wdy[2];
        if (!HOLD) load_wdy(k, at, wdy);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          s[k][i] = __fadd2_rn(s[k][i], nmean);
          q2 = __ffma2_rn(s[k][i], s[k][i], q2);
          d2 = __ffma2_rn(HOLD ? wdyh[HOLD ? k : 0][i] : wdy[i], s[k][i], d2);
        }
      }
    }
    float q = q2.x + q2.y, c1 = d2.x + d2.y;
    group_allsum2<G>(q, c1, scratch, turn);
    const float rstd = rsqrtf(q * inv + a.eps);
    // ds = rstd (w dy - xhat c1 - c2), xhat = rstd (s - mean), c1 = mean of w dy xhat, c2 = mean of w dy
    const float sc = -(c1 * inv * rstd) * rstd * rstd, off = -c2 * rstd;
    const float2 rs = make_float2(rstd, rstd), sc2 = make_float2(sc, sc), off2 = make_float2(off, off);
    const int64_t col = row * a.hidden + gt * 4;
#pragma unroll
    for (int k = 0; k < MG; ++k) {
      if (k < FULL || k * G + gt < ngran) {
        float2 dy[2], wdyl[2], ds[2];
        granule<T>(sx + at + (MG + k) * BLOCK * E, dy);
        if (!HOLD) load_wdy(k, at, wdyl);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          dw[k][i] = __ffma2_rn(dy[i], __fmul2_rn(s[k][i], rs), dw[k][i]);
          db[k][i] = __fadd2_rn(db[k][i], dy[i]);
          ds[i] = __ffma2_rn(s[k][i], sc2, __ffma2_rn(HOLD ? wdyh[HOLD ? k : 0][i] : wdyl[i], rs, off2));
        }
        if (has_g) {  // the gradient arriving through the x + residual output reaches x and residual unchanged
          float2 ga[2];
          granule_dyn(sg + at + k * BLOCK * ge, gtype, ga);
#pragma unroll
          for (int i = 0; i < 2; ++i) ds[i] = __fadd2_rn(ds[i], ga[i]), dy[i] = __fadd2_rn(dy[i], ga[i]);
        }
        granule_store(reinterpret_cast<T*>(g.dx) + col + k * G * 4, ds);
        if (STREAM || g.dresidual) {
          if (STREAM || a.prenorm) granule_store_dyn(g.dresidual, col + k * G * 4, rtype, ds);
          else granule_store_dyn(g.dresidual, col + k * G * 4, rtype, dy);
        }
      }
    }
    if (ST == 2) at ^= stage_bytes;
  }
  // fold the RPC row slots of this CTA (over the ring), then write the CTA's partial rows
  float4* const acc = reinterpret_cast<float4*>(norm_ring);
  if constexpr (RPC > 1) {
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
#pragma unroll
    for (int k = 0; k < MG; ++k) {
      acc[(2 * k) * BLOCK + tid] = make_float4(dw[k][0].x, dw[k][0].y, dw[k][1].x, dw[k][1].y);
      acc[(2 * k + 1) * BLOCK + tid] = make_float4(db[k][0].x, db[k][0].y, db[k][1].x, db[k][1].y);
    }
    __syncthreads();
  }
  if (slot == 0) {
    float* pw = g.partial + (int64_t)blockIdx.x * 2 * a.hidden + gt * 4;
#pragma unroll
    for (int k = 0; k < MG; ++k) {
      if (k < FULL || k * G + gt < ngran) {
        float4 tw = make_float4(dw[k][0].x, dw[k][0].y, dw[k][1].x, dw[k][1].y);
        float4 tb = make_float4(db[k][0].x, db[k][0].y, db[k][1].x, db[k][1].y);
        if constexpr (RPC > 1) {
#pragma unroll
          for (int o = 1; o < RPC; ++o) {
            const float4 x = acc[(2 * k) * BLOCK + o * G + gt], y = acc[(2 * k + 1) * BLOCK + o * G + gt];
            tw.x += x.x, tw.y += x.y, tw.z += x.z, tw.w += x.w;
            tb.x += y.x, tb.y += y.y, tb.z += y.z, tb.w += y.w;
          }
        }
        *reinterpret_cast<float4*>(pw + k * G * 4) = tw;
        *reinterpret_cast<float4*>(pw + a.hidden + k * G * 4) = tb;
      }
    }
  }
}

// Column sums of the per-CTA partial rows: 32 columns x kFoldLanes partial-row lanes per CTA,
// so the loads of a column are spread over many threads instead of one serial chain.
constexpr int kFoldLanes = 32;
__global__ void __launch_bounds__(32 * kFoldLanes) norm_fold_kernel(const float* __restrict__ partial, int nctas, int hidden,
                                                                   void* __restrict__ dweight, void* __restrict__ dbias, int dtype) {
  pdl_wait();
  pdl_trigger();
  __shared__ float sums[kFoldLanes][33];
  const int cx = threadIdx.x & 31, ky = threadIdx.x >> 5;
  const int col = blockIdx.x * 32 + cx;
  const float* __restrict__ p = partial + blockIdx.y * hidden + col;  // y: 0 the weight's gradient, 1 the bias's
  float t = 0.f;
  if (col < hidden) {
#pragma unroll 8
    for (int k = ky; k < nctas; k += kFoldLanes) t += __ldg(p + (int64_t)k * 2 * hidden);
  }
  sums[ky][cx] = t;
  __syncthreads();
  if (ky == 0 && col < hidden) {
#pragma unroll
    for (int k = 1; k < kFoldLanes; ++k) t += sums[k][cx];
    store_dyn(blockIdx.y ? dbias : dweight, col, dtype, t);
  }
}

// ---- fallback for rows that cannot be vectorised (hidden not a multiple of the vector, or
// ---- misaligned pointers): one CTA per row, strided scalar accesses, atomics for dw / db.
template <typename T>
__device__ __forceinline__ float norm_s_at(const ssm_norm_args& a, int64_t off) {
  float v = to_f<T>(reinterpret_cast<const T*>(a.x)[off]);
  if (a.residual && a.prenorm) v += load_dyn(a.residual, off, a.res_dtype);
  return v;
}
__device__ __forceinline__ float block_allsum128(float v, float* scratch) {
  v = warp_sum(v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = v;
  __syncthreads();
  return scratch[0] + scratch[1] + scratch[2] + scratch[3];
}
template <typename T, bool BWD>
__global__ void __launch_bounds__(128) norm_scalar_kernel(const ssm_norm_bwd_args g) {
  const ssm_norm_args& a = g.fwd;
  __shared__ float scratch[4];
  const int64_t row = blockIdx.x;
  const int64_t base = row * a.hidden;
  const float inv = 1.f / (float)a.hidden;
  float mean = 0.f;
  if (!a.is_rms) {
    float t = 0.f;
    for (int c = threadIdx.x; c < a.hidden; c += 128) t += norm_s_at<T>(a, base + c);
    mean = block_allsum128(t, scratch) * inv;
  }
  float q = 0.f;
  for (int c = threadIdx.x; c < a.hidden; c += 128) {
    const float d = norm_s_at<T>(a, base + c) - mean;
    q = fmaf(d, d, q);
  }
  const float rstd = rsqrtf(block_allsum128(q, scratch) * inv + a.eps);
  if (!BWD) {
    for (int c = threadIdx.x; c < a.hidden; c += 128) {
      const float sv = norm_s_at<T>(a, base + c);
      float y = (sv - mean) * rstd * load_dyn(a.weight, c, a.param_dtype);
      if (a.bias) y += load_dyn(a.bias, c, a.param_dtype);
      if (a.residual && !a.prenorm) y += load_dyn(a.residual, base + c, a.res_dtype);
      reinterpret_cast<T*>(a.y)[base + c] = from_f<T>(y);
      if (a.residual_out) {
        float ro = to_f<T>(reinterpret_cast<const T*>(a.x)[base + c]);
        if (a.residual) ro += load_dyn(a.residual, base + c, a.res_dtype);
        store_dyn(a.residual_out, base + c, a.resout_dtype, ro);
      }
    }
  } else {
    float c1 = 0.f, c2 = 0.f;
    for (int c = threadIdx.x; c < a.hidden; c += 128) {
      const float xh = (norm_s_at<T>(a, base + c) - mean) * rstd;
      const float dyv = to_f<T>(reinterpret_cast<const T*>(g.dy)[base + c]);
      const float wdy = dyv * load_dyn(a.weight, c, a.param_dtype);
      c1 = fmaf(wdy, xh, c1);
      c2 += wdy;
      atomicAdd(g.partial + c, dyv * xh);
      if (g.dbias) atomicAdd(g.partial + a.hidden + c, dyv);
    }
    c1 = block_allsum128(c1, scratch) * inv;
    c2 = a.is_rms ? 0.f : block_allsum128(c2, scratch) * inv;
    for (int c = threadIdx.x; c < a.hidden; c += 128) {
      const float xh = (norm_s_at<T>(a, base + c) - mean) * rstd;
      const float dyv = to_f<T>(reinterpret_cast<const T*>(g.dy)[base + c]);
      const float gro = g.dresidual_out ? load_dyn(g.dresidual_out, base + c, a.resout_dtype) : 0.f;
      const float ds = (dyv * load_dyn(a.weight, c, a.param_dtype) - xh * c1 - c2) * rstd + gro;
      reinterpret_cast<T*>(g.dx)[base + c] = from_f<T>(ds);
      if (g.dresidual) store_dyn(g.dresidual, base + c, a.res_dtype, a.prenorm ? ds : dyv + gro);
    }
  }
}

static int norm_validate(const ssm_norm_args* a) {
  SSM_REQUIRE(a != nullptr, SSM_ERR_NULL, "fused_layer_norm: args is NULL");
  SSM_REQUIRE(a->rows >= 0 && a->hidden >= 1, SSM_ERR_SHAPE, "fused_layer_norm: bad shape");
  SSM_REQUIRE(valid_dtype(a->io_dtype), SSM_ERR_DTYPE, "fused_layer_norm: unknown dtype");
  SSM_REQUIRE(!a->residual || valid_dtype(a->res_dtype), SSM_ERR_DTYPE, "fused_layer_norm: unknown residual dtype");
  SSM_REQUIRE(!a->residual_out || valid_dtype(a->resout_dtype), SSM_ERR_DTYPE, "fused_layer_norm: unknown residual_out dtype");
  SSM_REQUIRE(valid_dtype(a->param_dtype) && valid_dtype(a->dparam_dtype), SSM_ERR_DTYPE, "fused_layer_norm: unknown parameter dtype");
  SSM_REQUIRE(a->rows < (1ll << 31), SSM_ERR_TOO_LARGE, "fused_layer_norm: too many rows");
  return SSM_OK;
}

static bool norm_vec_ok(const ssm_norm_args& a, int maxchunks, const void* p1, const void* p2, const void* p3) {
  const int V = 16 / dtype_size(a.io_dtype);
  if (a.hidden % V != 0) return false;
  if (a.hidden > 512 * maxchunks * V) return false;
  auto ok = [](const void* p) { return p == nullptr || aligned_to(p, 16); };
  // residual / residual_out / dresidual rows of fp32 with hidden % V == 0 are 16-byte aligned too
  return ok(a.x) && ok(a.y) && ok(a.residual) && ok(a.residual_out) && ok(a.weight) && ok(a.bias) && ok(p1) && ok(p2) && ok(p3);
}

static int norm_bwd_ctas(const ssm_norm_args& a, int rpc) {
  const int64_t npass = (a.rows + rpc - 1) / rpc;
  return (int)(npass < kNormBwdMaxCtas ? npass : kNormBwdMaxCtas);
}

template <typename T, int G, int MC = kNormFwdChunks>
static int norm_fwd_launch(const ssm_norm_args& a, cudaStream_t st) {
  using Cfg = NormCfg<T, G>;
  const unsigned grid = (unsigned)((a.rows + Cfg::RPC - 1) / Cfg::RPC);
  return launch_overlapped("norm_fwd_kernel", a.residual ? norm_fwd_kernel<T, G, MC, true> : norm_fwd_kernel<T, G, MC, false>, dim3(grid), dim3(Cfg::BLOCK), 0, st, a);
}
static int norm_fold(const ssm_norm_bwd_args& g, int parts, cudaStream_t st) {
  return launch_overlapped("norm_fold_kernel", norm_fold_kernel, dim3((g.fwd.hidden + 31) / 32, g.dbias ? 2 : 1), dim3(32 * kFoldLanes), 0, st, g.partial, parts, g.fwd.hidden, g.dweight, g.dbias,
                           g.fwd.dparam_dtype);
}
constexpr size_t kNormRing = 200 * 1024;
template <typename T, int G, int MG, int FULL>
static int norm_bwd_launch(const ssm_norm_bwd_args& g, cudaStream_t st, int max_ctas) {
  using Cfg = NormCfg<T, G>;
  const ssm_norm_args& a = g.fwd;
  const int element = 2 * (int)sizeof(T) + (a.residual && a.prenorm ? dtype_bytes(a.res_dtype) : 0) + (g.dresidual_out ? dtype_bytes(a.resout_dtype) : 0);
  const size_t stage = (size_t)MG * 4 * Cfg::BLOCK * element, fold = Cfg::RPC > 1 ? (size_t)MG * Cfg::BLOCK * 32 : 0;
  const bool two = 2 * stage <= kNormRing;  // else (512 threads of the most granules) one row at a time
  const size_t smem = std::max(two ? 2 * stage : stage, fold);
  constexpr int ONE = G == 512 && MG * sizeof(T) == 16 ? 1 : 2;
  // the middle of a network: a residual stream of fp32, in and out
  const bool stream = a.prenorm && a.residual && g.dresidual && g.dresidual_out && a.res_dtype == SSM_F32 && a.resout_dtype == SSM_F32;
  auto kern = stream ? (two ? norm_bwd_kernel<T, G, MG, FULL, 2, true> : norm_bwd_kernel<T, G, MG, FULL, ONE, true>)
                     : (two ? norm_bwd_kernel<T, G, MG, FULL, 2, false> : norm_bwd_kernel<T, G, MG, FULL, ONE, false>);
  static_assert(ONE == 1 || 2 * MG * 4 * Cfg::BLOCK * (2 * sizeof(T) + 8) <= kNormRing, "two rows fit");
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  // persistent grid: exactly one resident wave (a second, partial wave would double the time)
  const int resident = std::min<int>(norm_bwd_ctas_per_sm<T, G, MG>(), (int)(228 * 1024 / (smem + 2048))) * sm_count();
  const int nctas = std::min(std::min(norm_bwd_ctas(a, Cfg::RPC), max_ctas), resident);
  if (int rc = launch_overlapped("norm_bwd_kernel", kern, dim3(nctas), dim3(Cfg::BLOCK), smem, st, g)) return rc;
  return norm_fold(g, nctas, st);
}

// As few granules of four columns per thread as the row needs: what a thread does not hold leaves room for more rows in flight
// (2560 columns of 16 bits: five, three CTAs per SM), and the number of them that all threads have (FULL) is known.  A warp owns a row while its lanes can hold it.
template <typename T>
static int norm_bwd_dispatch(const ssm_norm_bwd_args& g, cudaStream_t st, int max_ctas) {
  const int n = g.fwd.hidden / 4;
  if (n <= 32) return norm_bwd_launch<T, 32, 1, 0>(g, st, max_ctas);
  if (n <= 64) return norm_bwd_launch<T, 32, 2, 1>(g, st, max_ctas);
  if (n <= 96) return norm_bwd_launch<T, 32, 3, 2>(g, st, max_ctas);
  if (n <= 128) return norm_bwd_launch<T, 32, 4, 3>(g, st, max_ctas);
  if constexpr (sizeof(T) == 4) {
    if (n <= 256) return norm_bwd_launch<T, 128, 2, 1>(g, st, max_ctas);
    if (n <= 384) return norm_bwd_launch<T, 128, 3, 2>(g, st, max_ctas);
    if (n <= 512) return norm_bwd_launch<T, 128, 4, 3>(g, st, max_ctas);
    if (n <= 1024) return norm_bwd_launch<T, 512, 2, 1>(g, st, max_ctas);
    return norm_bwd_launch<T, 512, 4, 2>(g, st, max_ctas);
  } else {
    if (n <= 192) return norm_bwd_launch<T, 64, 3, 2>(g, st, max_ctas);
    if (n <= 256) return norm_bwd_launch<T, 64, 4, 3>(g, st, max_ctas);
    if (n <= 384) return norm_bwd_launch<T, 128, 3, 2>(g, st, max_ctas);
    if (n <= 512) return norm_bwd_launch<T, 128, 4, 3>(g, st, max_ctas);
    if (n <= 640) return norm_bwd_launch<T, 128, 5, 4>(g, st, max_ctas);
    if (n <= 768) return norm_bwd_launch<T, 128, 6, 5>(g, st, max_ctas);
    if (n <= 1024) return norm_bwd_launch<T, 256, 4, 3>(g, st, max_ctas);
    if (n <= 2048) return norm_bwd_launch<T, 512, 4, 2>(g, st, max_ctas);
    return norm_bwd_launch<T, 512, 8, 4>(g, st, max_ctas);
  }
}

template <typename T>
static int norm_fwd_t(const ssm_norm_args& a, cudaStream_t st) {
  if (!norm_vec_ok(a, kNormFwdChunks, nullptr, nullptr, nullptr)) {
    ssm_norm_bwd_args g{};
    g.fwd = a;
    norm_scalar_kernel<T, false><<<(unsigned)a.rows, 128, 0, st>>>(g);
    return launch_status("norm_scalar_kernel");
  }
  const int nchunk = a.hidden / (16 / (int)sizeof(T));
  // as few chunks per thread as the row needs: what a thread does not hold leaves room for more rows in flight
  if (nchunk <= 32) return norm_fwd_launch<T, 32, 1>(a, st);
  if (nchunk <= 64) return norm_fwd_launch<T, 32, 2>(a, st);
  if (nchunk <= 96) return norm_fwd_launch<T, 32, 3>(a, st);
  if (nchunk <= 128) return norm_fwd_launch<T, 32, 4>(a, st);
  if (nchunk <= 256) return norm_fwd_launch<T, 128, 2>(a, st);
  if (nchunk <= 384) return norm_fwd_launch<T, 128, 3>(a, st);
  if (nchunk <= 512) return norm_fwd_launch<T, 128, 4>(a, st);
  if (nchunk <= 768) return norm_fwd_launch<T, 128, 6>(a, st);
  return norm_fwd_launch<T, 512>(a, st);
}
// rows that cannot be vectorised: sums by atomics into one partial row, folded into the element type of the gradients
template <typename T>
static int norm_bwd_scalar(const ssm_norm_bwd_args& g, cudaStream_t st) {
  const int hidden = g.fwd.hidden;
  cudaMemsetAsync(g.partial, 0, sizeof(float) * 2 * hidden, st);
  norm_scalar_kernel<T, true><<<(unsigned)g.fwd.rows, 128, 0, st>>>(g);
  if (int rc = launch_status("norm_scalar_kernel")) return rc;
  return norm_fold(g, 1, st);
}
template <typename T>
static int norm_bwd_t(const ssm_norm_bwd_args& g, cudaStream_t st) {
  const ssm_norm_args& a = g.fwd;
  if (!norm_vec_ok(a, kNormBwdChunks, g.dy, g.dx, g.dresidual) || !aligned_to(g.dresidual_out, 16)) {
    return norm_bwd_scalar<T>(g, st);
  }
  return norm_bwd_dispatch<T>(g, st, kNormBwdMaxCtas);
}


// ---------------------------------------------------------------------------------------
// Backward variant for callers that must not allocate device memory.
//
// The persistent backward kernel needs a scratch area for its per-CTA partial weight / bias
// gradients.  Here that area is a fixed array that lives in the library's device image, so
// the call performs no cudaMalloc / cudaFree and asks no allocator for anything.  The price
// is a fixed capacity (hidden <= kNoAllocMaxHidden, at most kNoAllocCtas partial rows) and
// 9.25 MiB of device memory held on every GPU that loads the library until the process ends.
// ---------------------------------------------------------------------------------------
constexpr int kNoAllocMaxHidden = 8192;
constexpr int kNoAllocCtas = 148;  // one partial row per SM
constexpr size_t kNoAllocFloats = (size_t)2 * kNoAllocMaxHidden * kNoAllocCtas;
static __device__ __align__(256) float g_norm_noalloc_scratch[kNoAllocFloats];

constexpr int kNoAllocMaxDevices = 64;
static float* g_noalloc_addr[kNoAllocMaxDevices];  // device address of the array, per device; set once
static std::mutex g_noalloc_mutex;

// In host code the array's name is only a handle: the address a kernel can use has to be
// asked for, per device, with that device current.
static int noalloc_scratch_address(float** out) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) {
    set_error("fused_layer_norm_backward_noalloc: cudaGetDevice: %s", cudaGetErrorString(e));
    return (int)e;
  }
  if (dev < 0 || dev >= kNoAllocMaxDevices) return fail(SSM_ERR_UNSUPPORTED, "fused_layer_norm_backward_noalloc: device index out of range");
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  if (g_noalloc_addr[dev] == nullptr) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_norm_noalloc_scratch);
    if (e != cudaSuccess || p == nullptr) {
      set_error("fused_layer_norm_backward_noalloc: cudaGetSymbolAddress: %s", cudaGetErrorString(e));
      return e != cudaSuccess ? (int)e : SSM_ERR_DEVICE;
    }
    g_noalloc_addr[dev] = static_cast<float*>(p);
  }
  *out = g_noalloc_addr[dev];
  return SSM_OK;
}

template <typename T>
static int norm_bwd_noalloc_t(const ssm_norm_bwd_args& g, float* scratch, cudaStream_t st) {
  const ssm_norm_args& a = g.fwd;
  ssm_norm_bwd_args h = g;
  h.partial = scratch;
  if (!norm_vec_ok(a, kNormBwdChunks, g.dy, g.dx, g.dresidual) || !aligned_to(g.dresidual_out, 16)) {
    return norm_bwd_scalar<T>(h, st);
  }
  return norm_bwd_dispatch<T>(h, st, kNoAllocCtas);
}

}  // namespace ssmb

using namespace ssmb;

extern "C" int ssm_fused_add_norm_fwd(const ssm_norm_args* a, ssm_stream_t stream) {
  if (a && a->io_dtype == SSM_F64) {
    ssm_norm_bwd_args g{};
    g.fwd = *a;
    return f64_norm(g, false, reinterpret_cast<cudaStream_t>(stream));
  }
  if (int rc = norm_validate(a)) return rc;
  if (a->rows == 0) return SSM_OK;
  SSM_REQUIRE(a->x && a->y && a->weight, SSM_ERR_NULL, "fused_layer_norm: x, weight and y are required");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  switch (a->io_dtype) {
    case SSM_F32: return norm_fwd_t<float>(*a, st);
    case SSM_BF16: return norm_fwd_t<__nv_bfloat16>(*a, st);
    default: return norm_fwd_t<__half>(*a, st);
  }
}

extern "C" int64_t ssm_norm_bwd_scratch_floats(int64_t rows, int32_t hidden) {
  (void)rows;
  return (int64_t)2 * hidden * kNormBwdMaxCtas;
}

extern "C" int ssm_fused_add_norm_bwd(const ssm_norm_bwd_args* g, ssm_stream_t stream) {
  SSM_REQUIRE(g != nullptr, SSM_ERR_NULL, "fused_layer_norm_backward: args is NULL");
  const ssm_norm_args* a = &g->fwd;
  if (a->io_dtype == SSM_F64) return f64_norm(*g, true, reinterpret_cast<cudaStream_t>(stream));
  if (int rc = norm_validate(a)) return rc;
  SSM_REQUIRE(g->dweight, SSM_ERR_NULL, "fused_layer_norm_backward: dweight is required");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (a->rows == 0) {
    cudaMemsetAsync(g->dweight, 0, (size_t)dtype_size(a->dparam_dtype) * a->hidden, st);
    if (g->dbias) cudaMemsetAsync(g->dbias, 0, (size_t)dtype_size(a->dparam_dtype) * a->hidden, st);
    return SSM_OK;
  }
  SSM_REQUIRE(a->x && a->weight && g->dy && g->dx && g->partial, SSM_ERR_NULL, "fused_layer_norm_backward: missing pointer");
  SSM_REQUIRE(!a->residual == !g->dresidual || !g->dresidual, SSM_ERR_NULL, "fused_layer_norm_backward: dresidual without residual");
  SSM_REQUIRE(!g->dresidual_out || valid_dtype(a->resout_dtype), SSM_ERR_DTYPE, "fused_layer_norm_backward: dresidual_out needs resout_dtype");
  switch (a->io_dtype) {
    case SSM_F32: return norm_bwd_t<float>(*g, st);
    case SSM_BF16: return norm_bwd_t<__nv_bfloat16>(*g, st);
    default: return norm_bwd_t<__half>(*g, st);
  }
}

extern "C" int ssm_fused_add_norm_bwd_noalloc(const ssm_norm_bwd_args* g, ssm_stream_t stream) {
  SSM_REQUIRE(g != nullptr, SSM_ERR_NULL, "fused_layer_norm_backward_noalloc: args is NULL");
  const ssm_norm_args* a = &g->fwd;
  if (int rc = norm_validate(a)) return rc;
  SSM_REQUIRE(a->hidden <= kNoAllocMaxHidden, SSM_ERR_TOO_LARGE,
              "fused_layer_norm_backward_noalloc: hidden exceeds the built-in scratch capacity (8192); use ssm_fused_add_norm_bwd");
  SSM_REQUIRE(g->dweight, SSM_ERR_NULL, "fused_layer_norm_backward_noalloc: dweight is required");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (a->rows == 0) {
    cudaMemsetAsync(g->dweight, 0, (size_t)dtype_size(a->dparam_dtype) * a->hidden, st);
    if (g->dbias) cudaMemsetAsync(g->dbias, 0, (size_t)dtype_size(a->dparam_dtype) * a->hidden, st);
    return SSM_OK;
  }
  SSM_REQUIRE(a->x && a->weight && g->dy && g->dx, SSM_ERR_NULL, "fused_layer_norm_backward_noalloc: missing pointer");
  SSM_REQUIRE(a->residual || !g->dresidual, SSM_ERR_NULL, "fused_layer_norm_backward_noalloc: dresidual without residual");
  SSM_REQUIRE(!g->dresidual_out || valid_dtype(a->resout_dtype), SSM_ERR_DTYPE, "fused_layer_norm_backward_noalloc: dresidual_out needs resout_dtype");
  {
    // the built-in scratch is looked up for the CURRENT device; tensors that live on another one would be paired with the wrong GPU's array
    int cur = -1;
    cudaPointerAttributes attr{};
    if (cudaGetDevice(&cur) == cudaSuccess && cudaPointerGetAttributes(&attr, g->dy) == cudaSuccess && attr.type == cudaMemoryTypeDevice)
      SSM_REQUIRE(attr.device == cur, SSM_ERR_DEVICE, "fused_layer_norm_backward_noalloc: the tensors are not on the current device");
    else
      (void)cudaGetLastError();
  }
  float* scratch = nullptr;
  if (int rc = noalloc_scratch_address(&scratch)) return rc;
  switch (a->io_dtype) {
    case SSM_F32: return norm_bwd_noalloc_t<float>(*g, scratch, st);
    case SSM_BF16: return norm_bwd_noalloc_t<__nv_bfloat16>(*g, scratch, st);
    default: return norm_bwd_noalloc_t<__half>(*g, scratch, st);
  }
}
