// Single-token selective state step (decode), forward and backward, sm_100a.
//
// HBM-bound on the fp32 state: it is read once and written once per step, as float4, by a
// group of LPR lanes per (batch, channel) row that covers the row's states; everything
// else (softplus, dt bias, grouped B / C lookup, D skip, SiLU gate) is folded into the same
// pass.  No host synchronisation and no allocation.
#include "common.cuh"

namespace ssmb {

constexpr int kStepThreads = 128;

// A as stored, or from log(-A): a decode step then needs no pass of its own to form it
__device__ __forceinline__ float step_A(const ssm_step_args& a, float v) { return a.a_log ? -expf(v) : v; }

template <typename T, int LPR>
__global__ void __launch_bounds__(kStepThreads) step_fwd_kernel(const ssm_step_args a, int vec) {
  const int64_t gid = (int64_t)blockIdx.x * kStepThreads + threadIdx.x;
  const int64_t rows = (int64_t)a.batch * a.dim;
  const int64_t row_raw = gid / LPR;
  const bool live = row_raw < rows;
  const int64_t row = live ? row_raw : rows - 1;
  const int sg = (int)(gid % LPR);
  const int b = (int)(row / a.dim), d = (int)(row % a.dim);
  const int N = a.nstate;
  const int head = a.param_heads > 0 ? d / (a.dim / a.param_heads) : d;
  const int64_t prow = a.param_heads > 0 ? (int64_t)b * a.param_heads + head : row;

  const float x = to_f<T>(reinterpret_cast<const T*>(a.x)[row]);
  float dt = to_f<T>(reinterpret_cast<const T*>(a.dt)[prow]);
  if (a.dt_bias) dt += __ldg(a.dt_bias + head);
  if (a.dt_softplus) dt = softplus_f(dt);
  const float dtx = dt * x;
  const int g = d / (a.dim / a.bc_groups);
  const int64_t boff = (int64_t)b * a.b_sb + (int64_t)g * a.b_sg;
  const int64_t coff = (int64_t)b * a.c_sb + (int64_t)g * a.c_sg;
  float* st = a.state + row * N;
  float y = 0.f;
  if (vec) {
    for (int n0 = sg * 4; n0 < N; n0 += LPR * 4) {
      float4 s = *reinterpret_cast<const float4*>(st + n0);
      float sv[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int n = n0 + i;
        const float An = step_A(a, a.param_heads > 0 ? __ldg(a.A + head) : __ldg(a.A + (int64_t)d * N + n));
        const float Bn = load_dyn(a.Bm, boff + (int64_t)n * a.b_sn, a.bc_dtype);
        const float Cn = load_dyn(a.Cm, coff + (int64_t)n * a.c_sn, a.bc_dtype);
        sv[i] = fmaf(ex2_approx(dt * An * kLog2e), sv[i], dtx * Bn);
        y = fmaf(Cn, sv[i], y);
      }
      if (live) *reinterpret_cast<float4*>(st + n0) = make_float4(sv[0], sv[1], sv[2], sv[3]);
    }
  } else {
    for (int n = sg; n < N; n += LPR) {
      const float An = step_A(a, a.param_heads > 0 ? __ldg(a.A + head) : __ldg(a.A + (int64_t)d * N + n));
      const float Bn = load_dyn(a.Bm, boff + (int64_t)n * a.b_sn, a.bc_dtype);
      const float Cn = load_dyn(a.Cm, coff + (int64_t)n * a.c_sn, a.bc_dtype);
      const float s = fmaf(ex2_approx(dt * An * kLog2e), st[n], dtx * Bn);
      if (live) st[n] = s;
      y = fmaf(Cn, s, y);
    }
  }
  y = group_sum<LPR, 1>(y);
  if (sg == 0 && live) {
    if (a.D) y = fmaf(__ldg(a.D + head), x, y);
    if (a.z) y *= silu_fast(to_f<T>(reinterpret_cast<const T*>(a.z)[row]));
    reinterpret_cast<T*>(a.out)[row] = from_f<T>(y);
  }
}

// Fast path: every lane owns NV float4 groups of its row's state, all loaded before any is used so
// that each thread keeps NV * 16 bytes of the dominant stream in flight; the LPR lanes of a row
// read adjacent groups.  Needs nstate == 4 * NV * LPR.
template <typename T, int NV, int LPR>
__global__ void __launch_bounds__(kStepThreads) step_fwd_vec_kernel(const ssm_step_args a) {
  const int64_t gid = (int64_t)blockIdx.x * kStepThreads + threadIdx.x;
  const int64_t rows = (int64_t)a.batch * a.dim;
  const int64_t row_raw = gid / LPR;
  const bool live = row_raw < rows;
  const int64_t row = live ? row_raw : rows - 1;
  const int sg = (int)(gid % LPR);
  const int b = (int)(row / a.dim), d = (int)(row % a.dim);
  constexpr int N = 4 * NV * LPR;
  const int head = a.param_heads > 0 ? d / (a.dim / a.param_heads) : d;
  const int64_t prow = a.param_heads > 0 ? (int64_t)b * a.param_heads + head : row;
  float* st = a.state + row * N;
  float4 s[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) s[v] = *reinterpret_cast<const float4*>(st + (sg + v * LPR) * 4);
  const float x = to_f<T>(reinterpret_cast<const T*>(a.x)[row]);
  float dt = to_f<T>(reinterpret_cast<const T*>(a.dt)[prow]);
  if (a.dt_bias) dt += __ldg(a.dt_bias + head);
  if (a.dt_softplus) dt = softplus_fast(dt);
  const float dtx = dt * x;
  const int g = d / (a.dim / a.bc_groups);
  const int64_t boff = (int64_t)b * a.b_sb + (int64_t)g * a.b_sg;
  const int64_t coff = (int64_t)b * a.c_sb + (int64_t)g * a.c_sg;
  const float Ahead = a.param_heads > 0 ? step_A(a, __ldg(a.A + head)) * kLog2e : 0.f;
  float y = 0.f;
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int n0 = (sg + v * LPR) * 4;
    float An[4];
    if (a.param_heads > 0) {
      An[0] = An[1] = An[2] = An[3] = Ahead;
    } else {
      const float4 q = __ldg(reinterpret_cast<const float4*>(a.A + (int64_t)d * N + n0));
      An[0] = step_A(a, q.x) * kLog2e, An[1] = step_A(a, q.y) * kLog2e, An[2] = step_A(a, q.z) * kLog2e, An[3] = step_A(a, q.w) * kLog2e;
    }
    float sv[4] = {s[v].x, s[v].y, s[v].z, s[v].w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float Bn = load_dyn(a.Bm, boff + (int64_t)(n0 + i) * a.b_sn, a.bc_dtype);
      const float Cn = load_dyn(a.Cm, coff + (int64_t)(n0 + i) * a.c_sn, a.bc_dtype);
      sv[i] = fmaf(ex2_approx(dt * An[i]), sv[i], dtx * Bn);
      y = fmaf(Cn, sv[i], y);
    }
    if (live) *reinterpret_cast<float4*>(st + n0) = make_float4(sv[0], sv[1], sv[2], sv[3]);
  }
  y = group_sum<LPR, 1>(y);
  if (sg == 0 && live) {
    if (a.D) y = fmaf(__ldg(a.D + head), x, y);
    if (a.z) y *= silu_fast(to_f<T>(reinterpret_cast<const T*>(a.z)[row]));
    reinterpret_cast<T*>(a.out)[row] = from_f<T>(y);
  }
}

// Four consecutive B or C values of compile-time element type BT as fp32 (one 8- or 16-byte load).
template <typename BT>
__device__ __forceinline__ void load_bc4(const void* base, int64_t off, float (&v)[4]) {
  if constexpr (sizeof(BT) == 4) {
    const float4 q = __ldg(reinterpret_cast<const float4*>(reinterpret_cast<const float*>(base) + off));
    v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
  } else {
    const uint2 raw = __ldg(reinterpret_cast<const uint2*>(reinterpret_cast<const BT*>(base) + off));
    const BT* e = reinterpret_cast<const BT*>(&raw);
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = to_f<BT>(e[i]);
  }
}

// The same fast path with B / C rows read as vectors: unit state stride, every (batch, group) row of B and C aligned to the
// vector, element type BT known at compile time.  This is the layout decoding uses (B, C of shape (batch, groups, nstate));
// it replaces 2 x nstate scalar loads with run-time type dispatch per thread by 2 x nstate / 4 vector loads.
template <typename T, typename BT, int NV, int LPR>
__global__ void __launch_bounds__(kStepThreads) step_fwd_fast_kernel(const ssm_step_args a) {
  pdl_wait();
  pdl_trigger();
  const int64_t gid = (int64_t)blockIdx.x * kStepThreads + threadIdx.x;
  const int64_t rows = (int64_t)a.batch * a.dim;
  const int64_t row_raw = gid / LPR;
  const bool live = row_raw < rows;
  const int64_t row = live ? row_raw : rows - 1;
  const int sg = (int)(gid % LPR);
  const int b = (int)(row / a.dim), d = (int)(row % a.dim);
  constexpr int N = 4 * NV * LPR;
  const int head = a.param_heads > 0 ? d / (a.dim / a.param_heads) : d;
  const int64_t prow = a.param_heads > 0 ? (int64_t)b * a.param_heads + head : row;
  float* st = a.state + row * N;
  float4 s[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) s[v] = __ldcs(reinterpret_cast<const float4*>(st + (sg + v * LPR) * 4));
  const int g = d / (a.dim / a.bc_groups);
  const int64_t boff = (int64_t)b * a.b_sb + (int64_t)g * a.b_sg;
  const int64_t coff = (int64_t)b * a.c_sb + (int64_t)g * a.c_sg;
  float Bv[NV][4], Cv[NV][4], An[NV][4];
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int n0 = (sg + v * LPR) * 4;
    load_bc4<BT>(a.Bm, boff + n0, Bv[v]);
    load_bc4<BT>(a.Cm, coff + n0, Cv[v]);
    if (a.param_heads == 0) {
      const float4 q = __ldg(reinterpret_cast<const float4*>(a.A + (int64_t)d * N + n0));
      An[v][0] = step_A(a, q.x) * kLog2e, An[v][1] = step_A(a, q.y) * kLog2e, An[v][2] = step_A(a, q.z) * kLog2e, An[v][3] = step_A(a, q.w) * kLog2e;
    }
  }
  const float x = to_f<T>(reinterpret_cast<const T*>(a.x)[row]);
  float dt = to_f<T>(reinterpret_cast<const T*>(a.dt)[prow]);
  if (a.dt_bias) dt += __ldg(a.dt_bias + head);
  if (a.dt_softplus) dt = softplus_fast(dt);
  const float dtx = dt * x;
  float y = 0.f;
  if (a.param_heads > 0) {  // one decay for the whole head: a single ex2 per thread
    const float da = ex2_approx(dt * step_A(a, __ldg(a.A + head)) * kLog2e);
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      float sv[4] = {s[v].x, s[v].y, s[v].z, s[v].w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        sv[i] = fmaf(da, sv[i], dtx * Bv[v][i]);
        y = fmaf(Cv[v][i], sv[i], y);
      }
      if (live) __stcs(reinterpret_cast<float4*>(st + (sg + v * LPR) * 4), make_float4(sv[0], sv[1], sv[2], sv[3]));
    }
  } else {
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      float sv[4] = {s[v].x, s[v].y, s[v].z, s[v].w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        sv[i] = fmaf(ex2_approx(dt * An[v][i]), sv[i], dtx * Bv[v][i]);
        y = fmaf(Cv[v][i], sv[i], y);
      }
      if (live) __stcs(reinterpret_cast<float4*>(st + (sg + v * LPR) * 4), make_float4(sv[0], sv[1], sv[2], sv[3]));
    }
  }
  y = group_sum<LPR, 1>(y);
  if (sg == 0 && live) {
    if (a.D) y = fmaf(__ldg(a.D + head), x, y);
    if (a.z) y *= silu_fast(to_f<T>(reinterpret_cast<const T*>(a.z)[row]));
    reinterpret_cast<T*>(a.out)[row] = from_f<T>(y);
  }
}

// The same step for states that fill the GPU several times over: persistent warps, each with three 2 KB pieces of the state in
// flight (cp.async; a piece is 512 floats = 512 / N rows).  The copies and the write-back run over a piece in memory order, whole
// 128-byte lines per instruction whatever N is; the rows are picked out of shared memory.  The row-per-thread kernel above is
// bound by what its short-lived threads keep in flight (64 bytes each, only until they use it) and, at N = 16, reads half
// sectors.  (batch, heads x headdim, N) = (256, 80 x 64, 128), 1342 MB: 274 us with that kernel.
constexpr int kStreamThreads = 256, kStreamStages = 3, kStreamCtasPerSm = 3;
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
}
template <typename T, typename BT, int N, bool HEADS>
__global__ void __launch_bounds__(kStreamThreads, kStreamCtasPerSm) step_stream_kernel(const ssm_step_args a) {
  constexpr int kPiece = 512, RPW = kPiece / N, LPR = N / 16;
  __shared__ __align__(16) float buf[kStreamStages][kStreamThreads / 32][kPiece];
  pdl_wait();
  pdl_trigger();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rows = a.batch * a.dim;
  const int pieces = (rows + RPW - 1) / RPW, stride = gridDim.x * (kStreamThreads / 32);
  const int64_t total = (int64_t)rows * N;
  const int r = lane / LPR, sg = lane % LPR, rot = N == 16 ? r >> 1 : r;
  auto issue = [&](int piece, int st) {
    if (piece < pieces) {
      const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&buf[st][warp][lane * 4]);
      const int64_t at = (int64_t)piece * kPiece + lane * 4;
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (at + i * 128 < total) cp_async16(dst + i * 512, a.state + at + i * 128);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  int piece = blockIdx.x * (kStreamThreads / 32) + warp;
  issue(piece, 0);
  issue(piece + stride, 1);
  int st = 0;
  for (; piece < pieces; piece += stride) {
    __syncwarp();  // every lane has read the piece before last, whose buffer is refilled now
    issue(piece + 2 * stride, st >= 1 ? st - 1 : 2);
    const int row_raw = piece * RPW + r;
    const bool live = row_raw < rows;
    const int row = live ? row_raw : rows - 1;
    const int b = row / a.dim, d = row % a.dim;
    const int head = HEADS ? d / (a.dim / a.param_heads) : d;
    const float x = to_f<T>(reinterpret_cast<const T*>(a.x)[row]);
    float dt = to_f<T>(reinterpret_cast<const T*>(a.dt)[HEADS ? (int64_t)b * a.param_heads + head : row]);
    const float bias = a.dt_bias ? __ldg(a.dt_bias + head) : 0.f, Dv = a.D ? __ldg(a.D + head) : 0.f;
    const float zv = a.z ? to_f<T>(reinterpret_cast<const T*>(a.z)[row]) : 0.f;
    const float Ah = HEADS ? step_A(a, __ldg(a.A + head)) : 0.f;
    const int g = d / (a.dim / a.bc_groups);
    const int64_t boff = (int64_t)b * a.b_sb + (int64_t)g * a.b_sg, coff = (int64_t)b * a.c_sb + (int64_t)g * a.c_sg;
    float Bv[4][4], Cv[4][4];
    float4 Av[4];
    int at[4];
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      at[v] = (sg + LPR * ((v + rot) & 3)) * 4;  // rotated so that eight neighbouring lanes read 128 different bytes
      load_bc4<BT>(a.Bm, boff + at[v], Bv[v]);
      load_bc4<BT>(a.Cm, coff + at[v], Cv[v]);
      if (!HEADS) Av[v] = __ldg(reinterpret_cast<const float4*>(a.A + (int64_t)d * N + at[v]));
    }
    dt += bias;
    if (a.dt_softplus) dt = softplus_fast(dt);
    const float dtx = dt * x, dah = HEADS ? ex2_approx(dt * Ah * kLog2e) : 0.f;
    asm volatile("cp.async.wait_group 2;\n" ::: "memory");
    __syncwarp();
    float* mine = &buf[st][warp][r * N];
    float y = 0.f;
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const float4 s4 = *reinterpret_cast<const float4*>(mine + at[v]);
      float sv[4] = {s4.x, s4.y, s4.z, s4.w};
      const float An[4] = {Av[v].x, Av[v].y, Av[v].z, Av[v].w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float da = HEADS ? dah : ex2_approx(dt * (step_A(a, An[i]) * kLog2e));
        sv[i] = fmaf(da, sv[i], dtx * Bv[v][i]);
        y = fmaf(Cv[v][i], sv[i], y);
      }
      *reinterpret_cast<float4*>(mine + at[v]) = make_float4(sv[0], sv[1], sv[2], sv[3]);
    }
    __syncwarp();
    const int64_t out_at = (int64_t)piece * kPiece + lane * 4;
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (out_at + i * 128 < total) __stcs(reinterpret_cast<float4*>(a.state + out_at + i * 128), *reinterpret_cast<const float4*>(&buf[st][warp][lane * 4 + i * 128]));
    y = group_sum<LPR, 1>(y);
    if (sg == 0 && live) {
      y = fmaf(Dv, x, y);
      if (a.z) y *= silu_fast(zv);
      reinterpret_cast<T*>(a.out)[row] = from_f<T>(y);
    }
    st = st == 2 ? 0 : st + 1;
  }
}

// Four consecutive 16-bit B or C values as raw words, and as two pairs of fp32
template <typename BT>
struct Bc4 {
  uint2 raw;
  __device__ __forceinline__ void load(const void* base, int64_t off) { raw = __ldg(reinterpret_cast<const uint2*>(reinterpret_cast<const BT*>(base) + off)); }
  __device__ __forceinline__ float2 pair(int i) const {
    const uint32_t w = i ? raw.y : raw.x;
    if constexpr (std::is_same<BT, __nv_bfloat16>::value) return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
    else return __half22float2(*reinterpret_cast<const __half2*>(&w));
  }
};

// step_stream_kernel for parameters per channel and 16-bit operands: a warp keeps its 512 / N channels and walks over sequences, so that A (and
// its exponential, where log(-A) is given), D and the bias are formed once and no index is divided.  bf16, us of steps back to back against
// the kernel above: (256, 5120) x 16 26.1 and 28.9, (128, 5120) x 16 12.4 and 14.5, (256, 1024) x 64 19.8 and 22.9, (1024, 5120) x 16 116 and
// 120.  With fp32 operands it was the slower one: (256, 5120) x 16 36.6 and 30.2, (256, 512) x 128 26.0 and 22.3.
template <typename T, typename BT, int N>
__global__ void __launch_bounds__(kStreamThreads, kStreamCtasPerSm) step_channels_kernel(const ssm_step_args a) {
  constexpr int kPiece = 512, RPW = kPiece / N, LPR = N / 16;
  __shared__ __align__(16) float buf[kStreamStages][kStreamThreads / 32][kPiece];
  pdl_wait();
  pdl_trigger();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int per_seq = a.dim / RPW;  // pieces of a sequence
  const int w = blockIdx.x * (kStreamThreads / 32) + warp, warps = gridDim.x * (kStreamThreads / 32);
  const int slices = max(1, min(a.batch, warps / per_seq));  // warps that share the sequences of a piece's channels
  const int r = lane / LPR, sg = lane % LPR, rot = N == 16 ? r >> 1 : r;
  int at[4];
#pragma unroll
  for (int v = 0; v < 4; ++v) at[v] = (sg + LPR * ((v + rot) & 3)) * 4;  // rotated so that eight neighbouring lanes read 128 different bytes
  for (int item = w; item < per_seq * slices; item += warps) {
    const int pg = item % per_seq, slice = item / per_seq;
    const int b_begin = (int)((int64_t)a.batch * slice / slices), b_end = (int)((int64_t)a.batch * (slice + 1) / slices);
    const int d = pg * RPW + r, g = d / (a.dim / a.bc_groups);
    float2 A2[4][2];
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const float4 q = __ldg(reinterpret_cast<const float4*>(a.A + (int64_t)d * N + at[v]));
      A2[v][0] = make_float2(step_A(a, q.x) * kLog2e, step_A(a, q.y) * kLog2e), A2[v][1] = make_float2(step_A(a, q.z) * kLog2e, step_A(a, q.w) * kLog2e);
    }
    const float bias = a.dt_bias ? __ldg(a.dt_bias + d) : 0.f, Dv = a.D ? __ldg(a.D + d) : 0.f;
    float* state = a.state + (int64_t)pg * kPiece + lane * 4;  // of sequence 0
    const int64_t seq = (int64_t)a.dim * N;
    auto issue = [&](int b, int st) {
      if (b < b_end) {
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&buf[st][warp][lane * 4]);
        const float* src = state + b * seq;
#pragma unroll
        for (int i = 0; i < 4; ++i) cp_async16(dst + i * 512, src + i * 128);
      }
      asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    const T* px = reinterpret_cast<const T*>(a.x) + (int64_t)b_begin * a.dim + d;
    const T* pdt = reinterpret_cast<const T*>(a.dt) + (int64_t)b_begin * a.dim + d;
    const T* pz = a.z ? reinterpret_cast<const T*>(a.z) + (int64_t)b_begin * a.dim + d : nullptr;
    T* po = reinterpret_cast<T*>(a.out) + (int64_t)b_begin * a.dim + d;
    int64_t boff = (int64_t)b_begin * a.b_sb + (int64_t)g * a.b_sg, coff = (int64_t)b_begin * a.c_sb + (int64_t)g * a.c_sg;
    issue(b_begin, 0);
    issue(b_begin + 1, 1);
    int st = 0;
    for (int b = b_begin; b < b_end; ++b) {
      __syncwarp();  // every lane has read the piece before last, whose buffer is refilled now
      issue(b + 2, st >= 1 ? st - 1 : 2);
      const float x = to_f<T>(*px);
      float dt = to_f<T>(*pdt) + bias;
      const float zv = pz ? to_f<T>(*pz) : 0.f;
      Bc4<BT> B[4], C[4];
#pragma unroll
      for (int v = 0; v < 4; ++v) B[v].load(a.Bm, boff + at[v]), C[v].load(a.Cm, coff + at[v]);
      if (a.dt_softplus) dt = softplus_fast(dt);
      const float2 dt2 = make_float2(dt, dt), dtx = make_float2(dt * x, dt * x);
      asm volatile("cp.async.wait_group 2;\n" ::: "memory");
      __syncwarp();
      float* mine = &buf[st][warp][r * N];
      float2 y2 = make_float2(0.f, 0.f);
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        const float4 s4 = *reinterpret_cast<const float4*>(mine + at[v]);
        float2 sv[2] = {make_float2(s4.x, s4.y), make_float2(s4.z, s4.w)};
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float2 e = __fmul2_rn(dt2, A2[v][i]);
          sv[i] = __ffma2_rn(make_float2(ex2_approx(e.x), ex2_approx(e.y)), sv[i], __fmul2_rn(dtx, B[v].pair(i)));
          y2 = __ffma2_rn(C[v].pair(i), sv[i], y2);
        }
        *reinterpret_cast<float4*>(mine + at[v]) = make_float4(sv[0].x, sv[0].y, sv[1].x, sv[1].y);
      }
      __syncwarp();
      float* to = state + b * seq;
#pragma unroll
      for (int i = 0; i < 4; ++i) __stcs(reinterpret_cast<float4*>(to + i * 128), *reinterpret_cast<const float4*>(&buf[st][warp][lane * 4 + i * 128]));
      float y = group_sum<LPR, 1>(y2.x + y2.y);
      if (sg == 0) {
        y = fmaf(Dv, x, y);
        if (pz) y *= silu_fast(zv);
        *po = from_f<T>(y);
      }
      px += a.dim, pdt += a.dim, po += a.dim, boff += a.b_sb, coff += a.c_sb;
      if (pz) pz += a.dim;
      st = st == 2 ? 0 : st + 1;
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncwarp();
  }
}

// Backward of the plain step.  One group of LPR lanes per row, parameter gradients by atomics.
template <typename T, int LPR>
__global__ void __launch_bounds__(kStepThreads) step_bwd_kernel(const ssm_step_bwd_args g) {
  const ssm_step_args& a = g.fwd;
  const int64_t gid = (int64_t)blockIdx.x * kStepThreads + threadIdx.x;
  const int64_t rows = (int64_t)a.batch * a.dim;
  const int64_t row_raw = gid / LPR;
  const bool live = row_raw < rows;
  const int64_t row = live ? row_raw : rows - 1;
  const int sg = (int)(gid % LPR);
  const int b = (int)(row / a.dim), d = (int)(row % a.dim);
  const int N = a.nstate;
  const float x = to_f<T>(reinterpret_cast<const T*>(a.x)[row]);
  float pre = to_f<T>(reinterpret_cast<const T*>(a.dt)[row]);
  if (a.dt_bias) pre += __ldg(a.dt_bias + d);
  const float dt = a.dt_softplus ? softplus_f(pre) : pre;
  const float zv = a.z ? to_f<T>(reinterpret_cast<const T*>(a.z)[row]) : 0.f;
  const float gate = a.z ? silu_f(zv) : 1.f;
  const float dout = to_f<T>(reinterpret_cast<const T*>(g.dout)[row]);
  const float dy = dout * gate;
  const int grp = d / (a.dim / a.bc_groups);
  const int64_t boff = (int64_t)b * a.b_sb + (int64_t)grp * a.b_sg;
  const int64_t coff = (int64_t)b * a.c_sb + (int64_t)grp * a.c_sg;
  float y = 0.f, sum_gb = 0.f, sum_da = 0.f;
  for (int n = sg; n < N; n += LPR) {
    const float An = __ldg(a.A + (int64_t)d * N + n);
    const float Bn = load_dyn(a.Bm, boff + (int64_t)n * a.b_sn, a.bc_dtype);
    const float Cn = load_dyn(a.Cm, coff + (int64_t)n * a.c_sn, a.bc_dtype);
    const float s = a.state[row * N + n];
    const float da = expf(dt * An);
    const float nw = fmaf(da, s, dt * x * Bn);
    y = fmaf(Cn, nw, y);
    const float G = fmaf(Cn, dy, g.dnew_state ? g.dnew_state[row * N + n] : 0.f);
    if (live) {
      g.dstate[row * N + n] = G * da;
      atomicAdd(g.dC + coff + (int64_t)n * a.c_sn, dy * nw);
      atomicAdd(g.dB + boff + (int64_t)n * a.b_sn, G * dt * x);
      atomicAdd(g.dA + (int64_t)d * N + n, G * s * da * dt);
    }
    sum_gb = fmaf(G, Bn, sum_gb);
    sum_da = fmaf(G * s * da, An, sum_da);
  }
  y = group_sum<LPR, 1>(y);
  sum_gb = group_sum<LPR, 1>(sum_gb);
  sum_da = group_sum<LPR, 1>(sum_da);
  if (sg == 0 && live) {
    const float Dv = a.D ? __ldg(a.D + d) : 0.f;
    const float yfull = fmaf(Dv, x, y);
    if (g.dz) {
      const float s = sigmoid_f(zv);
      reinterpret_cast<T*>(g.dz)[row] = from_f<T>(dout * yfull * s * (1.f + zv * (1.f - s)));
    }
    reinterpret_cast<T*>(g.dx)[row] = from_f<T>(fmaf(dy, Dv, sum_gb * dt));
    const float ddl = fmaf(sum_gb, x, sum_da);
    const float dpre = a.dt_softplus ? ddl * softplus_grad_f(pre) : ddl;
    reinterpret_cast<T*>(g.ddt)[row] = from_f<T>(dpre);
    if (g.dD) atomicAdd(g.dD + d, dy * x);
    if (g.ddt_bias) atomicAdd(g.ddt_bias + d, dpre);
  }
}

static int step_validate(const ssm_step_args* a) {
  SSM_REQUIRE(a != nullptr, SSM_ERR_NULL, "selective_state_step: args is NULL");
  SSM_REQUIRE(a->batch >= 0 && a->dim >= 0 && a->nstate >= 1, SSM_ERR_SHAPE, "selective_state_step: bad shape");
  SSM_REQUIRE(valid_dtype(a->io_dtype) && valid_dtype(a->bc_dtype), SSM_ERR_DTYPE, "selective_state_step: unknown dtype");
  if (a->batch == 0 || a->dim == 0) return SSM_OK;
  SSM_REQUIRE(a->state && a->x && a->dt && a->A && a->Bm && a->Cm, SSM_ERR_NULL, "selective_state_step: missing pointer");
  SSM_REQUIRE(a->bc_groups >= 1 && a->dim % a->bc_groups == 0, SSM_ERR_SHAPE, "B group dimension must divide D.");
  SSM_REQUIRE(a->param_heads >= 0 && (a->param_heads == 0 || a->dim % a->param_heads == 0), SSM_ERR_SHAPE,
              "selective_state_step: param_heads must divide dim");
  return SSM_OK;
}

static int step_lpr(int n, bool vec) {
  const int per = vec ? (n + 3) / 4 : n;
  int l = 1;
  while (l < per && l < 32) l <<= 1;
  return l;
}

template <typename T, int LPR>
static int step_fwd_launch(const ssm_step_args& a, int vec, cudaStream_t st) {
  const int64_t threads = (int64_t)a.batch * a.dim * LPR;
  step_fwd_kernel<T, LPR><<<(unsigned)((threads + kStepThreads - 1) / kStepThreads), kStepThreads, 0, st>>>(a, vec);
  return launch_status("step_fwd_kernel");
}
template <typename T, int LPR>
static int step_bwd_launch(const ssm_step_bwd_args& g, cudaStream_t st) {
  const int64_t threads = (int64_t)g.fwd.batch * g.fwd.dim * LPR;
  step_bwd_kernel<T, LPR><<<(unsigned)((threads + kStepThreads - 1) / kStepThreads), kStepThreads, 0, st>>>(g);
  return launch_status("step_bwd_kernel");
}

template <typename T, int NV, int LPR>
static int step_fwd_vec_launch(const ssm_step_args& a, cudaStream_t st) {
  const int64_t threads = (int64_t)a.batch * a.dim * LPR;
  step_fwd_vec_kernel<T, NV, LPR><<<(unsigned)((threads + kStepThreads - 1) / kStepThreads), kStepThreads, 0, st>>>(a);
  return launch_status("step_fwd_vec_kernel");
}

template <typename T, typename BT, int NV, int LPR>
static int step_fwd_fast_launch(const ssm_step_args& a, cudaStream_t st) {
  const int64_t threads = (int64_t)a.batch * a.dim * LPR;
  return launch_overlapped("step_fwd_fast_kernel", step_fwd_fast_kernel<T, BT, NV, LPR>, dim3((unsigned)((threads + kStepThreads - 1) / kStepThreads)), dim3(kStepThreads), 0, st, a);
}
// Two pieces or more per warp of a full GPU, else the pipeline never gets going and one thread per row is the shorter path.
template <typename T, typename BT, int N>
static int step_stream_launch(const ssm_step_args& a, int sms, cudaStream_t st) {
  const int grid = sms * kStreamCtasPerSm;
  if (a.param_heads > 0) return launch_overlapped("step_stream_kernel", step_stream_kernel<T, BT, N, true>, dim3(grid), dim3(kStreamThreads), 0, st, a);
  if constexpr (sizeof(T) == 2 && sizeof(BT) == 2) {
    // whole pieces of channels per sequence, and warps that the channels' pieces do not leave idle
    const int per_seq = a.dim / (512 / N), warps = grid * (kStreamThreads / 32);
    if (a.dim % (512 / N) == 0 && a.batch >= 2 * (warps / per_seq) && (warps / per_seq) * per_seq * 8 >= 7 * warps)
      return launch_overlapped("step_channels_kernel", step_channels_kernel<T, BT, N>, dim3(grid), dim3(kStreamThreads), 0, st, a);
  }
  return launch_overlapped("step_stream_kernel", step_stream_kernel<T, BT, N, false>, dim3(grid), dim3(kStreamThreads), 0, st, a);
}
template <typename T, typename BT>
static int step_fwd_fast_n(const ssm_step_args& a, cudaStream_t st) {
  const int sms = sm_count();
  const int64_t rows = (int64_t)a.batch * a.dim;
  if (rows * a.nstate / 512 >= (int64_t)2 * sms * kStreamCtasPerSm * (kStreamThreads / 32) && rows < (1ll << 30)) {
    switch (a.nstate) {
      case 16: return step_stream_launch<T, BT, 16>(a, sms, st);
      case 32: return step_stream_launch<T, BT, 32>(a, sms, st);
      case 64: return step_stream_launch<T, BT, 64>(a, sms, st);
      case 128: return step_stream_launch<T, BT, 128>(a, sms, st);
      default: return step_stream_launch<T, BT, 256>(a, sms, st);
    }
  }
  switch (a.nstate) {
    case 16: return step_fwd_fast_launch<T, BT, 4, 1>(a, st);
    case 32: return step_fwd_fast_launch<T, BT, 4, 2>(a, st);
    case 64: return step_fwd_fast_launch<T, BT, 4, 4>(a, st);
    case 128: return step_fwd_fast_launch<T, BT, 4, 8>(a, st);
    default: return step_fwd_fast_launch<T, BT, 4, 16>(a, st);
  }
}

template <typename T>
static int step_fwd_t(const ssm_step_args& a, cudaStream_t st) {
  if (aligned_to(a.state, 16) && aligned_to(a.A, 16)) {
    // vector loads of B / C: unit state stride and rows that start on a vector boundary
    const int bcb = dtype_size(a.bc_dtype);
    const int64_t per = 16 / bcb / (bcb == 4 ? 1 : 2);  // elements per load: 4 (one 16-byte or one 8-byte load)
    const bool n_ok = a.nstate == 16 || a.nstate == 32 || a.nstate == 64 || a.nstate == 128 || a.nstate == 256;
    const bool bc_ok = a.b_sn == 1 && a.c_sn == 1 && a.b_sb % per == 0 && a.b_sg % per == 0 && a.c_sb % per == 0 && a.c_sg % per == 0 &&
                       aligned_to(a.Bm, 4 * bcb) && aligned_to(a.Cm, 4 * bcb);
    if (n_ok && bc_ok) {
      switch (a.bc_dtype) {
        case SSM_F32: return step_fwd_fast_n<T, float>(a, st);
        case SSM_BF16: return step_fwd_fast_n<T, __nv_bfloat16>(a, st);
        default: return step_fwd_fast_n<T, __half>(a, st);
      }
    }
    switch (a.nstate) {
      case 4: return step_fwd_vec_launch<T, 1, 1>(a, st);
      case 8: return step_fwd_vec_launch<T, 2, 1>(a, st);
      case 16: return step_fwd_vec_launch<T, 4, 1>(a, st);
      case 32: return step_fwd_vec_launch<T, 4, 2>(a, st);
      case 64: return step_fwd_vec_launch<T, 4, 4>(a, st);
      case 128: return step_fwd_vec_launch<T, 4, 8>(a, st);
      case 256: return step_fwd_vec_launch<T, 4, 16>(a, st);
      default: break;
    }
  }
  const int vec = (a.nstate % 4 == 0) && aligned_to(a.state, 16);
  switch (step_lpr(a.nstate, vec != 0)) {
    case 1: return step_fwd_launch<T, 1>(a, vec, st);
    case 2: return step_fwd_launch<T, 2>(a, vec, st);
    case 4: return step_fwd_launch<T, 4>(a, vec, st);
    case 8: return step_fwd_launch<T, 8>(a, vec, st);
    case 16: return step_fwd_launch<T, 16>(a, vec, st);
    default: return step_fwd_launch<T, 32>(a, vec, st);
  }
}
template <typename T>
static int step_bwd_t(const ssm_step_bwd_args& g, cudaStream_t st) {
  switch (step_lpr(g.fwd.nstate, false)) {
    case 1: return step_bwd_launch<T, 1>(g, st);
    case 2: return step_bwd_launch<T, 2>(g, st);
    case 4: return step_bwd_launch<T, 4>(g, st);
    case 8: return step_bwd_launch<T, 8>(g, st);
    case 16: return step_bwd_launch<T, 16>(g, st);
    default: return step_bwd_launch<T, 32>(g, st);
  }
}

}  // namespace ssmb

using namespace ssmb;

extern "C" int ssm_selective_state_step(const ssm_step_args* a, ssm_stream_t stream) {
  if (a && a->io_dtype == SSM_F64) {
    ssm_step_bwd_args g{};
    g.fwd = *a;
    return f64_step(g, false, reinterpret_cast<cudaStream_t>(stream));
  }
  if (int rc = step_validate(a)) return rc;
  if (a->batch == 0 || a->dim == 0) return SSM_OK;
  SSM_REQUIRE(a->out, SSM_ERR_NULL, "selective_state_step: out is required");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  switch (a->io_dtype) {
    case SSM_F32: return step_fwd_t<float>(*a, st);
    case SSM_BF16: return step_fwd_t<__nv_bfloat16>(*a, st);
    default: return step_fwd_t<__half>(*a, st);
  }
}

extern "C" int ssm_selective_state_step_bwd(const ssm_step_bwd_args* g, ssm_stream_t stream) {
  SSM_REQUIRE(g != nullptr, SSM_ERR_NULL, "selective_state_step_backward: args is NULL");
  const ssm_step_args* a = &g->fwd;
  if (a->io_dtype == SSM_F64) return f64_step(*g, true, reinterpret_cast<cudaStream_t>(stream));
  if (int rc = step_validate(a)) return rc;
  SSM_REQUIRE(a->param_heads == 0, SSM_ERR_UNSUPPORTED, "selective_state_step_backward: per-head parameters have no backward");
  SSM_REQUIRE(a->a_log == 0, SSM_ERR_UNSUPPORTED, "selective_state_step_backward: A must be given as it is");
  if (a->batch == 0 || a->dim == 0) return SSM_OK;
  SSM_REQUIRE(g->dout && g->dstate && g->dx && g->ddt && g->dA && g->dB && g->dC, SSM_ERR_NULL,
              "selective_state_step_backward: missing pointer");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  switch (a->io_dtype) {
    case SSM_F32: return step_bwd_t<float>(*g, st);
    case SSM_BF16: return step_bwd_t<__nv_bfloat16>(*g, st);
    default: return step_bwd_t<__half>(*g, st);
  }
}
