// Element-wise chunked diagonal recurrence over (batch, len, heads, proj), forward and
// backward, sm_100a.
//
//   s_t = exp(dt_t A) s_{t-1} + dt_t B_t X_t;   y_t = s_t C_t + D X_t;   y_t *= silu(z_t)
//
// Each (batch, head, proj) lane is an independent scalar recurrence, so with (head, proj)
// fastest in memory consecutive threads read consecutive addresses at every step; the kernels
// are HBM-bound streams.  The sequence axis is split into chunks that run in parallel:
//   forward   (1) every chunk integrates from a zero state and records its decay product,
//             (2) a short serial pass over chunks turns those into each chunk's incoming state,
//             (3) every chunk is replayed from its true incoming state and writes Y;
//   backward  the incoming states come from the forward call (or the same three phases), their
//             mirror image gives every chunk the adjoint that enters it from the right
//             (g_t = C_t dy_t + exp(dt_{t+1} A) g_{t+1} is a linear recurrence too), and one
//             final pass per chunk replays the states and walks back through them producing every
//             gradient.
// The usual layouts run on lanes of several projections (chunk_scan_vec.cuh); the kernels of this
// file take any broadcast.
// Every thread keeps raw pointers that advance by one time stride per step, and the loads of
// eight steps are issued before the first of them is used, so that enough bytes are in flight.
// Without scratch memory a single serial pass is used instead.
#include <type_traits>

#include "common.cuh"

namespace ssmb {

constexpr int kChunkThreads = 128;
constexpr int kChunkUnroll = 8;

__device__ __forceinline__ int64_t bc4_off(const ssm_bcast4& p, int b, int t, int h, int q) {
  return (int64_t)b * p.sb + (int64_t)t * p.st + (int64_t)h * p.sh + (int64_t)q * p.sq;
}
__device__ __forceinline__ float bc4_load_f32(const ssm_bcast4& p, int b, int t, int h, int q) {
  return __ldg(reinterpret_cast<const float*>(p.ptr) + bc4_off(p, b, t, h, q));
}
__device__ __forceinline__ float* bc4_ptr(const ssm_bcast4& p, int b, int t, int h, int q) {
  return const_cast<float*>(reinterpret_cast<const float*>(p.ptr)) + bc4_off(p, b, t, h, q);
}
// true when every (b, t, h, q) of a gradient buffer is a distinct element (no broadcast axis): plain stores suffice
__device__ __forceinline__ bool bc4_dense(const ssm_bcast4& p) { return p.sb != 0 && p.st != 0 && p.sh != 0 && p.sq != 0; }

__device__ __forceinline__ int chunk_valid_len(const ssm_chunk_args& a, int b) {
  if (!a.seq_lens) return a.len;
  const int64_t v = a.seq_lens[b];
  return (int)(v < 0 ? 0 : (v > a.len ? a.len : v));
}

// A time-strided stream of one lane: element offset at the lane's first step, stride per step (0: constant in time).
template <typename E>
struct Stream {
  const E* p;
  int64_t st;
  __device__ __forceinline__ float at(int k) const { return to_f<E>(__ldg(p + (int64_t)k * st)); }
};
// B / C / z stream of element type PT at (b, t, h, q)
template <typename PT>
__device__ __forceinline__ Stream<PT> par_stream(const ssm_bcast4& c, int b, int t, int h, int q) {
  return {reinterpret_cast<const PT*>(c.ptr) + bc4_off(c, b, t, h, q), c.st};
}

}  // namespace ssmb
#include "chunk_scan_vec.cuh"
namespace ssmb {

// per-lane context shared by all scalar kernels
template <typename T>
struct Lane {
  int b, h, q, hp, HP, valid;
  float Av, Dv;
  __device__ __forceinline__ bool init(const ssm_chunk_args& a) {
    HP = a.heads * a.proj;
    hp = blockIdx.x * kChunkThreads + threadIdx.x;
    if (hp >= HP) return false;
    h = hp / a.proj, q = hp % a.proj;
    b = blockIdx.z;
    valid = chunk_valid_len(a, b);
    Av = bc4_load_f32(a.A, 0, 0, h, q) * kLog2e;
    Dv = a.D.ptr ? bc4_load_f32(a.D, 0, 0, h, q) : 0.f;
    return true;
  }
  __device__ __forceinline__ Stream<T> x(const ssm_chunk_args& a, int t) const {
    return {reinterpret_cast<const T*>(a.X) + ((int64_t)b * a.len + t) * HP + hp, HP};
  }
  __device__ __forceinline__ Stream<T> dt(const ssm_chunk_args& a, int t) const {
    return {reinterpret_cast<const T*>(a.dt) + ((int64_t)b * a.len + t) * a.heads + h, a.heads};
  }
};

// ---------------------------------------------------------------------------------------------
// forward
// ---------------------------------------------------------------------------------------------
// mode 0: serial over the whole sequence (no scratch).  mode 1: phase 1 (local state + decay).  mode 3: phase 3.
template <typename T, typename PT, int MODE>
__global__ void __launch_bounds__(kChunkThreads) chunk_fwd_kernel(const ssm_chunk_args a, int nchunks, int chunk_len) {
  Lane<T> ln;
  if (!ln.init(a)) return;
  const int c = MODE == 0 ? 0 : blockIdx.y;
  const int t0 = MODE == 0 ? 0 : c * chunk_len;
  const int t1 = MODE == 0 ? a.len : min(a.len, t0 + chunk_len);
  const int te = max(t0, min(t1, ln.valid));
  float* P = a.scratch;                                                             // [batch][nchunks][HP] decay products
  float* S = a.scratch ? a.scratch + (int64_t)a.batch * nchunks * ln.HP : nullptr;  // local end state, then incoming state
  const int64_t slot = ((int64_t)ln.b * nchunks + c) * ln.HP + ln.hp;
  const Stream<T> sx = ln.x(a, t0), sdt = ln.dt(a, t0);
  const Stream<PT> sB = par_stream<PT>(a.Bm, ln.b, t0, ln.h, ln.q);
  const int n = te - t0;
  if (MODE == 1) {
    float s = 0.f, sumdt = 0.f;
    int k = 0;
    for (; k + kChunkUnroll <= n; k += kChunkUnroll) {
      float x[kChunkUnroll], d[kChunkUnroll], bv[kChunkUnroll];
#pragma unroll
      for (int i = 0; i < kChunkUnroll; ++i) x[i] = sx.at(k + i), d[i] = sdt.at(k + i), bv[i] = sB.at(k + i);
#pragma unroll
      for (int i = 0; i < kChunkUnroll; ++i) {
        s = fmaf(ex2_approx(d[i] * ln.Av), s, d[i] * bv[i] * x[i]);
        sumdt += d[i];
      }
    }
    for (; k < n; ++k) {
      const float d = sdt.at(k);
      s = fmaf(ex2_approx(d * ln.Av), s, d * sB.at(k) * sx.at(k));
      sumdt += d;
    }
    P[slot] = ex2_approx(sumdt * ln.Av);
    S[slot] = s;
    return;
  }
  const Stream<PT> sC = par_stream<PT>(a.Cm, ln.b, t0, ln.h, ln.q);
  const bool has_z = a.z.ptr != nullptr;
  const Stream<PT> sz = has_z ? par_stream<PT>(a.z, ln.b, t0, ln.h, ln.q) : Stream<PT>{nullptr, 0};
  T* Y = reinterpret_cast<T*>(a.Y) + ((int64_t)ln.b * a.len + t0) * ln.HP + ln.hp;
  float s;
  if (MODE == 0) s = a.initial.ptr ? bc4_load_f32(a.initial, ln.b, 0, ln.h, ln.q) : 0.f;
  else s = S[slot];
  auto step = [&](float x, float d, float bv, float cv, float zv) {
    s = fmaf(ex2_approx(d * ln.Av), s, d * bv * x);
    float y = fmaf(ln.Dv, x, s * cv);
    if (has_z) y *= silu_fast(zv);
    return y;
  };
  int k = 0;
  for (; k + kChunkUnroll <= n; k += kChunkUnroll) {
    float x[kChunkUnroll], d[kChunkUnroll], bv[kChunkUnroll], cv[kChunkUnroll], zv[kChunkUnroll];
#pragma unroll
    for (int i = 0; i < kChunkUnroll; ++i) {
      x[i] = sx.at(k + i), d[i] = sdt.at(k + i), bv[i] = sB.at(k + i), cv[i] = sC.at(k + i);
      zv[i] = has_z ? sz.at(k + i) : 0.f;
    }
#pragma unroll
    for (int i = 0; i < kChunkUnroll; ++i) Y[(int64_t)(k + i) * ln.HP] = from_f<T>(step(x[i], d[i], bv[i], cv[i], zv[i]));
  }
  for (; k < n; ++k) Y[(int64_t)k * ln.HP] = from_f<T>(step(sx.at(k), sdt.at(k), sB.at(k), sC.at(k), has_z ? sz.at(k) : 0.f));
  for (int t = te; t < t1; ++t) Y[(int64_t)(t - t0) * ln.HP] = from_f<T>(0.f);
  if (MODE == 0 && a.final_state) a.final_state[(int64_t)ln.b * ln.HP + ln.hp] = s;
}

// The carry over the pieces: v_{c+1} = P[c] v_c + L[c], and L[c] is replaced by v_c (what enters piece c).  One lane per hp,
// kCarryGroups threads per lane: each composes kCarryPer consecutive pieces (all their loads in flight at once), the
// composites of the groups meet in shared memory, and each group then replays its pieces from what enters it; a serial
// chain of 16 + 4 + 16 multiply-adds per 64 pieces instead of 64 dependent on 64 loads.  REVERSE walks the pieces from the
// right (the adjoint).  Returns the value that leaves the last piece.
constexpr int kCarryLanes = 128, kCarryGroups = 4, kCarryPer = 16;
template <bool REVERSE>
__device__ __forceinline__ float carry_pieces(const float* __restrict__ P, float* __restrict__ Lc, int nchunks, int64_t stride, float v_in, bool live) {
  __shared__ float sP[kCarryGroups][kCarryLanes], sS[kCarryGroups][kCarryLanes];
  const int lane = threadIdx.x % kCarryLanes, grp = threadIdx.x / kCarryLanes;
  for (int base = 0; base < nchunks; base += kCarryGroups * kCarryPer) {
    const int r0 = base + grp * kCarryPer;  // position in walking order
    float local[kCarryPer], pr[kCarryPer];
#pragma unroll
    for (int i = 0; i < kCarryPer; ++i) {
      const int r = min(r0 + i, nchunks - 1);
      const int64_t at = (int64_t)(REVERSE ? nchunks - 1 - r : r) * stride;
      local[i] = Lc[at], pr[i] = P[at];
    }
    float Pg = 1.f, Sg = 0.f;
#pragma unroll
    for (int i = 0; i < kCarryPer; ++i) {
      if (r0 + i < nchunks) Sg = fmaf(pr[i], Sg, local[i]), Pg *= pr[i];
    }
    sP[grp][lane] = Pg, sS[grp][lane] = Sg;
    __syncthreads();
    float v = v_in, v_next = v_in;
#pragma unroll
    for (int g2 = 0; g2 < kCarryGroups; ++g2) {
      if (g2 < grp) v = fmaf(sP[g2][lane], v, sS[g2][lane]);
      v_next = fmaf(sP[g2][lane], v_next, sS[g2][lane]);
    }
#pragma unroll
    for (int i = 0; i < kCarryPer; ++i) {
      const int r = r0 + i;
      if (r < nchunks) {
        if (live) Lc[(int64_t)(REVERSE ? nchunks - 1 - r : r) * stride] = v;
        v = fmaf(pr[i], v, local[i]);
      }
    }
    v_in = v_next;
    __syncthreads();
  }
  return v_in;
}

// phase 2: S[c] <- state entering piece c
__global__ void __launch_bounds__(kCarryLanes * kCarryGroups) chunk_carry_kernel(const ssm_chunk_args a, int nchunks) {
  pdl_wait();
  pdl_trigger();
  const int HP = a.heads * a.proj;
  const int hp_raw = blockIdx.x * kCarryLanes + threadIdx.x % kCarryLanes;
  const bool live = hp_raw < HP;
  const int hp = live ? hp_raw : HP - 1;  // idle lanes of the last CTA shadow a valid lane: they meet the barriers and write nothing
  const int b = blockIdx.z;
  const int h = hp / a.proj, q = hp % a.proj;
  const float* P = a.scratch + (int64_t)b * nchunks * HP + hp;
  float* S = a.scratch + (int64_t)a.batch * nchunks * HP + (int64_t)b * nchunks * HP + hp;
  const float s0 = a.initial.ptr ? bc4_load_f32(a.initial, b, 0, h, q) : 0.f;
  const float s = carry_pieces<false>(P, S, nchunks, HP, s0, live);
  if (live && threadIdx.x < kCarryLanes && a.final_state) a.final_state[(int64_t)b * HP + hp] = s;
}

// ---------------------------------------------------------------------------------------------
// backward
// ---------------------------------------------------------------------------------------------
// dy_t = dout_t * silu(z_t) (or dout_t)
__device__ __forceinline__ float gated_dy(float dout, bool has_z, float zv) { return has_z ? dout * silu_fast(zv) : dout; }

// reverse phase 1: per chunk, the adjoint that leaves the chunk on its left side when nothing enters on the right:
//   carry <- exp(dt_t A) (C_t dy_t + carry), t from the chunk's last valid step down to its first
template <typename T, typename PT>
__global__ void __launch_bounds__(kChunkThreads) chunk_bwd_local_kernel(const ssm_chunk_bwd_args g, int nchunks) {
  const ssm_chunk_args& a = g.fwd;
  Lane<T> ln;
  if (!ln.init(a)) return;
  const int c = blockIdx.y;
  const int t0 = c * a.chunk_size, t1 = min(a.len, t0 + a.chunk_size);
  const int te = max(t0, min(t1, ln.valid));
  const int n = te - t0;
  float* R = g.scratch + 2 * (int64_t)a.batch * nchunks * ln.HP;  // [batch][nchunks][HP] local adjoint, then the adjoint entering each chunk
  const int64_t slot = ((int64_t)ln.b * nchunks + c) * ln.HP + ln.hp;
  const Stream<T> sdt = ln.dt(a, t0);
  const Stream<T> sdy = {reinterpret_cast<const T*>(g.dY) + ((int64_t)ln.b * a.len + t0) * ln.HP + ln.hp, ln.HP};
  const Stream<PT> sC = par_stream<PT>(a.Cm, ln.b, t0, ln.h, ln.q);
  const bool has_z = a.z.ptr != nullptr;
  const Stream<PT> sz = has_z ? par_stream<PT>(a.z, ln.b, t0, ln.h, ln.q) : Stream<PT>{nullptr, 0};
  float carry = 0.f;
  int k = n;
  for (; k - kChunkUnroll >= 0; k -= kChunkUnroll) {
    float d[kChunkUnroll], dy[kChunkUnroll], cv[kChunkUnroll];
#pragma unroll
    for (int i = 0; i < kChunkUnroll; ++i) {
      const int kk = k - 1 - i;
      d[i] = sdt.at(kk), cv[i] = sC.at(kk);
      dy[i] = gated_dy(sdy.at(kk), has_z, has_z ? sz.at(kk) : 0.f);
    }
#pragma unroll
    for (int i = 0; i < kChunkUnroll; ++i) carry = ex2_approx(d[i] * ln.Av) * fmaf(cv[i], dy[i], carry);
  }
  for (; k > 0; --k) {
    const int kk = k - 1;
    carry = ex2_approx(sdt.at(kk) * ln.Av) * fmaf(sC.at(kk), gated_dy(sdy.at(kk), has_z, has_z ? sz.at(kk) : 0.f), carry);
  }
  R[slot] = carry;
}

// reverse phase 2: over the pieces from the right; R[c] <- adjoint entering piece c from piece c + 1
__global__ void __launch_bounds__(kCarryLanes * kCarryGroups) chunk_bwd_carry_kernel(const ssm_chunk_bwd_args g, const float* __restrict__ P_all, int nchunks) {
  pdl_wait();
  pdl_trigger();
  const ssm_chunk_args& a = g.fwd;
  const int HP = a.heads * a.proj;
  const int hp_raw = blockIdx.x * kCarryLanes + threadIdx.x % kCarryLanes;
  const bool live = hp_raw < HP;
  const int hp = live ? hp_raw : HP - 1;
  const int b = blockIdx.z;
  const float* P = P_all + (int64_t)b * nchunks * HP + hp;
  float* R = g.scratch + 2 * (int64_t)a.batch * nchunks * HP + (int64_t)b * nchunks * HP + hp;
  const float carry = carry_pieces<true>(P, R, nchunks, HP, 0.f, live);
  if (live && threadIdx.x < kCarryLanes && g.dinitial.ptr) {
    const int h = hp / a.proj, q = hp % a.proj;
    atomicAdd(bc4_ptr(g.dinitial, b, 0, h, q), carry);
  }
}

// sum over the lanes of a warp that share a head, then one atomic per group (proj a multiple of 32: the whole warp)
__device__ __forceinline__ void add_reduced(float* dst, float v, bool whole_warp) {
  if (whole_warp) {
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) atomicAdd(dst, v);
  } else {
    atomicAdd(dst, v);
  }
}

// final pass: MODE 0 = one thread walks the whole sequence (no scratch); MODE 1 = one chunk per blockIdx.y, the states entering the
// chunks taken from S, the adjoints from the scratch.
template <typename T, typename PT, int MODE>
__global__ void __launch_bounds__(kChunkThreads) chunk_bwd_kernel(const ssm_chunk_bwd_args g, const float* __restrict__ S, int nchunks) {
  const ssm_chunk_args& a = g.fwd;
  Lane<T> ln;
  if (!ln.init(a)) return;
  const int c = MODE == 0 ? 0 : blockIdx.y;
  const int t0 = MODE == 0 ? 0 : c * a.chunk_size;
  const int t1 = MODE == 0 ? a.len : min(a.len, t0 + a.chunk_size);
  const int te = max(t0, min(t1, ln.valid));
  const int n = te - t0;
  const int64_t slot = ((int64_t)ln.b * nchunks + c) * ln.HP + ln.hp;
  float s0, carry;
  if (MODE == 0) {
    s0 = a.initial.ptr ? bc4_load_f32(a.initial, ln.b, 0, ln.h, ln.q) : 0.f;
    carry = 0.f;
  } else {
    s0 = S[slot];
    carry = g.scratch[2 * (int64_t)a.batch * nchunks * ln.HP + slot];
  }
  const Stream<T> sx = ln.x(a, t0), sdt = ln.dt(a, t0);
  const Stream<T> sdy = {reinterpret_cast<const T*>(g.dY) + ((int64_t)ln.b * a.len + t0) * ln.HP + ln.hp, ln.HP};
  const Stream<PT> sB = par_stream<PT>(a.Bm, ln.b, t0, ln.h, ln.q);
  const Stream<PT> sC = par_stream<PT>(a.Cm, ln.b, t0, ln.h, ln.q);
  const bool has_z = a.z.ptr != nullptr;
  const Stream<PT> sz = has_z ? par_stream<PT>(a.z, ln.b, t0, ln.h, ln.q) : Stream<PT>{nullptr, 0};
  float* hist = g.history + ((int64_t)ln.b * a.len + t0) * ln.HP + ln.hp;
  T* dX = reinterpret_cast<T*>(g.dX) + ((int64_t)ln.b * a.len + t0) * ln.HP + ln.hp;

  // ---- states of the chunk, into the history ---------------------------------------------------------------
  {
    float s = s0;
    int k = 0;
    for (; k + kChunkUnroll <= n; k += kChunkUnroll) {
      float x[kChunkUnroll], d[kChunkUnroll], bv[kChunkUnroll];
#pragma unroll
      for (int i = 0; i < kChunkUnroll; ++i) x[i] = sx.at(k + i), d[i] = sdt.at(k + i), bv[i] = sB.at(k + i);
#pragma unroll
      for (int i = 0; i < kChunkUnroll; ++i) {
        s = fmaf(ex2_approx(d[i] * ln.Av), s, d[i] * bv[i] * x[i]);
        hist[(int64_t)(k + i) * ln.HP] = s;
      }
    }
    for (; k < n; ++k) {
      const float d = sdt.at(k);
      s = fmaf(ex2_approx(d * ln.Av), s, d * sB.at(k) * sx.at(k));
      hist[(int64_t)k * ln.HP] = s;
    }
  }
  // typed gradient buffers (a.typed_grads) are written in full, the rows beyond the sequence as zeros
  const bool typed_b = a.typed_grads & 1, typed_c = a.typed_grads & 2, typed_z = has_z && (a.typed_grads & 4);
  auto put = [&](const ssm_bcast4& p, bool typed, int t, float v) {
    const int64_t off = bc4_off(p, ln.b, t, ln.h, ln.q);
    if (typed) const_cast<PT*>(reinterpret_cast<const PT*>(p.ptr))[off] = from_f<PT>(v);
    else const_cast<float*>(reinterpret_cast<const float*>(p.ptr))[off] = v;
  };
  for (int t = te; t < t1; ++t) {
    dX[(int64_t)(t - t0) * ln.HP] = from_f<T>(0.f);
    if (typed_b) put(g.dB, true, t, 0.f);
    if (typed_c) put(g.dC, true, t, 0.f);
    if (typed_z) put(g.dz, true, t, 0.f);
  }

  // ---- reverse recurrence  g_t = C_t dy_t + exp(dt_{t+1} A) g_{t+1} -------------------------------------------
  const bool dense_b = bc4_dense(g.dB), dense_c = bc4_dense(g.dC), dense_z = has_z && bc4_dense(g.dz);
  const bool warp_heads = (a.proj & 31) == 0;  // a warp's 32 lanes share their head: (b, t, h) sums reduce in the warp first
  float dA_acc = 0.f, dD_acc = 0.f;
  const float A_nat = ln.Av * kLn2;
  auto back = [&](int k, float x, float d, float bv, float cv, float zv, float dout, float st, float sp) {
    const int t = t0 + k;
    float dyv = dout;
    if (has_z) {
      const float sg = sigmoid_fast(zv);
      const float yfull = fmaf(ln.Dv, x, st * cv);
      const float dzv = dout * yfull * sg * (1.f + zv * (1.f - sg));
      if (dense_z) put(g.dz, typed_z, t, dzv);
      else if (a.z.sq == 0) add_reduced(bc4_ptr(g.dz, ln.b, t, ln.h, 0), dzv, warp_heads);
      else atomicAdd(bc4_ptr(g.dz, ln.b, t, ln.h, ln.q), dzv);
      dyv = dout * zv * sg;
    }
    const float da = ex2_approx(d * ln.Av);
    const float G = fmaf(cv, dyv, carry);
    if (dense_c) put(g.dC, typed_c, t, dyv * st);
    else atomicAdd(bc4_ptr(g.dC, ln.b, t, ln.h, ln.q), dyv * st);
    if (dense_b) put(g.dB, typed_b, t, G * d * x);
    else atomicAdd(bc4_ptr(g.dB, ln.b, t, ln.h, ln.q), G * d * x);
    dX[(int64_t)k * ln.HP] = from_f<T>(fmaf(dyv, ln.Dv, G * d * bv));
    const float gsa = G * sp * da;
    add_reduced(reinterpret_cast<float*>(g.ddt) + ((int64_t)ln.b * a.len + t) * a.heads + ln.h, fmaf(G, bv * x, gsa * A_nat), warp_heads);
    dA_acc = fmaf(gsa, d, dA_acc);
    dD_acc = fmaf(dyv, x, dD_acc);
    carry = G * da;
  };
  int k = n;
  for (; k - kChunkUnroll >= 0; k -= kChunkUnroll) {
    float x[kChunkUnroll], d[kChunkUnroll], bv[kChunkUnroll], cv[kChunkUnroll], zv[kChunkUnroll], dout[kChunkUnroll], st[kChunkUnroll + 1];
#pragma unroll
    for (int i = 0; i < kChunkUnroll; ++i) {
      const int kk = k - 1 - i;
      x[i] = sx.at(kk), d[i] = sdt.at(kk), bv[i] = sB.at(kk), cv[i] = sC.at(kk), dout[i] = sdy.at(kk);
      zv[i] = has_z ? sz.at(kk) : 0.f;
      st[i] = hist[(int64_t)kk * ln.HP];
    }
    st[kChunkUnroll] = k - kChunkUnroll > 0 ? hist[(int64_t)(k - kChunkUnroll - 1) * ln.HP] : s0;
#pragma unroll
    for (int i = 0; i < kChunkUnroll; ++i) back(k - 1 - i, x[i], d[i], bv[i], cv[i], zv[i], dout[i], st[i], st[i + 1]);
  }
  for (; k > 0; --k) {
    const int kk = k - 1;
    back(kk, sx.at(kk), sdt.at(kk), sB.at(kk), sC.at(kk), has_z ? sz.at(kk) : 0.f, sdy.at(kk), hist[(int64_t)kk * ln.HP],
         kk > 0 ? hist[(int64_t)(kk - 1) * ln.HP] : s0);
  }
  atomicAdd(bc4_ptr(g.dA, 0, 0, ln.h, ln.q), dA_acc);
  if (g.dD.ptr) {
    if (a.D.sq == 0) add_reduced(bc4_ptr(g.dD, 0, 0, ln.h, 0), dD_acc, warp_heads);
    else atomicAdd(bc4_ptr(g.dD, 0, 0, ln.h, ln.q), dD_acc);
  }
  if (MODE == 0 && g.dinitial.ptr) atomicAdd(bc4_ptr(g.dinitial, ln.b, 0, ln.h, ln.q), carry);
}


static bool bc4_dense_host(const ssm_bcast4& p) { return p.ptr && p.sb != 0 && p.st != 0 && p.sh != 0 && p.sq != 0; }

static int chunk_validate(const ssm_chunk_args* a) {
  SSM_REQUIRE(a != nullptr, SSM_ERR_NULL, "ssd_chunk_scan: args is NULL");
  SSM_REQUIRE(a->batch >= 0 && a->len >= 0 && a->heads >= 0 && a->proj >= 0, SSM_ERR_SHAPE, "ssd_chunk_scan: negative size");
  SSM_REQUIRE(a->chunk_size >= 1, SSM_ERR_SHAPE, "chunk_size must be positive.");
  SSM_REQUIRE(valid_dtype(a->io_dtype) && valid_dtype(a->par_dtype), SSM_ERR_DTYPE, "ssd_chunk_scan: unknown dtype");
  SSM_REQUIRE(a->batch <= 65535, SSM_ERR_TOO_LARGE, "ssd_chunk_scan: batch exceeds 65535");
  return SSM_OK;
}

// The recurrence does not depend on where the sequence is cut, so the forward cuts it where it suits the machine: pieces of
// at most kFwdChunkMax steps (more pieces in flight than the caller's chunk size gives at short sequences).  The scratch size
// function uses the same length.
constexpr int kFwdChunkMax = 32;
static int chunk_fwd_len(int chunk_size, int len) {
  int piece = chunk_size < kFwdChunkMax ? chunk_size : kFwdChunkMax;
  while (piece < chunk_size && ((int64_t)len + piece - 1) / piece > 65535) piece *= 2;  // the pieces are a grid axis
  return piece < chunk_size ? piece : chunk_size;
}

// The layouts that the kernels on lanes of `v` projections read: the projection axis contiguous, every row a multiple of `v` elements and
// aligned to them; B, C, z of X's element type.
static bool chunk_vec_ok(const ssm_chunk_args& a, int piece, int v) {
  if (a.proj % v != 0 || a.scratch == nullptr || a.par_dtype != a.io_dtype || piece > kPiece) return false;
  const size_t al = v * dtype_size(a.io_dtype);
  auto rows = [&](const ssm_bcast4& p) { return p.sq == 1 && p.sb % v == 0 && p.st % v == 0 && p.sh % v == 0 && aligned_to(p.ptr, al); };
  if (!rows(a.Bm) || !rows(a.Cm) || (a.z.ptr && !rows(a.z))) return false;
  return aligned_to(a.X, al) && aligned_to(a.Y, al) && aligned_to(a.scratch, 16);
}

// chunk_len: steps per piece (the backward passes the caller's chunk size, which its own scratch and history are sized by)
template <typename T, typename PT>
static int chunk_fwd_t(const ssm_chunk_args& a, cudaStream_t st, int chunk_len, bool through_phase2_only = false) {
  const int HP = a.heads * a.proj;
  const unsigned gx = (HP + kChunkThreads - 1) / kChunkThreads;
  const int nchunks = (a.len + chunk_len - 1) / chunk_len;
  if (!a.scratch || nchunks <= 1) {
    chunk_fwd_kernel<T, PT, 0><<<dim3(gx, 1, a.batch), kChunkThreads, 0, st>>>(a, 1, chunk_len);
    return launch_status("chunk_fwd_kernel<serial>");
  }
  SSM_REQUIRE(nchunks <= 65535, SSM_ERR_TOO_LARGE, "ssd_chunk_scan: more than 65535 chunks");
  // projections per lane: what makes 16 bytes, else (16-bit rows on 8-byte boundaries) four, else one
  constexpr int kWide = 16 / sizeof(T);
  const int v = !std::is_same<T, PT>::value ? 1 : chunk_vec_ok(a, chunk_len, kWide) ? kWide : chunk_vec_ok(a, chunk_len, 4) ? 4 : 1;
  const dim3 grid((HP / v + kChunkThreads - 1) / kChunkThreads, nchunks, a.batch);
  const dim3 block(kChunkThreads);
  int rc;
  if (v == kWide) rc = launch_overlapped("chunk_fwd_row_kernel<local>", chunk_fwd_row_kernel<T, kWide, false>, grid, block, 0, st, a, nchunks, chunk_len);
  else if (v == 4) rc = launch_overlapped("chunk_fwd_row_kernel<local>", chunk_fwd_row_kernel<T, 4, false>, grid, block, 0, st, a, nchunks, chunk_len);
  else chunk_fwd_kernel<T, PT, 1><<<grid, kChunkThreads, 0, st>>>(a, nchunks, chunk_len), rc = launch_status("chunk_fwd_kernel<local>");
  if (rc) return rc;
  rc = launch_overlapped("chunk_carry_kernel", chunk_carry_kernel, dim3((HP + kCarryLanes - 1) / kCarryLanes, 1, a.batch), dim3(kCarryLanes * kCarryGroups), 0, st, a, nchunks);
  if (rc) return rc;
  if (through_phase2_only) return SSM_OK;
  if (v == kWide) return launch_overlapped("chunk_fwd_row_kernel<apply>", chunk_fwd_row_kernel<T, kWide, true>, grid, block, 0, st, a, nchunks, chunk_len);
  if (v == 4) return launch_overlapped("chunk_fwd_row_kernel<apply>", chunk_fwd_row_kernel<T, 4, true>, grid, block, 0, st, a, nchunks, chunk_len);
  chunk_fwd_kernel<T, PT, 3><<<grid, kChunkThreads, 0, st>>>(a, nchunks, chunk_len);
  return launch_status("chunk_fwd_kernel<apply>");
}

// The backward cuts the sequence into pieces of at most kBwdChunkMax steps, whatever the caller's chunk size: each piece is one
// serial walk per thread (replay, then the walk back), and short pieces are what puts enough of them in flight.
constexpr int kBwdChunkMax = 32;
static int chunk_bwd_len(int chunk_size, int len) {
  int piece = chunk_size < kBwdChunkMax ? chunk_size : kBwdChunkMax;
  while (piece < chunk_size && ((int64_t)len + piece - 1) / piece > 65535) piece *= 2;  // the pieces are a grid axis
  return piece < chunk_size ? piece : chunk_size;
}

// The call runs on the four-projection kernels: readable layouts, gradients of B, C, z written in full in their own type, and heads
// whose projections are a power of two of at most a warp's lanes (their sums for ddt then stay inside a warp).
static bool chunk_bwd_vec_ok(const ssm_chunk_bwd_args& g, int piece, int nchunks) {
  const ssm_chunk_args& a = g.fwd;
  const size_t al = 4 * dtype_size(a.io_dtype);
  const int share = a.proj / 4, need = 3 | (a.z.ptr ? 4 : 0);
  ssm_chunk_args f = a;
  f.scratch = g.scratch, f.Y = g.dX;  // only their alignment is looked at
  if (!chunk_vec_ok(f, piece, 4) || nchunks <= 1 || nchunks > 65535 || (a.typed_grads & need) != need || share > 32 || (share & (share - 1)) != 0) return false;
  auto rows4 = [&](const ssm_bcast4& p) { return p.sq == 1 && p.sb % 4 == 0 && p.st % 4 == 0 && p.sh % 4 == 0 && aligned_to(p.ptr, al); };
  return rows4(g.dB) && rows4(g.dC) && (!a.z.ptr || rows4(g.dz)) && aligned_to(g.dY, al) && aligned_to(g.fwd_scratch, 16);
}

// The rows that the local adjoint reads (dY, C, z), as chunk_vec_ok.
static bool chunk_bwd_wide_ok(const ssm_chunk_bwd_args& g, int v) {
  const ssm_chunk_args& a = g.fwd;
  const size_t al = v * dtype_size(a.io_dtype);
  auto rows = [&](const ssm_bcast4& p) { return p.sq == 1 && p.sb % v == 0 && p.st % v == 0 && p.sh % v == 0 && aligned_to(p.ptr, al); };
  return a.proj % v == 0 && rows(a.Cm) && (!a.z.ptr || rows(a.z)) && aligned_to(g.dY, al);
}

// Every row tensor of the call is contiguous like X, and a row's byte offset fits 32 bits.
static bool chunk_same_layout(const ssm_chunk_bwd_args& g) {
  const ssm_chunk_args& a = g.fwd;
  const int64_t HP = (int64_t)a.heads * a.proj, total = (int64_t)a.batch * a.len * HP;
  auto like_x = [&](const ssm_bcast4& p) { return p.sq == 1 && p.sh == a.proj && p.st == HP && p.sb == a.len * HP; };
  return total * dtype_size(a.io_dtype) < ((int64_t)1 << 32) && like_x(a.Bm) && like_x(a.Cm) && like_x(g.dB) && like_x(g.dC) &&
         (!a.z.ptr || (like_x(a.z) && like_x(g.dz)));
}

template <typename T, typename PT>
static int chunk_bwd_t(const ssm_chunk_bwd_args& g_in, cudaStream_t st) {
  ssm_chunk_bwd_args g = g_in;
  g.fwd.chunk_size = chunk_bwd_len(g_in.fwd.chunk_size, g_in.fwd.len);  // the kernels cut the sequence by this field
  const ssm_chunk_args& a = g.fwd;
  const int HP = a.heads * a.proj;
  const unsigned gx = (HP + kChunkThreads - 1) / kChunkThreads;
  const int nchunks = (a.len + a.chunk_size - 1) / a.chunk_size;
  const bool vec = std::is_same<T, PT>::value && chunk_bwd_vec_ok(g, a.chunk_size, nchunks);
  SSM_REQUIRE(vec || (g.history && !(a.typed_grads & 8)), SSM_ERR_UNSUPPORTED, "ssd_chunk_scan_backward: this call needs a history and an fp32 ddt");
  if (!g.scratch || nchunks <= 1 || nchunks > 65535) {
    chunk_bwd_kernel<T, PT, 0><<<dim3(gx, 1, a.batch), kChunkThreads, 0, st>>>(g, nullptr, 1);
    return launch_status("chunk_bwd_kernel<serial>");
  }
  // states entering every piece and the pieces' decay products: left by the forward call, or formed again (its phases 1 and 2 on
  // this call's scratch; no final state, no Y)
  const float* P = g.scratch;
  if (g.fwd_scratch && chunk_fwd_len(g_in.fwd.chunk_size, a.len) == a.chunk_size) {
    P = g.fwd_scratch;
  } else {
    ssm_chunk_args f = a;
    f.scratch = g.scratch, f.final_state = nullptr;
    if (int rc = chunk_fwd_t<T, PT>(f, st, a.chunk_size, true)) return rc;
  }
  const float* S = P + (int64_t)a.batch * nchunks * HP;
  float* R = g.scratch + 2 * (int64_t)a.batch * nchunks * HP;
  const unsigned gv = (HP / 4 + kChunkThreads - 1) / kChunkThreads;
  constexpr int kWide = 16 / sizeof(T);
  int rc;
  if (vec && chunk_bwd_wide_ok(g, kWide)) {
    rc = launch_overlapped("chunk_bwd_local_row_kernel", chunk_bwd_local_row_kernel<T, kWide>, dim3((HP / kWide + kChunkThreads - 1) / kChunkThreads, nchunks, a.batch),
                           dim3(kChunkThreads), 0, st, g, R, nchunks, a.chunk_size);
  } else if (vec) {
    rc = launch_overlapped("chunk_bwd_local_row_kernel", chunk_bwd_local_row_kernel<T, 4>, dim3(gv, nchunks, a.batch), dim3(kChunkThreads), 0, st, g, R, nchunks, a.chunk_size);
  } else {
    chunk_bwd_local_kernel<T, PT><<<dim3(gx, nchunks, a.batch), kChunkThreads, 0, st>>>(g, nchunks);
    rc = launch_status("chunk_bwd_local_kernel");
  }
  if (rc) return rc;
  rc = launch_overlapped("chunk_bwd_carry_kernel", chunk_bwd_carry_kernel, dim3((HP + kCarryLanes - 1) / kCarryLanes, 1, a.batch), dim3(kCarryLanes * kCarryGroups), 0, st, g, P,
                         nchunks);
  if (rc) return rc;
  if (vec) {
    const int64_t items = (int64_t)a.batch * nchunks, slots = (int64_t)bwd4_ctas<T>() * sm_count() / gv;  // one wave of CTAs, each looping over pieces
    const int64_t rounds = (items + (slots < 1 ? 1 : slots) - 1) / (slots < 1 ? 1 : slots);
    const unsigned gy = (unsigned)((items + rounds - 1) / rounds);  // as many CTAs as the longest of them makes worthwhile
    return launch_overlapped("chunk_bwd4_kernel", chunk_same_layout(g) ? chunk_bwd4_kernel<T, true> : chunk_bwd4_kernel<T, false>, dim3(gv, gy), dim3(kChunkThreads), 0, st, g, S, R,
                             nchunks, a.chunk_size, (int)((a.typed_grads & 8) != 0));
  }
  chunk_bwd_kernel<T, PT, 1><<<dim3(gx, nchunks, a.batch), kChunkThreads, 0, st>>>(g, S, nchunks);
  return launch_status("chunk_bwd_kernel");
}

}  // namespace ssmb

using namespace ssmb;

extern "C" int64_t ssm_chunk_scan_scratch_floats(int32_t batch, int32_t len, int32_t heads, int32_t proj, int32_t chunk_size) {
  if (chunk_size < 1) return 0;
  const int64_t piece = chunk_fwd_len(chunk_size, len);
  const int64_t nchunks = (len + piece - 1) / piece;
  return 2 * (int64_t)batch * nchunks * heads * proj;
}

extern "C" int64_t ssm_chunk_scan_bwd_scratch_floats(int32_t batch, int32_t len, int32_t heads, int32_t proj, int32_t chunk_size) {
  if (chunk_size < 1) return 0;
  const int64_t piece = chunk_bwd_len(chunk_size, len);
  const int64_t nchunks = (len + piece - 1) / piece;
  return 3 * (int64_t)batch * nchunks * heads * proj;  // decay products, states entering, adjoints entering every chunk
}

extern "C" int ssm_chunk_scan_bwd_fused(const ssm_chunk_bwd_args* g) {
  if (!g || g->fwd.io_dtype == SSM_F64 || chunk_validate(&g->fwd) || g->fwd.len == 0) return 0;
  const int piece = chunk_bwd_len(g->fwd.chunk_size, g->fwd.len);
  return chunk_bwd_vec_ok(*g, piece, (g->fwd.len + piece - 1) / piece);
}

extern "C" int ssm_chunk_scan_fwd(const ssm_chunk_args* a, ssm_stream_t stream) {
  if (a && a->io_dtype == SSM_F64) {
    ssm_chunk_bwd_args g{};
    g.fwd = *a;
    return f64_chunk(g, false, reinterpret_cast<cudaStream_t>(stream));
  }
  if (int rc = chunk_validate(a)) return rc;
  if (a->batch == 0 || a->heads == 0 || a->proj == 0) return SSM_OK;
  SSM_REQUIRE(a->A.ptr && a->Bm.ptr && a->Cm.ptr, SSM_ERR_NULL, "ssd_chunk_scan: A, B and C are required");
  SSM_REQUIRE(a->len == 0 || (a->X && a->dt && a->Y), SSM_ERR_NULL, "ssd_chunk_scan: X, dt and Y are required");
  SSM_REQUIRE(a->par_dtype == a->io_dtype || a->par_dtype == SSM_F32, SSM_ERR_UNSUPPORTED,
              "ssd_chunk_scan: B, C and z must have the element type of X, or float32");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const bool same = a->par_dtype == a->io_dtype;
  const int cl = chunk_fwd_len(a->chunk_size, a->len);
  switch (a->io_dtype) {
    case SSM_F32: return chunk_fwd_t<float, float>(*a, st, cl);
    case SSM_BF16: return same ? chunk_fwd_t<__nv_bfloat16, __nv_bfloat16>(*a, st, cl) : chunk_fwd_t<__nv_bfloat16, float>(*a, st, cl);
    default: return same ? chunk_fwd_t<__half, __half>(*a, st, cl) : chunk_fwd_t<__half, float>(*a, st, cl);
  }
}

extern "C" int ssm_chunk_scan_bwd(const ssm_chunk_bwd_args* g, ssm_stream_t stream) {
  SSM_REQUIRE(g != nullptr, SSM_ERR_NULL, "ssd_chunk_scan_backward: args is NULL");
  const ssm_chunk_args* a = &g->fwd;
  if (a->io_dtype == SSM_F64) return f64_chunk(*g, true, reinterpret_cast<cudaStream_t>(stream));
  if (int rc = chunk_validate(a)) return rc;
  if (a->batch == 0 || a->heads == 0 || a->proj == 0 || a->len == 0) return SSM_OK;
  SSM_REQUIRE(a->A.ptr && a->Bm.ptr && a->Cm.ptr && a->X && a->dt, SSM_ERR_NULL, "ssd_chunk_scan_backward: missing input");
  SSM_REQUIRE(g->dY && g->dX && g->ddt && g->dA.ptr && g->dB.ptr && g->dC.ptr, SSM_ERR_NULL,
              "ssd_chunk_scan_backward: missing gradient buffer");
  SSM_REQUIRE(!a->z.ptr || g->dz.ptr, SSM_ERR_NULL, "ssd_chunk_scan_backward: dz is required when z is given");
  SSM_REQUIRE((a->typed_grads & ~15) == 0 && (!(a->typed_grads & 1) || bc4_dense_host(g->dB)) && (!(a->typed_grads & 2) || bc4_dense_host(g->dC)) &&
                  (!(a->typed_grads & 4) || (a->z.ptr && bc4_dense_host(g->dz))),
              SSM_ERR_SHAPE, "ssd_chunk_scan_backward: a typed gradient buffer must have no broadcast axis");
  SSM_REQUIRE(a->par_dtype == a->io_dtype || a->par_dtype == SSM_F32, SSM_ERR_UNSUPPORTED,
              "ssd_chunk_scan_backward: B, C and z must have the element type of X, or float32");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const bool same = a->par_dtype == a->io_dtype;
  switch (a->io_dtype) {
    case SSM_F32: return chunk_bwd_t<float, float>(*g, st);
    case SSM_BF16: return same ? chunk_bwd_t<__nv_bfloat16, __nv_bfloat16>(*g, st) : chunk_bwd_t<__nv_bfloat16, float>(*g, st);
    default: return same ? chunk_bwd_t<__half, __half>(*g, st) : chunk_bwd_t<__half, float>(*g, st);
  }
}
