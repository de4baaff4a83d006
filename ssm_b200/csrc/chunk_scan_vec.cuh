// Element-wise chunked recurrence on lanes of neighbouring projections of one head: B, C (and z) of X's element type with the projection
// axis contiguous, as models use the operator.  A scalar lane moves 2 or 4 bytes per instruction and is bound by instruction
// issue.  The forward takes 16 bytes of a row per lane, four fp32 or eight 16-bit projections, and 8 bytes where only those are
// aligned; the backward, which keeps five rows of a step in registers, takes four projections in either element size.
//
// The sequence is cut into pieces of at most kPiece steps (whatever the caller's chunk size: the recurrence does not depend on
// the cut), which is what puts enough independent walks in flight.  Forward: local states, carry over the pieces, replay.
// Backward: the states that enter the pieces are kept from the forward pass (1/32 of X in fp32), so it starts with the local
// adjoints; the final pass then keeps the states of kBwdSub steps in registers while it walks them back, instead of writing
// an fp32 history of the whole sequence and reading it again.
#pragma once

#include "common.cuh"

namespace ssmb {

constexpr int kPiece = 32;  // longest piece of the sequence

// V consecutive elements of a row as one load or store of 8 or 16 bytes
template <typename T, int V>
struct RowRaw {
  static_assert(V * sizeof(T) == 8 || V * sizeof(T) == 16, "one access");
  using type = typename std::conditional<V * sizeof(T) == 16, uint4, uint2>::type;
};
template <typename T, int V>
__device__ __forceinline__ typename RowRaw<T, V>::type ld_row(const T* p) {
  return __ldg(reinterpret_cast<const typename RowRaw<T, V>::type*>(p));
}
// 16-bit elements word by word (see Vec16)
template <typename T, int V>
__device__ __forceinline__ void unpack_row(const typename RowRaw<T, V>::type& r, float (&f)[V]) {
  const uint32_t* w = reinterpret_cast<const uint32_t*>(&r);
#pragma unroll
  for (int i = 0; i < (int)sizeof(r) / 4; ++i) {
    if constexpr (std::is_same<T, float>::value) {
      f[i] = __uint_as_float(w[i]);
    } else if constexpr (std::is_same<T, __nv_bfloat16>::value) {
      f[2 * i] = __uint_as_float(w[i] << 16), f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    } else {
      const float2 v = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
      f[2 * i] = v.x, f[2 * i + 1] = v.y;
    }
  }
}
template <typename T, int V>
__device__ __forceinline__ void store_row(T* p, const float (&f)[V]) {
  typename RowRaw<T, V>::type r;
  uint32_t* w = reinterpret_cast<uint32_t*>(&r);
#pragma unroll
  for (int i = 0; i < (int)sizeof(r) / 4; ++i) {
    if constexpr (std::is_same<T, float>::value) {
      w[i] = __float_as_uint(f[i]);
    } else if constexpr (std::is_same<T, __nv_bfloat16>::value) {
      const __nv_bfloat162 v = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
      w[i] = *reinterpret_cast<const uint32_t*>(&v);
    } else {
      const __half2 v = __floats2half2_rn(f[2 * i], f[2 * i + 1]);
      w[i] = *reinterpret_cast<const uint32_t*>(&v);
    }
  }
  *reinterpret_cast<typename RowRaw<T, V>::type*>(p) = r;
}
__device__ __forceinline__ void load4f(const float* p, float (&f)[4]) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  f[0] = v.x, f[1] = v.y, f[2] = v.z, f[3] = v.w;
}
__device__ __forceinline__ void store4f(float* p, const float (&f)[4]) { *reinterpret_cast<float4*>(p) = make_float4(f[0], f[1], f[2], f[3]); }

template <int V>
__device__ __forceinline__ void load_f32(const float* p, float (&f)[V]) {
#pragma unroll
  for (int i = 0; i < V; i += 4) load4f(p + i, *reinterpret_cast<float(*)[4]>(&f[i]));
}
template <int V>
__device__ __forceinline__ void store_f32(float* p, const float (&f)[V]) {
#pragma unroll
  for (int i = 0; i < V; i += 4) store4f(p + i, *reinterpret_cast<const float(*)[4]>(&f[i]));
}

// Where a thread's piece lies: batch row b, first step t0, n valid steps, rows of X / dY / dX at `row`.
struct Piece4 {
  int b, t0, n, rows;  // rows: steps that exist (n plus those beyond the row's valid length)
  int64_t row, slot;
  __device__ __forceinline__ Piece4(const ssm_chunk_args& a, int nchunks, int len, int b_, int c, int hp) : b(b_) {
    const int HP = a.heads * a.proj;
    t0 = c * len;
    rows = min(a.len - t0, len);
    n = max(0, min(rows, chunk_valid_len(a, b) - t0));
    row = ((int64_t)b * a.len + t0) * HP + hp;
    slot = ((int64_t)b * nchunks + c) * HP + hp;
  }
};

// APPLY false: local end state and decay product of every piece.  APPLY true: the piece replayed from its incoming state, Y written.
// The loads of several steps go out before the first is used.  Bound by instruction issue.  bf16 with gate, us for all launches of
// the forward at (8, 2048, 16, 64) and (4, 4096, 32, 64): lanes of four projections 79 and 133, of eight 62 and 99.
template <typename T, int V, bool APPLY>
__global__ void __launch_bounds__(kChunkThreads) chunk_fwd_row_kernel(const ssm_chunk_args a, int nchunks, int len) {
  constexpr int U = 32 / V;
  using Raw = typename RowRaw<T, V>::type;
  const int HP = a.heads * a.proj;
  const int hp = (blockIdx.x * kChunkThreads + threadIdx.x) * V;
  if (hp >= HP) return;
  const int h = hp / a.proj, q = hp % a.proj;
  const Piece4 pc(a, nchunks, len, blockIdx.z, blockIdx.y, hp);
  float* P = a.scratch + pc.slot;                                    // decay products
  float* S = a.scratch + (int64_t)a.batch * nchunks * HP + pc.slot;  // local end states, then incoming states
  float Av[V], Dv[V], s[V], sumdt = 0.f;
#pragma unroll
  for (int e = 0; e < V; ++e) {
    s[e] = 0.f;
    Av[e] = bc4_load_f32(a.A, 0, 0, h, q + e) * kLog2e;
    Dv[e] = (APPLY && a.D.ptr) ? bc4_load_f32(a.D, 0, 0, h, q + e) : 0.f;
  }
  if (APPLY) load_f32<V>(S, s);
  const T* px = reinterpret_cast<const T*>(a.X) + pc.row;
  const T* pdt = reinterpret_cast<const T*>(a.dt) + ((int64_t)pc.b * a.len + pc.t0) * a.heads + h;
  const T* pB = reinterpret_cast<const T*>(a.Bm.ptr) + bc4_off(a.Bm, pc.b, pc.t0, h, q);
  const T* pC = reinterpret_cast<const T*>(a.Cm.ptr) + bc4_off(a.Cm, pc.b, pc.t0, h, q);
  const bool has_z = APPLY && a.z.ptr != nullptr;
  const T* pz = has_z ? reinterpret_cast<const T*>(a.z.ptr) + bc4_off(a.z, pc.b, pc.t0, h, q) : nullptr;
  T* Y = reinterpret_cast<T*>(a.Y) + pc.row;
  for (int k = 0; k < pc.n; k += U) {
    Raw xr[U], br[U], cr[U], zr[U];
    float d[U];
#pragma unroll
    for (int i = 0; i < U; ++i) {
      const int kk = min(k + i, pc.n - 1);  // beyond the piece: a valid row, dropped below
      xr[i] = ld_row<T, V>(px + (int64_t)kk * HP);
      br[i] = ld_row<T, V>(pB + (int64_t)kk * a.Bm.st);
      if (APPLY) cr[i] = ld_row<T, V>(pC + (int64_t)kk * a.Cm.st);
      if (has_z) zr[i] = ld_row<T, V>(pz + (int64_t)kk * a.z.st);
      d[i] = to_f<T>(__ldg(pdt + (int64_t)kk * a.heads));
    }
#pragma unroll
    for (int i = 0; i < U; ++i) {
      if (k + i >= pc.n) break;
      float x[V], bv[V];
      unpack_row<T, V>(xr[i], x), unpack_row<T, V>(br[i], bv);
#pragma unroll
      for (int e = 0; e < V; ++e) s[e] = fmaf(ex2_approx(d[i] * Av[e]), s[e], d[i] * bv[e] * x[e]);
      sumdt += d[i];
      if (APPLY) {
        float cv[V], y[V];
        unpack_row<T, V>(cr[i], cv);
#pragma unroll
        for (int e = 0; e < V; ++e) y[e] = fmaf(Dv[e], x[e], s[e] * cv[e]);
        if (has_z) {
          float zv[V];
          unpack_row<T, V>(zr[i], zv);
#pragma unroll
          for (int e = 0; e < V; ++e) y[e] *= silu_fast(zv[e]);
        }
        store_row<T, V>(Y + (int64_t)(k + i) * HP, y);
      }
    }
  }
  if (APPLY) {
    const float zero[V] = {};
    for (int k = pc.n; k < pc.rows; ++k) store_row<T, V>(Y + (int64_t)k * HP, zero);
  } else {
    float pr[V];
#pragma unroll
    for (int e = 0; e < V; ++e) pr[e] = ex2_approx(sumdt * Av[e]);
    store_f32<V>(P, pr), store_f32<V>(S, s);
  }
}

// Local adjoint of every piece: what leaves it on its left side when nothing enters on the right.
template <typename T>
__global__ void __launch_bounds__(kChunkThreads) chunk_bwd_local4_kernel(const ssm_chunk_bwd_args g, float* __restrict__ R, int nchunks, int len) {
  constexpr int U = 8;
  using Raw = typename RowRaw<T, 4>::type;
  const ssm_chunk_args& a = g.fwd;
  const int HP = a.heads * a.proj;
  const int hp = (blockIdx.x * kChunkThreads + threadIdx.x) * 4;
  if (hp >= HP) return;
  const int h = hp / a.proj, q = hp % a.proj;
  const Piece4 pc(a, nchunks, len, blockIdx.z, blockIdx.y, hp);
  float Av[4], carry[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int e = 0; e < 4; ++e) Av[e] = bc4_load_f32(a.A, 0, 0, h, q + e) * kLog2e;
  const T* pdy = reinterpret_cast<const T*>(g.dY) + pc.row;
  const T* pdt = reinterpret_cast<const T*>(a.dt) + ((int64_t)pc.b * a.len + pc.t0) * a.heads + h;
  const T* pC = reinterpret_cast<const T*>(a.Cm.ptr) + bc4_off(a.Cm, pc.b, pc.t0, h, q);
  const bool has_z = a.z.ptr != nullptr;
  const T* pz = has_z ? reinterpret_cast<const T*>(a.z.ptr) + bc4_off(a.z, pc.b, pc.t0, h, q) : nullptr;
  for (int k = pc.n; k > 0; k -= U) {
    Raw gr[U], cr[U], zr[U];
    float d[U];
#pragma unroll
    for (int i = 0; i < U; ++i) {
      const int kk = max(k - 1 - i, 0);
      gr[i] = ld_row<T, 4>(pdy + (int64_t)kk * HP);
      cr[i] = ld_row<T, 4>(pC + (int64_t)kk * a.Cm.st);
      if (has_z) zr[i] = ld_row<T, 4>(pz + (int64_t)kk * a.z.st);
      d[i] = to_f<T>(__ldg(pdt + (int64_t)kk * a.heads));
    }
#pragma unroll
    for (int i = 0; i < U; ++i) {
      if (k - 1 - i < 0) break;
      float dout[4], cv[4], zv[4];
      unpack_row<T, 4>(gr[i], dout), unpack_row<T, 4>(cr[i], cv);
      if (has_z) {
        unpack_row<T, 4>(zr[i], zv);
#pragma unroll
        for (int e = 0; e < 4; ++e) dout[e] *= silu_fast(zv[e]);
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) carry[e] = ex2_approx(d[i] * Av[e]) * fmaf(cv[e], dout[e], carry[e]);
    }
  }
  store4f(R + pc.slot, carry);
}

// Final backward pass.  A piece is walked back in groups of kBwdSub steps whose states stay in registers: the states that enter the
// groups come from one forward sweep over all but the last group, each group is then replayed and walked back while the loads
// of the group to its left are under way.  CTAs keep their projections and loop over pieces, so that the sums over batch and
// time (dA, dD) cost one addition per CTA and lane instead of one per piece (additions to one word are served one after the
// other, about 40 ns each).  Bound by latency: X, B (twice, the second time from the L2), C, z, dY in, dX, dB, dC, dz out, 302 MB
// in 110 us at (8, 2048, 16, 64) bf16.  The scalar pass with an fp32 history took 196 us; groups of 16 steps without requests
// ahead 163, of 8 131, of 4 123, of 2 with requests ahead 115, with rows converted word by word 110.
constexpr int kBwdSub = 2;    // steps of a group
constexpr int kBwdSweep = 8;  // steps per batch of loads of the forward sweep
template <typename T>
constexpr int bwd4_ctas() {  // resident CTAs per SM: what the registers of the rows in flight leave room for
  return sizeof(T) == 2 ? 4 : 3;
}
template <typename T>
__global__ void __launch_bounds__(kChunkThreads, bwd4_ctas<T>()) chunk_bwd4_kernel(const ssm_chunk_bwd_args g, const float* __restrict__ S, const float* __restrict__ R,
                                                                      int nchunks, int len, int typed_dt) {
  constexpr int SUB = kBwdSub, NG = kPiece / SUB, UF = kBwdSweep;
  using Raw = typename RowRaw<T, 4>::type;
  __shared__ float4 entry[NG][kChunkThreads];  // the state that enters each group of steps
  const ssm_chunk_args& a = g.fwd;
  const int HP = a.heads * a.proj;
  const int hp_raw = (blockIdx.x * kChunkThreads + threadIdx.x) * 4;
  const bool active = hp_raw < HP;
  const int hp = active ? hp_raw : HP - 4;  // idle threads of the last CTA shadow a valid lane and write nothing
  const int h = hp / a.proj, q = hp % a.proj;
  const int share = a.proj / 4;             // neighbouring threads with this head: a power of two, at most a warp (the launcher checks)
  const bool has_z = a.z.ptr != nullptr;
  float Av[4], Dv[4], dA[4] = {0.f, 0.f, 0.f, 0.f}, dD[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    Av[e] = bc4_load_f32(a.A, 0, 0, h, q + e) * kLog2e;
    Dv[e] = a.D.ptr ? bc4_load_f32(a.D, 0, 0, h, q + e) : 0.f;
  }
  const Raw zero_raw{};
  for (int item = blockIdx.y; item < a.batch * nchunks; item += gridDim.y) {
    const Piece4 pc(a, nchunks, len, item / nchunks, item % nchunks, hp);
    const T* px = reinterpret_cast<const T*>(a.X) + pc.row;
    const T* pdy = reinterpret_cast<const T*>(g.dY) + pc.row;
    const T* pdt = reinterpret_cast<const T*>(a.dt) + ((int64_t)pc.b * a.len + pc.t0) * a.heads + h;
    const T* pB = reinterpret_cast<const T*>(a.Bm.ptr) + bc4_off(a.Bm, pc.b, pc.t0, h, q);
    const T* pC = reinterpret_cast<const T*>(a.Cm.ptr) + bc4_off(a.Cm, pc.b, pc.t0, h, q);
    const T* pz = has_z ? reinterpret_cast<const T*>(a.z.ptr) + bc4_off(a.z, pc.b, pc.t0, h, q) : nullptr;
    T* dX = reinterpret_cast<T*>(g.dX) + pc.row;
    auto out = [&](const ssm_bcast4& p) { return const_cast<T*>(reinterpret_cast<const T*>(p.ptr)) + bc4_off(p, pc.b, pc.t0, h, q); };
    T *dB = out(g.dB), *dC = out(g.dC), *dZ = has_z ? out(g.dz) : nullptr;
    float s[4], carry[4];
    load4f(S + pc.slot, s), load4f(R + pc.slot, carry);
    // steps beyond the valid length enter as zeros: no decay, no input, no gradient, and zeros are what is written there
    const int groups = (pc.rows + SUB - 1) / SUB, sweep = (groups - 1) * SUB;
    entry[0][threadIdx.x] = make_float4(s[0], s[1], s[2], s[3]);
    for (int k = 0; k < sweep; k += UF) {
      Raw xr[UF], br[UF];
      float d[UF];
#pragma unroll
      for (int i = 0; i < UF; ++i) {
        const bool in = k + i < min(pc.n, sweep);
        xr[i] = in ? ld_row<T, 4>(px + (int64_t)(k + i) * HP) : zero_raw;
        br[i] = in ? ld_row<T, 4>(pB + (int64_t)(k + i) * a.Bm.st) : zero_raw;
        d[i] = in ? to_f<T>(__ldg(pdt + (int64_t)(k + i) * a.heads)) : 0.f;
      }
#pragma unroll
      for (int i = 0; i < UF; ++i) {
        float x[4], bv[4];
        unpack_row<T, 4>(xr[i], x), unpack_row<T, 4>(br[i], bv);
#pragma unroll
        for (int e = 0; e < 4; ++e) s[e] = fmaf(ex2_approx(d[i] * Av[e]), s[e], d[i] * bv[e] * x[e]);
        if ((i + 1) % SUB == 0 && k + i < sweep) entry[(k + i + 1) / SUB][threadIdx.x] = make_float4(s[0], s[1], s[2], s[3]);
      }
    }
    // the loads of the next group (to the left) go out before this one is worked on: X and B come back from the L2, C, z, dY from HBM
    Raw nx[SUB], nbr[SUB], nc[SUB], nz[SUB], ng[SUB];
    float nd[SUB];
    auto request = [&](int k0) {
#pragma unroll
      for (int i = 0; i < SUB; ++i) {
        const bool in = k0 + i >= 0 && k0 + i < pc.n;
        nx[i] = in ? ld_row<T, 4>(px + (int64_t)(k0 + i) * HP) : zero_raw;
        nbr[i] = in ? ld_row<T, 4>(pB + (int64_t)(k0 + i) * a.Bm.st) : zero_raw;
        nc[i] = in ? ld_row<T, 4>(pC + (int64_t)(k0 + i) * a.Cm.st) : zero_raw;
        ng[i] = in ? ld_row<T, 4>(pdy + (int64_t)(k0 + i) * HP) : zero_raw;
        nz[i] = in && has_z ? ld_row<T, 4>(pz + (int64_t)(k0 + i) * a.z.st) : zero_raw;
        nd[i] = in ? to_f<T>(__ldg(pdt + (int64_t)(k0 + i) * a.heads)) : 0.f;
      }
    };
    request((groups - 1) * SUB);
#pragma unroll 1
    for (int blk = groups - 1; blk >= 0; --blk) {
      const int k0 = blk * SUB;
      Raw xr[SUB], br[SUB], cr[SUB], zr[SUB], gr[SUB];
      float d[SUB], st[SUB + 1][4];  // st[i]: the state before step k0 + i
#pragma unroll
      for (int i = 0; i < SUB; ++i) xr[i] = nx[i], br[i] = nbr[i], cr[i] = nc[i], zr[i] = nz[i], gr[i] = ng[i], d[i] = nd[i];
      request(k0 - SUB);
      {
        const float4 v = entry[blk][threadIdx.x];
        st[0][0] = v.x, st[0][1] = v.y, st[0][2] = v.z, st[0][3] = v.w;
      }
#pragma unroll
      for (int i = 0; i < SUB; ++i) {
        float x[4], bv[4];
        unpack_row<T, 4>(xr[i], x), unpack_row<T, 4>(br[i], bv);
#pragma unroll
        for (int e = 0; e < 4; ++e) st[i + 1][e] = fmaf(ex2_approx(d[i] * Av[e]), st[i][e], d[i] * bv[e] * x[e]);
      }
#pragma unroll
      for (int i = SUB - 1; i >= 0; --i) {
        const int k = k0 + i;
        float x[4], bv[4], cv[4], dy[4], dxo[4], dbo[4], dco[4], ddt = 0.f;
        unpack_row<T, 4>(xr[i], x), unpack_row<T, 4>(br[i], bv), unpack_row<T, 4>(cr[i], cv), unpack_row<T, 4>(gr[i], dy);
        if (has_z) {
          float zv[4], dzo[4];
          unpack_row<T, 4>(zr[i], zv);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float sg = sigmoid_fast(zv[e]);
            dzo[e] = dy[e] * fmaf(Dv[e], x[e], st[i + 1][e] * cv[e]) * sg * (1.f + zv[e] * (1.f - sg));
            dy[e] *= zv[e] * sg;
          }
          if (active && k < pc.rows) store_row<T, 4>(dZ + (int64_t)k * g.dz.st, dzo);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float da = ex2_approx(d[i] * Av[e]);
          const float G = fmaf(cv[e], dy[e], carry[e]);
          dco[e] = dy[e] * st[i + 1][e];
          dbo[e] = G * d[i] * x[e];
          dxo[e] = fmaf(dy[e], Dv[e], G * d[i] * bv[e]);
          carry[e] = G * da;
          const float gsa = st[i][e] * carry[e];
          ddt += fmaf(G, bv[e] * x[e], gsa * (Av[e] * kLn2));
          dA[e] = fmaf(gsa, d[i], dA[e]);
          dD[e] = fmaf(dy[e], x[e], dD[e]);
        }
        if (active && k < pc.rows) {
          store_row<T, 4>(dC + (int64_t)k * g.dC.st, dco);
          store_row<T, 4>(dB + (int64_t)k * g.dB.st, dbo);
          store_row<T, 4>(dX + (int64_t)k * HP, dxo);
        }
        for (int o = 1; o < share; o <<= 1) ddt += __shfl_xor_sync(0xffffffffu, ddt, o);
        if (active && k < pc.rows && (threadIdx.x & (share - 1)) == 0) {
          const int64_t at = ((int64_t)pc.b * a.len + pc.t0 + k) * a.heads + h;
          const float v = k < pc.n ? ddt : 0.f;
          if (typed_dt) reinterpret_cast<T*>(g.ddt)[at] = from_f<T>(v);
          else reinterpret_cast<float*>(g.ddt)[at] = v;
        }
      }
    }
  }
  if (g.dD.ptr && a.D.sq == 0) {  // one skip weight per head
    float t = active ? (dD[0] + dD[1]) + (dD[2] + dD[3]) : 0.f;
    for (int o = 1; o < share; o <<= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (active && (threadIdx.x & (share - 1)) == 0) atomicAdd(bc4_ptr(g.dD, 0, 0, h, 0), t);
  }
  if (!active) return;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    atomicAdd(bc4_ptr(g.dA, 0, 0, h, q + e), dA[e]);
    if (g.dD.ptr && a.D.sq != 0) atomicAdd(bc4_ptr(g.dD, 0, 0, h, q + e), dD[e]);
  }
}

}  // namespace ssmb
