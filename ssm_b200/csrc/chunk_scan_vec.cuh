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
// the same as pairs of neighbouring projections, the operands of the packed fp32 instructions
template <typename T, int V>
__device__ __forceinline__ void unpack_pairs(const typename RowRaw<T, V>::type& r, float2 (&f)[V / 2]) {
  float v[V];
  unpack_row<T, V>(r, v);
#pragma unroll
  for (int i = 0; i < V / 2; ++i) f[i] = make_float2(v[2 * i], v[2 * i + 1]);
}
template <typename T, int V>
__device__ __forceinline__ void store_pairs(T* p, const float2 (&f)[V / 2]) {
  float v[V];
#pragma unroll
  for (int i = 0; i < V / 2; ++i) v[2 * i] = f[i].x, v[2 * i + 1] = f[i].y;
  store_row<T, V>(p, v);
}
__device__ __forceinline__ float2 both(float x) { return make_float2(x, x); }
__device__ __forceinline__ float2 ex2_pair(float2 e) { return make_float2(ex2_approx(e.x), ex2_approx(e.y)); }
__device__ __forceinline__ float2 sigmoid_pair(float2 z) {
  const float2 den = __fadd2_rn(ex2_pair(__fmul2_rn(z, both(-kLog2e))), both(1.f));
  return make_float2(rcp_approx(den.x), rcp_approx(den.y));
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
// The loads of U steps go out before the first is used, in the local pass (two rows per step, bound by the latency of its loads) while
// the U steps before them are worked on: (8, 2048, 16, 64) bf16, 67 MB, 29.6 -> 19.1 us.  The second pass moves 168 MB in 30 us.
// Lanes of four projections instead of eight take 19.3 and 32.0 us.
template <typename T, int V, bool APPLY>
__global__ void __launch_bounds__(kChunkThreads) chunk_fwd_row_kernel(const ssm_chunk_args a, int nchunks, int len) {
  pdl_wait();
  pdl_trigger();
  constexpr int U = 32 / V, P2 = V / 2;
  using Raw = typename RowRaw<T, V>::type;
  const int HP = a.heads * a.proj;
  const int hp = (blockIdx.x * kChunkThreads + threadIdx.x) * V;
  if (hp >= HP) return;
  const int h = hp / a.proj, q = hp % a.proj;
  const Piece4 pc(a, nchunks, len, blockIdx.z, blockIdx.y, hp);
  float* P = a.scratch + pc.slot;                                    // decay products
  float* S = a.scratch + (int64_t)a.batch * nchunks * HP + pc.slot;  // local end states, then incoming states
  float s0[V] = {}, sumdt = 0.f;
  float2 Av[P2], Dv[P2], s[P2];
  if (APPLY) load_f32<V>(S, s0);
#pragma unroll
  for (int e = 0; e < P2; ++e) {
    s[e] = make_float2(s0[2 * e], s0[2 * e + 1]);
    Av[e] = make_float2(bc4_load_f32(a.A, 0, 0, h, q + 2 * e) * kLog2e, bc4_load_f32(a.A, 0, 0, h, q + 2 * e + 1) * kLog2e);
    Dv[e] = (APPLY && a.D.ptr) ? make_float2(bc4_load_f32(a.D, 0, 0, h, q + 2 * e), bc4_load_f32(a.D, 0, 0, h, q + 2 * e + 1)) : both(0.f);
  }
  const T* px = reinterpret_cast<const T*>(a.X) + pc.row;
  const T* pdt = reinterpret_cast<const T*>(a.dt) + ((int64_t)pc.b * a.len + pc.t0) * a.heads + h;
  const T* pB = reinterpret_cast<const T*>(a.Bm.ptr) + bc4_off(a.Bm, pc.b, pc.t0, h, q);
  const T* pC = reinterpret_cast<const T*>(a.Cm.ptr) + bc4_off(a.Cm, pc.b, pc.t0, h, q);
  const bool has_z = APPLY && a.z.ptr != nullptr;
  const T* pz = has_z ? reinterpret_cast<const T*>(a.z.ptr) + bc4_off(a.z, pc.b, pc.t0, h, q) : nullptr;
  T* Y = reinterpret_cast<T*>(a.Y) + pc.row;
  Raw xr[U], br[U], cr[U], zr[U];
  float d[U];
  auto request = [&](int k) {
#pragma unroll
    for (int i = 0; i < U; ++i) {
      const int kk = min(k + i, pc.n - 1);  // beyond the piece: a valid row, dropped below
      xr[i] = ld_row<T, V>(px + (int64_t)kk * HP);
      br[i] = ld_row<T, V>(pB + (int64_t)kk * a.Bm.st);
      if (APPLY) cr[i] = ld_row<T, V>(pC + (int64_t)kk * a.Cm.st);
      if (has_z) zr[i] = ld_row<T, V>(pz + (int64_t)kk * a.z.st);
      d[i] = to_f<T>(__ldg(pdt + (int64_t)kk * a.heads));
    }
  };
  if (!APPLY && pc.n > 0) request(0);
#pragma unroll 1
  for (int k = 0; k < pc.n; k += U) {
    if (APPLY) request(k);
    Raw xc[U], bc[U];
    float dc[U];
#pragma unroll
    for (int i = 0; i < U; ++i) xc[i] = xr[i], bc[i] = br[i], dc[i] = d[i];
    if (!APPLY && k + U < pc.n) request(k + U);
#pragma unroll
    for (int i = 0; i < U; ++i) {
      if (k + i >= pc.n) break;
      float2 x[P2], bv[P2];
      unpack_pairs<T, V>(xc[i], x), unpack_pairs<T, V>(bc[i], bv);
#pragma unroll
      for (int e = 0; e < P2; ++e) s[e] = __ffma2_rn(ex2_pair(__fmul2_rn(both(dc[i]), Av[e])), s[e], __fmul2_rn(__fmul2_rn(both(dc[i]), bv[e]), x[e]));
      sumdt += dc[i];
      if (APPLY) {
        float2 cv[P2], y[P2];
        unpack_pairs<T, V>(cr[i], cv);
#pragma unroll
        for (int e = 0; e < P2; ++e) y[e] = __ffma2_rn(Dv[e], x[e], __fmul2_rn(s[e], cv[e]));
        if (has_z) {
          float2 zv[P2];
          unpack_pairs<T, V>(zr[i], zv);
#pragma unroll
          for (int e = 0; e < P2; ++e) y[e] = __fmul2_rn(y[e], __fmul2_rn(zv[e], sigmoid_pair(zv[e])));
        }
        store_pairs<T, V>(Y + (int64_t)(k + i) * HP, y);
      }
    }
  }
  if (APPLY) {
    const float zero[V] = {};
    for (int k = pc.n; k < pc.rows; ++k) store_row<T, V>(Y + (int64_t)k * HP, zero);
  } else {
    float pr[V];
#pragma unroll
    for (int e = 0; e < P2; ++e) {
      const float2 v = ex2_pair(__fmul2_rn(both(sumdt), Av[e]));
      pr[2 * e] = v.x, pr[2 * e + 1] = v.y, s0[2 * e] = s[e].x, s0[2 * e + 1] = s[e].y;
    }
    store_f32<V>(P, pr), store_f32<V>(S, s0);
  }
}

// Local adjoint of every piece: what leaves it on its left side when nothing enters on the right.  Three rows per step keep enough
// bytes in flight without requests ahead, and the registers these take cost resident warps: (8, 2048, 16, 64) bf16, 101 MB, 24.0 us,
// 29.0 with them; lanes of four projections 25.6.
template <typename T, int V>
__global__ void __launch_bounds__(kChunkThreads) chunk_bwd_local_row_kernel(const ssm_chunk_bwd_args g, float* __restrict__ R, int nchunks, int len) {
  pdl_wait();
  pdl_trigger();
  constexpr int U = 32 / V, P2 = V / 2;
  using Raw = typename RowRaw<T, V>::type;
  const ssm_chunk_args& a = g.fwd;
  const int HP = a.heads * a.proj;
  const int hp = (blockIdx.x * kChunkThreads + threadIdx.x) * V;
  if (hp >= HP) return;
  const int h = hp / a.proj, q = hp % a.proj;
  const Piece4 pc(a, nchunks, len, blockIdx.z, blockIdx.y, hp);
  float2 Av[P2], carry[P2];
#pragma unroll
  for (int e = 0; e < P2; ++e) {
    Av[e] = make_float2(bc4_load_f32(a.A, 0, 0, h, q + 2 * e) * kLog2e, bc4_load_f32(a.A, 0, 0, h, q + 2 * e + 1) * kLog2e);
    carry[e] = both(0.f);
  }
  const T* pdy = reinterpret_cast<const T*>(g.dY) + pc.row;
  const T* pdt = reinterpret_cast<const T*>(a.dt) + ((int64_t)pc.b * a.len + pc.t0) * a.heads + h;
  const T* pC = reinterpret_cast<const T*>(a.Cm.ptr) + bc4_off(a.Cm, pc.b, pc.t0, h, q);
  const bool has_z = a.z.ptr != nullptr;
  const T* pz = has_z ? reinterpret_cast<const T*>(a.z.ptr) + bc4_off(a.z, pc.b, pc.t0, h, q) : nullptr;
  Raw gr[U], cr[U], zr[U];
  float d[U];
  auto request = [&](int k) {  // steps k - 1, k - 2, ...
#pragma unroll
    for (int i = 0; i < U; ++i) {
      const int kk = max(k - 1 - i, 0);
      gr[i] = ld_row<T, V>(pdy + (int64_t)kk * HP);
      cr[i] = ld_row<T, V>(pC + (int64_t)kk * a.Cm.st);
      if (has_z) zr[i] = ld_row<T, V>(pz + (int64_t)kk * a.z.st);
      d[i] = to_f<T>(__ldg(pdt + (int64_t)kk * a.heads));
    }
  };
#pragma unroll 1
  for (int k = pc.n; k > 0; k -= U) {
    request(k);
#pragma unroll
    for (int i = 0; i < U; ++i) {
      if (k - 1 - i < 0) break;
      float2 dout[P2], cv[P2], zv[P2];
      unpack_pairs<T, V>(gr[i], dout), unpack_pairs<T, V>(cr[i], cv);
      if (has_z) {
        unpack_pairs<T, V>(zr[i], zv);
#pragma unroll
        for (int e = 0; e < P2; ++e) dout[e] = __fmul2_rn(dout[e], __fmul2_rn(zv[e], sigmoid_pair(zv[e])));
      }
#pragma unroll
      for (int e = 0; e < P2; ++e) carry[e] = __fmul2_rn(ex2_pair(__fmul2_rn(both(d[i]), Av[e])), __ffma2_rn(cv[e], dout[e], carry[e]));
    }
  }
  float out[V];
#pragma unroll
  for (int e = 0; e < P2; ++e) out[2 * e] = carry[e].x, out[2 * e + 1] = carry[e].y;
  store_f32<V>(R + pc.slot, out);
}

// Final backward pass.  A piece is walked back in groups of kBwdSub steps whose states stay in registers: the states that enter the
// groups come from one forward sweep over all but the last group, each group is then replayed and walked back while the loads
// of the group to its left are under way.  CTAs keep their projections and loop over pieces, so that the sums over batch and
// time (dA, dD) cost one addition per CTA and lane instead of one per piece (additions to one word are served one after the
// other, about 40 ns each).  Arithmetic on pairs of projections (packed fp32), no guards in the walk (rows beyond the piece are clamped
// and the one step that needs it is zeroed under a uniform branch).  SAME: every row tensor has X's layout and fits 32-bit byte
// offsets, so that a step has one offset for its nine rows instead of nine 64-bit addresses.
// Moves X, B (twice, the second time from the L2), C, z, dY in, dX, dB, dC, dz out: 302 MB at (8, 2048, 16, 64) bf16 in 75 us (scalar
// arithmetic, guards and an address per row: 126 instructions per element, 107 us).
constexpr int kBwdSub = 2;    // steps of a group
constexpr int kBwdSweep = 8;  // steps per batch of loads of the forward sweep
template <typename T>
constexpr int bwd4_ctas() {  // resident CTAs per SM: what the registers of the rows in flight leave room for
  return sizeof(T) == 2 ? 4 : 3;
}
template <typename T, bool SAME>
__global__ void __launch_bounds__(kChunkThreads, bwd4_ctas<T>()) chunk_bwd4_kernel(const ssm_chunk_bwd_args g, const float* __restrict__ S, const float* __restrict__ R,
                                                                      int nchunks, int len, int typed_dt) {
  pdl_wait();
  pdl_trigger();
  constexpr int SUB = kBwdSub, NG = kPiece / SUB, UF = kBwdSweep;
  static_assert(SUB == 2, "the sums of a group's two steps share their shuffles");
  using Raw = typename RowRaw<T, 4>::type;
  __shared__ float4 entry[NG][kChunkThreads];  // the state that enters each group of steps
  const ssm_chunk_args& a = g.fwd;
  const int HP = a.heads * a.proj;
  const int hp_raw = (blockIdx.x * kChunkThreads + threadIdx.x) * 4;
  const bool active = hp_raw < HP;
  const int hp = active ? hp_raw : HP - 4;  // idle threads of the last CTA shadow a valid lane and write nothing
  const int h = hp / a.proj, q = hp % a.proj;
  const int share = a.proj / 4;             // neighbouring threads with this head: a power of two, at most a warp (the launcher checks)
  const int at_share = threadIdx.x & (share - 1);
  const bool has_z = a.z.ptr != nullptr;
  float2 Av[2], Dv[2], dA[2], dD[2];
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    Av[e] = make_float2(bc4_load_f32(a.A, 0, 0, h, q + 2 * e) * kLog2e, bc4_load_f32(a.A, 0, 0, h, q + 2 * e + 1) * kLog2e);
    Dv[e] = a.D.ptr ? make_float2(bc4_load_f32(a.D, 0, 0, h, q + 2 * e), bc4_load_f32(a.D, 0, 0, h, q + 2 * e + 1)) : both(0.f);
    dA[e] = dD[e] = both(0.f);
  }
  const Raw zero_raw{};
  for (int item = blockIdx.y; item < a.batch * nchunks; item += gridDim.y) {
    const Piece4 pc(a, nchunks, len, item / nchunks, item % nchunks, hp);
    const int64_t dt0 = ((int64_t)pc.b * a.len + pc.t0) * a.heads + h;
    // this lane's row of step k of a tensor: `base` and the piece's offset in it
    const uint32_t off0 = (uint32_t)pc.row * (uint32_t)sizeof(T), pitch = (uint32_t)HP * (uint32_t)sizeof(T);
    auto at = [&](const void* base, int64_t off, int64_t st, int k) {
      if constexpr (SAME) return reinterpret_cast<const T*>(reinterpret_cast<const char*>(base) + (off0 + (uint32_t)k * pitch));
      else return reinterpret_cast<const T*>(base) + (off + (int64_t)k * st);
    };
    auto off4 = [&](const ssm_bcast4& p) { return SAME ? (int64_t)0 : bc4_off(p, pc.b, pc.t0, h, q); };
    const int64_t oB = off4(a.Bm), oC = off4(a.Cm), oz = off4(a.z), odB = off4(g.dB), odC = off4(g.dC), odz = off4(g.dz);
    auto out = [&](const void* base, int64_t off, int64_t st, int k) { return const_cast<T*>(at(base, off, st, k)); };
    if (active) {  // steps beyond the valid length
      const float2 zero[2] = {both(0.f), both(0.f)};
      for (int k = pc.n; k < pc.rows; ++k) {
        store_pairs<T, 4>(out(g.dX, pc.row, HP, k), zero), store_pairs<T, 4>(out(g.dB.ptr, odB, g.dB.st, k), zero), store_pairs<T, 4>(out(g.dC.ptr, odC, g.dC.st, k), zero);
        if (has_z) store_pairs<T, 4>(out(g.dz.ptr, odz, g.dz.st, k), zero);
        if (at_share == 0) {
          if (typed_dt) reinterpret_cast<T*>(g.ddt)[dt0 + (int64_t)k * a.heads] = from_f<T>(0.f);
          else reinterpret_cast<float*>(g.ddt)[dt0 + (int64_t)k * a.heads] = 0.f;
        }
      }
    }
    if (pc.n <= 0) continue;
    const T* pdt = reinterpret_cast<const T*>(a.dt) + dt0;
    auto load_dt = [&](int k) { return to_f<T>(__ldg(pdt + (SAME ? (uint32_t)k * (uint32_t)a.heads : (int64_t)k * a.heads))); };

    // the loads of the next group (to the left) go out before this one is worked on: X and B come back from the L2, C, z, dY from HBM
    Raw nx[SUB], nbr[SUB], nc[SUB], nz[SUB], ng[SUB];
    float nd[SUB];
    auto request = [&](int k0) {
#pragma unroll
      for (int i = 0; i < SUB; ++i) {
        const int k = min(max(k0 + i, 0), pc.n - 1);
        nx[i] = ld_row<T, 4>(at(a.X, pc.row, HP, k));
        nbr[i] = ld_row<T, 4>(at(a.Bm.ptr, oB, a.Bm.st, k));
        nc[i] = ld_row<T, 4>(at(a.Cm.ptr, oC, a.Cm.st, k));
        ng[i] = ld_row<T, 4>(at(g.dY, pc.row, HP, k));
        nz[i] = has_z ? ld_row<T, 4>(at(a.z.ptr, oz, a.z.st, k)) : zero_raw;
        nd[i] = load_dt(k);
      }
    };
    const int groups = (pc.n + SUB - 1) / SUB, sweep = (groups - 1) * SUB;
    request(sweep);
    if (sweep + SUB > pc.n) {  // the piece ends inside the group: no decay, no input, no gradient
#pragma unroll
      for (int i = 0; i < SUB; ++i)
        if (sweep + i >= pc.n) nx[i] = nbr[i] = nc[i] = ng[i] = nz[i] = zero_raw, nd[i] = 0.f;
    }
    float2 carry[2];
    {
      float s4[4], c4[4];
      load4f(S + pc.slot, s4), load4f(R + pc.slot, c4);
      float2 s[2] = {make_float2(s4[0], s4[1]), make_float2(s4[2], s4[3])};
      carry[0] = make_float2(c4[0], c4[1]), carry[1] = make_float2(c4[2], c4[3]);
      entry[0][threadIdx.x] = make_float4(s4[0], s4[1], s4[2], s4[3]);
      for (int k = 0; k < sweep; k += UF) {
        Raw xr[UF], br[UF];
        float d[UF];
#pragma unroll
        for (int i = 0; i < UF; ++i) {
          const int kk = min(k + i, pc.n - 1);
          xr[i] = ld_row<T, 4>(at(a.X, pc.row, HP, kk));
          br[i] = ld_row<T, 4>(at(a.Bm.ptr, oB, a.Bm.st, kk));
          d[i] = load_dt(kk);
        }
#pragma unroll
        for (int i = 0; i < UF; ++i) {
          if (k + i / SUB * SUB >= sweep) break;
          float2 x[2], bv[2];
          unpack_pairs<T, 4>(xr[i], x), unpack_pairs<T, 4>(br[i], bv);
#pragma unroll
          for (int e = 0; e < 2; ++e) s[e] = __ffma2_rn(ex2_pair(__fmul2_rn(both(d[i]), Av[e])), s[e], __fmul2_rn(__fmul2_rn(both(d[i]), bv[e]), x[e]));
          if ((i + 1) % SUB == 0) entry[(k + i + 1) / SUB][threadIdx.x] = make_float4(s[0].x, s[0].y, s[1].x, s[1].y);
        }
      }
    }
#pragma unroll 1
    for (int blk = groups - 1; blk >= 0; --blk) {
      const int k0 = blk * SUB;
      float2 x[SUB][2], bv[SUB][2], cv[SUB][2], dy[SUB][2], zv[SUB][2], st[SUB + 1][2], da[SUB][2];  // st[i]: the state before step k0 + i
      float d[SUB], ddt[SUB];
#pragma unroll
      for (int i = 0; i < SUB; ++i) {
        unpack_pairs<T, 4>(nx[i], x[i]), unpack_pairs<T, 4>(nbr[i], bv[i]), unpack_pairs<T, 4>(nc[i], cv[i]), unpack_pairs<T, 4>(ng[i], dy[i]);
        if (has_z) unpack_pairs<T, 4>(nz[i], zv[i]);
        d[i] = nd[i];
      }
      request(k0 - SUB);
      {
        const float4 v = entry[blk][threadIdx.x];
        st[0][0] = make_float2(v.x, v.y), st[0][1] = make_float2(v.z, v.w);
      }
#pragma unroll
      for (int i = 0; i < SUB; ++i) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          da[i][e] = ex2_pair(__fmul2_rn(both(d[i]), Av[e]));
          st[i + 1][e] = __ffma2_rn(da[i][e], st[i][e], __fmul2_rn(__fmul2_rn(both(d[i]), bv[i][e]), x[i][e]));
        }
      }
#pragma unroll
      for (int i = SUB - 1; i >= 0; --i) {
        const int k = k0 + i;
        const bool write = active && k < pc.n;
        if (has_z) {
          float2 dzo[2];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const float2 one = both(1.f), sg = sigmoid_pair(zv[i][e]);
            const float2 y = __ffma2_rn(Dv[e], x[i][e], __fmul2_rn(st[i + 1][e], cv[i][e]));
            const float2 zs = __fmul2_rn(zv[i][e], sg);                                   // silu(z)
            const float2 ds = __ffma2_rn(zs, __ffma2_rn(both(-1.f), sg, one), sg);        // silu'(z) = sg + z sg (1 - sg)
            dzo[e] = __fmul2_rn(__fmul2_rn(dy[i][e], y), ds);
            dy[i][e] = __fmul2_rn(dy[i][e], zs);
          }
          if (write) store_pairs<T, 4>(out(g.dz.ptr, odz, g.dz.st, k), dzo);
        }
        float2 dxo[2], dbo[2], dco[2], sum = both(0.f);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float2 G = __ffma2_rn(cv[i][e], dy[i][e], carry[e]), Gd = __fmul2_rn(G, both(d[i]));
          dco[e] = __fmul2_rn(dy[i][e], st[i + 1][e]);
          dbo[e] = __fmul2_rn(Gd, x[i][e]);
          dxo[e] = __ffma2_rn(Gd, bv[i][e], __fmul2_rn(dy[i][e], Dv[e]));
          carry[e] = __fmul2_rn(G, da[i][e]);
          const float2 gsa = __fmul2_rn(st[i][e], carry[e]);
          sum = __ffma2_rn(G, __fmul2_rn(bv[i][e], x[i][e]), sum);
          sum = __ffma2_rn(gsa, __fmul2_rn(Av[e], both(kLn2)), sum);
          dA[e] = __ffma2_rn(gsa, both(d[i]), dA[e]);
          dD[e] = __ffma2_rn(dy[i][e], x[i][e], dD[e]);
        }
        if (write) {
          store_pairs<T, 4>(out(g.dC.ptr, odC, g.dC.st, k), dco);
          store_pairs<T, 4>(out(g.dB.ptr, odB, g.dB.st, k), dbo);
          store_pairs<T, 4>(out(g.dX, pc.row, HP, k), dxo);
        }
        ddt[i] = sum.x + sum.y;
      }
      // over the head's projections: even lanes go on with the first step's sum, odd lanes with the second's
      auto put = [&](int k, float v) {
        if (!active || k >= pc.n) return;
        const int64_t to = dt0 + (int64_t)k * a.heads;
        if (typed_dt) reinterpret_cast<T*>(g.ddt)[to] = from_f<T>(v);
        else reinterpret_cast<float*>(g.ddt)[to] = v;
      };
      if (share > 1) {
        const bool odd = threadIdx.x & 1;
        float v = (odd ? ddt[1] : ddt[0]) + __shfl_xor_sync(0xffffffffu, odd ? ddt[0] : ddt[1], 1);
#pragma unroll
        for (int o = 2; o < 32; o <<= 1)
          if (o < share) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (at_share < 2) put(k0 + at_share, v);
      } else {
        put(k0, ddt[0]), put(k0 + 1, ddt[1]);
      }
    }
  }
  if (g.dD.ptr && a.D.sq == 0) {  // one skip weight per head
    float t = active ? (dD[0].x + dD[0].y) + (dD[1].x + dD[1].y) : 0.f;
    for (int o = 1; o < share; o <<= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (active && at_share == 0) atomicAdd(bc4_ptr(g.dD, 0, 0, h, 0), t);
  }
  if (!active) return;
  const float dAv[4] = {dA[0].x, dA[0].y, dA[1].x, dA[1].y}, dDv[4] = {dD[0].x, dD[0].y, dD[1].x, dD[1].y};
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    atomicAdd(bc4_ptr(g.dA, 0, 0, h, q + e), dAv[e]);
    if (g.dD.ptr && a.D.sq != 0) atomicAdd(bc4_ptr(g.dD, 0, 0, h, q + e), dDv[e]);
  }
}

}  // namespace ssmb
