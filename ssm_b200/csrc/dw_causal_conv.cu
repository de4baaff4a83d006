// Depthwise causal conv1d (+ optional SiLU), forward and backward, both layouts, sm_100a.
//
// The operator is HBM-bound: x is read once and y written once (backward: x, dy read once,
// dx written once).  Channels-first: one CTA per (batch, channel) row, 16-byte vector
// accesses along time, the K-1 element halo re-read through L1.  Channels-last: a thread
// owns a 16-byte group of channels and slides along time keeping the window in registers,
// so adjacent threads touch adjacent 16-byte groups of the same time step.
//
// Taps are held newest-first: wr[m] = weight[K-1-m] multiplies x[t-m], so that every
// register-array index below is a compile-time constant for any run-time width K <= 8.
#include <math.h>

#include <type_traits>

#include "common.cuh"
#include "decode_parts.h"

namespace ssmb {

__device__ __forceinline__ bool aligned_to_dev(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

constexpr int kConvMaxK = 8;  // widest supported kernel; kernels are built for KM = 4 and KM = 8
constexpr int kConvThreads = 128;
constexpr int kConvTimeTile = 128;  // channels-last: time steps per thread walk

// x[t] of one (batch, channel) row; before t = 0 the halo (or zero), beyond len zero.
template <typename T>
__device__ __forceinline__ float conv_x_at(const T* __restrict__ row, const float* __restrict__ halo, int K, int t, int L) {
  if (t >= 0) return t < L ? to_f<T>(row[t]) : 0.f;
  return (halo && t >= -(K - 1)) ? __ldg(halo + (K - 1) + t) : 0.f;
}

// ---------------------------------------------------------------------------------------
// channels-first forward
// ---------------------------------------------------------------------------------------
// How the rows of a channels-first tensor can be read: element by element (the tensor itself is off a 16-byte boundary), as 16-byte
// pieces from end to end, or as pieces with ragged ends.
enum { kRowScalar = 0, kRowPieces = 1, kRowRagged = 2 };

template <typename T, int KM, int ROW>
__global__ void __launch_bounds__(kConvThreads) conv_cf_fwd_kernel(const ssm_conv_args a) {
  constexpr int KH = KM - 1;
  constexpr int V = 16 / sizeof(T);
  const int64_t rowi = blockIdx.x;  // b * C + c
  const int c = (int)(rowi % a.channels);
  const int64_t roff = (rowi / a.channels) * a.row_sb + (int64_t)c * a.row_sc;
  const int L = a.len, K = a.width;
  const T* __restrict__ x = reinterpret_cast<const T*>(a.x) + roff;
  T* __restrict__ y = reinterpret_cast<T*>(a.y) + roff;
  const float* halo = a.halo ? a.halo + rowi * (K - 1) : nullptr;
  float wr[KM];
#pragma unroll
  for (int m = 0; m < KM; ++m) wr[m] = m < K ? load_dyn(a.weight, (int64_t)c * K + (K - 1 - m), a.param_dtype) : 0.f;
  const float bias = a.bias ? load_dyn(a.bias, c, a.param_dtype) : 0.f;
  int lo = 0, hi = 0;

  if constexpr (ROW != kRowScalar) {
    // A row may start anywhere: its 16-byte pieces are cut where they lie in memory, so piece ch holds the steps ch * V - sh ..,
    // sh = the row's offset from a 16-byte boundary (the same for x and y).  The loop below takes the pieces that lie inside the row
    // and whose earlier inputs do too, or precede the row altogether (sh = 0); the steps at ragged ends are left to the scalar
    // loop.
    // A thread takes UB vectors of 16 bytes per pass and issues their loads, and those of the vectors before them (the K - 1
    // earlier inputs: the neighbouring thread's vector, served by the L1), before the first value is used.  Vectors beyond the
    // end of the row are read at the last valid address and dropped.
    constexpr int UB = 4, NB = (KH + V - 1) / V;
    const int sh = ROW == kRowRagged ? (int)(roff % V) : 0, ch0 = sh ? NB + 1 : 0, nch = (L + sh) / V;
    const T* xg = x - sh;
    if (ch0 < nch) {
      lo = ch0 * V - sh, hi = nch * V - sh;
      for (int base = ch0 + threadIdx.x; base < nch; base += kConvThreads * UB) {
        uint4 curr[UB], prvr[UB][NB];
#pragma unroll
        for (int j = 0; j < UB; ++j) {
          const int ch = min(base + j * kConvThreads, nch - 1);
          curr[j] = __ldcs(reinterpret_cast<const uint4*>(xg + (int64_t)ch * V));
#pragma unroll
          for (int q = 0; q < NB; ++q) prvr[j][q] = __ldg(reinterpret_cast<const uint4*>(xg + (int64_t)max(ch - 1 - q, 0) * V));
        }
#pragma unroll
        for (int j = 0; j < UB; ++j) {
          const int ch = base + j * kConvThreads;
          if (ch >= nch) break;
          Vec16<T> v;
          float cur[V], prv[NB][V];  // prv[q][i] = x[t0 - (q + 1) V + i]
          v.raw = curr[j];
          v.unpack(cur);
#pragma unroll
          for (int q = 0; q < NB; ++q) {
            v.raw = prvr[j][q], v.unpack(prv[q]);
            if (ch - 1 - q < 0) {
#pragma unroll
              for (int i = 0; i < V; ++i) prv[q][i] = conv_x_at<T>(x, halo, K, (ch - 1 - q) * V + i, L);
            }
          }
          float out[V];
#pragma unroll
          for (int i = 0; i < V; ++i) {
            float acc = bias;
#pragma unroll
            for (int m = 0; m < KM; ++m) {
              constexpr int kLast = V - 1;
              const int back = m - i - 1;  // steps before the piece, when not inside it
              if (m < K) acc = fmaf(wr[m], i >= m ? cur[i >= m ? i - m : 0] : prv[back >= 0 ? back / V : 0][back >= 0 ? kLast - back % V : 0], acc);
            }
            out[i] = a.silu ? (sizeof(T) == 2 ? silu_half_io(acc) : silu_fast(acc)) : acc;
          }
          v.pack(out);
          v.store_stream(y - sh + (int64_t)ch * V);
        }
      }
    }
  }
  if constexpr (ROW == kRowPieces) return;
  // the steps outside [lo, hi): all of a row that cannot be read in pieces
  for (int u = threadIdx.x; u < L - (hi - lo); u += kConvThreads) {
    const int t = u < lo ? u : u + (hi - lo);
    float acc = bias;
#pragma unroll
    for (int m = 0; m < KM; ++m)
      if (m < K) acc = fmaf(wr[m], conv_x_at<T>(x, halo, K, t - m, L), acc);
    y[t] = from_f<T>(a.silu ? (sizeof(T) == 2 ? silu_half_io(acc) : silu_fast(acc)) : acc);
  }
}

// ---------------------------------------------------------------------------------------
// channels-first backward.  pre[t] = bias + sum_m wr[m] x[t-m];  dpre = dy * act'(pre)
//   dx[t] = sum_m wr[m] dpre[t+m];  dwr[m] += sum_t dpre[t] x[t-m];  dbias += sum_t dpre[t]
// ---------------------------------------------------------------------------------------
template <typename T, int KM, int ROW>
__global__ void __launch_bounds__(kConvThreads) conv_cf_bwd_kernel(const ssm_conv_bwd_args g) {
  constexpr int KH = KM - 1;
  const ssm_conv_args& a = g.fwd;
  const int64_t rowi = blockIdx.x;
  const int c = (int)(rowi % a.channels);
  const int64_t roff = (rowi / a.channels) * a.row_sb + (int64_t)c * a.row_sc;
  const int L = a.len, K = a.width;
  const T* __restrict__ x = reinterpret_cast<const T*>(a.x) + roff;
  const T* __restrict__ dy = reinterpret_cast<const T*>(g.dy) + roff;
  T* __restrict__ dx = reinterpret_cast<T*>(g.dx) + roff;
  const float* halo = a.halo ? a.halo + rowi * (K - 1) : nullptr;
  float wr[KM], dwr[KM];
#pragma unroll
  for (int m = 0; m < KM; ++m) wr[m] = m < K ? load_dyn(a.weight, (int64_t)c * K + (K - 1 - m), a.param_dtype) : 0.f, dwr[m] = 0.f;
  const float bias = a.bias ? load_dyn(a.bias, c, a.param_dtype) : 0.f;
  float db = 0.f;
  int lo = 0, hi = 0;

  if constexpr (ROW != kRowScalar) {
    // 16-byte pieces cut where they lie in memory, as in the forward kernel; a ragged end of the row is left to the scalar loop.  A
    // thread owns one piece of outputs and reads the neighbouring pieces of x (both sides) and dy (later side) through L1.
    // (Taking the neighbours' x and dpre from the neighbouring lanes by shuffles instead of forming the K - 1 later dpre again
    // needs fewer instructions but has fewer loads in flight: 101 us against 90 at (8, 1536, 4096) bf16.)
    constexpr int V = 16 / sizeof(T), NB = (KH + V - 1) / V;  // NB: neighbour pieces per side
    const int sh = ROW == kRowRagged ? (int)(roff % V) : 0, p1 = (L + sh) / V;
    const int ch0 = sh ? NB + 1 : 0, ch1 = ROW == kRowRagged && (L + sh) % V ? p1 - NB : p1;  // the pieces whose outputs are formed here
    if (ch0 < ch1) {
      lo = ch0 * V - sh, hi = ch1 * V - sh;
      const T *xg = x - sh, *dg = dy - sh;
      for (int ch = ch0 + threadIdx.x; ch < ch1; ch += kConvThreads) {
        // every load of the pass is issued before the first value is used
        uint4 xr[2 * NB + 1], dyr[NB + 1];
#pragma unroll
        for (int j = 0; j <= 2 * NB; ++j) xr[j] = __ldg(reinterpret_cast<const uint4*>(xg + (int64_t)min(max(ch + j - NB, 0), p1 - 1) * V));
#pragma unroll
        for (int j = 0; j <= NB; ++j) dyr[j] = __ldg(reinterpret_cast<const uint4*>(dg + (int64_t)min(ch + j, p1 - 1) * V));
        float xa[(2 * NB + 1) * V];  // xa[q] = x[t0 - NB * V + q]
#pragma unroll
        for (int j = 0; j <= 2 * NB; ++j) {
          const int cj = ch + j - NB;
          Vec16<T> v;
          v.raw = xr[j];
          float f[V];
          v.unpack(f);
          if (cj < 0 || cj >= p1) {  // beyond an end on a boundary: the halo, or nothing
#pragma unroll
            for (int i = 0; i < V; ++i) f[i] = cj < 0 ? conv_x_at<T>(x, halo, K, cj * V + i, L) : 0.f;
          }
#pragma unroll
          for (int i = 0; i < V; ++i) xa[j * V + i] = f[i];
        }
        float dp[(NB + 1) * V];  // dpre[t0 + i], first dy
#pragma unroll
        for (int j = 0; j <= NB; ++j) {
          Vec16<T> v;
          v.raw = ch + j < p1 ? dyr[j] : make_uint4(0, 0, 0, 0);
          v.unpack(*reinterpret_cast<float(*)[V]>(dp + j * V));
        }
#pragma unroll
        for (int i = 0; i < V + KH; ++i) {
          float pre = bias;
#pragma unroll
          for (int m = 0; m < KM; ++m)
            if (m < K) pre = fmaf(wr[m], xa[NB * V + i - m], pre);
          if (a.silu) dp[i] *= sizeof(T) == 2 ? silu_grad_half_io(pre) : silu_grad_fast(pre);
        }
        float out[V];
#pragma unroll
        for (int i = 0; i < V; ++i) {
          float acc = 0.f;
#pragma unroll
          for (int m = 0; m < KM; ++m)
            if (m < K) {
              acc = fmaf(wr[m], dp[i + m], acc);
              dwr[m] = fmaf(dp[i], xa[NB * V + i - m], dwr[m]);
            }
          out[i] = acc;
          db += dp[i];
        }
        Vec16<T> v;
        v.pack(out);
        v.store_stream(dx - sh + (int64_t)ch * V);
      }
    }
  }
  constexpr int S = 4;  // steps outside [lo, hi): outputs per thread per pass; x / dy re-reads hit L1
  const int head = (lo + S - 1) / S * S;  // the groups before lo, then those from hi on
  for (int u = ROW == kRowPieces ? L : threadIdx.x * S; u < head + L - hi; u += kConvThreads * S) {
    const int t0 = u < head ? u : hi + u - head, t1 = u < head ? min(lo, u + S) : L;  // this thread's outputs: t0 .. min(t0 + S, t1)
    float xw[S + 2 * KH];  // xw[q] = x[t0 - KH + q]
#pragma unroll
    for (int q = 0; q < S + 2 * KH; ++q) {
      const int t = t0 - KH + q;
      xw[q] = (t >= t0 - (K - 1) && t <= t0 + S - 1 + (K - 1)) ? conv_x_at<T>(x, halo, K, t, L) : 0.f;
    }
    float dp[S + KH];  // dpre[t0 + i]
#pragma unroll
    for (int i = 0; i < S + KH; ++i) {
      const int t = t0 + i;
      float v = 0.f;
      if (i < S + K - 1 && t < L) {
        float pre = bias;
#pragma unroll
        for (int m = 0; m < KM; ++m)
          if (m < K) pre = fmaf(wr[m], xw[i - m + KH], pre);
        v = to_f<T>(dy[t]);
        if (a.silu) v *= sizeof(T) == 2 ? silu_grad_half_io(pre) : silu_grad_fast(pre);
      }
      dp[i] = v;
    }
#pragma unroll
    for (int i = 0; i < S; ++i) {
      const int t = t0 + i;
      if (t < t1) {
        float acc = 0.f;
#pragma unroll
        for (int m = 0; m < KM; ++m)
          if (m < K) {
            acc = fmaf(wr[m], dp[i + m], acc);
            dwr[m] = fmaf(dp[i], xw[i - m + KH], dwr[m]);
          }
        dx[t] = from_f<T>(acc);
        db += dp[i];
      }
    }
  }
  // block reduce -> one atomic per CTA and tap
  __shared__ float red[kConvThreads / 32][KM + 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int m = 0; m < KM; ++m) dwr[m] = warp_sum(dwr[m]);
  db = warp_sum(db);
  if (lane == 0) {
#pragma unroll
    for (int m = 0; m < KM; ++m) red[warp][m] = dwr[m];
    red[warp][KM] = db;
  }
  __syncthreads();
  if (threadIdx.x <= KM) {
    float s = 0.f;
    for (int wv = 0; wv < kConvThreads / 32; ++wv) s += red[wv][threadIdx.x];
    const int m = threadIdx.x;
    if (m < K) atomicAdd(g.dweight + (int64_t)c * K + (K - 1 - m), s);
    if (m == KM && g.dbias) atomicAdd(g.dbias + c, s);
  }
}

// ---------------------------------------------------------------------------------------
// channels-last: x (B, L, C); a thread owns V consecutive channels (V*sizeof(T) = 16 or 8 bytes)
// ---------------------------------------------------------------------------------------
template <typename T, int V>
__device__ __forceinline__ void load_group(const T* __restrict__ p, bool vec, int nvalid, float (&f)[V]) {
  if (vec) {
    if constexpr (V * sizeof(T) == 16) {
      const uint4 raw = __ldcs(reinterpret_cast<const uint4*>(p));
      const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
      for (int i = 0; i < V; ++i) f[i] = to_f<T>(e[i]);
    } else {
      static_assert(V * sizeof(T) == 8, "group must be 8 or 16 bytes");
      const uint2 raw = __ldcs(reinterpret_cast<const uint2*>(p));
      const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
      for (int i = 0; i < V; ++i) f[i] = to_f<T>(e[i]);
    }
  } else {
#pragma unroll
    for (int i = 0; i < V; ++i) f[i] = i < nvalid ? to_f<T>(p[i]) : 0.f;
  }
}
template <typename T, int V>
__device__ __forceinline__ void store_group(T* __restrict__ p, bool vec, int nvalid, const float (&f)[V]) {
  if (vec) {
    if constexpr (V * sizeof(T) == 16) {
      uint4 raw;
      T* e = reinterpret_cast<T*>(&raw);
#pragma unroll
      for (int i = 0; i < V; ++i) e[i] = from_f<T>(f[i]);
      __stcs(reinterpret_cast<uint4*>(p), raw);
    } else {
      uint2 raw;
      T* e = reinterpret_cast<T*>(&raw);
#pragma unroll
      for (int i = 0; i < V; ++i) e[i] = from_f<T>(f[i]);
      __stcs(reinterpret_cast<uint2*>(p), raw);
    }
  } else {
#pragma unroll
    for (int i = 0; i < V; ++i)
      if (i < nvalid) p[i] = from_f<T>(f[i]);
  }
}

// x[b, t, c0 .. c0+V) with halo / zero outside [0, L); xb already points at (b, 0, c0)
template <typename T, int V>
__device__ __forceinline__ void load_x_cl(const ssm_conv_args& a, const T* __restrict__ xb, int b, int c0, int t, bool vec, int nvalid,
                                          float (&f)[V]) {
  const int K = a.width;
  if (t >= 0 && t < a.len) {
    load_group<T, V>(xb + (int64_t)t * a.channels, vec, nvalid, f);
    return;
  }
#pragma unroll
  for (int i = 0; i < V; ++i) f[i] = 0.f;
  if (t < 0 && t >= -(K - 1) && a.halo) {
#pragma unroll
    for (int i = 0; i < V; ++i)
      if (i < nvalid) f[i] = __ldg(a.halo + ((int64_t)b * a.channels + c0 + i) * (K - 1) + (K - 1) + t);
  }
}

// Channels-last forward: thread = V channels, walking `tile` consecutive steps with the K - 1 previous inputs in registers.
// Eight steps' loads are issued before their results are formed, so every thread keeps eight 16-byte loads in flight; the
// host picks `tile` so that narrow tensors (the 128-channel B / C inputs of a Mamba-2 layer) still fill the machine.
template <typename T, int KM>
__global__ void __launch_bounds__(kConvThreads, 3) conv_cl_fwd_kernel(const ssm_conv_args a, int vec, int tile) {
  constexpr int KH = KM - 1;
  constexpr int V = 16 / sizeof(T);
  constexpr int U = 8;  // steps per batch of loads
  const int C = a.channels, L = a.len, K = a.width;
  // work item = (time tile, channel vector), channel vectors fastest: a narrow tensor packs several time tiles into one CTA
  const int nvec = (C + V - 1) / V;
  const int64_t item = (int64_t)blockIdx.x * kConvThreads + threadIdx.x;
  const int c0 = (int)(item % nvec) * V;
  const int64_t tile_idx = item / nvec;
  const int64_t ts64 = tile_idx * tile;
  if (ts64 >= L) return;
  const int ts = (int)ts64, te = min(L, ts + tile);
  const int nvalid = min(V, C - c0);
  const int b = blockIdx.z;
  const T* __restrict__ x = reinterpret_cast<const T*>(a.x) + (int64_t)b * L * C + c0;
  T* __restrict__ y = reinterpret_cast<T*>(a.y) + (int64_t)b * L * C + c0;
  // channel pairs as float2 for the packed-fp32 multiply-adds
  float2 wr[KM][V / 2], bias[V / 2];
  if (K == KM && nvalid == V && (reinterpret_cast<uintptr_t>(a.weight) & 15) == 0 && (reinterpret_cast<uintptr_t>(a.bias) & 15) == 0) {
    // the thread's V x K weights are one contiguous run: vector loads (a scalar load per weight costs a sector request per lane,
    // more of them than the whole tile of x)
    float wf[V * KM], bf[V];
    load_param_vec<V * KM>(a.weight, (int64_t)c0 * KM, a.param_dtype, wf);
    if (a.bias) {
      load_param_vec<V>(a.bias, c0, a.param_dtype, bf);
    } else {
#pragma unroll
      for (int i = 0; i < V; ++i) bf[i] = 0.f;
    }
#pragma unroll
    for (int i = 0; i < V; i += 2) {
      bias[i / 2] = make_float2(bf[i], bf[i + 1]);
#pragma unroll
      for (int m = 0; m < KM; ++m) wr[m][i / 2] = make_float2(wf[i * KM + (KM - 1 - m)], wf[(i + 1) * KM + (KM - 1 - m)]);
    }
  } else {
    auto wat = [&](int ch, int m) { return load_dyn(a.weight, (int64_t)ch * K + (K - 1 - m), a.param_dtype); };
#pragma unroll
    for (int i = 0; i < V; i += 2) {
      const int c1 = min(c0 + i, C - 1), c2 = min(c0 + i + 1, C - 1);
      bias[i / 2] = a.bias ? make_float2(load_dyn(a.bias, c1, a.param_dtype), load_dyn(a.bias, c2, a.param_dtype)) : make_float2(0.f, 0.f);
#pragma unroll
      for (int m = 0; m < KM; ++m) wr[m][i / 2] = m < K ? make_float2(wat(c1, m), wat(c2, m)) : make_float2(0.f, 0.f);
    }
  }
  float2 hist[KH > 0 ? KH : 1][V / 2];  // hist[m] = x[t - 1 - m]
  // Where the K - 1 steps before the tile lie inside the tensor (every tile but the first of a sequence) and the rows can be
  // read as 16-byte pieces, they are not fetched here, one dependent load after the other, but run through the pipelined loop
  // below as steps without output.
  const bool warm = vec && ts >= K - 1;
#pragma unroll
  for (int m = 0; m < KH; ++m) {
    float f[V];
    if (m < K - 1 && !warm) {
      load_x_cl<T, V>(a, x, b, c0, ts - 1 - m, vec, nvalid, f);
    } else {
#pragma unroll
      for (int i = 0; i < V; ++i) f[i] = 0.f;
    }
#pragma unroll
    for (int i = 0; i < V; i += 2) hist[m][i / 2] = make_float2(f[i], f[i + 1]);
  }
  // one step: inputs f of step tt -> output row, then the window moves on
  auto step = [&](int tt, const float (&f)[V]) {
    if (tt < ts) {  // a step before the tile: it only enters the window
#pragma unroll
      for (int m = KH - 1; m >= 1; --m)
        if (m < K - 1) {
#pragma unroll
          for (int i = 0; i < V / 2; ++i) hist[m][i] = hist[m - 1][i];
        }
      if (KH > 0) {
#pragma unroll
        for (int i = 0; i < V / 2; ++i) hist[0][i] = make_float2(f[2 * i], f[2 * i + 1]);
      }
      return;
    }
    float out[V];
    float2 c2[V / 2];
#pragma unroll
    for (int i = 0; i < V; i += 2) {
      c2[i / 2] = make_float2(f[i], f[i + 1]);
      float2 acc = __ffma2_rn(wr[0][i / 2], c2[i / 2], bias[i / 2]);
#pragma unroll
      for (int m = 1; m < KM; ++m)
        if (m < K) acc = __ffma2_rn(wr[m][i / 2], hist[m - 1][i / 2], acc);
      if (a.silu) {
        out[i] = sizeof(T) == 2 ? silu_half_io(acc.x) : silu_fast(acc.x);
        out[i + 1] = sizeof(T) == 2 ? silu_half_io(acc.y) : silu_fast(acc.y);
      } else {
        out[i] = acc.x, out[i + 1] = acc.y;
      }
    }
    store_group<T, V>(y + (int64_t)tt * C, vec, nvalid, out);
#pragma unroll
    for (int m = KH - 1; m >= 1; --m)
      if (m < K - 1) {
#pragma unroll
        for (int i = 0; i < V / 2; ++i) hist[m][i] = hist[m - 1][i];
      }
    if (KH > 0) {
#pragma unroll
      for (int i = 0; i < V / 2; ++i) hist[0][i] = c2[i];
    }
  };
  if (vec) {
    // The loads of U steps are issued together and stay packed (16 bytes each) until their step is formed; the loads of the
    // next U steps go out before the current ones are used, so a thread always has loads in flight.
    uint4 raw[U], nxt[U];
    const int tb = warm ? ts - (K - 1) : ts;
#pragma unroll
    for (int j = 0; j < U; ++j)
      if (tb + j < te) nxt[j] = __ldcs(reinterpret_cast<const uint4*>(x + (int64_t)(tb + j) * C));
    for (int t = tb; t < te; t += U) {
#pragma unroll
      for (int j = 0; j < U; ++j) raw[j] = nxt[j];
#pragma unroll
      for (int j = 0; j < U; ++j)
        if (t + U + j < te) nxt[j] = __ldcs(reinterpret_cast<const uint4*>(x + (int64_t)(t + U + j) * C));
#pragma unroll
      for (int j = 0; j < U; ++j) {
        if (t + j < te) {
          float f[V];
          const T* e = reinterpret_cast<const T*>(&raw[j]);
#pragma unroll
          for (int i = 0; i < V; ++i) f[i] = to_f<T>(e[i]);
          step(t + j, f);
        }
      }
    }
  } else {
    for (int t = ts; t < te; ++t) {
      float f[V];
      load_group<T, V>(x + (int64_t)t * C, false, nvalid, f);
      step(t, f);
    }
  }
}

// 16-bit or fp32 elements of a piece of 8 or 16 bytes as pairs of channels, word by word (see Vec16), and back
template <typename T, int V>
__device__ __forceinline__ void unpack_cl(const uint32_t* w, float2 (&f)[V / 2]) {
#pragma unroll
  for (int i = 0; i < V / 2; ++i) {
    if constexpr (std::is_same<T, float>::value) f[i] = make_float2(__uint_as_float(w[2 * i]), __uint_as_float(w[2 * i + 1]));
    else if constexpr (std::is_same<T, __nv_bfloat16>::value) f[i] = make_float2(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xffff0000u));
    else f[i] = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
  }
}
template <typename T, int V>
__device__ __forceinline__ void pack_cl(const float2 (&f)[V / 2], uint32_t* w) {
#pragma unroll
  for (int i = 0; i < V / 2; ++i) {
    if constexpr (std::is_same<T, float>::value) {
      w[2 * i] = __float_as_uint(f[i].x), w[2 * i + 1] = __float_as_uint(f[i].y);
    } else if constexpr (std::is_same<T, __nv_bfloat16>::value) {
      const __nv_bfloat162 v = __floats2bfloat162_rn(f[i].x, f[i].y);
      w[i] = *reinterpret_cast<const uint32_t*>(&v);
    } else {
      const __half2 v = __floats2half2_rn(f[i].x, f[i].y);
      w[i] = *reinterpret_cast<const uint32_t*>(&v);
    }
  }
}
template <bool HALF>
__device__ __forceinline__ float2 silu2(float2 p) {
  if constexpr (HALF) {  // see silu_half_io
    const float2 h = __fmul2_rn(p, make_float2(0.5f, 0.5f));
    float2 t;
    asm("tanh.approx.f32 %0, %1;" : "=f"(t.x) : "f"(h.x));
    asm("tanh.approx.f32 %0, %1;" : "=f"(t.y) : "f"(h.y));
    return __ffma2_rn(h, t, h);
  } else {
    return make_float2(silu_fast(p.x), silu_fast(p.y));
  }
}

// The same for the width that state-space models use (4) and channels in whole 16-byte groups: the taps exist once, the window is
// the batch of rows itself (the steps of a batch are unrolled and nothing moves from step to step), the rows of the next batch are under
// way while this one is formed, and no step is guarded but those of a tile's last batch.  Bound by HBM.
template <typename T, bool SILU>
__global__ void __launch_bounds__(kConvThreads, 4) conv_cl_fwd4_kernel(const ssm_conv_args a, int tile) {
  constexpr int V = 16 / sizeof(T), P = V / 2;
  constexpr int U = 4;  // steps per batch of loads
  const int C = a.channels, L = a.len, nvec = C / V;
  const int64_t item = (int64_t)blockIdx.x * kConvThreads + threadIdx.x;  // channel groups fastest, then time tiles
  const int c0 = (int)(item % nvec) * V;
  const int64_t ts64 = item / nvec * tile;
  if (ts64 >= L) return;
  const int ts = (int)ts64, te = min(L, ts + tile), b = blockIdx.z;
  const T* __restrict__ x = reinterpret_cast<const T*>(a.x) + (int64_t)b * L * C + c0;
  T* __restrict__ y = reinterpret_cast<T*>(a.y) + (int64_t)b * L * C + c0;
  uint4 nxt[U];
  auto request = [&](int t) {  // beyond the sequence: its last row, dropped
#pragma unroll
    for (int j = 0; j < U; ++j) nxt[j] = __ldcs(reinterpret_cast<const uint4*>(x + (int64_t)min(t + j, L - 1) * C));
  };
  request(ts);
  float2 win[U + 3][P];  // win[j]: x of step t + j - 3
  if (ts >= 3) {
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const uint4 r = __ldcs(reinterpret_cast<const uint4*>(x + (int64_t)(ts - 3 + j) * C));
      unpack_cl<T, V>(reinterpret_cast<const uint32_t*>(&r), win[j]);
    }
  } else {  // (tiles are multiples of eight steps: the sequence's first)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
#pragma unroll
      for (int p = 0; p < P; ++p) {
        const float* h = a.halo + ((int64_t)b * C + c0 + 2 * p) * 3 + j;
        win[j][p] = a.halo ? make_float2(__ldg(h), __ldg(h + 3)) : make_float2(0.f, 0.f);
      }
    }
  }
  float2 w[4][P], bias[P];  // w[m]: the tap of x[t - m]
  {
    float wf[V * 4], bf[V];
    load_param_vec<V * 4>(a.weight, (int64_t)c0 * 4, a.param_dtype, wf);
    if (a.bias) load_param_vec<V>(a.bias, c0, a.param_dtype, bf);
#pragma unroll
    for (int p = 0; p < P; ++p) {
      bias[p] = a.bias ? make_float2(bf[2 * p], bf[2 * p + 1]) : make_float2(0.f, 0.f);
#pragma unroll
      for (int m = 0; m < 4; ++m) w[m][p] = make_float2(wf[8 * p + 3 - m], wf[8 * p + 7 - m]);
    }
  }
#pragma unroll 1
  for (int t = ts; t < te; t += U) {
#pragma unroll
    for (int j = 0; j < U; ++j) unpack_cl<T, V>(reinterpret_cast<const uint32_t*>(&nxt[j]), win[j + 3]);
    if (t + U < te) request(t + U);
    T* out = y + (int64_t)t * C;
#pragma unroll
    for (int j = 0; j < U; ++j) {
      if (t + j >= te) break;
      float2 o[P];
#pragma unroll
      for (int p = 0; p < P; ++p) {
        float2 acc = __ffma2_rn(w[0][p], win[j + 3][p], bias[p]);
#pragma unroll
        for (int m = 1; m < 4; ++m) acc = __ffma2_rn(w[m][p], win[j + 3 - m][p], acc);
        o[p] = SILU ? silu2<sizeof(T) == 2>(acc) : acc;
      }
      uint4 r;
      pack_cl<T, V>(o, reinterpret_cast<uint32_t*>(&r));
      __stcs(reinterpret_cast<uint4*>(out), r);
      out += C;
    }
#pragma unroll
    for (int j = 0; j < 3; ++j) {
#pragma unroll
      for (int p = 0; p < P; ++p) win[j][p] = win[U + j][p];
    }
  }
}

// channels-last backward.  Walk s over [ts, te + K - 1): dpre[s] needs x[s-(K-1) .. s];
// dx[t = s-(K-1)] = sum_q w[q] dpre[s - q] (w in stored order) needs dpre[s-(K-1) .. s].
// Four channels per thread keep both windows, both tap orders and the weight-gradient
// accumulators in registers.
template <typename T, int KM>
__global__ void __launch_bounds__(kConvThreads) conv_cl_bwd_kernel(const ssm_conv_bwd_args g, int vec) {
  constexpr int KH = KM - 1;
  const ssm_conv_args& a = g.fwd;
  constexpr int V = 4;
  const int C = a.channels, L = a.len, K = a.width;
  const int c0 = (blockIdx.x * kConvThreads + threadIdx.x) * V;
  if (c0 >= C) return;
  const int nvalid = min(V, C - c0);
  const int b = blockIdx.z;
  const int ts = blockIdx.y * kConvTimeTile, te = min(L, ts + kConvTimeTile);
  const T* __restrict__ x = reinterpret_cast<const T*>(a.x) + (int64_t)b * L * C + c0;
  const T* __restrict__ dy = reinterpret_cast<const T*>(g.dy) + (int64_t)b * L * C + c0;
  T* __restrict__ dx = reinterpret_cast<T*>(g.dx) + (int64_t)b * L * C + c0;
  float w[KM][V], wr[KM][V], bias[V];  // w[q] = weight[c][q];  wr[m] = weight[c][K-1-m]
#pragma unroll
  for (int i = 0; i < V; ++i) {
    const int cc = min(c0 + i, C - 1);
    bias[i] = a.bias ? load_dyn(a.bias, cc, a.param_dtype) : 0.f;
#pragma unroll
    for (int q = 0; q < KM; ++q) {
      w[q][i] = q < K ? load_dyn(a.weight, (int64_t)cc * K + q, a.param_dtype) : 0.f;
      wr[q][i] = q < K ? load_dyn(a.weight, (int64_t)cc * K + (K - 1 - q), a.param_dtype) : 0.f;
    }
  }
  float dwr[KM][V], db[V];
#pragma unroll
  for (int i = 0; i < V; ++i) {
    db[i] = 0.f;
#pragma unroll
    for (int m = 0; m < KM; ++m) dwr[m][i] = 0.f;
  }
  float xh[KH > 0 ? KH : 1][V], dph[KH > 0 ? KH : 1][V];  // xh[m] = x[s-1-m], dph[m] = dpre[s-1-m]
  // Where the K - 1 steps before the tile lie inside the tensor and the rows can be read as whole pieces, they run through the
  // batched loop below as steps that only enter the window, instead of being fetched here one dependent load after the other.
  const bool warm = vec && ts >= K - 1;
#pragma unroll
  for (int m = 0; m < KH; ++m) {
#pragma unroll
    for (int i = 0; i < V; ++i) dph[m][i] = 0.f;  // dx[ts..] never needs dpre before ts
    if (m < K - 1 && !warm) load_x_cl<T, V>(a, x, b, c0, ts - 1 - m, vec, nvalid, xh[m]);
    else {
#pragma unroll
      for (int i = 0; i < V; ++i) xh[m][i] = 0.f;
    }
  }
  // the loads of U steps (x and dy, as packed pieces) go out together; steps beyond the sequence read its last row and drop it
  constexpr int U = 8;
  using Raw = typename std::conditional<sizeof(T) == 2, uint2, uint4>::type;
  const int sb = warm ? ts - (K - 1) : ts, se = te + K - 1;
  for (int s0 = sb; s0 < se; s0 += U) {
    Raw xr[U], gr[U];
    if (vec) {
#pragma unroll
      for (int j = 0; j < U; ++j) {
        const int sc = min(s0 + j, L - 1);
        xr[j] = __ldcs(reinterpret_cast<const Raw*>(x + (int64_t)sc * C));
        gr[j] = __ldcs(reinterpret_cast<const Raw*>(dy + (int64_t)sc * C));
      }
    }
#pragma unroll
    for (int j = 0; j < U; ++j) {
    const int s = s0 + j;
    if (s >= se) break;
    float cur[V], dyv[V], dp[V];
    if (vec) {
      const T* ex = reinterpret_cast<const T*>(&xr[j]);
      const T* eg = reinterpret_cast<const T*>(&gr[j]);
#pragma unroll
      for (int i = 0; i < V; ++i) cur[i] = s < L ? to_f<T>(ex[i]) : 0.f, dyv[i] = (s < L && s >= ts) ? to_f<T>(eg[i]) : 0.f;
    } else {
      load_x_cl<T, V>(a, x, b, c0, s, vec, nvalid, cur);
      if (s < L) load_group<T, V>(dy + (int64_t)s * C, vec, nvalid, dyv);
      else {
#pragma unroll
        for (int i = 0; i < V; ++i) dyv[i] = 0.f;
      }
    }
#pragma unroll
    for (int i = 0; i < V; ++i) {
      float pre = fmaf(wr[0][i], cur[i], bias[i]);
#pragma unroll
      for (int m = 1; m < KM; ++m)
        if (m < K) pre = fmaf(wr[m][i], xh[m - 1][i], pre);
      dp[i] = s < L ? (a.silu ? dyv[i] * (sizeof(T) == 2 ? silu_grad_half_io(pre) : silu_grad_fast(pre)) : dyv[i]) : 0.f;
      if (s >= ts && s < te) {  // each position's parameter gradient is counted by the tile that owns it
        db[i] += dp[i];
        dwr[0][i] = fmaf(dp[i], cur[i], dwr[0][i]);
#pragma unroll
        for (int m = 1; m < KM; ++m)
          if (m < K) dwr[m][i] = fmaf(dp[i], xh[m - 1][i], dwr[m][i]);
      }
    }
    const int t = s - (K - 1);
    if (t >= ts && t < te) {
      float out[V];
#pragma unroll
      for (int i = 0; i < V; ++i) {
        float acc = w[0][i] * dp[i];
#pragma unroll
        for (int q = 1; q < KM; ++q)
          if (q < K) acc = fmaf(w[q][i], dph[q - 1][i], acc);
        out[i] = acc;
      }
      store_group<T, V>(dx + (int64_t)t * C, vec, nvalid, out);
    }
#pragma unroll
    for (int m = KH - 1; m >= 1; --m)
      if (m < K - 1) {
#pragma unroll
        for (int i = 0; i < V; ++i) xh[m][i] = xh[m - 1][i], dph[m][i] = dph[m - 1][i];
      }
    if (KH > 0) {
#pragma unroll
      for (int i = 0; i < V; ++i) xh[0][i] = cur[i], dph[0][i] = dp[i];
    }
    }
  }
#pragma unroll
  for (int i = 0; i < V; ++i) {
    if (i < nvalid) {
      if (g.dbias) atomicAdd(g.dbias + c0 + i, db[i]);
#pragma unroll
      for (int m = 0; m < KM; ++m)
        if (m < K) atomicAdd(g.dweight + (int64_t)(c0 + i) * K + (K - 1 - m), dwr[m][i]);
    }
  }
}

// SiLU gradient of a pair of pre-activations
template <bool HALF>
__device__ __forceinline__ float2 silu_grad2(float2 p) {
  float2 s;
  if constexpr (HALF) {  // sigmoid(x) = 0.5 + 0.5 tanh(x / 2), one special-function instruction (see silu_grad_half_io)
    const float2 h = __fmul2_rn(p, make_float2(0.5f, 0.5f));
    float2 t;
    asm("tanh.approx.f32 %0, %1;" : "=f"(t.x) : "f"(h.x));
    asm("tanh.approx.f32 %0, %1;" : "=f"(t.y) : "f"(h.y));
    s = __ffma2_rn(t, make_float2(0.5f, 0.5f), make_float2(0.5f, 0.5f));
  } else {
    s = make_float2(sigmoid_fast(p.x), sigmoid_fast(p.y));
  }
  const float2 r = __ffma2_rn(s, make_float2(-1.f, -1.f), make_float2(1.f, 1.f));
  return __ffma2_rn(__fmul2_rn(p, s), r, s);
}

// The same walk for the width that state-space models use (4) and channels in whole groups of four: taps, windows and
// accumulators are pairs of channels for the packed-fp32 instructions, the taps exist once, rows travel through a ring in shared memory, and
// the four steps of a batch run without any check unless they touch an end of the tile.  512 threads per SM, half of their issue slots
// busy, and a tile length that fills whole waves (conv_cl_tile).
// (4, 4093, 2560) bf16, 251 MB: 154 us with the kernel above, 63 us with this one (4.0 TB/s).  Narrow tensors, NT = 512: (2, 16384, 128) bf16
// 72 -> 14 us.
constexpr int kConvRing = 4, kConvBatch = 4;  // batches of the ring, steps of a batch
constexpr size_t conv_ring_bytes(int threads) { return (size_t)kConvRing * kConvBatch * 2 * 8 * threads; }
__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
template <typename T, int V, int NT, bool SILU>
__global__ void __launch_bounds__(NT, 512 / NT) conv_cl_bwd4_kernel(const ssm_conv_bwd_args g, int tile) {
  const ssm_conv_args& a = g.fwd;
  constexpr int U = kConvBatch;
  constexpr int P = V / 2;
  static_assert(V * sizeof(T) == 8, "a thread's channels of a step are one load of 8 bytes");
  using Raw = uint2;
  const int C = a.channels, L = a.len, nvec = C / V;
  const int64_t item = (int64_t)blockIdx.x * NT + threadIdx.x;  // channel groups fastest, then time tiles
  const int c0 = (int)(item % nvec) * V;
  const int64_t ts64 = item / nvec * tile;
  const bool live = ts64 < L;
  const int ts = live ? (int)ts64 : 0, te = live ? min(L, ts + tile) : -3, b = blockIdx.z;
  const T* __restrict__ x = reinterpret_cast<const T*>(a.x) + (int64_t)b * L * C + c0;
  const T* __restrict__ dy = reinterpret_cast<const T*>(g.dy) + (int64_t)b * L * C + c0;
  T* __restrict__ dx = reinterpret_cast<T*>(g.dx) + (int64_t)b * L * C + c0;
  float2 w[4][P], bias[P], dw[4][P], db[P];  // w[m], dw[m]: the tap of x[t - m]
  {
    float wf[V * 4], bf[V];
    load_param_vec<V * 4>(a.weight, (int64_t)c0 * 4, a.param_dtype, wf);
#pragma unroll
    for (int i = 0; i < V; ++i) bf[i] = a.bias ? load_dyn(a.bias, c0 + i, a.param_dtype) : 0.f;
#pragma unroll
    for (int p = 0; p < P; ++p) {
      bias[p] = make_float2(bf[2 * p], bf[2 * p + 1]), db[p] = make_float2(0.f, 0.f);
#pragma unroll
      for (int m = 0; m < 4; ++m) w[m][p] = make_float2(wf[8 * p + 3 - m], wf[8 * p + 7 - m]), dw[m][p] = make_float2(0.f, 0.f);
    }
  }
  // rows travel through a ring of batches in shared memory, each thread's own 8 bytes of x and of dy: no barrier, and twelve steps
  // are under way without a register
  extern __shared__ __align__(16) unsigned char conv_ring[];
  Raw* ring = reinterpret_cast<Raw*>(conv_ring) + threadIdx.x;  // [stage][step][x | dy][NT]
  auto request = [&](int s, int stage) {
    if (s < te + 3) {
      const T *px = x + (int64_t)min(s, L - 1) * C, *pg = dy + (int64_t)min(s, L - 1) * C;
#pragma unroll
      for (int j = 0; j < U; ++j) {
        cp_async8(ring + ((stage * U + j) * 2) * NT, px), cp_async8(ring + ((stage * U + j) * 2 + 1) * NT, pg);
        if (s + j + 1 < L) px += C, pg += C;  // beyond the sequence: its last row, dropped
      }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
#pragma unroll
  for (int q = 0; q < kConvRing - 1; ++q) request(ts + q * U, q);
  float2 win[U + 3][P], dwin[U + 3][P];  // x and the pre-activation gradient of step s + j - 3
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const int t = ts - 3 + j;
    if (t >= 0) {
      const Raw r = __ldcs(reinterpret_cast<const Raw*>(x + (int64_t)t * C));
      unpack_cl<T, V>(reinterpret_cast<const uint32_t*>(&r), win[j]);
    }
#pragma unroll
    for (int p = 0; p < P; ++p) {
      if (t < 0) {
        const float* h = a.halo + ((int64_t)b * C + c0 + 2 * p) * 3 + 3 + t;
        win[j][p] = a.halo ? make_float2(__ldg(h), __ldg(h + 3)) : make_float2(0.f, 0.f);
      }
      dwin[j][p] = make_float2(0.f, 0.f);
    }
  }
  // a batch of steps; not inner: those that touch an end of the tile (each position's parameter gradient is counted by the tile
  // that owns it, each dx written by the tile that owns it) or lie beyond the sequence
  auto batch = [&](auto inner, int s0) {
    constexpr bool kInner = decltype(inner)::value;
    T* to = dx + (int64_t)(s0 - 3) * C;
#pragma unroll
    for (int j = 0; j < U; ++j) {
      const int s = s0 + j;
#pragma unroll
      for (int p = 0; p < P; ++p) {
        if (!kInner && s >= L) win[j + 3][p] = dwin[j + 3][p] = make_float2(0.f, 0.f);
        float2 pre = __ffma2_rn(w[0][p], win[j + 3][p], bias[p]);
#pragma unroll
        for (int m = 1; m < 4; ++m) pre = __ffma2_rn(w[m][p], win[j + 3 - m][p], pre);
        float2& dp = dwin[j + 3][p];
        if (SILU) dp = __fmul2_rn(dp, silu_grad2<sizeof(T) == 2>(pre));
        if (kInner || s < te) {
          db[p] = __fadd2_rn(db[p], dp);
#pragma unroll
          for (int m = 0; m < 4; ++m) dw[m][p] = __ffma2_rn(dp, win[j + 3 - m][p], dw[m][p]);
        }
      }
      if (kInner || (s - 3 >= ts && s - 3 < te)) {  // dx[s - 3] = w[3] dpre[s] + w[2] dpre[s - 1] + w[1] dpre[s - 2] + w[0] dpre[s - 3]
        float2 o[P];
#pragma unroll
        for (int p = 0; p < P; ++p) {
          o[p] = __fmul2_rn(w[3][p], dwin[j + 3][p]);
#pragma unroll
          for (int m = 0; m < 3; ++m) o[p] = __ffma2_rn(w[m][p], dwin[j + m][p], o[p]);
        }
        Raw r;
        pack_cl<T, V>(o, reinterpret_cast<uint32_t*>(&r));
        __stcs(reinterpret_cast<Raw*>(to), r);
      }
      to += C;
    }
  };
  int stage = 0;
#pragma unroll 1
  for (int s0 = ts; s0 < te + 3; s0 += U) {
    request(s0 + (kConvRing - 1) * U, stage == 0 ? kConvRing - 1 : stage - 1);
    asm volatile("cp.async.wait_group %0;\n" ::"n"(kConvRing - 1) : "memory");
#pragma unroll
    for (int j = 0; j < U; ++j) {
      const Raw xr = ring[((stage * U + j) * 2) * NT], gr = ring[((stage * U + j) * 2 + 1) * NT];
      unpack_cl<T, V>(reinterpret_cast<const uint32_t*>(&xr), win[j + 3]);
      unpack_cl<T, V>(reinterpret_cast<const uint32_t*>(&gr), dwin[j + 3]);
    }
    stage = stage == kConvRing - 1 ? 0 : stage + 1;
    if (s0 >= ts + 3 && s0 + U <= te) batch(std::true_type{}, s0);
    else batch(std::false_type{}, s0);
#pragma unroll
    for (int j = 0; j < 3; ++j) {
#pragma unroll
      for (int p = 0; p < P; ++p) win[j][p] = win[U + j][p], dwin[j][p] = dwin[U + j][p];
    }
  }
  auto comp = [](const float2 (&v)[P], int i) { return i & 1 ? v[i / 2].y : v[i / 2].x; };
  // Narrow tensors: the threads of a CTA that share channels meet in shared memory, one global addition per CTA and gradient (an
  // addition to a word that many CTAs want takes about 40 ns).
  __shared__ float sums[NT > 128 ? NT * 5 : 1];
  if constexpr (NT > 128) {
    for (int i = threadIdx.x; i < C * 5; i += NT) sums[i] = 0.f;
    __syncthreads();
    if (live) {
#pragma unroll
      for (int i = 0; i < V; ++i) {
        atomicAdd(sums + (c0 + i) * 5 + 4, comp(db, i));
#pragma unroll
        for (int m = 0; m < 4; ++m) atomicAdd(sums + (c0 + i) * 5 + 3 - m, comp(dw[m], i));
      }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < C * 5; i += NT) {
      const int c = i / 5, q = i % 5;
      if (q < 4) atomicAdd(g.dweight + c * 4 + q, sums[i]);
      else if (g.dbias) atomicAdd(g.dbias + c, sums[i]);
    }
  } else if (live) {
#pragma unroll
    for (int i = 0; i < V; ++i) {
      if (g.dbias) atomicAdd(g.dbias + c0 + i, comp(db, i));
#pragma unroll
      for (int m = 0; m < 4; ++m) atomicAdd(g.dweight + (int64_t)(c0 + i) * 4 + (3 - m), comp(dw[m], i));
    }
  }
}

// Decode-time update of up to three windows.  A thread takes one channel of U sequences: its weights once, and U states in flight (one
// state per thread kept too few bytes under way: (256, 5120) 11.3 us, 84 MB/ms of 42 MB).
struct ConvUpdates {
  ssm_conv_update_args a[3];
  int blocks_end[3];  // thread blocks of the windows so far
};
template <typename T, int U>
__global__ void __launch_bounds__(256) conv_update_kernel(const __grid_constant__ ConvUpdates all) {
  pdl_wait();
  pdl_trigger();
  const int which = (int)blockIdx.x >= all.blocks_end[0] ? (int)blockIdx.x >= all.blocks_end[1] ? 2 : 1 : 0;
  const ssm_conv_update_args& a = all.a[which];
  const int64_t i = (int64_t)(blockIdx.x - (which ? all.blocks_end[which - 1] : 0)) * 256 + threadIdx.x;
  const int C = a.channels, K = a.width;
  const int c = (int)(i % C), b0 = (int)(i / C) * U;
  if (b0 >= a.batch) return;
  const float bias = a.bias ? load_dyn(a.bias, c, a.param_dtype) : 0.f;
  if (K == 4 && aligned_to_dev(a.conv_state)) {
    float4 v[U];
    float xn[U], w[4];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t at = (int64_t)min(b0 + u, a.batch - 1) * C + c;
      v[u] = *reinterpret_cast<const float4*>(a.conv_state + at * 4);
      xn[u] = to_f<T>(reinterpret_cast<const T*>(a.x)[at]);
    }
    load_param_vec<4>(a.weight, (int64_t)c * 4, a.param_dtype, w);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (b0 + u >= a.batch) break;
      const int64_t at = (int64_t)(b0 + u) * C + c;
      const float4 n = make_float4(v[u].y, v[u].z, v[u].w, xn[u]);
      *reinterpret_cast<float4*>(a.conv_state + at * 4) = n;
      const float acc = fmaf(n.x, w[0], fmaf(n.y, w[1], fmaf(n.z, w[2], fmaf(n.w, w[3], bias))));
      reinterpret_cast<T*>(a.out)[at] = from_f<T>(a.silu ? silu_fast(acc) : acc);
    }
    return;
  }
  for (int b = b0; b < min(b0 + U, a.batch); ++b) {
    const int64_t at = (int64_t)b * C + c;
    float* cs = a.conv_state + at * K;
    const float xn = to_f<T>(reinterpret_cast<const T*>(a.x)[at]);
    float acc = bias;
    for (int j = 0; j < K; ++j) {
      const float v = j + 1 < K ? cs[j + 1] : xn;
      cs[j] = v;
      acc = fmaf(v, load_dyn(a.weight, (int64_t)c * K + j, a.param_dtype), acc);
    }
    reinterpret_cast<T*>(a.out)[at] = from_f<T>(a.silu ? silu_fast(acc) : acc);
  }
}

template <typename T, int U>
static int conv_update_launch(const ssm_conv_update_args* a, int n, cudaStream_t st) {
  ConvUpdates all{};
  int blocks = 0;
  for (int i = 0; i < 3; ++i) {
    if (i < n) {
      all.a[i] = a[i];
      blocks += (int)(((int64_t)((a[i].batch + U - 1) / U) * a[i].channels + 255) / 256);
    }
    all.blocks_end[i] = i < n - 1 ? blocks : INT32_MAX;
  }
  return launch_overlapped("conv_update_kernel", conv_update_kernel<T, U>, dim3(blocks), dim3(256), 0, st, all);
}
template <typename T>
static int conv_update_t(const ssm_conv_update_args* a, int n, cudaStream_t st) {
  int64_t items = 0;
  for (int i = 0; i < n; ++i) items += (int64_t)a[i].batch * a[i].channels;
  // four sequences per thread once that still gives every SM a thousand threads
  return items >= (int64_t)sm_count() * 4096 ? conv_update_launch<T, 4>(a, n, st) : conv_update_launch<T, 1>(a, n, st);
}

static int conv_validate(const ssm_conv_args* a) {
  SSM_REQUIRE(a != nullptr, SSM_ERR_NULL, "dw_causal_conv: args is NULL");
  SSM_REQUIRE(a->batch >= 0 && a->channels >= 0 && a->len >= 0, SSM_ERR_SHAPE, "dw_causal_conv: negative size");
  SSM_REQUIRE(a->width >= 1 && a->width <= kConvMaxK, SSM_ERR_UNSUPPORTED, "dw_causal_conv: kernel width must be in [1, 8]");
  SSM_REQUIRE(valid_dtype(a->io_dtype) && valid_dtype(a->param_dtype), SSM_ERR_DTYPE, "dw_causal_conv: unknown dtype");
  SSM_REQUIRE(a->batch <= 65535, SSM_ERR_TOO_LARGE, "dw_causal_conv: batch exceeds 65535");
  SSM_REQUIRE(!a->channels_first || (a->row_sb >= 0 && a->row_sc >= a->len), SSM_ERR_SHAPE, "dw_causal_conv: bad row strides");
  SSM_REQUIRE((int64_t)a->batch * a->channels < (1ll << 31), SSM_ERR_TOO_LARGE, "dw_causal_conv: batch*channels too large");
  return SSM_OK;
}

static dim3 conv_cl_grid(const ssm_conv_args& a, int V) {
  return dim3(((a.channels + V - 1) / V + kConvThreads - 1) / kConvThreads, (a.len + kConvTimeTile - 1) / kConvTimeTile, a.batch);
}

// Steps per thread of a channels-last walk: the tile length with the least (waves of resident CTAs) x (steps per CTA), where a
// walk costs about `extra` steps more than its tile (the window and weight loads of its start, the sums at its end).
static int64_t conv_cl_ctas(const ssm_conv_args& a, int V, int threads, int tile) {
  const int64_t items = (int64_t)((a.channels + V - 1) / V) * ((a.len + tile - 1) / tile);
  return (items + threads - 1) / threads;
}
static int conv_cl_tile(const ssm_conv_args& a, int V, int threads, int ctas_per_sm, int extra, int longest) {
  const int64_t slots = (int64_t)sm_count() * ctas_per_sm;
  int best = 8;
  double cost = 1e300;
  for (int tile = 8; tile <= longest; tile += 8) {
    const int64_t n = conv_cl_ctas(a, V, threads, tile) * a.batch;
    if (n >= (1ll << 31)) continue;
    // a last wave costs what it holds, but no less than half a wave: its CTAs run alone and cannot hide their latencies
    const double waves = (double)(n / slots) + (n % slots ? fmax(0.5, (double)(n % slots) / slots) : 0.0);
    const double c = fmax(1.0, waves) * (tile + extra);
    if (c < cost) cost = c, best = tile;
  }
  return best;
}

// every row a whole number of 16-byte pieces, starting on a boundary
static bool conv_rows_whole(const ssm_conv_args& a, int V) { return a.len % V == 0 && a.row_sb % V == 0 && a.row_sc % V == 0; }

template <typename T, int KM>
static int conv_fwd_launch(const ssm_conv_args& a, cudaStream_t st) {
  constexpr int V = 16 / sizeof(T);
  if (a.channels_first) {
    const unsigned grid = (unsigned)((int64_t)a.batch * a.channels);
    if (!(aligned_to(a.x, 16) && aligned_to(a.y, 16))) conv_cf_fwd_kernel<T, KM, kRowScalar><<<grid, kConvThreads, 0, st>>>(a);
    else if (conv_rows_whole(a, V)) conv_cf_fwd_kernel<T, KM, kRowPieces><<<grid, kConvThreads, 0, st>>>(a);
    else conv_cf_fwd_kernel<T, KM, kRowRagged><<<grid, kConvThreads, 0, st>>>(a);
  } else {
    const int vec = (a.channels % V == 0) && aligned_to(a.x, 16) && aligned_to(a.y, 16);
    if (a.width == 4 && vec && aligned_to(a.weight, 16) && aligned_to(a.bias, 16)) {
      const int tile = conv_cl_tile(a, V, kConvThreads, 4, 12, 128);
      const dim3 grid((unsigned)conv_cl_ctas(a, V, kConvThreads, tile), 1, a.batch);
      if (a.silu) conv_cl_fwd4_kernel<T, true><<<grid, kConvThreads, 0, st>>>(a, tile);
      else conv_cl_fwd4_kernel<T, false><<<grid, kConvThreads, 0, st>>>(a, tile);
      return launch_status("dw_causal_conv_fwd");
    }
    const int tile = conv_cl_tile(a, V, kConvThreads, 3, 12, 128);
    conv_cl_fwd_kernel<T, KM><<<dim3((unsigned)conv_cl_ctas(a, V, kConvThreads, tile), 1, a.batch), kConvThreads, 0, st>>>(a, vec, tile);
  }
  return launch_status("dw_causal_conv_fwd");
}

template <typename T, int KM>
static int conv_bwd_launch(const ssm_conv_bwd_args& g, cudaStream_t st) {
  const ssm_conv_args& a = g.fwd;
  if (a.channels_first) {
    const unsigned grid = (unsigned)((int64_t)a.batch * a.channels);
    if (!(aligned_to(a.x, 16) && aligned_to(g.dy, 16) && aligned_to(g.dx, 16))) conv_cf_bwd_kernel<T, KM, kRowScalar><<<grid, kConvThreads, 0, st>>>(g);
    else if (conv_rows_whole(a, 16 / sizeof(T))) conv_cf_bwd_kernel<T, KM, kRowPieces><<<grid, kConvThreads, 0, st>>>(g);
    else conv_cf_bwd_kernel<T, KM, kRowRagged><<<grid, kConvThreads, 0, st>>>(g);
  } else {
    constexpr int V = 4;
    const size_t gb = V * sizeof(T);
    const int vec = (a.channels % V == 0) && aligned_to(a.x, gb) && aligned_to(g.dy, gb) && aligned_to(g.dx, gb);
    if (a.width == 4 && vec && aligned_to(a.weight, 16) && aligned_to(a.bias, 16)) {
      constexpr int VB = 8 / sizeof(T), kPerSm = 512;  // channels and resident threads per SM
      // up to 512 channels: CTAs of 512 threads, each holding all channels at several time tiles
      constexpr int kWide = 512;
      auto launch = [&](auto kern, int threads, int tile) {
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)conv_ring_bytes(threads));
        kern<<<dim3((unsigned)conv_cl_ctas(a, VB, threads, tile), 1, a.batch), threads, conv_ring_bytes(threads), st>>>(g, tile);
      };
      if (a.channels <= kWide) {
        const int tile = conv_cl_tile(a, VB, kWide, kPerSm / kWide, 16, 256);
        launch(a.silu ? conv_cl_bwd4_kernel<T, VB, kWide, true> : conv_cl_bwd4_kernel<T, VB, kWide, false>, kWide, tile);
      } else {
        const int tile = conv_cl_tile(a, VB, kConvThreads, kPerSm / kConvThreads, 16, 256);
        launch(a.silu ? conv_cl_bwd4_kernel<T, VB, kConvThreads, true> : conv_cl_bwd4_kernel<T, VB, kConvThreads, false>, kConvThreads, tile);
      }
    } else {
      conv_cl_bwd_kernel<T, KM><<<conv_cl_grid(a, V), kConvThreads, 0, st>>>(g, vec);
    }
  }
  return launch_status("dw_causal_conv_bwd");
}

template <typename T>
static int conv_fwd_k(const ssm_conv_args& a, cudaStream_t st) {
  return a.width <= 4 ? conv_fwd_launch<T, 4>(a, st) : conv_fwd_launch<T, 8>(a, st);
}
template <typename T>
static int conv_bwd_k(const ssm_conv_bwd_args& g, cudaStream_t st) {
  return g.fwd.width <= 4 ? conv_bwd_launch<T, 4>(g, st) : conv_bwd_launch<T, 8>(g, st);
}

}  // namespace ssmb

using namespace ssmb;

extern "C" int ssm_dw_causal_conv_fwd(const ssm_conv_args* a, ssm_stream_t stream) {
  if (a && a->io_dtype == SSM_F64) {
    ssm_conv_bwd_args g{};
    g.fwd = *a;
    return f64_conv(g, false, reinterpret_cast<cudaStream_t>(stream));
  }
  if (int rc = conv_validate(a)) return rc;
  if (a->batch == 0 || a->channels == 0 || a->len == 0) return SSM_OK;
  SSM_REQUIRE(a->x && a->y && a->weight, SSM_ERR_NULL, "dw_causal_conv: x, weight and y are required");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  switch (a->io_dtype) {
    case SSM_F32: return conv_fwd_k<float>(*a, st);
    case SSM_BF16: return conv_fwd_k<__nv_bfloat16>(*a, st);
    default: return conv_fwd_k<__half>(*a, st);
  }
}

extern "C" int ssm_dw_causal_conv_bwd(const ssm_conv_bwd_args* g, ssm_stream_t stream) {
  SSM_REQUIRE(g != nullptr, SSM_ERR_NULL, "dw_causal_conv_backward: args is NULL");
  const ssm_conv_args* a = &g->fwd;
  if (a->io_dtype == SSM_F64) return f64_conv(*g, true, reinterpret_cast<cudaStream_t>(stream));
  if (int rc = conv_validate(a)) return rc;
  if (a->batch == 0 || a->channels == 0 || a->len == 0) return SSM_OK;
  SSM_REQUIRE(a->x && a->weight && g->dy && g->dx && g->dweight, SSM_ERR_NULL, "dw_causal_conv_backward: missing pointer");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  switch (a->io_dtype) {
    case SSM_F32: return conv_bwd_k<float>(*g, st);
    case SSM_BF16: return conv_bwd_k<__nv_bfloat16>(*g, st);
    default: return conv_bwd_k<__half>(*g, st);
  }
}

static int conv_update_check(const ssm_conv_update_args* a) {
  SSM_REQUIRE(a != nullptr, SSM_ERR_NULL, "dw_causal_conv_update: args is NULL");
  SSM_REQUIRE(a->batch >= 0 && a->channels >= 0 && a->width >= 1, SSM_ERR_SHAPE, "dw_causal_conv_update: bad shape");
  SSM_REQUIRE(valid_dtype(a->io_dtype), SSM_ERR_DTYPE, "dw_causal_conv_update: unknown dtype");
  if ((int64_t)a->batch * a->channels == 0) return SSM_OK;
  SSM_REQUIRE(a->conv_state && a->x && a->weight && a->out, SSM_ERR_NULL, "dw_causal_conv_update: missing pointer");
  SSM_REQUIRE(valid_dtype(a->param_dtype), SSM_ERR_DTYPE, "dw_causal_conv_update: unknown parameter dtype");
  SSM_REQUIRE(a->width != 4 || aligned_to(a->weight, 4 * dtype_size(a->param_dtype)), SSM_ERR_ALIGN, "dw_causal_conv_update: weight must be aligned to four elements");
  return SSM_OK;
}

extern "C" int ssmb_conv_update_many(const ssm_conv_update_args* a, int32_t n, void* stream) {
  SSM_REQUIRE(n >= 1 && n <= 3, SSM_ERR_UNSUPPORTED, "dw_causal_conv_update: one to three windows");
  for (int i = 0; i < n; ++i) {
    if (int rc = conv_update_check(a + i)) return rc;
    if ((int64_t)a[i].batch * a[i].channels == 0) return SSM_OK;  // (the windows share the batch)
  }
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  switch (a->io_dtype) {
    case SSM_F32: return conv_update_t<float>(a, n, st);
    case SSM_BF16: return conv_update_t<__nv_bfloat16>(a, n, st);
    default: return conv_update_t<__half>(a, n, st);
  }
}

extern "C" int ssm_dw_causal_conv_update(const ssm_conv_update_args* a, ssm_stream_t stream) { return ssmb_conv_update_many(a, 1, stream); }
