// One decode token through a whole mixer in one launch, for small batches (up to 16 sequences), sm_100a.
//
// A decode step at batch 1 reads a few MB of weights once and does almost no arithmetic; as separate calls it was bound by
// launches (a Mamba-1 block of d_model 768: 13 launches, 39 us of device time and 130 us of host time for 8 MB of
// weights and states).  Here the phases between the matrix-vector products are separated by a grid barrier instead of a
// launch: one cooperative kernel, one CTA of 32 warps per SM.
//
//   Mamba-1:  [x | z] = W_in t, conv window, SiLU -> u | x_proj u | dt_proj, softplus, state step, gate -> y | out_proj y | add + RMSNorm
//   Mamba-2:  [z | x | B | C | dt] = W_in t, conv windows | state step, gate -> y | RMSNorm folded into the staging of y, out_proj
//
// The products are bound by the weight stream.  A tile is 8 weight rows; each lane reads 16 contiguous bytes of a row per
// 32 columns and hands them to mma.m16n8k16 as the N operand (the token rows are M: up to 16 sequences cost the same as
// one).  K runs over the columns in the order in which the lanes hold them, the same for both operands, so no element
// moves between lanes.  A tile's columns are split over S warps, whose partial sums meet in shared memory: S is chosen
// per phase so that the tiles fill the GPU in few rounds.  Every value that the separate operators round to the
// activation type (projections, u, delta, y) is rounded here too.
//
// 16 sequences fill the M of one mma; more would stream the weights again.  us per step, CUDA-graph replays, this kernel at 1, 8 and 16
// sequences against library GEMMs around the single-step kernels at 1, 16, 17, 32 and 64:
//   Mamba-1 d_model  768   15.6  17.0  18.7   against  24.6  24.0  23.5  24.2   25.5
//   Mamba-1 d_model 2560   31.4  37.2  45.1   against  44.2  42.5  45.3  49.2   51.9
//   Mamba-2 d_model  768   16.7  19.2  23.8   against  33.4  37.8  38.2  37.8   45.1
//   Mamba-2 d_model 2560   31.6  45.6  63.7   against  56.2  75.9  77.0  89.1  115.6
// Without a graph the separate calls take 70 to 100 us of host time.
// 17 to 256 sequences take a few overlapped launches instead, with products of their own (decode_parts.h): a Mamba-1 step of 256 sequences at
// d_model 2560 97 us, against 110 with library GEMMs.
#include <cooperative_groups.h>

#include <algorithm>

#include "common.cuh"

namespace ssmb {

namespace cg = cooperative_groups;

constexpr int kDecThreads = 1024;
constexpr int kDecWarps = kDecThreads / 32;
constexpr int kDecRows = 8;       // weight rows per tile
constexpr int kDecMaxBatch = 16;  // token rows of one mma

template <typename T>
__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1);
template <>
__device__ __forceinline__ void mma_16816<__nv_bfloat16>(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
template <>
__device__ __forceinline__ void mma_16816<__half>(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint4 ld_weights(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// bytes between the staged token rows: half a 128-byte line off a whole number of lines, so that the two rows that a
// quarter-warp reads lie in different banks
__host__ __device__ inline int dec_pitch(int k) { return (k * 2) % 128 == 0 ? k * 2 + 64 : k * 2; }

// token rows (nb, k) -> shared memory.  CG: written by other CTAs earlier in this kernel, read through the L2.
template <bool CG>
__device__ __forceinline__ void stage_rows(const void* src, unsigned char* dst, int nb, int k, int pitch) {
  const int per = k / 8;
  for (int i = threadIdx.x; i < nb * per; i += kDecThreads) {
    const int b = i / per, u = i % per;
    const uint4* p = reinterpret_cast<const uint4*>(src) + (size_t)b * per + u;
    *reinterpret_cast<uint4*>(dst + (size_t)b * pitch + u * 16) = CG ? __ldcg(p) : __ldg(p);
  }
}

// Up to five weight matrices of one input, stacked: tiles of 8 rows, every matrix starting a new tile.
template <int NSEG>
struct DecMats {
  const void* w[NSEG];
  int rows[NSEG];
  __device__ __forceinline__ int tiles() const {
    int t = 0;
#pragma unroll
    for (int s = 0; s < NSEG; ++s) t += (rows[s] + kDecRows - 1) / kDecRows;
    return t;
  }
};

// out[b][r] = <w row r, token row b> for all rows of `m`; epi(segment, b, row, value) receives every result once.
// `split` warps share a tile; called by the whole CTA.
template <typename T, int NSEG, typename Epi>
__device__ __forceinline__ void dec_gemv(const DecMats<NSEG>& m, int nb, int k, int split, const unsigned char* xs, int pitch, float* red, const Epi& epi) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int grp = warp / split, part = warp % split;
  const int groups = kDecWarps / split;
  const int tiles = m.tiles(), slots = gridDim.x * groups;
  const int g = lane >> 2, t4 = lane & 3;
  const int nchunk = k / 32, per = (nchunk + split - 1) / split;
  const int c_begin = min(part * per, nchunk), c_end = min(c_begin + per, nchunk);
  const bool two = nb > 8;  // token rows 8..15 in use
  for (int first = blockIdx.x; first < tiles; first += slots) {  // the same number of rounds for every warp of the CTA
    int tile = first + grp * gridDim.x, seg = -1, row0 = 0;
    if (tile < tiles) {
      int at = 0;
#pragma unroll
      for (int s = 0; s < NSEG; ++s) {
        const int n = (m.rows[s] + kDecRows - 1) / kDecRows;
        if (tile >= at && tile < at + n) seg = s, row0 = (tile - at) * kDecRows;
        at += n;
      }
    }
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    int rows = 0;
    if (seg >= 0) {
      const void* wbase = nullptr;
#pragma unroll
      for (int s = 0; s < NSEG; ++s)
        if (s == seg) wbase = m.w[s], rows = m.rows[s];
      const int r = min(row0 + g, rows - 1);  // rows beyond the matrix read its last row and are dropped
      const T* wp = reinterpret_cast<const T*>(wbase) + (size_t)r * k + t4 * 8;
      const unsigned char* x0 = xs + (size_t)min(g, nb - 1) * pitch + t4 * 16;
      const unsigned char* x1 = xs + (size_t)min(g + 8, nb - 1) * pitch + t4 * 16;
      for (int c = c_begin; c < c_end; c += 6) {
        uint4 w[6];
#pragma unroll
        for (int j = 0; j < 6; ++j)
          if (c + j < c_end) w[j] = ld_weights(wp + (size_t)(c + j) * 32);
#pragma unroll
        for (int j = 0; j < 6; ++j)
          if (c + j < c_end) {
            const uint4 a = *reinterpret_cast<const uint4*>(x0 + (c + j) * 64);
            uint4 b = make_uint4(0u, 0u, 0u, 0u);
            if (two) b = *reinterpret_cast<const uint4*>(x1 + (c + j) * 64);
            mma_16816<T>(acc, a.x, b.x, a.y, b.y, w[j].x, w[j].y);
            mma_16816<T>(acc, a.z, b.z, a.w, b.w, w[j].z, w[j].w);
          }
      }
    }
    // partial sums of this warp: [token row][weight row]
    float* mine = red + warp * (kDecMaxBatch * kDecRows);
    *reinterpret_cast<float2*>(mine + g * kDecRows + t4 * 2) = make_float2(acc[0], acc[1]);
    if (two) *reinterpret_cast<float2*>(mine + (g + 8) * kDecRows + t4 * 2) = make_float2(acc[2], acc[3]);
    __syncthreads();
    if (seg >= 0) {
      const float* base = red + grp * split * (kDecMaxBatch * kDecRows);
      for (int o = part * 32 + lane; o < nb * kDecRows; o += split * 32) {
        float v = 0.f;
        for (int s = 0; s < split; ++s) v += base[s * (kDecMaxBatch * kDecRows) + o];
        const int row = row0 + (o & (kDecRows - 1));
        if (row < rows) epi(seg, o / kDecRows, row, v);
      }
    }
    __syncthreads();
  }
}

// push one value into a conv window of four and return act(bias + <window, weights>)
template <typename T>
__device__ __forceinline__ float dec_conv4(float* state, float x, const T* w, const T* bias, int channel) {
  float4 v = *reinterpret_cast<const float4*>(state);
  v = make_float4(v.y, v.z, v.w, x);
  *reinterpret_cast<float4*>(state) = v;
  const T* wr = w + (size_t)channel * 4;
  float acc = bias ? to_f<T>(__ldg(bias + channel)) : 0.f;
  acc = fmaf(v.x, to_f<T>(__ldg(wr)), fmaf(v.y, to_f<T>(__ldg(wr + 1)), fmaf(v.z, to_f<T>(__ldg(wr + 2)), fmaf(v.w, to_f<T>(__ldg(wr + 3)), acc))));
  return silu_fast(acc);
}
template <typename T>
__device__ __forceinline__ float round_to(float v) {
  return to_f<T>(from_f<T>(v));
}
template <typename T>
__device__ __forceinline__ T ldcg_t(const T* p) {
  const unsigned short u = __ldcg(reinterpret_cast<const unsigned short*>(p));
  return *reinterpret_cast<const T*>(&u);
}

__device__ __forceinline__ float block_sum(float v, float* scratch) {
  v = warp_sum(v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = scratch[threadIdx.x & 31];
  return warp_sum(t);
}

struct DecSplits {
  int s[4];
};

// ---------------------------------------------------------------------------------------------
// Mamba-1
// ---------------------------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(kDecThreads, 1) mamba1_decode_kernel(const ssm_mamba1_decode_args a, const DecSplits sp) {
  extern __shared__ __align__(16) unsigned char dsm[];
  __shared__ float sum_scratch[32];
  float* red = reinterpret_cast<float*>(dsm);
  unsigned char* xs = dsm + kDecWarps * kDecMaxBatch * kDecRows * 4;
  cg::grid_group grid = cg::this_grid();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nb = a.batch, dm = a.d_model, di = a.d_inner, R = a.dt_rank, xw = R + 2 * a.nstate;
  T* zb = reinterpret_cast<T*>(a.scratch);
  T* ub = zb + (size_t)nb * di;
  T* yb = ub + (size_t)nb * di;
  T* ob = yb + (size_t)nb * di;
  T* xd = ob + (size_t)nb * dm;
  const int gtid = blockIdx.x * kDecThreads + tid, gsize = gridDim.x * kDecThreads;

  // weights of the later phases on their way into the L2 while the first phase runs
  {
    const size_t n1 = (size_t)xw * di * 2 / 128, n2 = (size_t)di * R * 2 / 128, n3 = (size_t)dm * di * 2 / 128;
    for (size_t i = gtid; i < n1 + n2 + n3; i += gsize) {
      const char* p = i < n1 ? reinterpret_cast<const char*>(a.x_proj) + i * 128
                             : (i < n1 + n2 ? reinterpret_cast<const char*>(a.dt_proj) + (i - n1) * 128 : reinterpret_cast<const char*>(a.out_proj) + (i - n1 - n2) * 128);
      prefetch_l2(p);
    }
  }
  // ---- x and z projections; conv window and SiLU on x --------------------------------------------------------
  const int pm = dec_pitch(dm), pi = dec_pitch(di);
  stage_rows<false>(a.hidden, xs, nb, dm, pm);
  __syncthreads();
  {
    DecMats<2> m{{a.in_x, a.in_z}, {di, di}};
    dec_gemv<T>(m, nb, dm, sp.s[0], xs, pm, red, [&](int seg, int b, int row, float v) {
      const size_t at = (size_t)b * di + row;
      if (seg == 0)
        ub[at] = from_f<T>(dec_conv4<T>(a.conv_state + at * 4, round_to<T>(v), reinterpret_cast<const T*>(a.conv_w), reinterpret_cast<const T*>(a.conv_b), row));
      else
        zb[at] = from_f<T>(v);
    });
  }
  grid.sync();
  // ---- dt_low, B, C = x_proj u -------------------------------------------------------------------------------
  {
    DecMats<1> m{{a.x_proj}, {xw}};
    if ((int)blockIdx.x < m.tiles()) {
      stage_rows<true>(ub, xs, nb, di, pi);
      __syncthreads();
      dec_gemv<T>(m, nb, di, sp.s[1], xs, pi, red, [&](int, int b, int row, float v) { xd[(size_t)b * xw + row] = from_f<T>(v); });
    }
  }
  grid.sync();
  // ---- delta, state step, gate: a warp takes eight channels of one sequence, four lanes per channel --------------
  {
    float* sx = reinterpret_cast<float*>(xs);  // dt_low | B | C of every sequence in fp32
    for (int i = tid; i < nb * xw; i += kDecThreads) sx[i] = to_f<T>(ldcg_t<T>(xd + i));
    __syncthreads();
    const int oct = (di + 7) / 8, q = lane & 3;
    for (int it = blockIdx.x + gridDim.x * warp; it < oct * nb; it += gridDim.x * kDecWarps) {
      const int b = it / oct, d = (it % oct) * 8 + (lane >> 2);
      const bool live = d < di;
      const int dd = live ? d : di - 1;
      const size_t at = (size_t)b * di + dd;
      float* st = a.ssm_state + at * 16 + q * 4;
      const float4 s4 = *reinterpret_cast<const float4*>(st);
      const float4 A4 = __ldg(reinterpret_cast<const float4*>(a.A + (size_t)dd * 16 + q * 4));
      const float u = to_f<T>(ldcg_t<T>(ub + at)), z = to_f<T>(ldcg_t<T>(zb + at));
      const float* xb = sx + b * xw;
      const T* w = reinterpret_cast<const T*>(a.dt_proj) + (size_t)dd * R;
      float dt = 0.f;
      for (int k = q * 4; k < R; k += 16) {  // R is a multiple of 4: 8-byte pieces
        const uint2 raw = __ldg(reinterpret_cast<const uint2*>(w + k));
        const T* e = reinterpret_cast<const T*>(&raw);
        const float4 x4 = *reinterpret_cast<const float4*>(xb + k);
        dt = fmaf(to_f<T>(e[0]), x4.x, fmaf(to_f<T>(e[1]), x4.y, fmaf(to_f<T>(e[2]), x4.z, fmaf(to_f<T>(e[3]), x4.w, dt))));
      }
      dt = round_to<T>(group_sum<4, 1>(dt)) + __ldg(a.dt_bias + dd);
      dt = softplus_fast(dt);
      const float4 B4 = *reinterpret_cast<const float4*>(xb + R + q * 4);
      const float4 C4 = *reinterpret_cast<const float4*>(xb + R + 16 + q * 4);
      const float dtx = dt * u;
      float sv[4] = {s4.x, s4.y, s4.z, s4.w};
      const float Av[4] = {A4.x, A4.y, A4.z, A4.w}, Bv[4] = {B4.x, B4.y, B4.z, B4.w}, Cv[4] = {C4.x, C4.y, C4.z, C4.w};
      float y = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float An = a.a_log ? -expf(Av[i]) : Av[i];
        sv[i] = fmaf(ex2_approx(dt * An * kLog2e), sv[i], dtx * Bv[i]);
        y = fmaf(Cv[i], sv[i], y);
      }
      if (live) *reinterpret_cast<float4*>(st) = make_float4(sv[0], sv[1], sv[2], sv[3]);
      y = group_sum<4, 1>(y);
      if (q == 0 && live) yb[at] = from_f<T>(fmaf(__ldg(a.D + dd), u, y) * silu_fast(z));
    }
  }
  grid.sync();
  // ---- out projection ----------------------------------------------------------------------------------------
  {
    DecMats<1> m{{a.out_proj}, {dm}};
    T* dst = a.norm_w ? ob : reinterpret_cast<T*>(a.out);
    if ((int)blockIdx.x < m.tiles()) {
      stage_rows<true>(yb, xs, nb, di, pi);
      __syncthreads();
      dec_gemv<T>(m, nb, di, sp.s[2], xs, pi, red, [&](int, int b, int row, float v) { dst[(size_t)b * dm + row] = from_f<T>(v); });
    }
  }
  if (!a.norm_w) return;
  grid.sync();
  // ---- residual add and RMSNorm: one CTA per sequence ----------------------------------------------------------
  for (int b = blockIdx.x; b < nb; b += gridDim.x) {
    float* row = reinterpret_cast<float*>(xs);
    float q = 0.f;
    for (int i = tid; i < dm; i += kDecThreads) {
      const size_t at = (size_t)b * dm + i;
      float v = to_f<T>(ldcg_t<T>(ob + at));
      if (a.residual) v += load_dyn(a.residual, at, a.res_dtype);
      store_dyn(a.residual_out, at, a.resout_dtype, v);
      row[i] = v;
      q = fmaf(v, v, q);
    }
    const float rstd = rsqrtf(block_sum(q, sum_scratch) / (float)dm + a.eps);
    for (int i = tid; i < dm; i += kDecThreads)
      reinterpret_cast<T*>(a.out)[(size_t)b * dm + i] = from_f<T>(row[i] * rstd * to_f<T>(__ldg(reinterpret_cast<const T*>(a.norm_w) + i)));
  }
}

// ---------------------------------------------------------------------------------------------
// Mamba-2
// ---------------------------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(kDecThreads, 1) mamba2_decode_kernel(const ssm_mamba2_decode_args a, const DecSplits sp) {
  extern __shared__ __align__(16) unsigned char dsm[];
  __shared__ float sum_scratch[32];
  float* red = reinterpret_cast<float*>(dsm);
  unsigned char* xs = dsm + kDecWarps * kDecMaxBatch * kDecRows * 4;
  cg::grid_group grid = cg::this_grid();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nb = a.batch, dm = a.d_model, nh = a.heads, di = nh * 64, gn = a.groups * 128;
  T* zb = reinterpret_cast<T*>(a.scratch);
  T* ub = zb + (size_t)nb * di;
  T* yb = ub + (size_t)nb * di;
  T* bb = yb + (size_t)nb * di;
  T* cb = bb + (size_t)nb * gn;
  T* db = cb + (size_t)nb * gn;
  {
    const size_t n = (size_t)dm * di * 2 / 128;
    for (size_t i = blockIdx.x * kDecThreads + tid; i < n; i += (size_t)gridDim.x * kDecThreads) prefetch_l2(reinterpret_cast<const char*>(a.out_proj) + i * 128);
  }
  // ---- z, x, B, C, dt projections; conv windows and SiLU on x, B, C ----------------------------------------------
  const int pm = dec_pitch(dm), pi = dec_pitch(di);
  stage_rows<false>(a.hidden, xs, nb, dm, pm);
  __syncthreads();
  {
    DecMats<5> m{{a.in_x, a.in_z, a.in_B, a.in_C, a.in_dt}, {di, di, gn, gn, nh}};
    dec_gemv<T>(m, nb, dm, sp.s[0], xs, pm, red, [&](int seg, int b, int row, float v) {
      auto conv = [&](float* state, const void* w, const void* bias, int width) {
        return from_f<T>(dec_conv4<T>(state + ((size_t)b * width + row) * 4, round_to<T>(v), reinterpret_cast<const T*>(w), reinterpret_cast<const T*>(bias), row));
      };
      switch (seg) {
        case 0: ub[(size_t)b * di + row] = conv(a.conv_state_x, a.conv_x_w, a.conv_x_b, di); break;
        case 1: zb[(size_t)b * di + row] = from_f<T>(v); break;
        case 2: bb[(size_t)b * gn + row] = conv(a.conv_state_B, a.conv_B_w, a.conv_B_b, gn); break;
        case 3: cb[(size_t)b * gn + row] = conv(a.conv_state_C, a.conv_C_w, a.conv_C_b, gn); break;
        default: db[(size_t)b * nh + row] = from_f<T>(v); break;
      }
    });
  }
  grid.sync();
  // ---- state step and gate: a warp takes eight rows of one head, a lane four of the 128 states ---------------------
  {
    constexpr int RPW = 8;
    const int items = nb * nh * (64 / RPW);
    for (int it = blockIdx.x + gridDim.x * warp; it < items; it += gridDim.x * kDecWarps) {
      const int p0 = (it % (64 / RPW)) * RPW, h = (it / (64 / RPW)) % nh, b = it / (64 / RPW * nh);
      const int grp = h / (nh / a.groups);
      float* st = a.ssm_state + (((size_t)b * nh + h) * 64 + p0) * 128 + lane * 4;
      float4 s4[RPW];
#pragma unroll
      for (int r = 0; r < RPW; ++r) s4[r] = __ldcs(reinterpret_cast<const float4*>(st + r * 128));
      const uint2 braw = __ldcg(reinterpret_cast<const uint2*>(bb + (size_t)b * gn + grp * 128 + lane * 4));
      const uint2 craw = __ldcg(reinterpret_cast<const uint2*>(cb + (size_t)b * gn + grp * 128 + lane * 4));
      const T *be = reinterpret_cast<const T*>(&braw), *ce = reinterpret_cast<const T*>(&craw);
      const float dt = softplus_fast(to_f<T>(ldcg_t<T>(db + (size_t)b * nh + h)) + __ldg(a.dt_bias + h));
      const float Ah = a.a_log ? -expf(__ldg(a.A + h)) : __ldg(a.A + h);
      const float da = ex2_approx(dt * Ah * kLog2e);
      const size_t at0 = (size_t)b * di + h * 64 + p0;
      float y[RPW];
#pragma unroll
      for (int r = 0; r < RPW; ++r) {
        const float dtx = dt * to_f<T>(ldcg_t<T>(ub + at0 + r));
        float sv[4] = {s4[r].x, s4[r].y, s4[r].z, s4[r].w};
        y[r] = 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          sv[i] = fmaf(da, sv[i], dtx * to_f<T>(be[i]));
          y[r] = fmaf(to_f<T>(ce[i]), sv[i], y[r]);
        }
        __stcs(reinterpret_cast<float4*>(st + r * 128), make_float4(sv[0], sv[1], sv[2], sv[3]));
      }
      // eight sums over the 32 lanes: after the scatter a group of four lanes shares row lane / 4
      reduce_scatter<8, 4, RPW>(y, lane);
      const float ys = group_sum<4, 1>(y[0]);
      if ((lane & 3) == 0) {
        const int r = lane >> 2;
        const float u = to_f<T>(ldcg_t<T>(ub + at0 + r)), z = to_f<T>(ldcg_t<T>(zb + at0 + r));
        yb[at0 + r] = from_f<T>(fmaf(__ldg(a.D + h), u, ys) * silu_fast(z));
      }
    }
  }
  grid.sync();
  // ---- RMSNorm over d_inner while y is staged (every CTA that has a tile forms it again: no barrier), out projection ----
  {
    DecMats<1> m{{a.out_proj}, {dm}};
    if ((int)blockIdx.x < m.tiles()) {
      stage_rows<true>(yb, xs, nb, di, pi);
      __syncthreads();
      // two warps per sequence, both of which sum the whole row; the rescale below goes over all rows by thread
      const int wpb = kDecWarps / kDecMaxBatch;  // 2
      for (int b = warp / wpb; b < nb; b += kDecMaxBatch) {
        T* row = reinterpret_cast<T*>(xs + (size_t)b * pi);
        float q = 0.f;
        for (int i = lane; i < di; i += 32) {
          const float v = to_f<T>(row[i]);
          q = fmaf(v, v, q);
        }
        const float rstd = rsqrtf(warp_sum(q) / (float)di + a.eps);
        if (lane == 0) sum_scratch[b] = rstd;  // both warps of a sequence write the same value
      }
      __syncthreads();
      for (int i = tid; i < nb * di; i += kDecThreads) {
        const int b = i / di, c = i % di;
        T* e = reinterpret_cast<T*>(xs + (size_t)b * pi) + c;
        *e = from_f<T>(to_f<T>(*e) * sum_scratch[b] * to_f<T>(__ldg(reinterpret_cast<const T*>(a.norm_w) + c)));
      }
      __syncthreads();
      dec_gemv<T>(m, nb, di, sp.s[1], xs, pi, red, [&](int, int b, int row, float v) { reinterpret_cast<T*>(a.out)[(size_t)b * dm + row] = from_f<T>(v); });
    }
  }
}

// Warps per tile: the split with the least rounds x (columns per warp + a round's fixed cost, which is worth about eight
// 32-column pieces: two CTA barriers, the exchange of the partial sums, the epilogue).
static int dec_split(int tiles, int k, int sms) {
  int best = 1;
  double cost = 1e300;
  for (int s = 1; s <= kDecWarps; s *= 2) {
    const int slots = sms * (kDecWarps / s), per = (k / 32 + s - 1) / s;
    const double c = (double)((tiles + slots - 1) / slots) * (per + 8.0);
    if (c < cost) cost = c, best = s;
  }
  return best;
}
static int tiles_of(int rows) { return (rows + kDecRows - 1) / kDecRows; }
static size_t dec_smem(int batch, int kmax) { return (size_t)kDecWarps * kDecMaxBatch * kDecRows * 4 + (size_t)batch * dec_pitch(kmax); }
constexpr size_t kDecMaxSmem = 220 * 1024;

template <typename K, typename A>
static int dec_launch(K kernel, const A& a, const DecSplits& sp, int sms, size_t smem, cudaStream_t st, const char* name) {
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  A arg = a;
  DecSplits s = sp;
  void* params[] = {&arg, &s};
  const cudaError_t e = cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(kernel), dim3(sms), dim3(kDecThreads), params, smem, st);
  if (e != cudaSuccess) {
    cudaGetLastError();  // reported here; the next launch starts clean
    set_error("%s: %s", name, cudaGetErrorString(e));
    // a CTA per SM of the device, but the context may have fewer to give (green contexts, partitions): the separate calls serve it
    return e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported ? SSM_ERR_UNSUPPORTED : (int)e;
  }
  return launch_status(name);
}

}  // namespace ssmb

using namespace ssmb;

extern "C" int ssm_mamba1_decode_supported(int32_t batch, int32_t d_model, int32_t d_inner, int32_t nstate, int32_t dt_rank, int32_t width, int32_t io_dtype) {
  return batch >= 1 && batch <= kDecMaxBatch && d_model >= 32 && d_model % 32 == 0 && d_inner >= 32 && d_inner % 32 == 0 && nstate == 16 && dt_rank >= 4 &&
         dt_rank % 4 == 0 && width == 4 && (io_dtype == SSM_BF16 || io_dtype == SSM_F16) && d_model <= 16384 &&
         dec_smem(batch, d_inner > 2 * d_model ? d_inner : 2 * d_model) <= kDecMaxSmem && (size_t)batch * (dt_rank + 32) * 4 <= (size_t)batch * d_inner * 2;
}
extern "C" int64_t ssm_mamba1_decode_scratch_bytes(int32_t batch, int32_t d_model, int32_t d_inner, int32_t nstate, int32_t dt_rank) {
  return 2 * (int64_t)batch * (3 * (int64_t)d_inner + d_model + dt_rank + 2 * nstate);
}
extern "C" int ssm_mamba1_decode(const ssm_mamba1_decode_args* a, ssm_stream_t stream) {
  SSM_REQUIRE(a != nullptr, SSM_ERR_NULL, "mamba1_decode: args is NULL");
  if (a->batch == 0) return SSM_OK;
  SSM_REQUIRE(ssm_mamba1_decode_supported(a->batch, a->d_model, a->d_inner, a->nstate, a->dt_rank, a->width, a->io_dtype), SSM_ERR_UNSUPPORTED,
              "mamba1_decode: built for up to 16 sequences, d_state 16, conv width 4, bf16 / fp16");
  SSM_REQUIRE(a->hidden && a->in_x && a->in_z && a->conv_w && a->x_proj && a->dt_proj && a->dt_bias && a->A && a->D && a->out_proj && a->conv_state &&
                  a->ssm_state && a->out && a->scratch && (!a->norm_w || a->residual_out),
              SSM_ERR_NULL, "mamba1_decode: missing tensor");
  SSM_REQUIRE(aligned_to(a->hidden, 16) && aligned_to(a->in_x, 16) && aligned_to(a->in_z, 16) && aligned_to(a->x_proj, 16) && aligned_to(a->dt_proj, 8) &&
                  aligned_to(a->out_proj, 16) && aligned_to(a->conv_state, 16) && aligned_to(a->ssm_state, 16) && aligned_to(a->A, 16) && aligned_to(a->scratch, 16),
              SSM_ERR_ALIGN, "mamba1_decode: tensors must be 16-byte aligned");
  const int sms = sm_count();
  DecSplits sp{};
  sp.s[0] = dec_split(2 * tiles_of(a->d_inner), a->d_model, sms);
  sp.s[1] = dec_split(tiles_of(a->dt_rank + 2 * a->nstate), a->d_inner, sms);
  sp.s[2] = dec_split(tiles_of(a->d_model), a->d_inner, sms);
  const size_t smem = dec_smem(a->batch, a->d_inner > 2 * a->d_model ? a->d_inner : 2 * a->d_model);  // the last phase keeps a row of d_model floats
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (a->io_dtype == SSM_BF16) return dec_launch(mamba1_decode_kernel<__nv_bfloat16>, *a, sp, sms, smem, st, "mamba1_decode_kernel");
  return dec_launch(mamba1_decode_kernel<__half>, *a, sp, sms, smem, st, "mamba1_decode_kernel");
}

extern "C" int ssm_mamba2_decode_supported(int32_t batch, int32_t d_model, int32_t heads, int32_t headdim, int32_t nstate, int32_t groups, int32_t width,
                                           int32_t io_dtype) {
  return batch >= 1 && batch <= kDecMaxBatch && d_model >= 32 && d_model % 32 == 0 && heads >= 1 && headdim == 64 && nstate == 128 && groups >= 1 &&
         heads % groups == 0 && width == 4 && (io_dtype == SSM_BF16 || io_dtype == SSM_F16) &&
         dec_smem(batch, heads * 64 > d_model ? heads * 64 : d_model) <= kDecMaxSmem;
}
extern "C" int64_t ssm_mamba2_decode_scratch_bytes(int32_t batch, int32_t heads, int32_t groups) {
  return 2 * (int64_t)batch * (3 * (int64_t)heads * 64 + 2 * (int64_t)groups * 128 + heads);
}
extern "C" int ssm_mamba2_decode(const ssm_mamba2_decode_args* a, ssm_stream_t stream) {
  SSM_REQUIRE(a != nullptr, SSM_ERR_NULL, "mamba2_decode: args is NULL");
  if (a->batch == 0) return SSM_OK;
  SSM_REQUIRE(ssm_mamba2_decode_supported(a->batch, a->d_model, a->heads, a->headdim, a->nstate, a->groups, a->width, a->io_dtype), SSM_ERR_UNSUPPORTED,
              "mamba2_decode: built for up to 16 sequences, headdim 64, d_state 128, conv width 4, bf16 / fp16");
  SSM_REQUIRE(a->hidden && a->in_z && a->in_x && a->in_B && a->in_C && a->in_dt && a->conv_x_w && a->conv_B_w && a->conv_C_w && a->dt_bias && a->A && a->D &&
                  a->norm_w && a->out_proj && a->conv_state_x && a->conv_state_B && a->conv_state_C && a->ssm_state && a->out && a->scratch,
              SSM_ERR_NULL, "mamba2_decode: missing tensor");
  SSM_REQUIRE(aligned_to(a->hidden, 16) && aligned_to(a->in_z, 16) && aligned_to(a->in_x, 16) && aligned_to(a->in_B, 16) && aligned_to(a->in_C, 16) &&
                  aligned_to(a->in_dt, 16) && aligned_to(a->out_proj, 16) && aligned_to(a->conv_state_x, 16) && aligned_to(a->conv_state_B, 16) &&
                  aligned_to(a->conv_state_C, 16) && aligned_to(a->ssm_state, 16) && aligned_to(a->scratch, 16),
              SSM_ERR_ALIGN, "mamba2_decode: tensors must be 16-byte aligned");
  const int sms = sm_count(), di = a->heads * 64;
  DecSplits sp{};
  sp.s[0] = dec_split(2 * tiles_of(di) + 2 * tiles_of(a->groups * 128) + tiles_of(a->heads), a->d_model, sms);
  sp.s[1] = dec_split(tiles_of(a->d_model), di, sms);
  const size_t smem = dec_smem(a->batch, di > a->d_model ? di : a->d_model);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (a->io_dtype == SSM_BF16) return dec_launch(mamba2_decode_kernel<__nv_bfloat16>, *a, sp, sms, smem, st, "mamba2_decode_kernel");
  return dec_launch(mamba2_decode_kernel<__half>, *a, sp, sms, smem, st, "mamba2_decode_kernel");
}
