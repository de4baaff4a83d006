// Mamba-1 selective scan, backward, for calls of 5 to 16 states whose CTAs' rows share one B / C group.
//
// A lane keeps four states of TWO rows, and every packed fp32 (f32x2) instruction works on the same state of both: a step's B_n and
// C_n are broadcast operands (free in hardware), delta, u and dy lie in shared memory as pairs of rows, and nothing is moved
// between registers to form operands.  Time is walked in reverse in tiles of one checkpoint interval, by two kinds of warps:
//   producers  rebuild the states of a tile from the checkpoint the forward stored, and keep them after every fourth step; delta after
//              softplus, u, <C, h>, from which dy = dout silu(z) and dz, which they write out;
//   consumers  the adjoint G_t = C_t dy_t + a_{t+1} G_{t+1}, four steps at a time, the states in between rebuilt from the kept
//              ones; du, ddelta and the parameter gradients.
// A tile does not need the one before it to be rebuilt, so the producers work a tile ahead: this doubles the warps that a call's rows
// give the GPU without a second pass.  Buffers are half tiles (16 steps): a tile's upper half, which the consumers take first, has one;
// lower halves alternate between two.
// Sums over states (du, ddelta, y) are reduce-scatters across the lanes of a row.  Sums over rows (dB, dC): the lane's two rows in a
// register, the warp's row pairs through a staging area, then one 16-byte reduction per output to global memory.
//
// Bound by the issue of the schedulers that hold consumers, about half of whose slots wait for fixed latencies (26 instructions per
// (row, state, step), of which 2.5 ex2 and 14 on the fp32 pipe; 33 in the kernel with one row per lane).  Whole backward, us:
//   8 x 1536 rows of 4096 steps, 16 states: bf16 1662 -> 1390, fp32 (two CTAs per SM) 2380 -> 1834;  2 x 1536 bf16, cut in time: 548 -> 485
//   4 x 2048 rows of 2048 steps,  8 states: bf16 680 -> 567
// One kind of warp that does both (six warps per SM): 1784; two states per lane and twelve warps: 1750.
#pragma once

#include "scan_common.cuh"

namespace ssmb {

template <typename T, int LPR, bool PIECES>
struct BwdPairs {
  static constexpr int NS = 4, NP = NS * LPR;      // states of a lane, of a row
  static constexpr int RPW = 32 / LPR;             // row pairs of a warp
  static constexpr int NW = 2;                     // warps of a kind
  static constexpr int ROWS = NW * 2 * RPW;
  static constexpr int TL = kScanCkpt, HL = TL / 2;
  static constexpr int PITCH = HL + 2;  // pairs of a row pair's half tile: 16 bytes more, so that eight of them cover all banks
  static constexpr int V = 16 / (int)sizeof(T), RP = TL + V;  // pitch of a raw row (PIECES: rows that start anywhere take one piece more)
  // floats
  static constexpr int ROW_ARRAY = RPW * PITCH * 2;
  static constexpr int HIST = (HL / 4) * 32 * 2 * NS;  // states before every fourth step of a half
  static constexpr int BC = 2 * HL * NP;               // B, C as [HL][NP]
  static constexpr int HALF = BC + NW * (3 * ROW_ARRAY + HIST);
  static constexpr int STAGE = 2 * NP * RPW * 4;       // dB / dC products of four steps: [2 * NP][RPW][4]
  static constexpr int LAST = 32 * 2 * NS;             // states after the call's (segment's) last step
  // bytes
  static constexpr int BC_RAW_BYTES = 2 * NP * (TL + (PIECES ? 4 : 0)) * 4;
  static constexpr int WARP_RAW_BYTES = 4 * 2 * RPW * RP * (int)sizeof(T);
  static constexpr size_t kBytes = sizeof(float) * (3 * HALF + NW * (STAGE + LAST)) + BC_RAW_BYTES + NW * WARP_RAW_BYTES;
  static_assert(kBytes <= 227 * 1024, "shared memory budget");
};

// Sums over the lanes of a row pair.  In: eight values of four steps, entry 2 * step + row.  Out: lane group g = (lane / RPW) % LPR
// holds entries g * 8 / LPR ...
template <int LPR, int RPW>
__device__ __forceinline__ void pair_sums(float (&p)[8], int lane) { reduce_scatter<LPR, RPW, 8>(p, lane); }

// 16-byte pieces of the rows of a warp (row pair p: rows p and p + RPW); dst pitch TL + V
template <typename T, int ROWS, int TL>
__device__ __forceinline__ void fill_rows_pitched(T* __restrict__ raw, const T* __restrict__ g, int b, int D, int L, int drow0, int t0, bool vec, int lane,
                                                  int64_t sb, int64_t sd) {
  constexpr int V = 16 / sizeof(T), CH = TL / V, RP = TL + V;
  if (vec) {
    for (int c = lane; c < ROWS * CH; c += 32) {
      const int rr = c / CH, ch = c % CH;
      const int t = t0 + ch * V;
      const bool ok = t < L;
      cp_async16(raw + rr * RP + ch * V, g + (int64_t)b * sb + (int64_t)min(drow0 + rr, D - 1) * sd + (ok ? t : 0), ok);
    }
  } else {
    for (int i = lane; i < ROWS * TL; i += 32) {
      const int rr = i / TL, tt = i % TL, t = t0 + tt;
      raw[rr * RP + tt] = t < L ? g[(int64_t)b * sb + (int64_t)min(drow0 + rr, D - 1) * sd + t] : from_f<T>(0.f);
    }
  }
}

// Named barriers of a CTA: one kind of warp arrives, the other waits.
template <int THREADS>
__device__ __forceinline__ void named_sync(int id) { __syncwarp(); asm volatile("bar.sync %0, %1;\n" ::"r"(id), "n"(THREADS) : "memory"); }
template <int THREADS>
__device__ __forceinline__ void named_arrive(int id) { __syncwarp(); asm volatile("bar.arrive %0, %1;\n" ::"r"(id), "n"(THREADS) : "memory"); }
enum { kBarProducers = 1, kBarFull = 2, kBarHi = 3, kBarLo = 4 };  // kBarLo + 0 / 1: lower halves of alternate tiles

// A call whose rows alone cannot fill the machine is cut in time into gridDim.z segments of `seg_tiles` tiles.  The states need
// nothing for it (every tile starts from its checkpoint); the adjoint that enters a segment from the right does: scan_bwd_kernel's CARRY
// pass finds it.
// PIECES: ragged rows or coefficients (see fill_rows_pieces); an instance of its own, because the offsets cost the aligned form 5-10 %
template <typename T, int LPR, bool PIECES>
__global__ void __launch_bounds__(BwdPairs<T, LPR, PIECES>::NW * 64, 3)
    scan_bwd_pairs_kernel(const ssm_scan_bwd_args g, const ScanFlags fl, int seg_tiles, int sms) {
  using S = BwdPairs<T, LPR, PIECES>;
  constexpr int NS = S::NS, NP = S::NP, RPW = S::RPW, ROWS = S::ROWS, TL = S::TL, HL = S::HL, PITCH = S::PITCH, NW = S::NW, V = S::V, RP = S::RP;
  constexpr int NT = NW * 64, NPROD = NW * 32;
  constexpr int PER = 8 / LPR;  // (step, row) entries of a lane after pair_sums
  static_assert(PER >= 2, "whole steps of a row pair per lane");
  const ssm_scan_fwd_args& a = g.fwd;

  extern __shared__ __align__(16) float smem[];
  // warps alternate over the schedulers of an SM by their number: CTAs that follow each other onto an SM take the two kinds in turn
  const int cta = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
  const int lane = threadIdx.x & 31, wid = (threadIdx.x >> 5) ^ ((cta / sms & 1) * NW);
  const bool producer = wid >= NW;
  const int warp = producer ? wid - NW : wid;
  float* last = smem + 3 * S::HALF + warp * (S::LAST + S::STAGE);
  float* stage = last + S::LAST;
  char* rawbase = reinterpret_cast<char*>(smem + 3 * S::HALF + NW * (S::LAST + S::STAGE));
  char* rawB = rawbase;
  char* rawC = rawbase + S::BC_RAW_BYTES / 2;
  T* rawU = reinterpret_cast<T*>(rawbase + S::BC_RAW_BYTES + warp * S::WARP_RAW_BYTES);
  T* rawD = rawU + 2 * RPW * RP;
  T* rawZ = rawD + 2 * RPW * RP;
  T* rawO = rawZ + 2 * RPW * RP;
  // a half tile's buffer: B, C [HL][NP], then per warp delta, u (overwritten step by step with ddelta), dy (with du) as pairs [RPW][PITCH]
  // and the states [slot][2][32]
  struct Half {
    float *B, *C;
    float2 *dl, *u, *dy;
    float4* hist;
  };
  auto half = [&](int slot) {
    float* base = smem + slot * S::HALF;
    float* w = base + S::BC + warp * (3 * S::ROW_ARRAY + S::HIST);
    return Half{base, base + S::BC / 2, reinterpret_cast<float2*>(w), reinterpret_cast<float2*>(w + S::ROW_ARRAY), reinterpret_cast<float2*>(w + 2 * S::ROW_ARRAY),
                reinterpret_cast<float4*>(w + 3 * S::ROW_ARRAY) + lane};
  };

  const int b = blockIdx.y;
  const int d0 = blockIdx.x * ROWS;
  const int N = a.nstate, L = a.len, D = a.dim;
  const int r = lane % RPW, sg = lane / RPW;  // row pair (low lane bits: the eight lanes of a quarter warp share their states), state group
  const int drow0 = d0 + warp * 2 * RPW;
  const int dr[2] = {drow0 + r, drow0 + r + RPW};  // within D: the rows of a CTA share a group, so its size divides D
  const int64_t row[2] = {(int64_t)b * D + dr[0], (int64_t)b * D + dr[1]};
  const int seg = blockIdx.z, nseg = gridDim.z;
  const int ntiles = (L + TL - 1) / TL;
  const int k_begin = seg * seg_tiles, k_end = min(ntiles, k_begin + seg_tiles);
  const float2 Dv = a.D ? make_float2(__ldg(a.D + dr[0]), __ldg(a.D + dr[1])) : make_float2(0.f, 0.f);
  float2 A2[NS];
#pragma unroll
  for (int j = 0; j < NS; ++j) {
    const int n = sg * NS + j;
    A2[j] = n < N ? make_float2(__ldg(a.A + (int64_t)dr[0] * N + n) * kLog2e, __ldg(a.A + (int64_t)dr[1] * N + n) * kLog2e) : make_float2(0.f, 0.f);
  }
  // four steps of a row pair's array
  auto load4 = [](const float2* p, float2 (&v)[4]) {
    const float4 x = *reinterpret_cast<const float4*>(p), y = *reinterpret_cast<const float4*>(p + 2);
    v[0] = make_float2(x.x, x.y), v[1] = make_float2(x.z, x.w), v[2] = make_float2(y.x, y.y), v[3] = make_float2(y.z, y.w);
  };
  auto both = [](float x) { return make_float2(x, x); };  // a broadcast operand
  auto decay = [](float2 dl, float2 A) {
    const float2 e = __fmul2_rn(dl, A);
    return make_float2(ex2_approx(e.x), ex2_approx(e.y));
  };
  const bool io_vec = fl.io_vec != 0;

  if (producer) {
    const int ptid = warp * 32 + lane;
    const T* __restrict__ gz = reinterpret_cast<const T*>(a.z);
    T* __restrict__ gdz = reinterpret_cast<T*>(g.dz);
    const int rpg = fl.rows_per_group;
    const int64_t boff = bc_row_offset(b, d0, rpg, a.b_sb, a.b_sg);
    const int64_t coff = bc_row_offset(b, d0, rpg, a.c_sb, a.c_sg);
    const int bcsz = a.bc_dtype == SSM_F32 ? 4 : 2;
    const bool bc_vec = fl.bc_vec != 0;
    // ragged rows and coefficients: the same asynchronous copies in 16-byte pieces, read at the row's own offset.  (With scalar loads
    // between two barriers the tile's DRAM latency was exposed: 2 x 1024 rows, fp16, 3999 steps 2364 us against 1008 for 4000.)
    const bool io_pieces = PIECES && !io_vec && fl.io_pieces, bc_pieces = PIECES && !bc_vec && fl.bc_pieces;
    const int raw_bc_dtype = bc_vec || bc_pieces ? a.bc_dtype : SSM_F32;
    const int bc_per = bc_pieces ? 16 / bcsz : 0;
    const int shift[2] = {io_pieces ? row_shift<T>((int64_t)b * a.row_sb + (int64_t)dr[0] * a.row_sd) : 0,
                          io_pieces ? row_shift<T>((int64_t)b * a.row_sb + (int64_t)dr[1] * a.row_sd) : 0};
    auto fill_rows = [&](T* raw, const void* src, int t0) {
      const T* p = reinterpret_cast<const T*>(src);
      if (io_pieces) fill_rows_pieces<T, 2 * RPW, TL>(raw, p, b, D, L, drow0, t0, lane, a.row_sb, a.row_sd);
      else fill_rows_pitched<T, 2 * RPW, TL>(raw, p, b, D, L, drow0, t0, io_vec, lane, a.row_sb, a.row_sd);
    };
    auto fill_raw = [&](int t0) {
      fill_rows(rawU, a.u, t0), fill_rows(rawD, a.delta, t0), fill_rows(rawO, g.dout, t0);
      if (gz) fill_rows(rawZ, a.z, t0);
      if (bc_pieces) {
        fill_bc_pieces<TL>(rawB, a.Bm, a.bc_dtype, boff, a.b_sn, N, t0, L, ptid, NPROD);
        fill_bc_pieces<TL>(rawC, a.Cm, a.bc_dtype, coff, a.c_sn, N, t0, L, ptid, NPROD);
      } else {
        fill_bc_raw<TL>(rawB, reinterpret_cast<const char*>(a.Bm) + boff * bcsz, a.bc_dtype, a.b_sn, a.b_st, N, t0, L, bc_vec, ptid, NPROD);
        fill_bc_raw<TL>(rawC, reinterpret_cast<const char*>(a.Cm) + coff * bcsz, a.bc_dtype, a.c_sn, a.c_st, N, t0, L, bc_vec, ptid, NPROD);
      }
      cp_async_commit();
    };
    // raw [n][pitch] -> fp32 [HL][NP], steps `from` .. from + HL - 1
    auto convert_half = [&](float* dst, const char* raw, int64_t start, int64_t sn, int from) {
      constexpr int NQ = NP / 4;
      for (int i = ptid; i < NQ * HL; i += NPROD) {
        const int nq = i % NQ, tt = i / NQ;
        float v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int n = nq * 4 + q;
          const int at = (PIECES ? n * (TL + bc_per) + ((int)(start + n * sn) & max(bc_per - 1, 0)) : n * TL) + from + tt;
          v[q] = n < N ? raw_bc_at(raw, at, raw_bc_dtype) : 0.f;
        }
        *reinterpret_cast<float4*>(dst + tt * NP + nq * 4) = make_float4(v[0], v[1], v[2], v[3]);
      }
    };
    // the checkpoint a tile starts from is fetched one tile ahead
    float2 h[NS], hck[NS];
    auto load_checkpoint = [&](int kt) {
      const float* ck[2] = {a.checkpoints + (row[0] * ntiles + kt) * N + sg * NS, a.checkpoints + (row[1] * ntiles + kt) * N + sg * NS};
#pragma unroll
      for (int j = 0; j < NS; ++j) hck[j] = sg * NS + j < N ? make_float2(__ldg(ck[0] + j), __ldg(ck[1] + j)) : make_float2(0.f, 0.f);
    };
    if (k_begin < k_end) {
      fill_raw((k_end - 1) * TL);
      load_checkpoint(k_end - 1);
    }
    for (int k = k_end - 1; k >= k_begin; --k) {
      const int t0 = k * TL, order = k_end - 1 - k;
      cp_async_wait_all();
      named_sync<NPROD>(kBarProducers);  // the producers' shares of the raw tile have landed
#pragma unroll
      for (int j = 0; j < NS; ++j) h[j] = hck[j];
      if (k > k_begin) load_checkpoint(k - 1);
#pragma unroll 1
      for (int hf = 0; hf < 2; ++hf) {
        const Half w = half(hf ? 1 : (order & 1) * 2);
        // the buffer's last user: the upper half of the tile before, the lower half of the tile before that
        if (hf ? order > 0 : order > 1) named_sync<NT>(hf ? kBarHi : kBarLo + (order & 1));
        // ---- delta, u (and dy where nothing gates it) as pairs
        constexpr int CH = HL / V;
        for (int c = lane; c < RPW * CH; c += 32) {
          const int p = c % RPW, ch = c / RPW, t = t0 + hf * HL + ch * V;
          float fu[2][V], fd[2][V], fo[2][V];
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int rr = p + q * RPW, dd = drow0 + rr;
            const int at = rr * RP + hf * HL + ch * V + (io_pieces ? row_shift<T>((int64_t)b * a.row_sb + (int64_t)dd * a.row_sd) : 0);
            if (io_pieces) {
#pragma unroll
              for (int i = 0; i < V; ++i) {
                fu[q][i] = to_f<T>(rawU[at + i]), fd[q][i] = to_f<T>(rawD[at + i]);
                if (!gz) fo[q][i] = to_f<T>(rawO[at + i]);
              }
            } else {
              Vec16<T> v;
              v.raw = *reinterpret_cast<const uint4*>(rawU + at);
              v.unpack(fu[q]);
              v.raw = *reinterpret_cast<const uint4*>(rawD + at);
              v.unpack(fd[q]);
              if (!gz) {
                v.raw = *reinterpret_cast<const uint4*>(rawO + at);
                v.unpack(fo[q]);
              }
            }
            const float bias = a.dt_bias ? __ldg(a.dt_bias + dd) : 0.f;
#pragma unroll
            for (int i = 0; i < V; ++i) {
              float x = fd[q][i] + bias;
              if (a.delta_softplus) x = softplus_fast(x);
              fd[q][i] = t + i >= L ? 0.f : x;
            }
          }
          const int o = p * PITCH + ch * V;
#pragma unroll
          for (int i = 0; i < V; i += 2) {
            *reinterpret_cast<float4*>(w.dl + o + i) = make_float4(fd[0][i], fd[1][i], fd[0][i + 1], fd[1][i + 1]);
            *reinterpret_cast<float4*>(w.u + o + i) = make_float4(fu[0][i], fu[1][i], fu[0][i + 1], fu[1][i + 1]);
            if (!gz) *reinterpret_cast<float4*>(w.dy + o + i) = make_float4(fo[0][i], fo[1][i], fo[0][i + 1], fo[1][i + 1]);
          }
        }
        convert_half(w.B, rawB, boff, a.b_sn, hf * HL);
        convert_half(w.C, rawC, coff, a.c_sn, hf * HL);
        named_sync<NPROD>(kBarProducers);
        // ---- the states of this half
        const float2 *rDl = w.dl + r * PITCH, *rU = w.u + r * PITCH;
        float2* rDy = w.dy + r * PITCH;
#pragma unroll 2
        for (int tt = 0; tt < HL; tt += 4) {
          float2 dl[4], u[4];
          float p[8];
          load4(rDl + tt, dl), load4(rU + tt, u);
          w.hist[(tt / 4 * 2) * 32] = make_float4(h[0].x, h[0].y, h[1].x, h[1].y);
          w.hist[(tt / 4 * 2 + 1) * 32] = make_float4(h[2].x, h[2].y, h[3].x, h[3].y);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float4 b4 = *reinterpret_cast<const float4*>(w.B + (tt + i) * NP + sg * NS);
            const float bv[4] = {b4.x, b4.y, b4.z, b4.w};
            float4 c4 = make_float4(0.f, 0.f, 0.f, 0.f);
            if (gz) c4 = *reinterpret_cast<const float4*>(w.C + (tt + i) * NP + sg * NS);
            const float cv[4] = {c4.x, c4.y, c4.z, c4.w};
            const float2 du = __fmul2_rn(dl[i], u[i]);
            float2 acc = make_float2(0.f, 0.f);
#pragma unroll
            for (int j = 0; j < NS; ++j) {
              h[j] = __ffma2_rn(decay(dl[i], A2[j]), h[j], __fmul2_rn(du, both(bv[j])));
              if (gz) acc = __ffma2_rn(both(cv[j]), h[j], acc);
            }
            p[2 * i] = acc.x, p[2 * i + 1] = acc.y;
          }
          if (gz) {  // dy = dout silu(z), dz = dout silu'(z) (sum_n C h + D u)
            pair_sums<LPR, RPW>(p, lane);
#pragma unroll
            for (int i = 0; i < PER; i += 2) {
              const int at = tt + (sg * PER + i) / 2;
              const float2 uv = rU[at];
              float dyv[2];
#pragma unroll
              for (int q = 0; q < 2; ++q) {
                const int ra = (r + q * RPW) * RP + hf * HL + at + shift[q];
                const float zv = to_f<T>(rawZ[ra]), ov = to_f<T>(rawO[ra]), s = sigmoid_fast(zv);
                dyv[q] = ov * zv * s;
                rawZ[ra] = from_f<T>(ov * s * (1.f + zv * (1.f - s)) * fmaf(q ? Dv.y : Dv.x, q ? uv.y : uv.x, p[i + q]));
              }
              rDy[at] = make_float2(dyv[0], dyv[1]);
            }
          }
        }
      }
      if (k == k_end - 1) {
        *reinterpret_cast<float4*>(last + lane * 8) = make_float4(h[0].x, h[0].y, h[1].x, h[1].y);
        *reinterpret_cast<float4*>(last + lane * 8 + 4) = make_float4(h[2].x, h[2].y, h[3].x, h[3].y);
      }
      named_arrive<NT>(kBarFull);
      if (gdz) {  // finished in the places of z
        __syncwarp();
        if (io_vec) {
          constexpr int CH = TL / V;
          for (int c = lane; c < 2 * RPW * CH; c += 32) {
            const int rr = c / CH, ch = c % CH, t = t0 + ch * V;
            if (t < L)
              __stcs(reinterpret_cast<uint4*>(gdz + (int64_t)b * a.row_sb + (int64_t)(drow0 + rr) * a.row_sd + t), *reinterpret_cast<const uint4*>(rawZ + rr * RP + ch * V));
          }
        } else {
          for (int i = lane; i < 2 * RPW * TL; i += 32) {
            const int rr = i / TL, tt = i % TL, t = t0 + tt;
            const int64_t at = (int64_t)b * a.row_sb + (int64_t)(drow0 + rr) * a.row_sd;
            if (t < L) gdz[at + t] = rawZ[rr * RP + tt + (io_pieces ? row_shift<T>(at) : 0)];
          }
        }
      }
      named_sync<NPROD>(kBarProducers);  // raw tile consumed
      if (k > k_begin) fill_raw(t0 - TL);
    }
    return;
  }

  // ---- consumers -------------------------------------------------------------------------------------------
  T* __restrict__ gdu = reinterpret_cast<T*>(g.du);
  T* __restrict__ gdd = reinterpret_cast<T*>(g.ddelta);
  float2 carry[NS], dAacc[NS], hc[NS];
#pragma unroll
  for (int j = 0; j < NS; ++j) {
    const int n = sg * NS + j;
    carry[j] = dAacc[j] = make_float2(0.f, 0.f);
    if (seg == nseg - 1) {
      if (n < N && g.dlast_state) carry[j] = make_float2(__ldg(g.dlast_state + row[0] * N + n), __ldg(g.dlast_state + row[1] * N + n));
    } else if (n < N) {  // split scratch, after the combine: the adjoint that enters a segment from the right, [batch][dim][nseg][N]
      carry[j] = make_float2(a.split_scratch[(row[0] * nseg + seg) * N + n], a.split_scratch[(row[1] * nseg + seg) * N + n]);
    }
  }
  float2 dDacc = make_float2(0.f, 0.f), dBiasAcc = dDacc;
  // dB / dC: the output (state n of dB, then of dC) that this lane sums over the warp's row pairs, four steps at a time
  constexpr int O = 2 * NP;
  constexpr int PARTS = 32 / O, RPP = RPW / PARTS;  // lanes that share an output, each summing RPP row pairs
  static_assert(O <= 32 && RPP == 8, "one output and eight 16-byte loads per lane and group");
  const int part = lane / O, out_o = lane % O, out_n = out_o % NP;
  const int64_t red_st = out_o < NP ? g.db_st : g.dc_st;
  float* red_dst = out_o < NP ? g.dB + bc_row_offset(b, d0, fl.rows_per_group, g.db_sb, g.db_sg) + (int64_t)out_n * g.db_sn
                              : g.dC + bc_row_offset(b, d0, fl.rows_per_group, g.dc_sb, g.dc_sg) + (int64_t)out_n * g.dc_sn;
  const bool red_vec = red_st == 1 && (reinterpret_cast<uintptr_t>(red_dst) & 15) == 0;
  const bool red_on = part == 0 && out_n < N;

  for (int k = k_end - 1; k >= k_begin; --k) {
    const int t0 = k * TL, order = k_end - 1 - k;
    named_sync<NT>(kBarFull);
    if (order == 0) {
      const float4 x = *reinterpret_cast<const float4*>(last + lane * 8), y = *reinterpret_cast<const float4*>(last + lane * 8 + 4);
      hc[0] = make_float2(x.x, x.y), hc[1] = make_float2(x.z, x.w), hc[2] = make_float2(y.x, y.y), hc[3] = make_float2(y.z, y.w);
    }
#pragma unroll 1
    for (int hf = 1; hf >= 0; --hf) {
      const Half w = half(hf ? 1 : (order & 1) * 2);
      const float2* rDl = w.dl + r * PITCH;
      float2 *rU = w.u + r * PITCH, *rDy = w.dy + r * PITCH;
      const int th = t0 + hf * HL;
#pragma unroll 1
      for (int tt = HL - 4; tt >= 0; tt -= 4) {
        float2 dl[4], du[4], dy[4], s1[4], s2[4];
        load4(rDl + tt, dl), load4(rU + tt, du), load4(rDy + tt, dy);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          du[i] = __fmul2_rn(dl[i], du[i]);
          s1[i] = s2[i] = make_float2(0.f, 0.f);
        }
#pragma unroll
        for (int jh = 0; jh < NS; jh += 2) {
          // states before steps tt .. tt + 3 (hs[0] from the rebuild, the rest formed again) and the four decays
          float2 hs[4][2], da[4][2], bv[4], cv[4];
          float vB[2][4], vC[2][4];
          const float4 h0 = w.hist[(tt / 4 * 2 + jh / 2) * 32];
          hs[0][0] = make_float2(h0.x, h0.y), hs[0][1] = make_float2(h0.z, h0.w);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            bv[i] = *reinterpret_cast<const float2*>(w.B + (tt + i) * NP + sg * NS + jh);
            cv[i] = *reinterpret_cast<const float2*>(w.C + (tt + i) * NP + sg * NS + jh);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              da[i][j] = decay(dl[i], A2[jh + j]);
              if (i < 3) hs[i + 1][j] = __ffma2_rn(da[i][j], hs[i][j], __fmul2_rn(du[i], both(j ? bv[i].y : bv[i].x)));
            }
          }
#pragma unroll
          for (int i = 3; i >= 0; --i) {
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              const float2 hcur = i == 3 ? hc[jh + j] : hs[i == 3 ? 0 : i + 1][j];  // the state after this step
              const float2 G = __ffma2_rn(both(j ? cv[i].y : cv[i].x), dy[i], carry[jh + j]);
              // (two scalar operations: a packed product and the sum of its halves hold the pipe half as long again)
              vC[j][i] = fmaf(dy[i].y, hcur.y, dy[i].x * hcur.x), vB[j][i] = fmaf(G.y, du[i].y, G.x * du[i].x);
              s1[i] = __ffma2_rn(G, both(j ? bv[i].y : bv[i].x), s1[i]);
              carry[jh + j] = __fmul2_rn(da[i][j], G);
              const float2 gha = __fmul2_rn(carry[jh + j], hs[i][j]);
              s2[i] = __ffma2_rn(gha, A2[jh + j], s2[i]);
              dAacc[jh + j] = __ffma2_rn(gha, dl[i], dAacc[jh + j]);
            }
          }
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            hc[jh + j] = hs[0][j];
            const int o = sg * NS + jh + j;
            *reinterpret_cast<float4*>(stage + ((o * RPW + r) << 2)) = make_float4(vB[j][0], vB[j][1], vB[j][2], vB[j][3]);
            *reinterpret_cast<float4*>(stage + (((NP + o) * RPW + r) << 2)) = make_float4(vC[j][0], vC[j][1], vC[j][2], vC[j][3]);
          }
        }
        __syncwarp();  // the products are in the staging area, and every lane has read this group's u / dy
        float4 sv[8];
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) sv[kk] = *reinterpret_cast<const float4*>(stage + ((out_o * RPW + part * RPP + ((kk + out_o) & (RPP - 1))) << 2));
        float p1[8], p2[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) p1[2 * i] = s1[i].x, p1[2 * i + 1] = s1[i].y, p2[2 * i] = s2[i].x, p2[2 * i + 1] = s2[i].y;
        pair_sums<LPR, RPW>(p1, lane);
        pair_sums<LPR, RPW>(p2, lane);
        {
          float2 lo = make_float2(0.f, 0.f), hi = lo;
#pragma unroll
          for (int kk = 0; kk < 8; ++kk) lo = __fadd2_rn(lo, make_float2(sv[kk].x, sv[kk].y)), hi = __fadd2_rn(hi, make_float2(sv[kk].z, sv[kk].w));
#pragma unroll
          for (int off = O; off < 32; off <<= 1) {
            lo.x += __shfl_xor_sync(0xffffffffu, lo.x, off), lo.y += __shfl_xor_sync(0xffffffffu, lo.y, off);
            hi.x += __shfl_xor_sync(0xffffffffu, hi.x, off), hi.y += __shfl_xor_sync(0xffffffffu, hi.y, off);
          }
          const int t = th + tt;
          if (red_on && t < L) {
            float* dst = red_dst + (int64_t)t * red_st;
            if (red_vec && t + 3 < L) {
              asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(lo.x), "f"(lo.y), "f"(hi.x), "f"(hi.y) : "memory");
            } else {
              const float av[4] = {lo.x, lo.y, hi.x, hi.y};
#pragma unroll
              for (int i = 0; i < 4; ++i)
                if (t + i < L) atomicAdd(dst + i * red_st, av[i]);
            }
          }
        }
        // ddelta and du of this lane's steps from the sums over states
        auto dstep = [&](float dlv, float uv, float q1, float q2) {
          const float dd = fmaf(q1, uv, q2 * kLn2);
          // d softplus(pre) / d pre = sigmoid(pre) = 1 - exp(-softplus(pre))
          return a.delta_softplus ? dd * one_minus_exp_neg(dlv) : dd;
        };
#pragma unroll
        for (int i = 0; i < PER; i += 2) {
          const int at = tt + (sg * PER + i) / 2;
          const float2 dlv = rDl[at], uv = rU[at], dyv = rDy[at];
          const float2 dd = make_float2(dstep(dlv.x, uv.x, p1[i], p2[i]), dstep(dlv.y, uv.y, p1[i + 1], p2[i + 1]));
          dDacc = __ffma2_rn(dyv, uv, dDacc);
          if (th + at < L) dBiasAcc = __fadd2_rn(dBiasAcc, dd);
          rDy[at] = __ffma2_rn(make_float2(p1[i], p1[i + 1]), dlv, __fmul2_rn(dyv, Dv));
          rU[at] = dd;
        }
        __syncwarp();  // staging area read; du and ddelta of the half are complete after its last group
      }
      // ---- write du / ddelta
      if (io_vec) {
        constexpr int CH = HL / V;
        for (int c = lane; c < RPW * CH; c += 32) {
          const int p = c / CH, ch = c % CH;
          const int t = th + ch * V;
          if (t < L) {
            auto put = [&](const float2* src, T* dst) {
              float f[2][V];
#pragma unroll
              for (int i = 0; i < V; i += 2) {
                const float4 q = *reinterpret_cast<const float4*>(src + p * PITCH + ch * V + i);
                f[0][i] = q.x, f[1][i] = q.y, f[0][i + 1] = q.z, f[1][i + 1] = q.w;
              }
#pragma unroll
              for (int q = 0; q < 2; ++q) {
                Vec16<T> v;
                v.pack(f[q]);
                v.store_stream(dst + (int64_t)b * a.row_sb + (int64_t)(drow0 + p + q * RPW) * a.row_sd + t);
              }
            };
            put(w.dy, gdu), put(w.u, gdd);
          }
        }
      } else {
        for (int i = lane; i < 2 * RPW * HL; i += 32) {
          const int rr = i / HL, tt = i % HL, t = th + tt;
          if (t < L) {
            const int o = ((rr % RPW) * PITCH + tt) * 2 + rr / RPW;
            const int64_t base = (int64_t)b * a.row_sb + (int64_t)(drow0 + rr) * a.row_sd + t;
            gdu[base] = from_f<T>(reinterpret_cast<const float*>(w.dy)[o]);
            gdd[base] = from_f<T>(reinterpret_cast<const float*>(w.u)[o]);
          }
        }
      }
      // the buffer's next user: this half of the next tile, or (lower halves) of the one after it
      if (hf ? k > k_begin : k > k_begin + 1) named_arrive<NT>(hf ? kBarHi : kBarLo + (order & 1));
    }
  }

#pragma unroll
  for (int j = 0; j < NS; ++j) {
    const int n = sg * NS + j;
    if (n < N) {
      if (g.dinitial_state && seg == 0) {  // what the adjoint carries past step 0 is the gradient of the state before it
        g.dinitial_state[row[0] * N + n] = carry[j].x;
        g.dinitial_state[row[1] * N + n] = carry[j].y;
      }
      atomicAdd(g.dA + (int64_t)dr[0] * N + n, dAacc[j].x);
      atomicAdd(g.dA + (int64_t)dr[1] * N + n, dAacc[j].y);
    }
  }
  float sums[4] = {dDacc.x, dDacc.y, dBiasAcc.x, dBiasAcc.y};
#pragma unroll
  for (int i = 0; i < 4; ++i) sums[i] = group_sum<LPR, RPW>(sums[i]);
  if (sg == 0) {
    if (g.dD) atomicAdd(g.dD + dr[0], sums[0]), atomicAdd(g.dD + dr[1], sums[1]);
    if (g.ddt_bias) atomicAdd(g.ddt_bias + dr[0], sums[2]), atomicAdd(g.ddt_bias + dr[1], sums[3]);
  }
}

}  // namespace ssmb
