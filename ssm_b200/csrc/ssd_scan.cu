// State-space-dual (Mamba-2) chunked scan with a d_state axis, forward, for sm_100a.
//
//   delta_t = softplus?(dt_t + dt_bias);  S_t = exp(delta_t A) S_{t-1} + delta_t x_t B_t^T;  y_t = S_t C_t + D x_t;  y_t *= silu(z_t)
//
// evaluated chunk by chunk (Q = 256 steps) in the dual, matrix form, with every contraction on
// the tcgen05 tensor cores (bf16 / fp16 operands in shared memory, staged by TMA, fp32 accumulators in TMEM):
//
//   ssd_cumsum_kernel   per chunk the running decay exponent  c_i = log2(e) sum_{k<=i} delta_k A  and  c_i - log2(delta_i)
//   ssd_state_kernel    per (batch, a few heads), chunks in order: local state  S_c = sum_j exp2(c_last - c_j) delta_j x_j B_j^T
//                       [N x P GEMM, K = Q] folded into the running state in registers; writes the state before every
//                       chunk (in the operand dtype and order of the GEMM below), the final state in fp32, and what a
//                       sequence shard hands to the other ranks
//   ssd_fold_shards_kernel / ssd_fold_init_kernel   (sequence shards only) fold the other ranks' summaries into this
//                       shard's incoming state, and add that late-arriving state to the per-chunk states by linearity
//   ssd_scan_kernel     per (batch, chunk, 128-row block, part of a head group):  G = C B^T once (TMEM -> registers), then per
//                       head the decay mask exp2(c_i - c_j) delta_j [j <= i] (+ D on the diagonal) written back to TMEM
//                       (tcgen05.st) as the A operand of Y_intra = (G o L) X, plus  Y_inter = C S_in;
//                       y = Y_intra + exp2(c_i) Y_inter, gated, stored by TMA.  Sixteen warps form masks and epilogues, one
//                       issues the MMAs and the copies.
//
// Exponent differences are always formed before exp2 (never exp2(c_i) / exp2(c_j)), so long
// sequences stay finite.  Every wait on an mbarrier is bounded and reports through the status word.
#include "seq_table.h"
#include "ssd_common.cuh"

#include <algorithm>
#include <cmath>

namespace ssmb {

// floats of the shard summary (final state, then total log-decay), rounded up to whole 256-byte lines
__host__ __device__ inline int64_t ssd_summary_floats_padded(int batch, int heads) {
  return ((int64_t)batch * heads * (kP * kN + 1) + 63) / 64 * 64;
}

// ---------------------------------------------------------------------------------------------
// delta and within-chunk cumulative log-decay.  One CTA per (batch, chunk, 32 heads): the step sizes are read the way they
// lie in memory (heads innermost: each thread the 32 heads of one step), activated, transposed through shared memory, and
// each warp then scans whole heads, a lane owning 8 consecutive steps and writing them as 16-byte pieces.
// ---------------------------------------------------------------------------------------------
constexpr int kCumHeads = 32;
constexpr int kCumLd = kQ + 8;  // row pitch of the transposed tile (floats): rows stay 16-byte aligned, lanes 32 bytes apart

// first step of a chunk, and the first step beyond its sequence: of packed sequences they come from the table
__device__ __forceinline__ int chunk_begin(const ssm_ssd_args& a, int c) { return a.seq_table ? __ldg(a.seq_table + 2 * c) : c * kQ; }
__device__ __forceinline__ int chunk_limit(const ssm_ssd_args& a, int c) { return a.seq_table ? __ldg(a.seq_table + 2 * c + 1) : a.len; }

template <typename T>
__global__ void __launch_bounds__(kQ) ssd_cumsum_kernel(const ssm_ssd_args a, int nchunks) {
  __shared__ __align__(16) float sD[kCumHeads * kCumLd];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int h0 = blockIdx.x * kCumHeads, c = blockIdx.y, b = blockIdx.z;
  const int nh = min(kCumHeads, a.heads - h0);
  if (a.seq_table && chunk_begin(a, c) >= chunk_limit(a, c)) return;  // no chunk: the table has room to spare
  {
    const int t = chunk_begin(a, c) + tid;
    if (t < chunk_limit(a, c)) {
      const int64_t at = ((int64_t)b * a.len + t) * a.heads + h0;
      {
        const T* p = reinterpret_cast<const T*>(a.dt) + at;
        if (nh == kCumHeads && (reinterpret_cast<uintptr_t>(p) & 15) == 0) {
#pragma unroll
          for (int q = 0; q < kCumHeads / 8; ++q) {
            Vec16<T> v;
            v.load(p + q * 8);
            float f[8];
            v.unpack(f);
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              float x = f[e] + (a.dt_bias ? __ldg(a.dt_bias + h0 + q * 8 + e) : 0.f);
              if (a.dt_softplus) x = softplus_f(x);
              sD[(q * 8 + e) * kCumLd + tid] = x;
            }
          }
        } else {
          for (int hh = 0; hh < nh; ++hh) {
            float x = to_f<T>(p[hh]) + (a.dt_bias ? __ldg(a.dt_bias + h0 + hh) : 0.f);
            if (a.dt_softplus) x = softplus_f(x);
            sD[hh * kCumLd + tid] = x;
          }
        }
      }
    } else {
      for (int hh = 0; hh < nh; ++hh) sD[hh * kCumLd + tid] = 0.f;  // steps beyond the sequence: no decay, no input
    }
  }
  __syncthreads();
  for (int hh = warp; hh < nh; hh += kQ / 32) {
    const int h = h0 + hh;
    const float Ah = __ldg(a.A + h);
    float* odt = a.ws_dt + (((int64_t)b * a.heads + h) * nchunks + c) * kQ + lane * 8;
    float* ocum = a.ws_cum + (((int64_t)b * a.heads + h) * nchunks + c) * kQ + lane * 8;
    float d[8], run = 0.f;  // each lane owns 8 consecutive steps
    {
      const float4 d0 = *reinterpret_cast<const float4*>(sD + hh * kCumLd + lane * 8);
      const float4 d1 = *reinterpret_cast<const float4*>(sD + hh * kCumLd + lane * 8 + 4);
      d[0] = d0.x, d[1] = d0.y, d[2] = d0.z, d[3] = d0.w, d[4] = d1.x, d[5] = d1.y, d[6] = d1.z, d[7] = d1.w;
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) run += d[k] * Ah;
    // exclusive prefix of the lane sums
    float pre = run;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const float o = __shfl_up_sync(0xffffffffu, pre, off);
      if (lane >= off) pre += o;
    }
    float acc = pre - run;
    float oc[8], od[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      acc += d[k] * Ah;
      const float c2 = acc * kLog2e;
      oc[k] = c2;                      // running decay exponent, base 2
      // the same with delta folded in: exp2(x - odt[j]) = exp2(x - c2_j) * delta_j  (delta 0 -> +inf -> weight 0)
      od[k] = c2 - lg2_approx(d[k]);
    }
    reinterpret_cast<float4*>(ocum)[0] = make_float4(oc[0], oc[1], oc[2], oc[3]);
    reinterpret_cast<float4*>(ocum)[1] = make_float4(oc[4], oc[5], oc[6], oc[7]);
    reinterpret_cast<float4*>(odt)[0] = make_float4(od[0], od[1], od[2], od[3]);
    reinterpret_cast<float4*>(odt)[1] = make_float4(od[4], od[5], od[6], od[7]);
  }
}

// ---------------------------------------------------------------------------------------------
// chunk states, local and carried, in one pass:  one CTA per (batch, a few heads) walks the chunks in order.
// Per chunk the tensor cores form  S_c[n][p] = sum_j B[j][n] * (w_j x[j][p]),  w_j = exp2(c_last - (c_j - log2 delta_j)),
// in four stages of 64 steps from a ring of TMA-filled buffers:
//   A operand = B^T, MN-major;  B operand = w x of the CTA's heads side by side, MN-major;  M = 128 (n), N = 64 per head (p),
//   K = 64 per stage.  (Units that are neighbours along M / N are 128 bytes apart, so the tensor core's reads of one K slice
//   fall on different banks; with units 2 KB apart the MMAs ran 4-5x slower.)
// Eight compute warps scale the x rows of the landed stages in place, four of them the even and four the odd stages (a stage costs a
// warp a fixed chain of waits, shared-memory round trips and fences, whatever the number of rows: half as many stages per warp,
// each with twice the rows; sixteen warps on four groups were slower), and keep the running state in registers (thread = state n,
// 32 of the 64 columns p):  state <- exp2(c_last) * state + S_c ;  the state BEFORE each chunk goes out in the operand dtype,
// in the operand order of the scan kernel (MN-major units [p/8][n][8]).  The per-chunk local states never touch global memory.
// A ninth warp issues the copies (a buffer is refilled once the MMAs that read it have completed: tcgen05.commit -> mbarrier),
// a tenth the MMAs (once the eight compute warps have arrived on the stage's barrier).
// ---------------------------------------------------------------------------------------------
// HPC heads of one B / C group per CTA share the B^T tile of every stage (the grid is sized to about one CTA per SM).
// Tiles are rows of 128 bytes (64 elements along M / N) written by TMA with the 128-byte swizzle, 64 steps each:
// B^T as two blocks (states 0..63, 64..127), then one x block per head; blocks are 8 KB apart.
template <int HPC, int NST>
struct StateSmem {
  static constexpr int kStep = 64;                            // steps per stage
  static constexpr int BLK_BYTES = kStep * 128;               // 8 KB: 64 steps x 64 elements
  static constexpr int A_BYTES = 2 * BLK_BYTES;               // 16 KB
  static constexpr int STAGE = A_BYTES + HPC * BLK_BYTES;
  static constexpr int NSTAGE = NST;
  // exponents that come with a stage, per head: those of its steps, the chunk's first four (REV) and its last four
  static constexpr int kVec = kStep + 8;
  static constexpr int VEC_BYTES = HPC * kVec * 4;
  static constexpr int TOTAL = NSTAGE * (STAGE + VEC_BYTES);
  static constexpr int ALLOC = TOTAL + 1024;
};

// tensor maps of the state kernel: B rows (box 64 states x 64 steps) and x rows (box 64 p x 64 steps)
struct StateMaps {
  CUtensorMap b, x;
};

// Threads: eight warps scale the x rows and keep the running states; one warp issues the copies, one the MMAs.  The stages pass
// from role to role through mbarriers only (landed -> scaled -> multiplied -> free), so no warp waits for another role's
// instruction issue.
constexpr int kStateComputeThreads = 256;
constexpr int kStateGroupThreads = kStateComputeThreads / 2;  // one group scales the even stages, the other the odd ones
constexpr int kStateThreads = kStateComputeThreads + 64;
constexpr int kStateCopyWarp = 8, kStateMmaWarp = 9;

// REV: the adjoint recurrence.  The chunks are walked from the last to the first with dy, C and B in the places of x, B and C; the
// local sum is taken to a chunk's first step, sum_i exp2(c_i - c_0) C_i dy_i^T, and what is handed out is the adjoint that enters a
// chunk from the right (the adjoint state at the next chunk's first step; the decay of that step belongs to the walk).
// PACKED: the walk covers one of several sequences that follow one another along the time axis.  Rows behind its end belong to the next
// one and must not reach the sums in any form (0 x Inf is NaN): K slices of 16 steps beyond the end are not multiplied, and the
// rows of the slice in which it ends are overwritten with zeros, in x and in B.
template <typename T, int HPC, int NST, bool REV, bool PACKED>
__global__ void __launch_bounds__(kStateThreads, 1) ssd_state_kernel(const ssm_ssd_args a, const __grid_constant__ StateMaps maps, int nchunks) {
  using M = StateSmem<HPC, NST>;
  constexpr int kStep = M::kStep, NS = M::NSTAGE;
  constexpr int SPC = kQ / kStep;  // stages per chunk
  extern __shared__ unsigned char smdyn[];
  unsigned char* smraw = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smdyn) + 1023) & ~(uintptr_t)1023);
  float* sVec = reinterpret_cast<float*>(smraw + NS * M::STAGE);  // [NS][HPC][kVec]
  static_assert(SPC % 2 == 0 && NS >= 2, "a group's stages are the same parts of every chunk");
  __shared__ __align__(8) uint64_t mbar_full[NS];   // a stage's copies have landed
  __shared__ __align__(8) uint64_t mbar_scaled[NS]; // every warp of the stage's group has scaled its part of the x rows
  __shared__ __align__(8) uint64_t mbar_free[NS];   // the MMAs that read a stage's buffer have completed
  __shared__ __align__(8) uint64_t mbar_acc[2];     // a chunk's accumulators are complete
  __shared__ __align__(8) uint64_t mbar_read[2];    // every compute warp has read them
  __shared__ uint32_t tmem_slot;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wg = tid >> 7;
  const int h0 = blockIdx.x * HPC;
  const int g = h0 / (a.heads / a.groups);
  // b: batch element of the operands; sb: whose state this is (the packed sequence, or b); the walk covers chunks c_off ..
  // c_off + nwalk, whose first step is t_off
  constexpr bool packed = PACKED;
  const int sb = blockIdx.y, b = packed ? 0 : sb;
  const int* seq_first = packed ? a.seq_table + 2 * a.num_chunks + sb : nullptr;
  const int c_off = packed ? __ldg(seq_first) : 0;
  const int nwalk = packed ? __ldg(seq_first + 1) - c_off : nchunks;
  const int t_off = packed && nwalk > 0 ? __ldg(a.seq_table + 2 * c_off) : 0;
  const int walk_len = packed && nwalk > 0 ? __ldg(a.seq_table + 2 * c_off + 1) - t_off : 0;
  const int n_states = packed ? a.num_seqs : a.batch;  // batch extent of the states
  const int n = (warp & 3) * 32 + lane;  // this thread's state index = TMEM lane
  constexpr int fmt = std::is_same<T, __nv_bfloat16>::value ? 1 : 0;
  constexpr uint32_t kCols = HPC <= 1 ? 128 : (HPC == 2 ? 256 : 512);  // 2 accumulators of 64 columns per head, a power of two

  if (warp == 0) tc::tmem_alloc(tc::smem_u32(&tmem_slot), kCols);
  if (tid == 0) {
    for (int i = 0; i < NS; ++i) {
      tc::mbar_init(tc::smem_u32(&mbar_full[i]), 1);
      tc::mbar_init(tc::smem_u32(&mbar_scaled[i]), kStateGroupThreads / 32);
      tc::mbar_init(tc::smem_u32(&mbar_free[i]), 1);
    }
    tc::mbar_init(tc::smem_u32(&mbar_acc[0]), 1);
    tc::mbar_init(tc::smem_u32(&mbar_acc[1]), 1);
    tc::mbar_init(tc::smem_u32(&mbar_read[0]), kStateComputeThreads / 32);
    tc::mbar_init(tc::smem_u32(&mbar_read[1]), kStateComputeThreads / 32);
  }
  __syncthreads();  // TMEM address and barriers are set up
  const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_slot, 0);
  const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
  const int role = __shfl_sync(0xffffffffu, warp, 0);  // the same in every lane, and visibly so

  const int64_t vrow0 = (((int64_t)b * a.heads + h0) * nchunks + c_off) * kQ;  // exponent vectors of head h0 (next head: + nchunks * kQ)
  const int nst = SPC * nwalk;
  // steps of the sequence from the first step of a stage on (packed sequences only; the first stage of a chunk has at least one)
  auto steps_left = [&](int c, int part) { return walk_len - c * kQ - part * kStep; };
  auto chunk_of = [&](int c) { return REV ? nwalk - 1 - c : c; };  // c-th chunk of the walk
  // stage s = steps [s * 64, s * 64 + 64), issued by one thread: two boxes of B, one box of x per head, and the exponents.
  // Steps beyond the sequence read as zero.
  auto copy_stage = [&](int s) {
    const uint32_t base = tc::smem_u32(smraw + (s % NS) * M::STAGE);
    const uint32_t full = tc::smem_u32(&mbar_full[s % NS]);
    const int c = chunk_of(s / SPC), part = s % SPC;
    const int t = t_off + c * kQ + part * kStep;
    tc::mbar_expect_tx(full, M::STAGE + HPC * (kStep * 4 + (REV ? 32 : 16)));
    tc::tma_load_4d(base, &maps.b, full, 0, g, t, b);
    tc::tma_load_4d(base + M::BLK_BYTES, &maps.b, full, 64, g, t, b);
#pragma unroll
    for (int hh = 0; hh < HPC; ++hh) {
      tc::tma_load_4d(base + M::A_BYTES + hh * M::BLK_BYTES, &maps.x, full, 0, h0 + hh, t, b);
      const int64_t at = vrow0 + ((int64_t)hh * nchunks + c) * kQ;
      const uint32_t dv = tc::smem_u32(sVec + ((s % NS) * HPC + hh) * M::kVec);
      tc::bulk_load(dv, (REV ? a.ws_cum : a.ws_dt) + at + part * kStep, kStep * 4, full);
      if (REV) tc::bulk_load(dv + kStep * 4, a.ws_cum + at, 16, full);
      tc::bulk_load(dv + kStep * 4 + 16, a.ws_cum + at + kQ - 4, 16, full);
    }
  };
  int fail = 0;
  if (role == kStateCopyWarp) {
    // ---- copies: a buffer is refilled once the MMAs of the stage that used it before have completed ------------
#pragma unroll 1
    for (int s = 0; s < nst; ++s) {
      bool okf = true;
      if (s >= NS) okf = __all_sync(0xffffffffu, tc::mbar_wait(tc::smem_u32(&mbar_free[s % NS]), ((s - NS) / NS) & 1));
      if (!okf) {  // the stage never lands and the waits of the other warps report it too
        fail = 1;
        break;
      }
      if (tc::elect_one()) copy_stage(s);
      __syncwarp();
    }
  } else if (role == kStateMmaWarp) {
    // ---- MMAs: S_c (+)= B^T (w x) over the 64 steps of a stage, as soon as the eight compute warps have scaled it ----
    float ctot[HPC];
#pragma unroll
    for (int hh = 0; hh < HPC; ++hh) ctot[hh] = 0.f;
#pragma unroll 1
    for (int s = 0; s < nst; ++s) {
      const int c = s / SPC, part = s % SPC;
      bool okm = true;
      // the accumulators of the chunk before last have been read
      if (part == 0 && c >= 2) okm = __all_sync(0xffffffffu, tc::mbar_wait(tc::smem_u32(&mbar_read[c & 1]), ((c - 2) >> 1) & 1));
      okm = okm && __all_sync(0xffffffffu, tc::mbar_wait(tc::smem_u32(&mbar_scaled[s % NS]), (s / NS) & 1));
      if (!okm) {
        fail = 1;
        break;
      }
      float last[HPC];  // read before the commit that lets the stage's buffer be refilled
#pragma unroll
      for (int hh = 0; hh < HPC; ++hh) last[hh] = sVec[((s % NS) * HPC + hh) * M::kVec + kStep + 7];
      tc::fence_after_sync();
      if (tc::elect_one()) {
        // M = 128 states = two 64-element blocks, N = 64 HPC = one block per head; blocks 8 KB apart, 8 steps 1 KB apart
        unsigned char* base = smraw + (s % NS) * M::STAGE;
        constexpr uint32_t idesc = tc::instr_desc(kN, HPC * kP, fmt, 1, 1);
        const uint64_t da0 = tc::smem_desc_sw128(tc::smem_u32(base), M::BLK_BYTES, 1024);
        const uint64_t db0 = tc::smem_desc_sw128(tc::smem_u32(base + M::A_BYTES), M::BLK_BYTES, 1024);
        const int live = packed && c == nwalk - 1 ? steps_left(c, part) : kStep;
#pragma unroll
        for (int kk = 0; kk < kStep / 16; ++kk)  // 16 steps = 16 rows of 128 bytes
          if (kk * 16 < live) tc::mma_ss(tmem + (c & 1) * HPC * 64, da0 + (uint64_t)(kk * (2048 >> 4)), db0 + (uint64_t)(kk * (2048 >> 4)), idesc, part > 0 || kk > 0);
        tc::commit(tc::smem_u32(&mbar_free[s % NS]));
        if (part == SPC - 1) tc::commit(tc::smem_u32(&mbar_acc[c & 1]));
      }
      __syncwarp();
      if (!REV && part == 0) {
#pragma unroll
        for (int hh = 0; hh < HPC; ++hh) {
          // exponent (base 2) of the decay from the start of the sequence to the start of this chunk: what a state
          // that arrives later (phase 2 of a sequence shard) is multiplied by before it joins this chunk's state
          if (lane == 0 && !packed) a.ws_state[ssd_summary_floats_padded(a.batch, a.heads) + ((int64_t)b * a.heads + h0 + hh) * nchunks + c] = ctot[hh];
          ctot[hh] += last[hh];
        }
      }
    }
    // the shard's total log-decay (natural log) follows the states in the scratch: together they are what a sequence shard sends to
    // the other ranks
    if (!REV && !fail && lane == 0) {
#pragma unroll
      for (int hh = 0; hh < HPC; ++hh) a.ws_state[(int64_t)n_states * a.heads * kP * kN + (int64_t)sb * a.heads + h0 + hh] = ctot[hh] * kLn2;
    }
  } else {
  // ======== compute warps ========================================================================================
  // running states: st[hh][i] = S_{h0 + hh}[n][wg * 32 + i]
  float st[HPC][32];
#pragma unroll
  for (int hh = 0; hh < HPC; ++hh) {
    const float* init = a.initial_states ? a.initial_states + (((int64_t)sb * a.heads + h0 + hh) * kP + wg * 32) * kN + n : nullptr;
#pragma unroll
    for (int i = 0; i < 32; ++i) st[hh][i] = init ? __ldg(init + (int64_t)i * kN) : 0.f;
  }
  T* sin = reinterpret_cast<T*>(a.ws_state_in);
  // the states before chunk c, in the operand dtype: unit (p / 8, n) of the (batch, chunk, head) tile
  auto emit_state_in = [&](int c) {
#pragma unroll
    for (int hh = 0; hh < HPC; ++hh) {
      T* blk = sin + (((int64_t)b * nchunks + c_off + chunk_of(c)) * a.heads + h0 + hh) * (int64_t)(kP * kN);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        Vec16<T> o;
        o.pack(*reinterpret_cast<const float(*)[8]>(&st[hh][q * 8]));
        *reinterpret_cast<uint4*>(blk + ((size_t)(wg * 4 + q) * kN + n) * 8) = o.raw;
      }
      if (a.ws_state_in_f32) {  // the same tile unrounded (the backward pass forms <adjoint state, state> from it)
        float* blk32 = a.ws_state_in_f32 + (((int64_t)b * nchunks + c_off + chunk_of(c)) * a.heads + h0 + hh) * (int64_t)(kP * kN);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          float4* dst = reinterpret_cast<float4*>(blk32 + ((size_t)(wg * 4 + q) * kN + n) * 8);
          dst[0] = make_float4(st[hh][q * 8], st[hh][q * 8 + 1], st[hh][q * 8 + 2], st[hh][q * 8 + 3]);
          dst[1] = make_float4(st[hh][q * 8 + 4], st[hh][q * 8 + 5], st[hh][q * 8 + 6], st[hh][q * 8 + 7]);
        }
      }
    }
  };
  // last exponent of the current / previous chunk per head (the decay across the chunk is exp2 of it)
  float clast[HPC], clast_prev[HPC];
#pragma unroll
  for (int hh = 0; hh < HPC; ++hh) clast[hh] = 0.f, clast_prev[hh] = 0.f;
  float cfirst[HPC];  // REV: the running exponent at the current chunk's first step
#pragma unroll
  for (int hh = 0; hh < HPC; ++hh) cfirst[hh] = 0.f;
  // fold chunk c's finished accumulators into the running states
  auto fold_chunk = [&](int c, const float (&cl)[HPC]) -> bool {
    const bool ok = __all_sync(0xffffffffu, tc::mbar_wait(tc::smem_u32(&mbar_acc[c & 1]), (c >> 1) & 1));
    tc::fence_after_sync();
    if (ok) {
#pragma unroll
      for (int hh = 0; hh < HPC; ++hh) {
        const float decay = ex2_approx(cl[hh]);
        float v[32];
        tc::tmem_ld32(tmem + lane_base + ((c & 1) * HPC + hh) * 64 + wg * 32, v);
#pragma unroll
        for (int i = 0; i < 32; ++i) st[hh][i] = fmaf(decay, st[hh][i], v[i]);
      }
    }
    tc::fence_before_sync();
    __syncwarp();
    if (lane == 0) tc::mbar_arrive(tc::smem_u32(&mbar_read[c & 1]));  // also by a warp whose wait ran out
    return ok;
  };

  const int gtid = tid & (kStateGroupThreads - 1);
#pragma unroll 1
  for (int s = wg; s < nst; s += 2) {  // a warp's group is its half of the columns, too
    const int c = s / SPC, part = s % SPC;
    if (s == wg) emit_state_in(0);
    if (!fail) fail = !__all_sync(0xffffffffu, tc::mbar_wait(tc::smem_u32(&mbar_full[s % NS]), (s / NS) & 1));  // this stage's copies
    const float* vs = sVec + (s % NS) * HPC * M::kVec;
    if (part < 2) {  // this group's first stage of a chunk
#pragma unroll
      for (int hh = 0; hh < HPC; ++hh) {
        const float* edge = vs + hh * M::kVec + kStep;  // c at the chunk's first four and last four steps
        clast_prev[hh] = clast[hh];
        clast[hh] = edge[7];
        if (REV) {  // from the first step of the chunk to its right, which was walked before, down to this one's
          clast[hh] += cfirst[hh] - edge[0];
          cfirst[hh] = edge[0];
        }
      }
    }

    // ---- scale the x rows in place: w_j x_j (a row is one step, whatever the swizzle does inside it).  Every load of a head (or
    // of two) before its first store: the compiler cannot tell that the units are distinct, and one after the other would put a
    // shared-memory round trip per unit on the critical path of the stage
    unsigned char* xs = smraw + (s % NS) * M::STAGE + M::A_BYTES;
    constexpr int UPT = M::BLK_BYTES / 16 / kStateGroupThreads;  // 16-byte units of a head's tile per thread; 8 units per step
    constexpr int HB = HPC == 2 ? 2 : 1;                         // heads at a time: what the registers allow
#pragma unroll
    for (int h2 = 0; h2 < HPC; h2 += HB) {
      uint4 raw[HB][UPT];
      float wt[HB][UPT];
#pragma unroll
      for (int hh = h2; hh < h2 + HB && hh < HPC; ++hh) {
#pragma unroll
        for (int k = 0; k < UPT; ++k) {
          const int u = gtid + kStateGroupThreads * k;
          wt[hh - h2][k] = vs[hh * M::kVec + (u >> 3)];
          raw[hh - h2][k] = *reinterpret_cast<const uint4*>(xs + hh * M::BLK_BYTES + (size_t)u * 16);
        }
      }
#pragma unroll
      for (int hh = h2; hh < h2 + HB && hh < HPC; ++hh) {
#pragma unroll
        for (int k = 0; k < UPT; ++k) {
          const float e = wt[hh - h2][k];
          const float w = ex2_approx(REV ? e - cfirst[hh] : clast[hh] - e);  // 0 for steps beyond the sequence
          Vec16<T> v;
          v.raw = raw[hh - h2][k];
          float f[8];
          v.unpack(f);
#pragma unroll
          for (int i = 0; i < 8; ++i) f[i] *= w;
          v.pack(f);
          *reinterpret_cast<uint4*>(xs + hh * M::BLK_BYTES + (size_t)(gtid + kStateGroupThreads * k) * 16) = v.raw;
        }
      }
    }
    if (packed && c == nwalk - 1) {  // the last chunk: zeros behind the sequence, by the threads that have scaled these units of x
      const int live = steps_left(c, part);
      if (live > 0 && live < kStep && (gtid >> 3) >= (live & 15)) {
#pragma unroll
        for (int blk = 0; blk < 2 + HPC; ++blk)
          *reinterpret_cast<uint4*>(smraw + (s % NS) * M::STAGE + blk * M::BLK_BYTES + (size_t)(gtid + kStateGroupThreads * (live >> 4)) * 16) = make_uint4(0, 0, 0, 0);
      }
    }
    // the scaled rows become visible to the tensor cores' reads.  A warp whose wait ran out still arrives, so that the others do
    // not wait for it.
    tc::fence_async_smem();
    __syncwarp();
    if (lane == 0) tc::mbar_arrive(tc::smem_u32(&mbar_scaled[s % NS]));
    // ---- its second stage is on its way, and the MMAs of the chunk before are surely finished: fold them, hand out the states
    // ---- before this chunk
    if (part >= 2 && c >= 1) {
      if (!fold_chunk(c - 1, clast_prev)) fail = 1;
      emit_state_in(c);
    }
  }
  if (nwalk > 0 && !fold_chunk(nwalk - 1, clast)) fail = 1;
  // final states in fp32, (p, n) order: to the caller, and kept in scratch for a later phase 2
  if (!fail) {
#pragma unroll
    for (int hh = 0; hh < HPC; ++hh) {
      const int64_t off = (((int64_t)sb * a.heads + h0 + hh) * kP + wg * 32) * kN + n;
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        if (a.final_states) a.final_states[off + (int64_t)i * kN] = st[hh][i];
        a.ws_state[off + (int64_t)i * kN] = st[hh][i];
      }
    }
  }
  }  // compute warps
  if (fail && lane == 0 && a.status) *(volatile int32_t*)a.status = 1;
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, kCols);
}

// ---------------------------------------------------------------------------------------------
// phase 2 of a sequence shard: the shard's incoming state S0 arrives after the chunk states were
// formed from a zero state.  By linearity  state_before_chunk_c += exp2(sum_{c' < c} c_last[c']) * S0
// and  final += exp2(sum_c c_last[c]) * S0.  One thread per element, operand order of the scan kernel.
// ---------------------------------------------------------------------------------------------
constexpr int kFoldChunks = 8;  // chunks per thread: the eight values of S0 are read once for them, their loads go out together
template <typename T>
__global__ void __launch_bounds__(256) ssd_fold_init_kernel(const ssm_ssd_args a, int nchunks) {
  // thread = one 16-byte unit (p / 8, n) of the states before kFoldChunks chunks; blockIdx.y = group of chunks (the row after
  // the last chunk: final states)
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;  // unit of one (batch, head): 1024 units each
  const int64_t units = (int64_t)a.batch * a.heads * (kP * kN / 8);
  if (i >= units) return;
  const int64_t bh = i / (kP * kN / 8);
  const int u = (int)(i % (kP * kN / 8));
  const int n = u % kN, pc = u / kN;
  const int b = (int)(bh / a.heads), h = (int)(bh % a.heads);
  const int c0 = blockIdx.y * kFoldChunks;
  const float* s0p = a.initial_states + bh * (int64_t)(kP * kN) + (int64_t)(pc * 8) * kN + n;  // 8 values p = 8 pc .. 8 pc + 7 of state n
  const float* pre = a.ws_state + ssd_summary_floats_padded(a.batch, a.heads);
  float s0[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) s0[e] = __ldg(s0p + (int64_t)e * kN);
  T* blk0 = reinterpret_cast<T*>(a.ws_state_in) + (((int64_t)b * nchunks) * a.heads + h) * (int64_t)(kP * kN) + (int64_t)u * 8;
  const int64_t cstride = (int64_t)a.heads * (kP * kN);
  uint4 raw[kFoldChunks];
  float wl[kFoldChunks];
#pragma unroll
  for (int k = 0; k < kFoldChunks; ++k) {
    const int c = min(c0 + k, nchunks - 1);  // beyond the last chunk: a valid address, dropped below
    raw[k] = *reinterpret_cast<const uint4*>(blk0 + c * cstride);
    wl[k] = __ldg(pre + bh * nchunks + c);
  }
#pragma unroll
  for (int k = 0; k < kFoldChunks; ++k) {
    const int c = c0 + k;
    if (c < nchunks) {
      const float w = ex2_approx(wl[k]);
      Vec16<T> v;
      v.raw = raw[k];
      float f[8];
      v.unpack(f);
#pragma unroll
      for (int e = 0; e < 8; ++e) f[e] = fmaf(w, s0[e], f[e]);
      v.pack(f);
      *reinterpret_cast<uint4*>(blk0 + c * cstride) = v.raw;
    } else if (c == nchunks && a.final_states) {
      const float w = __expf(__ldg(a.ws_state + (int64_t)a.batch * a.heads * kP * kN + bh));  // total log-decay of the call
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int64_t off = bh * (int64_t)(kP * kN) + (int64_t)(pc * 8 + e) * kN + n;
        a.final_states[off] = fmaf(w, s0[e], a.ws_state[off]);
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------
// chunk scan: one CTA (512 threads) per (batch, chunk, 128-row block m, part of the heads of one
// B / C group).  Heads of a group share B and C, so  G = C_m B^T  (128 x 128 (m+1), causal: only
// steps before the block's last row) is formed ONCE per CTA; every thread then keeps its part of
// G (one row, a quarter of the steps) in registers while the CTA walks its heads:
//   per head:  G times the head's decay mask exp2(c_i - c_j) delta_j [j <= i], packed as the A
//              operand (in tensor memory, over the dead G columns);  Y_intra = (G o L) X  and
//              Y_inter = C_m S_in accumulate in TMEM while the previous head's result is read
//              back, gated and staged.
//   Copies (TMA and bulk copies issued by one warp, the MMAs too) run one head ahead into the other half of a
//   double buffer: x, the incoming state, the exponent vectors; z and the y that leaves by a TMA store have two
//   tiles each over the dead B tile.
//   TMEM columns: G [0,256), later the masked operands of two heads [128b, +128); per buffer b: Y_intra [256+128b, +64),
//   Y_inter [320+128b, +64).
// No CTA-wide barrier per head: the warps pass mbarriers (operands landed, operand written, MMAs done, epilogue done, y read), so
// that one warp's mask runs beside another's epilogue.  Before, two CTA-wide barriers per head kept the warps in step, the cut on the
// diagonal cost its four warps 128 compares and adds a head, and all waited for them.  8 x 8192 steps of 48 heads, gate and D: 390 us,
// now 347; 24 packed sequences in 16384 steps 125, now 107; 2 x 4001 steps 63, now 56.5, adjoint 62.5, now 57.
// Tried: column factors formed once per CTA by idle warps (353, 113, 57); operands two heads ahead with y stored from registers in sectors of
// 32 bytes (401, 103, 76: the row-strided stores); the issuing done by a seventeenth warp without the register split (spills).
// ---------------------------------------------------------------------------------------------
template <typename T>
struct ScanSmem {
  static constexpr int C_BYTES = kBlk * kN * 2;     // C rows of the block: two blocks (states 0..63, 64..127) of [i][128 B], swizzled   32 KB
  static constexpr int B_BYTES = kQ * kN * 2;       // B rows likewise, [j][128 B] per block; later the gate tiles of two heads  64 KB
  static constexpr int X_BYTES = kQ * kP * 2;       // x rows [j][64 p], 128-byte rows, TMA 128-byte swizzle  32 KB (x2)
  static constexpr int S_BYTES = kP * kN * 2;       // incoming state, MN-major [p/8][n][8]                 16 KB (x2)
  static constexpr int VEC_BYTES = 2 * kQ * 4;      // c and c - log2(delta) of the chunk                     2 KB (x2)
  static constexpr int Z_BYTES = kBlk * kP * 2;     // gate rows of a head, or y on its way out: [row][64 p], same swizzle; 4 x 16 KB over the B tile
  static_assert(4 * Z_BYTES <= B_BYTES, "two gate tiles and two of y fit over the B tile");
  static constexpr int W_BYTES = 1024 * 4;          // per warp: the column factors of its mask chunks (16 warps x 64)          4 KB
  static constexpr int TOTAL = C_BYTES + B_BYTES + 2 * (X_BYTES + S_BYTES + VEC_BYTES) + W_BYTES;
  static constexpr int ALLOC = TOTAL + 1024;        // the tiles TMA swizzles must start on 1024-byte boundaries
};

constexpr int kScanCompute = 512;                // threads of the mask and the epilogue
// ... and a warpgroup whose first warp issues the copies and the MMAs.  Launched with 96 registers a thread (640 x 96 = 61440): the
// issuing group keeps 32, the others take 112 (128 x 32 + 512 x 112 = 61440).
constexpr int kScanThreads = kScanCompute + 128;
constexpr int kScanIssueRegs = 32, kScanComputeRegs = 112;
static_assert(128 * kScanIssueRegs + kScanCompute * kScanComputeRegs <= kScanThreads * 96, "the split draws on what the block was launched with");
constexpr int kScanWG = kScanCompute / 128;  // warpgroups: each owns every kScanWG-th 32-step column chunk of the mask and kP / kScanWG output columns
constexpr int kEC = kP / kScanWG;             // epilogue columns per thread
constexpr int kEU = kEC / 8;                  // ... in 16-byte units
// tensor maps of one call: x (box of 128 or 256 steps), z and y (boxes of 128 rows); rank 4 (p, head, step, batch)
struct ScanMaps {
  CUtensorMap x0, x1, z, y;
  CUtensorMap c, bm;  // C and B rows: rank 4 (state, group, step, batch), boxes of 64 states x 128 steps
};

// Body for row block MB (0: rows 0..127, steps 0..127; 1: rows 128..255, steps 0..255).  XSKIP: the skip term D x is added
// in the epilogue (a weight per channel, or the row sums of the backward pass are wanted), which carries each thread's x row
// from one iteration to the next; without it a weight per head rides on the diagonal of the masked operand.
// REV: the adjoint pass, dx_j = dt_j (sum_{i >= j} exp2(c_i - c_j) (B_j . C_i) dy_i + exp2(off - c_j) G B_j), with B, C and dy in the places of C, B
// and x, and G the adjoint that enters the chunk from the right (off: the decay of the chunk and of the step after it).  It is the
// mirror image in time: columns at or after the row's step, the long block is rows 0..127.
// PACKED: several sequences along the time axis; rows behind the end of a chunk's sequence belong to the next one.  Their columns of the
// mask are zero, but 0 x Inf is NaN: the x rows under them are overwritten with zeros.  Kernel us without / with that, 24 sequences in
// 16384 steps of 48 heads 121 / 123, 4 in 6344 of 28 heads 39.3 / 39.8 (by all warps in front of the mask 124 and 42; with an instance of
// the body for ragged blocks, which the instruction cache does not hold beside the other two, 131 and 49).
template <typename T, int MB, bool XSKIP, bool REV, bool PACKED>
__device__ __forceinline__ void ssd_scan_body(const ssm_ssd_args& a, const ScanMaps& maps, int nchunks, int hpc, int nparts, unsigned char* smraw,
                                              uint64_t* mbar, uint32_t* tmem_slot) {
  using M = ScanSmem<T>;
  constexpr int KJ = (MB + 1) * kBlk;  // steps that can reach this block's rows
  constexpr int NCH = KJ / (32 * kScanWG);  // 32-step column chunks per thread (the warpgroups interleave chunks)
  constexpr int ROW0 = (REV ? 1 - MB : MB) * kBlk;  // first row and first column of the block within the chunk
  constexpr int COL0 = REV ? ROW0 : 0;
  constexpr int VLEN = REV ? kQ : KJ;               // exponents of the chunk that are needed
  unsigned char* sC = smraw;
  unsigned char* sBA = sC + M::C_BYTES;
  unsigned char* sX = sBA + M::B_BYTES;        // two buffers
  unsigned char* sS = sX + 2 * M::X_BYTES;     // two buffers
  float* sVec = reinterpret_cast<float*>(sS + 2 * M::S_BYTES);  // two buffers of [c | c - log2 delta]
  // mbar: 0 G done; 1 C and B tiles landed; per buffer b of a head: 2 + b its MMAs done; 4 + b its operands landed; 6 + b masked operand
  // written; 8 + b epilogue done; 10 + b its y has been read from the staging tile; 12 + b its gate rows landed
  const uint32_t mb_g = tc::smem_u32(&mbar[0]), mb_cb = tc::smem_u32(&mbar[1]);
  auto mb_mma = [&](int bf) { return tc::smem_u32(&mbar[2 + bf]); };
  auto mb_full = [&](int bf) { return tc::smem_u32(&mbar[4 + bf]); };
  auto mb_mask = [&](int bf) { return tc::smem_u32(&mbar[6 + bf]); };
  auto mb_epi = [&](int bf) { return tc::smem_u32(&mbar[8 + bf]); };
  auto mb_out = [&](int bf) { return tc::smem_u32(&mbar[10 + bf]); };
  auto mb_z = [&](int bf) { return tc::smem_u32(&mbar[12 + bf]); };

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wg = tid >> 7;                     // column chunks wg, wg + kScanWG, ... in the mask stage; column slice in the epilogue
  float* sW = sVec + 2 * (M::VEC_BYTES / 4) + (warp & 15) * (NCH * 32);  // this warp's column factors
  // The gate rows of a head and its y on the way out have two buffers each, over the B tile (dead once G is formed: the masked
  // operand lives in tensor memory).
  auto sZin = [&](int bf) { return sBA + bf * M::Z_BYTES; };
  auto sY = [&](int bf) { return sBA + (2 + bf) * M::Z_BYTES; };
  const int half_grid = gridDim.x >> 1;
  const int rem = (int)blockIdx.x % half_grid;
  const int part = rem % nparts, bc = rem / nparts;
  const int c = bc % nchunks, b = bc / nchunks;
  const int h0 = part * hpc;
  const int nh = min(hpc, a.heads - h0);
  const int g = h0 / (a.heads / a.groups);
  const int t0 = PACKED ? chunk_begin(a, c) : c * kQ;
  // rows of this block that exist; a ragged block of a packed sequence stores its rows by hand (what follows them belongs to
  // the next sequence), everything else leaves through TMA, which cuts at the end of the tensor
  const int t_live = PACKED ? chunk_limit(a, c) - t0 - ROW0 : kBlk;
  const bool ragged = PACKED && t_live < kBlk;
  const int k_live = ragged ? t_live + ROW0 - COL0 : KJ;  // columns that belong to the sequence
  const int i_loc = (warp & 3) * 32 + lane;    // row within the block = TMEM lane
  const int i_chunk = ROW0 + i_loc;            // row within the chunk
  const int rc = (ROW0 - COL0) / 32 + (warp & 3);  // this warp's rows as a 32-step chunk index, counted like the columns
  auto reached = [&](int cc) { return REV ? cc >= rc : cc <= rc; };  // column chunks that reach this warp's rows
  constexpr int fmt = std::is_same<T, __nv_bfloat16>::value ? 1 : 0;
  const bool has_z = a.z != nullptr;
  const CUtensorMap* mapx = MB ? &maps.x1 : &maps.x0;

  // ---- C rows of the block, B rows of the reachable steps, by TMA: per half of the states one block of 128-byte rows
  if (tid == kScanCompute) {
    tc::mbar_expect_tx(mb_cb, M::C_BYTES + KJ * kN * 2);
#pragma unroll
    for (int nb2 = 0; nb2 < 2; ++nb2) {
      tc::tma_load_4d(tc::smem_u32(sC + nb2 * (kBlk * 128)), &maps.c, mb_cb, nb2 * 64, g, t0 + ROW0, b);
#pragma unroll
      for (int jb2 = 0; jb2 <= MB; ++jb2)
        tc::tma_load_4d(tc::smem_u32(sBA + nb2 * (KJ * 128) + jb2 * (kBlk * 128)), &maps.bm, mb_cb, nb2 * 64, g, t0 + COL0 + jb2 * kBlk, b);
    }
  }

  // One head's operands, by bulk copies issued from one thread: x rows through the tensor map (128-byte rows, swizzled),
  // the incoming state and the two exponent vectors as contiguous pieces.  Steps beyond the sequence read as zero.
  constexpr uint32_t kOperandBytes = KJ * kP * 2 + M::S_BYTES + 2 * VLEN * 4;
  auto prefetch = [&](int h, int buf) {
    const uint32_t full = mb_full(buf);
    tc::mbar_expect_tx(full, kOperandBytes);
    tc::tma_load_4d(tc::smem_u32(sX + buf * M::X_BYTES), mapx, full, 0, h, t0 + COL0, b);
    const T* ss = reinterpret_cast<const T*>(a.ws_state_in) + (((int64_t)b * nchunks + c) * a.heads + h) * (int64_t)(kP * kN);
    tc::bulk_load(tc::smem_u32(sS + buf * M::S_BYTES), ss, M::S_BYTES, full);
    const int64_t voff = (((int64_t)b * a.heads + h) * nchunks + c) * kQ;
    float* dV = sVec + buf * (2 * kQ);
    tc::bulk_load(tc::smem_u32(dV), a.ws_cum + voff, VLEN * 4, full);
    tc::bulk_load(tc::smem_u32(dV + kQ), a.ws_dt + voff, VLEN * 4, full);
  };
  // slot of (row, 16-byte chunk) in a tile of 128-byte rows written / read by TMA with the 128-byte swizzle
  auto swz = [&](unsigned char* tile, int row, int chunk) { return tile + ((size_t)row * 8 + (chunk ^ (row & 7))) * 16; };

  if (tid == kScanCompute) prefetch(h0, 0);

  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
  const bool issuer = __shfl_sync(0xffffffffu, warp, 0) == kScanCompute / 32;  // the same in every lane, and visibly so
  auto wait = [&](uint32_t bar, int n) { return (bool)__all_sync(0xffffffffu, tc::mbar_test(bar, n & 1) || tc::mbar_wait(bar, n & 1)); };  // the n-th completion; warp-uniform
  const int t_blk = t0 + ROW0;  // first step of this block's rows

  // ---- G = C_m B^T ------------------------------------------------------------------------------------
  // K-major operands in 128-byte-swizzled rows: 16 states = 32 bytes further along the row, 64 states = the next block
  const uint64_t dc0 = tc::smem_desc_sw128(tc::smem_u32(sC), 16, 1024);
  bool ok = true;
  if (issuer) {
    ok = wait(mb_cb, 0);
    if (ok && tc::elect_one()) {
      const uint64_t db0 = tc::smem_desc_sw128(tc::smem_u32(sBA), 16, 1024);
      constexpr uint32_t idG = tc::instr_desc(kBlk, KJ, fmt, 0, 0);
#pragma unroll
      for (int kk = 0; kk < kN / 16; ++kk)
        tc::mma_ss(tmem, dc0 + (uint64_t)(((kk >> 2) * (kBlk * 128) + (kk & 3) * 32) >> 4), db0 + (uint64_t)(((kk >> 2) * (KJ * 128) + (kk & 3) * 32) >> 4), idG,
                   kk > 0);
      tc::commit(mb_g);
    }
    __syncwarp();
  }
  ok = wait(mb_g, 0) && ok;
  tc::fence_after_sync();

  // ======== copies and MMAs: one warp, which the others never wait for but through what it issues ====================
  if (wg == kScanWG) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(kScanIssueRegs));
    __syncthreads();  // G has been read: its columns and the B tile are free
    if (!issuer) return;
    int fail = ok ? 0 : 1;
#pragma unroll 1
    for (int hi = 0; hi < nh && !fail; ++hi) {
      const int h = h0 + hi, buf = hi & 1;
      // the other buffer's tiles are free once the MMAs of the head before are done (its exponents were read before those began)
      if (hi >= 1 && !wait(mb_mma(buf ^ 1), (hi - 1) >> 1)) {
        fail = 1;
        break;
      }
      if (hi + 1 < nh && lane == 0) prefetch(h + 1, buf ^ 1);
      __syncwarp();
      // accumulators, gate tile and staged y of this buffer: the epilogue of the head before last
      if ((hi >= 2 && !wait(mb_epi(buf), (hi - 2) >> 1)) || !wait(mb_full(buf), hi >> 1)) {
        fail = 1;
        break;
      }
      tc::fence_after_sync();
      if (tc::elect_one()) {
        // Y_inter = C_m S_in needs nothing of the mask: issued first, it runs on the tensor cores while the mask is formed
        const uint64_t ds0 = tc::smem_desc(tc::smem_u32(sS + buf * M::S_BYTES), 128, kN * 16);
        constexpr uint32_t idS = tc::instr_desc(kBlk, kP, fmt, 0, 1);
        const uint32_t dS = tmem + 256 + buf * 128 + 64;
#pragma unroll
        for (int kk = 0; kk < kN / 16; ++kk)
          tc::mma_ss(dS, dc0 + (uint64_t)(((kk >> 2) * (kBlk * 128) + (kk & 3) * 32) >> 4), ds0 + (uint64_t)(kk * (256 >> 4)), idS, kk > 0);
      }
      __syncwarp();
      if (lane == 0) {
        if (has_z) {
          tc::mbar_expect_tx(mb_z(buf), M::Z_BYTES);
          tc::tma_load_4d(tc::smem_u32(sZin(buf)), &maps.z, mb_z(buf), 0, h, t_blk, b);
        }
        if (hi >= 2 && !ragged) {
          tc::tma_store_4d(&maps.y, tc::smem_u32(sY(buf)), 0, h - 2, t_blk, b);
          tc::bulk_commit();
        }
        if (hi + 2 < nh) {  // the tiles of the head after next on their way into the L2: one iteration alone does not cover the latency
          tc::tma_prefetch_4d(mapx, 0, h + 2, t0 + COL0, b);
          if (has_z) tc::tma_prefetch_4d(&maps.z, 0, h + 2, t_blk, b);
          tc::bulk_prefetch(reinterpret_cast<const T*>(a.ws_state_in) + (((int64_t)b * nchunks + c) * a.heads + h + 2) * (int64_t)(kP * kN), M::S_BYTES);
        }
      }
      __syncwarp();
      if (!wait(mb_mask(buf), hi >> 1)) {
        fail = 1;
        break;
      }
      tc::fence_after_sync();
      // ---- Y_intra = (G o L) X  for this head; the commit also covers the Y_inter MMAs issued above
      if (tc::elect_one()) {
        // descriptors differ from instruction to instruction only in the start address (16-byte units, low bits)
        const uint64_t dx0 = tc::smem_desc_sw128(tc::smem_u32(sX + buf * M::X_BYTES), 16, 1024);
        constexpr uint32_t idY = tc::instr_desc(kBlk, kP, fmt, 0, 1);
        const uint32_t dY = tmem + 256 + buf * 128, dA = tmem + buf * 128;
#pragma unroll
        for (int kk = 0; kk < KJ / 16; ++kk)  // 16 steps = 16 rows of 128 bytes of the x tile
          tc::mma_ts(dY, dA + kk * 8, dx0 + (uint64_t)(kk * (2048 >> 4)), idY, kk > 0);  // A: 16 steps = 8 columns of the masked rows
        tc::commit(mb_mma(buf));
      }
      __syncwarp();
      if (hi >= 2 && !ragged && lane == 0) {  // (the store's reads queue behind this iteration's copies: never in front of the MMAs)
        tc::bulk_wait_read();
        tc::mbar_arrive(mb_out(buf));
      }
      __syncwarp();
    }
    for (int hi = max(nh - 2, 0); hi < nh && !fail && !ragged; ++hi) {
      if (!wait(mb_epi(hi & 1), hi >> 1)) {
        fail = 1;
      } else if (lane == 0) {
        tc::tma_store_4d(&maps.y, tc::smem_u32(sY(hi & 1)), 0, h0 + hi, t_blk, b);
        tc::bulk_commit();
      }
    }
    if (lane == 0) {
      tc::bulk_wait_all();  // the staging tiles must outlive the stores that read them
      if (fail && a.status) *(volatile int32_t*)a.status = 2;
    }
    return;
  }

  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(kScanComputeRegs));

  // This thread's part of G stays in registers for all heads: row i_loc, chunks wg, wg + kScanWG, ...
  const bool fold_d = !XSKIP && !REV && a.D;  // see below
  float vG[NCH][32], gdiag = 0.f;
#pragma unroll
  for (int k = 0; k < NCH; ++k) {
    const int cc = wg + kScanWG * k;
    if (ok && reached(cc)) {
      tc::tmem_ld32(tmem + lane_base + cc * 32, vG[k]);
    } else {
#pragma unroll
      for (int e = 0; e < 32; ++e) vG[k][e] = 0.f;
    }
    if (cc == rc) {  // the chunk of this warp's own rows: steps after the row are cut
#pragma unroll
      for (int e = 0; e < 32; ++e) {
        if (e == lane) gdiag = vG[k][e];
        if (REV ? e < lane : (fold_d ? e >= lane : e > lane)) vG[k][e] = 0.f;
      }
    }
  }
  tc::fence_before_sync();
  __syncthreads();  // every part of G has been read: the masked operands take its columns, the gate tiles and y the B tile
  tc::fence_after_sync();

  // A skip weight per head (not per channel) rides on the diagonal of the masked operand: (G o L + D I) X = Y_intra + D x.
  // The row sums for the backward pass want y without the skip term, so that mode keeps the explicit form.
  constexpr bool skip_explicit = XSKIP;

  // epilogue of head h from accumulator pair `buf`: y = Y_intra + exp2(c_i) Y_inter (+ D x where it is not folded), gated by
  // the z row, staged for the bulk store.  Thread = row i_loc, this warpgroup's 16 columns; the arithmetic runs on pairs.
  constexpr int kXR = XSKIP ? kEU : 1;  // x row registers exist only where the explicit skip term needs them
  auto epilogue = [&](int h, int buf, float ct, const uint4 (&xr)[kXR]) {
    const float escale = ex2_approx(ct);
    const float2 es2 = make_float2(escale, escale);
    const float Dh = (skip_explicit && !a.d_has_p) ? __ldg(a.D + h) : 0.f;
    const bool dots = a.row_dots != nullptr;
    float dot = 0.f;  // row_dots: this thread's 16 columns of  sum_p y[p] z[p]  (y before the skip term and unrounded)
#pragma unroll
    for (int q = 0; q < kEU; ++q) {
      // eight columns at a time: sixteen left too few registers, and the instance with a skip weight per channel spilled 130 bytes (1 x 1024 steps of
      // 24 heads 11.8 us, 10.1 so; mirrored 2 x 4001 of 48 55.0 and 52.6; the others equal)
      float2 f2[4];
      float yi[8], ys[8];
      tc::tmem_ld8_pair(tmem + lane_base + 256 + buf * 128 + wg * kEC + q * 8, tmem + lane_base + 320 + buf * 128 + wg * kEC + q * 8, yi, ys);
#pragma unroll
      for (int e = 0; e < 4; ++e)
        f2[e] = __ffma2_rn(es2, make_float2(ys[2 * e], ys[2 * e + 1]), make_float2(yi[2 * e], yi[2 * e + 1]));
      float zv[8];
      if (has_z) {
        Vec16<T> zz;
        zz.raw = *reinterpret_cast<const uint4*>(swz(sZin(buf), i_loc, wg * kEU + q));
        zz.unpack(zv);
        if (dots) {
#pragma unroll
          for (int e = 0; e < 4; ++e) dot = fmaf(f2[e].x, zv[2 * e], dot), dot = fmaf(f2[e].y, zv[2 * e + 1], dot);
        }
      }
      if (skip_explicit) {
        float xv[8];
        Vec16<T> xx;
        xx.raw = xr[XSKIP ? q : 0];
        xx.unpack(xv);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 d2 = a.d_has_p ? make_float2(__ldg(a.D + h * kP + wg * kEC + q * 8 + 2 * e), __ldg(a.D + h * kP + wg * kEC + q * 8 + 2 * e + 1))
                                      : make_float2(Dh, Dh);
          f2[e] = __ffma2_rn(d2, make_float2(xv[2 * e], xv[2 * e + 1]), f2[e]);
        }
      }
      if (has_z && !dots) {  // y silu(z), silu(z) = h + h tanh(h) with h = z / 2
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 h2 = __fmul2_rn(make_float2(zv[2 * e], zv[2 * e + 1]), make_float2(0.5f, 0.5f));
          float2 t2;
          asm("tanh.approx.f32 %0, %1;" : "=f"(t2.x) : "f"(h2.x));
          asm("tanh.approx.f32 %0, %1;" : "=f"(t2.y) : "f"(h2.y));
          f2[e] = __fmul2_rn(f2[e], __ffma2_rn(h2, t2, h2));
        }
      }
      float f[8];
#pragma unroll
      for (int e = 0; e < 4; ++e) f[2 * e] = f2[e].x, f[2 * e + 1] = f2[e].y;
      Vec16<T> o;
      o.pack(f);
      *reinterpret_cast<uint4*>(swz(sY(buf), i_loc, wg * kEU + q)) = o.raw;
    }
    if (dots && has_z) {
      const int t = t0 + ROW0 + i_loc;
      // the four threads of a row (column slices) add to one zero-initialised word, in any order: its last bits vary from run to run
      if (t < a.len) atomicAdd(a.row_dots + ((int64_t)b * a.len + t) * a.heads + h, dot);
    }
    tc::fence_async_smem();  // the staged rows leave through a bulk store
  };
  auto store_rows = [&](int h, int buf) {  // the staged rows of a ragged block, 16 bytes a thread
    for (int u = tid; u < t_live * 8; u += kScanCompute)
      *reinterpret_cast<uint4*>(reinterpret_cast<T*>(a.Y) + (((int64_t)b * a.len + t_blk + (u >> 3)) * a.heads + h) * kP + (u & 7) * 8) =
          *reinterpret_cast<const uint4*>(swz(sY(buf), u >> 3, u & 7));
  };

  float ct_prev = 0.f;   // the previous head's row exponent and x row, carried into its (deferred) epilogue
  uint4 xr_prev[kXR];
#pragma unroll
  for (int q = 0; q < kXR; ++q) xr_prev[q] = make_uint4(0, 0, 0, 0);
  int fail = ok ? 0 : 1;
  // No CTA-wide barrier in the loop: a warp tells the issuing warp when its rows of the masked operand are written and when its
  // epilogue is done, and waits only for what it reads next.  With two masked operands a warp's mask needs the MMAs of the head before last,
  // and its epilogue those of the head before, which have had a whole mask to run.
#pragma unroll 1
  for (int hi = 0; hi <= nh && !fail; ++hi) {
    const int h = h0 + hi, buf = hi & 1;
    float ct = 0.f;
    uint4 xr[kXR];
#pragma unroll
    for (int q = 0; q < kXR; ++q) xr[q] = make_uint4(0, 0, 0, 0);
    if (hi < nh) {
      if (!wait(mb_full(buf), hi >> 1)) {  // this head's operands
        fail = 1;
        break;
      }
      const float* vc = sVec + buf * (2 * kQ);
      const float* vcp = vc + kQ;
      const float Dfold = fold_d ? __ldg(a.D + h) : 0.f;
      // exponents of the decay mask, weight = exp2(re - col(j)), and of the carried state's row weight, exp2(ct)
      float re;
      if constexpr (REV) {
        const float next = c + 1 < nchunks ? __ldg(a.ws_cum + (((int64_t)b * a.heads + h) * nchunks + c + 1) * kQ) : 0.f;
        re = -vcp[i_chunk], ct = vc[kQ - 1] + next + re;
      } else {
        re = ct = vc[i_chunk];
      }
      auto col = [&](int j) { return REV ? -vc[COL0 + j] : vcp[j]; };
      // The weight exp2(c_i - c'_j) of a 32-step chunk factors as exp2(c_i - r) * exp2(r - c'_j) with r = c at the
      // chunk's first step (row factor <= 1 for causal rows, column factor bounded by the decay inside the chunk).
      // Each lane forms one column factor per chunk, each thread one row factor per chunk: 2 ex2 per 32 elements
      // instead of 32.  Chunks whose internal decay exceeds 2^60 keep the exact per-element form.
      float arow[NCH], bdiag = 0.f;
      bool fast[NCH];
#pragma unroll
      for (int k = 0; k < NCH; ++k) {
        const int cc = wg + kScanWG * k;
        arow[k] = 0.f, fast[k] = false;
        if (reached(cc)) {
          const float first = vc[COL0 + cc * 32], r = REV ? -first : first;
          fast[k] = first - vc[COL0 + cc * 32 + 31] < 60.f;  // same for every lane
          arow[k] = ex2_approx(re - r);
          const float bcol = ex2_approx(r - col(cc * 32 + lane));
          sW[k * 32 + lane] = bcol;
          // on the diagonal the steps after a row are cut by a zero in its G, which needs finite factors (a step size may be anything)
          if (cc == rc) bdiag = bcol, fast[k] = __all_sync(0xffffffffu, fast[k] && fabsf(bcol) < __int_as_float(0x7f800000));
        }
      }
      __syncwarp();  // the column factors are read by other lanes
      if (ragged && hi >= 2) {  // before this head's mask is reported, and thereby before the staging tile is written again
        if (!wait(mb_epi(buf), (hi - 2) >> 1)) {
          fail = 1;
          break;
        }
        store_rows(h - 2, buf);
      }
      // ---- decay mask: G (registers) x the factors formed above -> the A operand in tensor memory
#pragma unroll
      for (int k = 0; k < NCH; ++k) {
        const int cc = wg + kScanWG * k;  // chunk of 32 steps: whole, diagonal (cc == rc) or empty for this warp's rows
        const int jb = cc * 32;
        // the masked row goes to tensor memory as the A operand: 32 steps = 16 columns of two 16-bit values
        const uint32_t dst = tmem + lane_base + buf * 128 + cc * 16;
        uint32_t packed[16];
        if (!reached(cc)) {
#pragma unroll
          for (int q = 0; q < 16; ++q) packed[q] = 0u;
          tc::tmem_st16(dst, packed);
          continue;
        }
        const bool diag = cc == rc;
        if (fast[k]) {
          const float2 a2 = make_float2(arow[k], arow[k]);
#pragma unroll
          for (int q = 0; q < 32; q += 8) {
            const float4 b0 = *reinterpret_cast<const float4*>(sW + k * 32 + q);
            const float4 b1 = *reinterpret_cast<const float4*>(sW + k * 32 + q + 4);
            const float2 bp[4] = {make_float2(b0.x, b0.y), make_float2(b0.z, b0.w), make_float2(b1.x, b1.y), make_float2(b1.z, b1.w)};
            float f[8];
#pragma unroll
            for (int e = 0; e < 8; e += 2) {
              const float2 w = __fmul2_rn(__fmul2_rn(make_float2(vG[k][q + e], vG[k][q + e + 1]), bp[e / 2]), a2);
              f[e] = w.x, f[e + 1] = w.y;
            }
            Vec16<T> o;
            o.pack(f);
            packed[q / 2] = o.raw.x, packed[q / 2 + 1] = o.raw.y, packed[q / 2 + 2] = o.raw.z, packed[q / 2 + 3] = o.raw.w;
          }
          if (diag && fold_d) {  // the diagonal with its D, formed once per row and merged into the word that has been left zero there
            Vec16<T> d;
            const float one[8] = {fmaf(gdiag * bdiag, arow[k], Dfold), 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            d.pack(one);
            const uint32_t word = lane & 1 ? d.raw.x << 16 : d.raw.x & 0xffffu;
            const int at = lane >> 1;
#pragma unroll
            for (int q = 0; q < 16; ++q) packed[q] |= q == at ? word : 0u;
          }
        } else {
#pragma unroll
          for (int q = 0; q < 32; q += 8) {
            float f[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              f[e] = vG[k][q + e] * ex2_approx(re - col(jb + q + e));
              if (diag && (REV ? q + e < lane : q + e > lane)) f[e] = 0.f;  // after the product: G may be Inf there
              if (diag && fold_d && q + e == lane) f[e] = fmaf(gdiag, ex2_approx(re - col(jb + q + e)), Dfold);
            }
            Vec16<T> o;
            o.pack(f);
            packed[q / 2] = o.raw.x, packed[q / 2 + 1] = o.raw.y, packed[q / 2 + 2] = o.raw.z, packed[q / 2 + 3] = o.raw.w;
          }
        }
        tc::tmem_st16(dst, packed);
      }
      tc::tmem_wait_st();
      if constexpr (XSKIP) {  // this row of x (for D x in the epilogue one iteration later)
#pragma unroll
        for (int q = 0; q < kXR; ++q) xr[q] = *reinterpret_cast<const uint4*>(swz(sX + buf * M::X_BYTES, i_chunk, wg * kEU + q));
      }
      if (ragged && (warp == 13 || warp == 14)) {  // x rows of the next sequence, by two of the warps that have had the least mask work
#pragma unroll 1
        for (int u = k_live * 8 + tid - 13 * 32; u < KJ * 8; u += 64) *reinterpret_cast<uint4*>(sX + buf * M::X_BYTES + (size_t)u * 16) = make_uint4(0, 0, 0, 0);
        tc::fence_async_smem();
      }
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(mb_mask(buf));
    }
    // ---- the previous head's result, while the tensor cores work on this one ---------------------------------
    if (hi > 0) {
      const int ob = buf ^ 1, hp = hi - 1;
      // its MMAs, its gate rows, and the staging tile: y of two heads ago has left it (a barrier that has completed no phase passes
      // parity 1).  Mostly complete by now: the probes overlap.
      const uint32_t par = (hp >> 1) & 1, zb = has_z ? mb_z(ob) : mb_mma(ob), yb = ragged ? mb_mma(ob) : mb_out(ob), yp = ragged ? par : par ^ 1;
      const uint32_t t0 = tc::mbar_test(mb_mma(ob), par), t1 = tc::mbar_test(zb, par), t2 = tc::mbar_test(yb, yp);
      bool there = (t0 & t1 & t2) != 0;
      if (!there) there = tc::mbar_wait(mb_mma(ob), par) && tc::mbar_wait(zb, par) && tc::mbar_wait(yb, yp);
      if (!__all_sync(0xffffffffu, there)) {
        fail = 1;
        break;
      }
      tc::fence_after_sync();
      epilogue(h - 1, ob, ct_prev, xr_prev);
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(mb_epi(ob));
    }
    ct_prev = ct;
#pragma unroll
    for (int q = 0; q < kXR; ++q) xr_prev[q] = xr[q];
  }
  if (ragged) {
    for (int hi = max(nh - 2, 0); hi < nh && !fail; ++hi) {
      if (wait(mb_epi(hi & 1), hi >> 1)) store_rows(h0 + hi, hi & 1);
      else fail = 1;
    }
  }
  if (fail && lane == 0 && a.status) *(volatile int32_t*)a.status = 2;
}

template <typename T, bool XSKIP, bool REV, bool PACKED>
__global__ void __launch_bounds__(kScanThreads, 1)
    ssd_scan_kernel(const ssm_ssd_args a, const __grid_constant__ ScanMaps maps, int nchunks, int hpc, int nparts) {
  extern __shared__ unsigned char smdyn[];
  unsigned char* smraw = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smdyn) + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t mbar[14];
  __shared__ uint32_t tmem_slot;
  const int warp = threadIdx.x >> 5;
  const bool long_block = (int)blockIdx.x < (int)(gridDim.x >> 1);
  if constexpr (PACKED) {  // no rows: the sequence ends before them, or the table has room to spare
    const int c = (int)blockIdx.x % (int)(gridDim.x >> 1) / nparts % nchunks;
    if (chunk_limit(a, c) - chunk_begin(a, c) <= (long_block ? kBlk : 0)) return;
  }
  if (warp == 0) tc::tmem_alloc(tc::smem_u32(&tmem_slot), 512);
  if (threadIdx.x == 0) {
    for (int i = 0; i < 14; ++i) tc::mbar_init(tc::smem_u32(&mbar[i]), i >= 6 && i < 10 ? kScanCompute / 32 : 1);
  }
  __syncthreads();  // barriers and the TMEM address are set up before anyone arms or polls them
  // the heavier blocks (rows 128..255; REV: rows 0..127) are scheduled first
  if (long_block) ssd_scan_body<T, 1, XSKIP, REV, PACKED>(a, maps, nchunks, hpc, nparts, smraw, mbar, &tmem_slot);
  else ssd_scan_body<T, 0, XSKIP, REV, PACKED>(a, maps, nchunks, hpc, nparts, smraw, mbar, &tmem_slot);
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem_slot, 512);
}

// One CTA: sequences are taken kTableThreads at a time, a thread counting the chunks of one, a warp writing them out.
constexpr int kTableThreads = 1024;
__global__ void __launch_bounds__(kTableThreads) seq_table_kernel(const void* __restrict__ cu, int wide, int num_seqs, int len, int num_chunks, int* __restrict__ table) {
  __shared__ int from[kTableThreads], to[kTableThreads], at[kTableThreads], warp_sum[32];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  auto bound = [&](int i) {
    const int64_t v = wide ? __ldg(reinterpret_cast<const long long*>(cu) + i) : (int64_t)__ldg(reinterpret_cast<const int*>(cu) + i);
    return (int)min(max(v, (int64_t)0), (int64_t)len);
  };
  int* first = table + 2 * num_chunks;
  int base = 0;  // chunks of the sequences so far
  for (int s0 = 0; s0 < num_seqs; s0 += kTableThreads) {
    const int s = s0 + tid, b = s < num_seqs ? bound(s) : 0, e = s < num_seqs ? bound(s + 1) : 0;
    const int n = e > b ? (e - b + kQ - 1) / kQ : 0;
    int sum = n;  // inclusive prefix over the warp, then over the warps
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, sum, off);
      if (lane >= off) sum += v;
    }
    if (lane == 31) warp_sum[warp] = sum;
    __syncthreads();
    int before = 0, total = 0;
    for (int w = 0; w < 32; ++w) {
      if (w < warp) before += warp_sum[w];
      total += warp_sum[w];
    }
    from[tid] = b, to[tid] = e, at[tid] = min(base + before + sum - n, num_chunks);
    if (s < num_seqs) first[s] = at[tid];
    __syncthreads();
    for (int q = warp; q < kTableThreads && s0 + q < num_seqs; q += 32) {
      for (int c = lane; from[q] + c * kQ < to[q] && at[q] + c < num_chunks; c += 32) table[2 * (at[q] + c)] = from[q] + c * kQ, table[2 * (at[q] + c) + 1] = to[q];
    }
    base = min(base + total, num_chunks);
    __syncthreads();
  }
  if (tid == 0) first[num_seqs] = base;
  for (int c = base + tid; c < num_chunks; c += kTableThreads) table[2 * c] = table[2 * c + 1] = len;
}

template <typename T, int HPC, int NST, bool REV, bool PACKED>
static int ssd_state_launch(const ssm_ssd_args& a, int nchunks, cudaStream_t st) {
  StateMaps maps;
  using M = StateSmem<HPC, NST>;
  if (int rc = encode_rows_map(&maps.b, a.Bm, a.batch, a.len, a.groups, kN, M::kStep, a.io_dtype)) return rc;
  if (int rc = encode_rows_map(&maps.x, a.X, a.batch, a.len, a.heads, kP, M::kStep, a.io_dtype)) return rc;
  cudaFuncSetAttribute(ssd_state_kernel<T, HPC, NST, REV, PACKED>, cudaFuncAttributeMaxDynamicSharedMemorySize, M::ALLOC);
  ssd_state_kernel<T, HPC, NST, REV, PACKED><<<dim3(a.heads / HPC, a.num_seqs ? a.num_seqs : a.batch), kStateThreads, M::ALLOC, st>>>(a, maps, nchunks);
  return launch_status("ssd_state_kernel");
}

// ---------------------------------------------------------------------------------------------
// incoming state of sequence shard `rank` from every rank's (final state from a zero start | total log-decay):
//   S_in = sum_{q < rank} exp(sum_{q < m < rank} logP_m) S_q  (+ exp(sum_{m < rank} logP_m) initial)
// `gathered`: world x per_rank floats, each rank's block = batch_heads * elems states then batch_heads log-decays.
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) ssd_fold_shards_kernel(const float* __restrict__ gathered, int rank, int64_t per_rank, int batch_heads, int elems,
                                                              const float* __restrict__ initial, float* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= (int64_t)batch_heads * elems) return;
  const int bh = (int)(i / elems);
  float s = initial ? __ldg(initial + i) : 0.f;
  for (int q = 0; q < rank; ++q) {
    const float* blk = gathered + (int64_t)q * per_rank;
    s = fmaf(__expf(__ldg(blk + (int64_t)batch_heads * elems + bh)), s, __ldg(blk + i));
  }
  out[i] = s;
}

// Self-test of the bounded waits: one warp waits on an mbarrier that nothing ever arms, with a limit of `probes` probes
// (about a microsecond each).  The wait runs out, the kernel records status 3 and returns normally: the path every
// kernel above takes if one of its copies or MMAs never completes, exercised without a fault.
__global__ void __launch_bounds__(32) ssd_wait_selftest_kernel(int32_t* status, int probes) {
  __shared__ __align__(8) uint64_t mbar;
  if (threadIdx.x == 0) tc::mbar_init(tc::smem_u32(&mbar), 1);
  __syncwarp();
  const bool ok = tc::mbar_wait(tc::smem_u32(&mbar), 0, probes);
  if (!ok && threadIdx.x == 0 && status) *(volatile int32_t*)status = 3;
}

template <typename T, bool REV, bool PACKED>
static int ssd_state_dispatch(const ssm_ssd_args& a, int hpc, int nchunks, cudaStream_t st) {
  // as many stages as fit: the ring's round trip (a copy's 2300 cycles, the waits and fences of three roles) is what bounds the walk.
  // 96 walks of 4001 steps: 39 us with four stages and eight warps per stage, 38 with four per stage, 32 with eight stages
  if (hpc == 1) return ssd_state_launch<T, 1, 8, REV, PACKED>(a, nchunks, st);
  if (PACKED || hpc == 2) return ssd_state_launch<T, 2, 6, REV, PACKED>(a, nchunks, st);  // packed sequences: at most two
  if constexpr (!PACKED) {
    if (hpc == 3) return ssd_state_launch<T, 3, 5, REV, false>(a, nchunks, st);
    return ssd_state_launch<T, 4, 4, REV, false>(a, nchunks, st);
  }
}

template <typename T, bool XSKIP, bool REV, bool PACKED>
static int ssd_scan_launch(const ssm_ssd_args& a, const ScanMaps& maps, unsigned ctas, int nchunks, int hpc, int nparts, cudaStream_t st) {
  const size_t smem = ScanSmem<T>::ALLOC;
  cudaFuncSetAttribute(ssd_scan_kernel<T, XSKIP, REV, PACKED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  ssd_scan_kernel<T, XSKIP, REV, PACKED><<<ctas, kScanThreads, smem, st>>>(a, maps, nchunks, hpc, nparts);
  return launch_status("ssd_scan_kernel");
}

// Heads per scan CTA: a divisor of the heads of one B / C group, so that a CTA's heads share their G.  One CTA runs per SM; the
// long row blocks go first, then the short ones, each to the first SM that is free.  A long block costs 3 + d and a short one
// 1.9 + 0.82 d head times (C / B tiles, G, pipeline fill; fitted to all divisors of 13 dense shapes, rms 2.3 %).  Taken is the d with the
// earliest end: within 3 % of the best divisor in those shapes, from 1 x 178 steps of 20 heads (8.2 us) over 3 x 777 of 40 in two groups (22.3;
// 25.6 with the next one) to 8 x 8192 of 48 (343), and in seven packed ones from 64 sequences in 512 steps of 8 heads (13.8; 19.0 with half as
// many) to 24 in 16384 of 48 (105); of those 64 sequences in 16384 are 3 % off.
static int scan_heads_per_cta(int hpg, int64_t longs, int64_t shorts) {
  const int64_t sms = sm_count();
  double best = 1e300;
  int heads = 1;
  for (int d = 1; d <= hpg && d <= 32; ++d) {
    if (hpg % d) continue;
    const double lng = 3.0 + d, shrt = 1.9 + 0.82 * d;
    const int64_t n = shorts * (hpg / d), q = longs * (hpg / d) / sms, r = longs * (hpg / d) % sms;  // r SMs run q + 1 long blocks, the others q
    // how many short blocks can have ended by t
    auto room = [&](double t) {
      auto fit = [&](double from) { return t < from ? (int64_t)0 : (int64_t)((t - from) / shrt + 1e-9); };
      return r * fit((q + 1) * lng) + (sms - r) * fit(q * lng);
    };
    for (int64_t more = 0; more < (r ? 2 : 1); ++more) {  // the last short block follows q or q + 1 long ones
      int64_t lo = 0, hi = n + 1;                        // the fewest short blocks on one SM that make room for all of them
      while (lo < hi) {
        const int64_t mid = (lo + hi) / 2;
        if (room((q + more) * lng + mid * shrt) >= n) hi = mid;
        else lo = mid + 1;
      }
      double end = (q + more) * lng + lo * shrt;
      if (r && end < (q + 1) * lng) end = (q + 1) * lng;
      if (end < best) best = end, heads = d;
    }
  }
  return heads;
}

template <typename T>
static int ssd_launch(const ssm_ssd_args& a, cudaStream_t st) {
  const int nchunks = a.num_seqs ? a.num_chunks : (a.len + kQ - 1) / kQ;
  const int walks = a.num_seqs ? a.num_seqs : a.batch;  // sequences that the state kernel walks
  const int hpg = a.heads / a.groups;
  int64_t shorts = (int64_t)a.batch * nchunks, longs = shorts;
  if (a.num_seqs) {  // as many as sequences have that are cut at random: where they are cut is not known here
    const double mean = (double)a.len / a.num_seqs, chunks = a.num_seqs / (1.0 - std::exp(-kQ / mean));
    shorts = std::min<int64_t>(nchunks, std::llround(chunks)), longs = std::min<int64_t>(shorts, std::llround(chunks * std::exp(-kBlk / mean)));
  }
  const int hpc = scan_heads_per_cta(hpg, longs * a.groups, shorts * a.groups);
  const int nparts = a.heads / hpc;
  if (a.phase != 2 && !a.reverse) {
    ssd_cumsum_kernel<T><<<dim3((a.heads + kCumHeads - 1) / kCumHeads, nchunks, a.batch), kQ, 0, st>>>(a, nchunks);
    if (int rc = launch_status("ssd_cumsum_kernel")) return rc;
  }
  if (a.phase != 2) {
    // heads per CTA of the sequential state kernel: enough to bring the grid down to about one CTA per SM (its CTAs all run
    // for the whole sequence, so a second, partial wave would double the time), at most 4, and a divisor of the heads of one
    // B / C group.  Packed sequences differ in length, so their walks spread over the SMs by themselves as long as there are
    // many; two heads share a B tile, four make the longest walk longer.  us with one / two / three / four heads, 48 heads unless
    // stated: 24 sequences in 16384 steps 77 / 57 / 57 / 72, 2 in 16384 72 / 86 / 128 / 269 (one is taken), 64 in 16384 137 / 98 / 92 / 101,
    // 200 in 16384 353 / 244 / 214 / 228, 64 in 65536 225 / 165 / 153 / 200, 8 in 4096 with 24 heads 18.5 / 22.5 / 31 / 50, 32 short ones and one
    // of 14336 steps 148 / 151 / 203 / 405.
    const int most = a.num_seqs ? 2 : 4;
    int shpc = (int)(((int64_t)walks * a.heads + sm_count() - 1) / sm_count());
    shpc = shpc < 1 ? 1 : (shpc > most ? most : shpc);
    while (hpg % shpc != 0) --shpc;
    const int rc = a.reverse    ? ssd_state_dispatch<T, true, false>(a, shpc, nchunks, st)
                   : a.num_seqs ? ssd_state_dispatch<T, false, true>(a, shpc, nchunks, st)
                                : ssd_state_dispatch<T, false, false>(a, shpc, nchunks, st);
    if (rc) return rc;
  } else if (a.initial_states) {
    const int64_t units = (int64_t)a.batch * a.heads * (kP * kN / 8);
    ssd_fold_init_kernel<T><<<dim3((unsigned)((units + 255) / 256), (nchunks + 1 + kFoldChunks - 1) / kFoldChunks), 256, 0, st>>>(a, nchunks);
    if (int rc = launch_status("ssd_fold_init_kernel")) return rc;
  } else if (a.final_states) {  // nothing arrives: the final state is the one phase 1 left in the scratch
    const cudaError_t e = cudaMemcpyAsync(a.final_states, a.ws_state, sizeof(float) * (size_t)a.batch * a.heads * kP * kN, cudaMemcpyDeviceToDevice, st);
    if (e != cudaSuccess) return ::ssmb::fail((int)e, "ssd_scan: copying the final state failed");
  }
  if (a.phase != 1) {
    ScanMaps maps;
    if (int rc = encode_rows_map(&maps.x0, a.X, a.batch, a.len, a.heads, kP, kBlk, a.io_dtype)) return rc;
    if (int rc = encode_rows_map(&maps.x1, a.X, a.batch, a.len, a.heads, kP, kQ, a.io_dtype)) return rc;
    if (int rc = encode_rows_map(&maps.z, a.z ? a.z : a.Y, a.batch, a.len, a.heads, kP, kBlk, a.io_dtype)) return rc;
    if (int rc = encode_rows_map(&maps.y, a.Y, a.batch, a.len, a.heads, kP, kBlk, a.io_dtype)) return rc;
    if (int rc = encode_rows_map(&maps.c, a.Cm, a.batch, a.len, a.groups, kN, kBlk, a.io_dtype)) return rc;
    if (int rc = encode_rows_map(&maps.bm, a.Bm, a.batch, a.len, a.groups, kN, kBlk, a.io_dtype)) return rc;
    const unsigned ctas = 2u * nparts * a.batch * nchunks;
    if (a.reverse) return ssd_scan_launch<T, false, true, false>(a, maps, ctas, nchunks, hpc, nparts, st);
    const bool xskip = a.D && (a.d_has_p || a.row_dots);
    if (a.num_seqs)
      return xskip ? ssd_scan_launch<T, true, false, true>(a, maps, ctas, nchunks, hpc, nparts, st)
                   : ssd_scan_launch<T, false, false, true>(a, maps, ctas, nchunks, hpc, nparts, st);
    return xskip ? ssd_scan_launch<T, true, false, false>(a, maps, ctas, nchunks, hpc, nparts, st)
                 : ssd_scan_launch<T, false, false, false>(a, maps, ctas, nchunks, hpc, nparts, st);
  }
  return SSM_OK;
}

}  // namespace ssmb

using namespace ssmb;

extern "C" int ssm_ssd_supported(int32_t headdim, int32_t nstate, int32_t chunk_size, int32_t io_dtype) {
  return headdim == kP && nstate == kN && chunk_size == kQ && (io_dtype == SSM_BF16 || io_dtype == SSM_F16);
}

extern "C" int64_t ssm_ssd_state_scratch_bytes(int32_t batch, int32_t len, int32_t heads) {
  const int64_t nchunks = (len + kQ - 1) / kQ;
  return ((ssd_summary_floats_padded(batch, heads) + (int64_t)batch * heads * nchunks) * 4 + 255) / 256 * 256;
}

extern "C" int64_t ssm_ssd_scratch_bytes(int32_t batch, int32_t len, int32_t heads) {
  const int64_t nchunks = (len + kQ - 1) / kQ;
  const int64_t vec = (int64_t)batch * heads * nchunks * kQ * 4;      // delta, cum (each)
  const int64_t fin = ssm_ssd_state_scratch_bytes(batch, len, heads);  // shard-local final state, total log-decay, per-chunk decay prefixes
  const int64_t st = (int64_t)batch * nchunks * heads * kP * kN * 2;  // state before every chunk, operand dtype
  return 2 * vec + fin + st;
}

extern "C" int64_t ssm_ssd_packed_scratch_bytes(int32_t num_seqs, int32_t num_chunks, int32_t heads, int64_t* state_bytes) {
  const int64_t fin = (ssd_summary_floats_padded(num_seqs, heads) * 4 + 255) / 256 * 256;
  if (state_bytes) *state_bytes = fin;
  return 2 * (int64_t)heads * num_chunks * kQ * 4 + fin + (int64_t)num_chunks * heads * kP * kN * 2;
}

extern "C" int64_t ssm_ssd_shard_summary_floats(int32_t batch, int32_t heads) { return (int64_t)batch * heads * (kP * kN + 1); }

extern "C" int ssm_ssd_fold_shards(const float* gathered, int32_t world, int32_t rank, int32_t batch, int32_t heads, const float* initial_states,
                                   float* incoming, ssm_stream_t stream) {
  SSM_REQUIRE(gathered && incoming, SSM_ERR_NULL, "ssd_fold_shards: missing tensor");
  SSM_REQUIRE(world >= 1 && rank >= 0 && rank < world && batch >= 0 && heads >= 1, SSM_ERR_SHAPE, "ssd_fold_shards: bad shape");
  const int64_t total = (int64_t)batch * heads * kP * kN;
  if (total == 0) return SSM_OK;
  ssd_fold_shards_kernel<<<(unsigned)((total + 255) / 256), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      gathered, rank, ssm_ssd_shard_summary_floats(batch, heads), batch * heads, kP * kN, initial_states, incoming);
  return launch_status("ssd_fold_shards_kernel");
}

extern "C" int ssmb_seq_table(const void* cu, int32_t wide, int32_t num_seqs, int32_t len, int32_t num_chunks, int32_t* table, void* stream) {
  SSM_REQUIRE(cu && table, SSM_ERR_NULL, "seq_table: missing tensor");
  SSM_REQUIRE(num_seqs >= 1 && len >= 0 && num_chunks >= 0, SSM_ERR_SHAPE, "seq_table: bad shape");
  seq_table_kernel<<<1, kTableThreads, 0, reinterpret_cast<cudaStream_t>(stream)>>>(cu, wide, num_seqs, len, num_chunks, table);
  return launch_status("seq_table_kernel");
}

extern "C" int ssm_ssd_wait_selftest(int32_t* status, int32_t probes, ssm_stream_t stream) {
  SSM_REQUIRE(status != nullptr, SSM_ERR_NULL, "ssd_wait_selftest: status is NULL");
  SSM_REQUIRE(probes >= 1 && probes <= 100000, SSM_ERR_SHAPE, "ssd_wait_selftest: probes must be in [1, 100000]");
  ssd_wait_selftest_kernel<<<1, 32, 0, reinterpret_cast<cudaStream_t>(stream)>>>(status, probes);
  return launch_status("ssd_wait_selftest_kernel");
}

extern "C" int ssm_ssd_fwd(const ssm_ssd_args* a, ssm_stream_t stream) {
  SSM_REQUIRE(a != nullptr, SSM_ERR_NULL, "ssd_scan: args is NULL");
  SSM_REQUIRE(a->batch >= 0 && a->len >= 0 && a->heads >= 1 && a->groups >= 1, SSM_ERR_SHAPE, "ssd_scan: bad shape");
  SSM_REQUIRE(a->heads % a->groups == 0, SSM_ERR_SHAPE, "Group dimension must divide H.");
  SSM_REQUIRE(ssm_ssd_supported(a->headdim, a->nstate, a->chunk_size, a->io_dtype), SSM_ERR_UNSUPPORTED,
              "ssd_scan: the tensor-core path is built for headdim 64, d_state 128, chunk 256, bf16 / fp16");
  if (a->batch == 0 || a->len == 0) return SSM_OK;
  SSM_REQUIRE(a->phase >= 0 && a->phase <= 2, SSM_ERR_SHAPE, "ssd_scan: phase must be 0, 1 or 2");
  SSM_REQUIRE(!a->reverse || (a->phase == 0 && !a->D && !a->num_seqs), SSM_ERR_UNSUPPORTED, "ssd_scan: the adjoint pass has no skip term, shards or packed sequences");
  SSM_REQUIRE(a->X && a->dt && a->A && a->Bm && a->Cm && (a->Y || a->phase == 1), SSM_ERR_NULL, "ssd_scan: missing tensor");
  SSM_REQUIRE(a->ws_dt && a->ws_cum && a->ws_state && a->ws_state_in, SSM_ERR_NULL, "ssd_scan: missing scratch");
  SSM_REQUIRE(aligned_to(a->X, 16) && aligned_to(a->Bm, 16) && aligned_to(a->Cm, 16) && (!a->Y || aligned_to(a->Y, 16)) && aligned_to(a->ws_state_in, 16) &&
                  (!a->z || aligned_to(a->z, 16)),
              SSM_ERR_ALIGN, "ssd_scan: tensors must be 16-byte aligned");
  if (a->num_seqs) {
    SSM_REQUIRE(a->num_seqs > 0 && a->num_seqs <= 65535 && a->num_chunks > 0 && a->seq_table && a->batch == 1, SSM_ERR_SHAPE,
                "ssd_scan: packed sequences need a batch of one and a table");
    SSM_REQUIRE(a->phase != 2 && !a->initial_states && !a->row_dots, SSM_ERR_UNSUPPORTED, "ssd_scan: not built for packed sequences");
  }
  const int64_t nchunks = a->num_seqs ? a->num_chunks : (a->len + kQ - 1) / kQ;
  SSM_REQUIRE((a->num_seqs == 0) == (a->seq_table == nullptr), SSM_ERR_NULL, "ssd_scan: num_seqs without a table");
  SSM_REQUIRE((int64_t)a->batch * nchunks <= 65535 && a->heads <= 65535 && (int64_t)a->batch * nchunks * a->heads * 2 < (1ll << 31), SSM_ERR_TOO_LARGE,
              "ssd_scan: grid too large");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (a->io_dtype == SSM_BF16) return ssd_launch<__nv_bfloat16>(*a, st);
  return ssd_launch<__half>(*a, st);
}
