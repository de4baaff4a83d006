/*
 * ssm_b200 — C ABI of the B200 (sm_100a) backend for the five state-space operators
 * of the b-vitamins/ssm package.
 *
 * Every entry point takes a plain argument struct (raw device pointers, sizes, element
 * strides, dtype codes) plus a CUDA stream handle, enqueues its kernels on that stream and
 * returns without synchronising.  The library never allocates: outputs and scratch are
 * passed in by the caller.  Return value: 0 on success; a negative SSM_ERR_* code when an
 * argument is rejected (nothing was launched); a positive value is a cudaError_t from the
 * launch.  ssm_b200_last_error() returns a thread-local description of the last failure.
 *
 * The functions replace, one for one, the compiled operators that the upstream package
 * binds in src/ssm/ops/cuda/bindings.cpp:96-152 (the citation beside each declaration
 * names the host function there whose device work it takes over).  Layouts follow the
 * upstream Python specification src/ssm/ops/python/reference.py.
 */
#ifndef SSM_B200_H_
#define SSM_B200_H_

#include <stdint.h>

#ifdef __cplusplus
extern "C" {
#endif

/* Raised with every change of a struct's layout, of an entry point's signature or of the set of entry points.
 * 4: entry points and fields of the earlier SSD backward removed; log(-A) in the state step; packed sequences, decode steps. */
#define SSM_B200_ABI_VERSION 4

/* element types of activation tensors.  SSM_F64 selects the double-precision variants of the five operators (forward and
 * backward; written for gradient checking as in upstream's tests/ops/test_backend_gradients.py:1172-1612, not for speed): with
 * io_dtype == SSM_F64 EVERY floating-point tensor of the call -- activations, A, B, C, D, biases, weights, states, gradients --
 * is double, whatever C type the argument struct gives its pointer; bc_dtype, par_dtype, res_dtype, resout_dtype and last_dtype
 * are ignored; d_state <= 256; the scan backward takes batch * dim * len * nstate doubles of scratch through fwd.checkpoints (no
 * forward checkpoints are needed); the chunk-scan history is double; the norm backward ACCUMULATES into dweight / dbias (the
 * caller zero-fills them) and needs no `partial`.  The decode-time conv update, the SSD entry points and the allocation-free norm
 * backward have no fp64 variant. */
enum { SSM_F32 = 0, SSM_BF16 = 1, SSM_F16 = 2, SSM_F64 = 3 };

enum {
  SSM_OK = 0,
  SSM_ERR_NULL = -1,        /* a required pointer is NULL */
  SSM_ERR_SHAPE = -2,       /* a size is negative/zero where it may not be, or sizes disagree */
  SSM_ERR_DTYPE = -3,       /* unknown dtype code */
  SSM_ERR_ALIGN = -4,       /* a pointer misses its natural alignment */
  SSM_ERR_UNSUPPORTED = -5, /* valid in the operator's contract but outside what is built */
  SSM_ERR_TOO_LARGE = -6,   /* exceeds a documented capacity */
  SSM_ERR_DEVICE = -7       /* device-side status word reported a bounded wait that ran out */
};

/* The stream is a cudaStream_t passed as an opaque pointer so that this header needs no CUDA include. */
typedef void* ssm_stream_t;

int ssm_b200_abi_version(void);
const char* ssm_b200_last_error(void);
/* kernels launched by this library since the process started, over all devices and threads */
int64_t ssm_b200_launch_count(void);

/* ---------------------------------------------------------------------------------------
 * Selective scan (Mamba-1), forward.   Replaces selective_scan_cuda
 * (src/ssm/ops/cuda/selective_scan.cu:1034-1161; spec reference.py:87-194).
 *
 *   dl_t = softplus?(delta_t + dt_bias);  h_t = exp(dl_t*A) .* h_{t-1} + dl_t*B_t*u_t
 *   y_t  = <C_t, h_t> + D*u_t;            out_t = y_t * silu(z_t)
 *
 * u, delta, z, out: (batch, dim, len) with contiguous time axis and the batch / channel strides
 * row_sb / row_sd, element type io_dtype.  A: (dim, nstate)
 * fp32.  Bm / Cm are addressed as  base[b*sb + g*sg + n*sn + t*st]  (element strides, type
 * bc_dtype) with g = d / (dim / bc_groups); this one form covers the (D,N), (B,D,N) and
 * grouped time-varying (B,G,N,L) layouts of reference.py:22-56.  D, dt_bias: (dim) fp32
 * or NULL.  initial_state: (batch, dim, nstate) fp32 or NULL (zeros).  last_state: optional
 * output (batch, dim, nstate) of type last_dtype.  checkpoints: optional output
 * (batch, dim, ceil(len / ssm_scan_checkpoint_interval()), nstate) fp32 holding the state
 * before every interval; the backward pass needs it.
 * ------------------------------------------------------------------------------------- */
typedef struct {
  int32_t batch, dim, len, nstate;
  int32_t io_dtype, bc_dtype, last_dtype, delta_softplus;
  const void* u;
  const void* delta;
  const void* z; /* nullable */
  const float* A;
  const void* Bm;
  const void* Cm;
  int32_t bc_groups, reserved0;
  int64_t b_sb, b_sg, b_sn, b_st;
  int64_t c_sb, c_sg, c_sn, c_st;
  const float* D;             /* nullable */
  const float* dt_bias;       /* nullable */
  const float* initial_state; /* nullable */
  void* out;
  void* last_state;   /* nullable */
  float* checkpoints; /* nullable */
  /* Element strides of the batch and channel axes of u, delta, z, out (and of dout, du, ddelta,
   * dz in the backward call); the time axis is contiguous.  Dense (B, D, L) is {dim*len, len};
   * a (D, B, L) buffer viewed as (B, D, L) is {len, batch*len}, which lets the projections
   * around the scan be plain 2-D GEMMs with no transposing copies. */
  int64_t row_sb, row_sd;
  /* Optional time-parallel execution for calls whose (batch x dim) rows alone cannot fill the GPU (e.g. batch 1): the sequence
   * is cut into split_segments pieces that are integrated in parallel and stitched by a short serial pass (the block-level
   * prefix over the (A, B u) recurrence).  split_scratch: 2 * batch * dim * split_segments * nstate floats.  NULL or
   * split_segments <= 1: one pass over the whole sequence.  ssm_scan_split_segments() suggests the count. */
  float* split_scratch;
  int32_t split_segments, reserved1;
} ssm_scan_fwd_args;

int ssm_scan_checkpoint_interval(void);
int ssm_scan_split_segments(int32_t batch, int32_t dim, int32_t len, int32_t nstate);
/* the same for the backward (its fwd.split_scratch / split_segments; d_state <= 32) */
int ssm_scan_bwd_split_segments(int32_t batch, int32_t dim, int32_t len, int32_t nstate);
int ssm_selective_scan_fwd(const ssm_scan_fwd_args* args, ssm_stream_t stream);

/* ---------------------------------------------------------------------------------------
 * Selective scan, backward.   Replaces selective_scan_backward_cuda
 * (src/ssm/ops/cuda/selective_scan.cu:1696-1875) and, because grad_last_state is
 * handled on the device, the Python fall-back in src/ssm/ops/__init__.py:365-436.
 *
 * fwd holds the forward call's arguments (out/last_state unused; checkpoints required).
 * dout: (batch, dim, len) io_dtype.  dlast_state: (batch, dim, nstate) fp32 or NULL.
 * du, ddelta, dz: io_dtype (dz NULL iff fwd.z is NULL).  dA (dim, nstate), dD, ddt_bias
 * (dim): fp32, ACCUMULATED into (caller zero-fills); dD / ddt_bias may be NULL.
 * dB / dC: fp32 buffers addressed with db_* / dc_* strides exactly like Bm / Cm,
 * accumulated into (caller zero-fills).
 * ------------------------------------------------------------------------------------- */
typedef struct {
  ssm_scan_fwd_args fwd;
  const void* dout;
  const float* dlast_state; /* nullable */
  void* du;
  void* ddelta;
  void* dz; /* nullable */
  float* dA;
  float* dB;
  float* dC;
  int64_t db_sb, db_sg, db_sn, db_st;
  int64_t dc_sb, dc_sg, dc_sn, dc_st;
  float* dD;       /* nullable */
  float* ddt_bias; /* nullable */
  float* dinitial_state; /* nullable: (batch, dim, nstate) fp32, written: gradient of fwd.initial_state (additive extension) */
} ssm_scan_bwd_args;

int ssm_selective_scan_bwd(const ssm_scan_bwd_args* args, ssm_stream_t stream);

/* ---------------------------------------------------------------------------------------
 * Single-token state step (decode).   Replaces selective_state_step_cuda
 * (src/ssm/ops/cuda/state_step.cu:310-434; spec reference.py:197-309).
 *
 * state: (batch, dim, nstate) fp32, updated in place.  x, z, out: (batch, dim) io_dtype.
 * Parameters are per channel when param_heads == 0: dt (batch, dim), A (dim, nstate),
 * D / dt_bias (dim).  With param_heads = H > 0 (Mamba-2 layout, channel d belongs to head
 * d / (dim / H)) they are per head: dt (batch, H), A (H), D / dt_bias (H).  Bm / Cm:
 * base[b*sb + g*sg + n*sn], type bc_dtype, g = d / (dim / bc_groups), which covers (D,N),
 * (B,D,N) and grouped (B,G,N).
 * ------------------------------------------------------------------------------------- */
typedef struct {
  int32_t batch, dim, nstate, io_dtype;
  int32_t bc_dtype, bc_groups, dt_softplus, param_heads;
  float* state;
  const void* x;
  const void* dt;
  const void* z; /* nullable */
  const float* A;
  const void* Bm;
  const void* Cm;
  int64_t b_sb, b_sg, b_sn;
  int64_t c_sb, c_sg, c_sn;
  const float* D;       /* nullable */
  const float* dt_bias; /* nullable */
  void* out;
  int32_t a_log, reserved0; /* a_log: A holds log(-A) (forward only) */
} ssm_step_args;

int ssm_selective_state_step(const ssm_step_args* args, ssm_stream_t stream);

/* Backward of the step (per-channel parameters only).  Replaces
 * selective_state_step_backward_cuda (src/ssm/ops/cuda/state_step.cu:436-693).
 * state is the state BEFORE the step.  dout (batch, dim) io_dtype; dnew_state
 * (batch, dim, nstate) fp32 or NULL.  dstate (batch, dim, nstate) fp32; dx, ddt, dz
 * io_dtype; dA, dD, ddt_bias, dB, dC fp32 accumulated into (caller zero-fills);
 * dB / dC use the Bm / Cm strides of fwd. */
typedef struct {
  ssm_step_args fwd;
  const void* dout;
  const float* dnew_state; /* nullable */
  float* dstate;
  void* dx;
  void* ddt;
  void* dz; /* nullable */
  float* dA;
  float* dB;
  float* dC;
  float* dD;       /* nullable */
  float* ddt_bias; /* nullable */
} ssm_step_bwd_args;

int ssm_selective_state_step_bwd(const ssm_step_bwd_args* args, ssm_stream_t stream);

/* ---------------------------------------------------------------------------------------
 * Element-wise chunked recurrence ("ssd_chunk_scan" upstream).   Replaces
 * ssd_chunk_scan_cuda (src/ssm/ops/cuda/ssd_chunk_scan.cu:637-860; spec reference.py:312-463).
 *
 * X, Y: (batch, len, heads, proj) io_dtype.  dt: (batch, len, heads) io_dtype.  Every
 * parameter p in {A, Bm, Cm, D, z, initial} is addressed  base[b*sb + t*st + h*sh + q*sq]
 * with zero strides for broadcast axes (A/D/initial fp32; Bm/Cm/z of type par_dtype).
 * seq_lens: (batch) int64 on the device or NULL; outputs beyond a row's length are zero.
 * final_state: optional output (batch, heads, proj) fp32 (additive; upstream returns none).
 * chunk_size splits the sequence into independently processed chunks (it has no numerical
 * effect beyond rounding).  scratch: fp32 workspace of ssm_chunk_scan_scratch_floats()
 * elements; when NULL the sequence is walked serially by one thread per (batch, head, proj).
 * ------------------------------------------------------------------------------------- */
typedef struct {
  const void* ptr;
  int64_t sb, st, sh, sq;
} ssm_bcast4;

typedef struct {
  int32_t batch, len, heads, proj;
  int32_t io_dtype, par_dtype, reserved0, typed_grads; /* typed_grads: backward only, see ssm_chunk_bwd_args */
  const void* X;
  const void* dt;
  ssm_bcast4 A, Bm, Cm, D, z, initial; /* D, z, initial: ptr may be NULL */
  const int64_t* seq_lens;             /* nullable */
  void* Y;
  float* final_state; /* nullable */
  float* scratch;     /* nullable */
  int32_t chunk_size, reserved2;
} ssm_chunk_args;

int64_t ssm_chunk_scan_scratch_floats(int32_t batch, int32_t len, int32_t heads, int32_t proj, int32_t chunk_size);
int ssm_chunk_scan_fwd(const ssm_chunk_args* args, ssm_stream_t stream);

/* Backward.  Replaces ssd_chunk_scan_backward_cuda (src/ssm/ops/cuda/ssd_chunk_scan.cu:341-635).
 * dY io_dtype.  dX (io_dtype), ddt fp32 (batch, len, heads), and fp32 gradient buffers
 * dA/dB/dC/dD/dz/dinitial addressed with the strides given here (broadcast axes = stride 0),
 * accumulated into (caller zero-fills).  history: scratch (batch, len, heads, proj) fp32.
 * fwd.typed_grads, bits 0 / 1 / 2: dB / dC / dz is instead a buffer of par_dtype elements with no broadcast axis (every
 * (b, t, h, q) a distinct element) that the call WRITES, every element of it, zeros beyond a row's length included: no zero-fill
 * by the caller, no fp32 copy to convert afterwards.
 * ssm_chunk_scan_bwd_fused(args) tells whether a call with these arguments (typed_grads bits 0 - 2, layouts, pointers of the
 * gradients of B, C, z) keeps its states in registers: it then needs no history, and bit 3 may be set.  Such a call reads
 * `scratch` and `fwd_scratch` in 16-byte pieces: set them before asking. */
typedef struct {
  ssm_chunk_args fwd;
  const void* dY;
  void* dX;
  void* ddt; /* fp32, accumulated into; with bit 3 of typed_grads io_dtype, written */
  ssm_bcast4 dA, dB, dC, dD, dz, dinitial; /* ptr as float*; NULL to skip where fwd's is NULL */
  float* history;
  float* scratch; /* nullable: ssm_chunk_scan_bwd_scratch_floats() floats; with it the chunks run in parallel, without it one thread
                     per (batch, head, proj) walks the whole sequence */
  float* fwd_scratch; /* nullable: the scratch that the forward call with the same arguments left behind */
} ssm_chunk_bwd_args;

int64_t ssm_chunk_scan_bwd_scratch_floats(int32_t batch, int32_t len, int32_t heads, int32_t proj, int32_t chunk_size);
int ssm_chunk_scan_bwd_fused(const ssm_chunk_bwd_args* args);
int ssm_chunk_scan_bwd(const ssm_chunk_bwd_args* args, ssm_stream_t stream);

/* ---------------------------------------------------------------------------------------
 * Depthwise causal conv1d.   Replaces dw_causal_conv_cuda / dw_causal_conv_backward_cuda
 * (src/ssm/ops/cuda/dw_causal_conv.cu:771-857, 859-965; spec reference.py:466-537).
 *
 * x, y: channels_first ? (batch, channels, len) : (batch, len, channels), io_dtype.
 * weight: (channels, width), tap j multiplies x[t - (width-1) + j].  bias (channels) or NULL; both param_dtype.
 * 1 <= width <= 8.  Optional halo: (batch, channels, width-1) fp32 inputs that precede
 * t = 0 (sequence-sharded prefill; NULL means zeros, the upstream behaviour).
 * Backward: dx io_dtype; dweight (channels, width), dbias (channels) fp32 accumulated into.
 * ------------------------------------------------------------------------------------- */
typedef struct {
  int32_t batch, channels, len, width;
  int32_t io_dtype, channels_first, silu;
  int32_t param_dtype; /* element type of weight and bias (0: fp32); their gradients are fp32 */
  const void* x;
  const void* weight;
  const void* bias;  /* nullable */
  const float* halo; /* nullable */
  void* y;
  /* channels_first only: element strides of the batch and channel axes of x, y (and dy, dx);
   * dense is {channels*len, len}.  Ignored for the channels-last layout. */
  int64_t row_sb, row_sc;
} ssm_conv_args;

int ssm_dw_causal_conv_fwd(const ssm_conv_args* args, ssm_stream_t stream);

typedef struct {
  ssm_conv_args fwd;
  const void* dy;
  void* dx;
  float* dweight;
  float* dbias; /* nullable */
} ssm_conv_bwd_args;

int ssm_dw_causal_conv_bwd(const ssm_conv_bwd_args* args, ssm_stream_t stream);

/* Decode-time form of the same convolution: push one token into the rolling window and take
 * the dot product.  Upstream does this with torch.roll in Python
 * (src/ssm/modules/mamba1.py:345-353).  conv_state: (batch, channels, width) fp32, shifted
 * left by one and x appended, in place.  x, out: (batch, channels) io_dtype;
 * out = silu?(bias + <conv_state, weight>). */
typedef struct {
  int32_t batch, channels, width, io_dtype;
  int32_t silu, param_dtype; /* param_dtype: element type of weight and bias (0: fp32) */
  float* conv_state;
  const void* x;
  const void* weight;
  const void* bias; /* nullable */
  void* out;
} ssm_conv_update_args;

int ssm_dw_causal_conv_update(const ssm_conv_update_args* args, ssm_stream_t stream);

/* ---------------------------------------------------------------------------------------
 * Residual add fused with LayerNorm / RMSNorm.   Replaces fused_layer_norm_cuda /
 * fused_layer_norm_backward_cuda (src/ssm/ops/cuda/layer_norm.cu:372-496, 498-676; spec
 * reference.py:540-609).
 *
 * x, y: (rows, hidden) io_dtype.  residual: res_dtype or NULL.  weight, bias: param_dtype.
 * prenorm: y = norm(x + residual)*w + b, else y = norm(x)*w + b + residual.
 * All arithmetic is fp32 (upstream's residual_in_fp32 only matters for fp64 inputs, which
 * are not built).  hidden <= 16384 (16-bit) / 8192 (fp32).  residual_out: optional
 * (rows, hidden) of resout_dtype receiving x + residual (additive extension).
 * Backward: dx io_dtype, dresidual res_dtype (NULL iff residual NULL); dweight, dbias
 * (hidden), dparam_dtype, written (not accumulated); partial: scratch fp32 of
 * ssm_norm_bwd_scratch_floats(rows, hidden) floats.
 * ------------------------------------------------------------------------------------- */
typedef struct {
  int64_t rows;
  int32_t hidden, io_dtype, res_dtype, resout_dtype;
  int32_t is_rms, prenorm;
  int32_t param_dtype; /* element type of weight and bias (0: fp32) */
  int32_t dparam_dtype; /* backward: element type of dweight and dbias as written (0: fp32) */
  float eps, reserved1;
  const void* x;
  const void* residual; /* nullable */
  const void* weight; /* param_dtype */
  const void* bias;   /* param_dtype, nullable */
  void* y;
  void* residual_out; /* nullable */
} ssm_norm_args;

int ssm_fused_add_norm_fwd(const ssm_norm_args* args, ssm_stream_t stream);

typedef struct {
  ssm_norm_args fwd;
  const void* dy;
  void* dx;
  void* dresidual; /* nullable */
  void* dweight; /* fwd.dparam_dtype */
  void* dbias;   /* fwd.dparam_dtype, nullable */
  float* partial;
  const void* dresidual_out; /* nullable: gradient arriving through residual_out, (rows, hidden) of fwd.resout_dtype; added to dx and dresidual */
} ssm_norm_bwd_args;

int64_t ssm_norm_bwd_scratch_floats(int64_t rows, int32_t hidden);
int ssm_fused_add_norm_bwd(const ssm_norm_bwd_args* args, ssm_stream_t stream);

/* Backward of the fused add + norm for callers that are not allowed to allocate device memory
 * (it has no counterpart in the upstream package).  Code that runs inside someone else's memory
 * plan -- an inference server that hands out one fixed arena at start-up, a plugin that must not
 * touch the CUDA allocator of its host process, a real-time loop that cannot risk the implicit
 * synchronisation of cudaMalloc / cudaFree -- cannot provide the `partial` scratch that
 * ssm_fused_add_norm_bwd needs.  This entry point computes the same result but keeps that
 * scratch in a fixed array inside the library's own device image: `args->partial` is ignored
 * and neither this call nor anything it launches allocates or frees memory.
 *
 * Limits and rules:
 *  - hidden <= 8192 (larger rows are rejected with SSM_ERR_TOO_LARGE); the array takes
 *    9.25 MiB on every GPU that loads the library, for the life of the process;
 *  - the first call on each device looks up the array's device address (with that device
 *    current) and remembers it; make that first call outside any stream capture.  The tensors
 *    must live on the current device (checked: SSM_ERR_DEVICE otherwise);
 *  - all calls on a device share the one array.  Nothing in it has to start at zero (every
 *    launch overwrites the part it later reads), but two calls whose kernels overlap on
 *    the GPU (different streams, no ordering) race on it: serialise them on one stream or
 *    with events;
 *  - weight / bias gradients are summed over at most 148 partial rows instead of up to 592, so
 *    they can differ from ssm_fused_add_norm_bwd in the last bits; dx / dresidual are identical. */
int ssm_fused_add_norm_bwd_noalloc(const ssm_norm_bwd_args* args, ssm_stream_t stream);

/* ---------------------------------------------------------------------------------------
 * State-space-dual scan with a d_state axis (Mamba-2), forward, on the tcgen05 tensor cores.
 * Upstream has no operator of this shape (its ssd_chunk_scan has no state axis,
 * src/ssm/ops/python/reference.py:312-463); the semantics are those of its selective_scan
 * (reference.py:87-194) on channel h*P+p with delta[b,h*P+p,t] = dt[b,t,h], A[h*P+p,:] = A[h]
 * and B, C shared per group, the final state being selective_scan's last state kept in fp32.
 *
 * X, z, Y: (batch, len, heads, headdim) io_dtype.  dt: (batch, len, heads) io_dtype.  A: (heads)
 * fp32.  Bm, Cm: (batch, len, groups, nstate) io_dtype.  D: (heads) or, with d_has_p,
 * (heads, headdim) fp32, nullable.  dt_bias: (heads) fp32, nullable.  initial_states /
 * final_states: (batch, heads, headdim, nstate) fp32, nullable.  Built for headdim 64,
 * nstate 128, chunk_size 256, bf16 / fp16 (ssm_ssd_supported()).  Scratch, in this order, is
 * carved by the caller from one buffer of ssm_ssd_scratch_bytes() bytes:
 *   ws_dt, ws_cum : (batch, heads, nchunks * 256) fp32 each; per chunk ws_cum[i] = log2(e) * sum_{k<=i} delta_k A
 *                   (running decay exponent, base 2) and ws_dt[i] = ws_cum[i] - log2(delta_i)
 *   ws_state      : (batch, heads, headdim, nstate) fp32 — the final state reached from the given (or zero)
 *                   initial state, kept for a later phase-2 call on the same scratch — followed by (batch, heads)
 *                   fp32, the total log-decay sum(delta A) of the call; the two together (ssm_ssd_shard_summary_floats()
 *                   floats) are what a sequence shard sends to the other ranks; then, from the next 256-byte boundary,
 *                   (batch, heads, nchunks) fp32 decay exponents from the start of the call to each chunk.  The whole
 *                   region takes ssm_ssd_state_scratch_bytes() bytes
 *   ws_state_in   : (batch, nchunks, heads, headdim * nstate) in io_dtype — the state before every chunk, in
 *                   the operand order of the scan kernel
 * status: optional device int, set non-zero when a bounded device-side wait ran out.
 * phase: 0 runs everything.  1 stops after the chunk states (it fills the scratch and
 * final_states from the given, normally absent, initial_states and writes no Y); 2 adds the
 * given initial_states on top of what phase 1 left in the scratch (by linearity), writes
 * the corrected final_states and produces Y.  A sequence shard uses 1, exchanges final
 * states with its neighbours, then 2.
 * reverse: the adjoint pass of the backward.  X, Bm and Cm hold dy, C and B; ws_dt and ws_cum are those of the forward call on
 * the same step sizes (nothing is recomputed), initial_states the gradient of the final state.  Y receives
 * dx_j = dt_j (G_j B_j) without the skip term, G_j the adjoint state of step j; ws_state_in, for every chunk, the adjoint that enters it from
 * the right (that of the next chunk's first step); final_states the adjoint state of step 0.
 * row_dots: (batch, len, heads) fp32, zero-filled by the caller.  When given, z is not a gate: Y is written ungated and
 * row_dots[b, t, h] receives sum_p y[p] z[p], with y taken before the D x term and before rounding to io_dtype (the
 * backward pass forms dy . y and d(dt x) . x this way).
 * ws_state_in_f32: optional (batch, nchunks, heads, headdim * nstate) fp32: ws_state_in before rounding, same element order.
 * ------------------------------------------------------------------------------------- */
typedef struct {
  int32_t batch, len, heads, headdim;
  int32_t nstate, groups, chunk_size, io_dtype;
  int32_t dt_softplus, d_has_p, phase, reverse;
  const void* X;
  const void* dt;
  const float* A;
  const void* Bm;
  const void* Cm;
  const float* D;              /* nullable */
  const void* z;               /* nullable */
  const float* dt_bias;        /* nullable */
  const float* initial_states; /* nullable */
  void* Y;
  float* final_states; /* nullable */
  float* ws_dt;
  float* ws_cum;
  float* ws_state;
  void* ws_state_in;
  int32_t* status; /* nullable */
  float* row_dots; /* nullable */
  float* ws_state_in_f32; /* nullable */
  /* Packed sequences: num_seqs > 0 sequences lie end to end along len of a batch of one, each scanned from a zero state with
   * chunks counted from its first step.  seq_table (device): num_chunks pairs {first step, end of the sequence}, sequence by
   * sequence, then num_seqs + 1 chunk offsets.  final_states, and the state and shard-summary part of the scratch, are per
   * sequence; scratch: ssm_ssd_packed_scratch_bytes().  phase 0 (states and Y) or 1 (states only), no initial_states. */
  const int32_t* seq_table; /* nullable */
  int32_t num_seqs, num_chunks;
} ssm_ssd_args;

int ssm_ssd_supported(int32_t headdim, int32_t nstate, int32_t chunk_size, int32_t io_dtype);

/* Self-test of the bounded device-side waits (no counterpart upstream).  Launches one warp that waits on a barrier nothing
 * arms, with a limit of `probes` probes of about a microsecond each (1 .. 100000); when the limit runs out the kernel
 * writes 3 to *status (device int) and returns normally -- the error path of ssm_ssd_fwd's kernels, without a fault. */
int ssm_ssd_wait_selftest(int32_t* status, int32_t probes, ssm_stream_t stream);
int64_t ssm_ssd_scratch_bytes(int32_t batch, int32_t len, int32_t heads);
int64_t ssm_ssd_state_scratch_bytes(int32_t batch, int32_t len, int32_t heads);
/* scratch of a packed call: ws_dt, ws_cum (num_chunks * 256 * heads floats each), ws_state, ws_state_in as above; the offset of
 * ws_state_in from ws_state is written to *state_bytes */
int64_t ssm_ssd_packed_scratch_bytes(int32_t num_seqs, int32_t num_chunks, int32_t heads, int64_t* state_bytes);
int ssm_ssd_fwd(const ssm_ssd_args* args, ssm_stream_t stream);

/* Sequence shards (no reference counterpart: the reference is single-device).  After phase 1 every rank all-gathers its
 * summary (ws_state: final state from a zero start, then total log-decay; ssm_ssd_shard_summary_floats() floats) into
 * `gathered` (world x that many floats).  ssm_ssd_fold_shards writes the incoming state (batch, heads, headdim, nstate)
 * fp32 of shard `rank`:  sum_{q<rank} exp(sum_{q<m<rank} logP_m) S_q  (+ the decayed `initial_states`, nullable),
 * which is the initial_states of the phase-2 call. */
int64_t ssm_ssd_shard_summary_floats(int32_t batch, int32_t heads);
int ssm_ssd_fold_shards(const float* gathered, int32_t world, int32_t rank, int32_t batch, int32_t heads, const float* initial_states,
                        float* incoming, ssm_stream_t stream);

/* ---------------------------------------------------------------------------------------
 * Backward of the state-space-dual scan in the dual form (no counterpart upstream, whose Mamba-2 scan has no d_state
 * axis), in this order:
 *   ssm_ssd_bwd_gate    dy = gY * silu(z) (needed only with a gate)
 *   ssm_ssd_fwd         again, without skip and gate: y, row_dots u = dy . y (z = dy), states before the chunks, also in fp32
 *   ssm_ssd_fwd         reverse = 1: dx without the skip term, row_dots qd = delta d(delta x) . x (z = X), adjoints, also in fp32
 *   ssm_ssd_bwd_bc      dB, dC (fp32, zero-filled by the caller) from dy, X, B, C, the exponents and both sets of states
 *   ssm_ssd_bwd_finish  dz = gY (y + D x) silu'(z);  dX = dx + D dy;  dD (heads) or (heads, headdim) += sum dy x (zero-filled
 *                       by the caller; NULL when D is NULL)
 *   ssm_ssd_bwd_steps   ddt in dt's type, and dA (heads), ddt_bias (heads) += (fp32, zero-filled by the caller), from u, qd and the
 *                       products <state, adjoint> at the chunk boundaries: the gradient of the decay exponent obeys
 *                       da_{t+1} = da_t + qd_t - u_t
 * --------------------------------------------------------------------------------------- */
typedef struct {
  int32_t batch, len, heads, headdim;
  int32_t io_dtype, d_has_p;
  const void* gY;      /* (batch, len, heads, headdim) */
  const void* z;       /* nullable */
  const void* X;       /* finish */
  const void* y_plain; /* finish, with z */
  const void* dx;      /* finish: output of the adjoint pass */
  const float* D;      /* nullable */
  void* dy;            /* gate: out; finish: in */
  void* dX;            /* finish: out */
  void* dz;            /* finish: out, with z */
  float* dD;           /* finish: accumulated, nullable */
} ssm_ssd_bwd_args;

int ssm_ssd_bwd_gate(const ssm_ssd_bwd_args* args, ssm_stream_t stream);
int ssm_ssd_bwd_finish(const ssm_ssd_bwd_args* args, ssm_stream_t stream);

typedef struct {
  int32_t batch, len, heads, groups;
  int32_t io_dtype, reserved0;
  const void* X;  /* (batch, len, heads, 64) */
  const void* dy; /* (batch, len, heads, 64) */
  const void* Bm; /* (batch, len, groups, 128) */
  const void* Cm;
  const float* ws_dt; /* exponents and states as the two runs of ssm_ssd_fwd left them */
  const float* ws_cum;
  const void* state_in;
  const void* adjoint_in;
  float* dB; /* (batch, len, groups, 128), accumulated */
  float* dC;
  int32_t* status; /* nullable */
} ssm_ssd_bc_args;
int ssm_ssd_bwd_bc(const ssm_ssd_bc_args* args, ssm_stream_t stream);

typedef struct {
  int32_t batch, len, heads, io_dtype;
  int32_t dt_softplus, reserved0;
  const void* dt;       /* (batch, len, heads) io_dtype */
  const float* dt_bias; /* nullable */
  const float* A;
  const float* u;  /* (batch, len, heads) */
  const float* qd;
  const float* ws_cum;
  const float* state_f32;   /* (batch, nchunks, heads, 64 * 128): states before the chunks */
  const float* adjoint_f32; /* likewise: adjoints entering them from the right */
  const float* start0;      /* (batch, heads): <d initial state, initial state>; nullable */
  void* ddt;                /* (batch, len, heads) io_dtype, written */
  float* dA;
  float* ddt_bias; /* nullable */
} ssm_ssd_steps_args;
int ssm_ssd_bwd_steps(const ssm_ssd_steps_args* args, ssm_stream_t stream);

/* ---------------------------------------------------------------------------------------
 * One decode token through a whole mixer in one launch (no counterpart upstream, whose step methods are sequences of
 * operator calls: src/ssm/modules/mamba1.py:324-385).  For up to 16 sequences, bf16 / fp16 activations and projection
 * weights (io_dtype), conv width 4; ssm_mamba*_decode_supported() says whether a shape is built.  hidden (batch, d_model).
 * Weights as in ssm_b200/mixer.py, row-major (out, in): io_dtype; dt_bias, A, D fp32.  a_log: A holds log(-A).  States fp32,
 * updated in place.  scratch: ssm_mamba*_decode_scratch_bytes() bytes.
 * Mamba-1: out is the mixer's output (batch, d_model), or, with norm_w, RMSNorm(residual + mixer output) * norm_w with the
 * sum written to residual_out (residual nullable).  The state is (batch, d_inner, 16).
 * Mamba-2: out is the mixer's output; norm_w (d_inner) is the gated norm in front of the out projection.  The state is
 * (batch, heads, 64, 128).
 * ------------------------------------------------------------------------------------- */
typedef struct {
  int32_t batch, d_model, d_inner, nstate;
  int32_t dt_rank, width, io_dtype, a_log;
  int32_t res_dtype, resout_dtype;
  float eps;
  int32_t reserved0;
  const void* hidden;
  const void* in_x;
  const void* in_z;
  const void* conv_w;
  const void* conv_b; /* nullable */
  const void* x_proj;
  const void* dt_proj;
  const float* dt_bias;
  const float* A;
  const float* D;
  const void* out_proj;
  const void* norm_w;   /* nullable */
  const void* residual; /* nullable */
  float* conv_state;
  float* ssm_state;
  void* out;
  void* residual_out; /* with norm_w */
  void* scratch;
} ssm_mamba1_decode_args;

int ssm_mamba1_decode_supported(int32_t batch, int32_t d_model, int32_t d_inner, int32_t nstate, int32_t dt_rank, int32_t width, int32_t io_dtype);
int64_t ssm_mamba1_decode_scratch_bytes(int32_t batch, int32_t d_model, int32_t d_inner, int32_t nstate, int32_t dt_rank);
int ssm_mamba1_decode(const ssm_mamba1_decode_args* args, ssm_stream_t stream);

typedef struct {
  int32_t batch, d_model, heads, headdim;
  int32_t nstate, groups, width, io_dtype;
  int32_t a_log, reserved0;
  float eps;
  int32_t reserved1;
  const void* hidden;
  const void* in_z;
  const void* in_x;
  const void* in_B;
  const void* in_C;
  const void* in_dt;
  const void* conv_x_w;
  const void* conv_x_b; /* nullable, as the other two biases */
  const void* conv_B_w;
  const void* conv_B_b;
  const void* conv_C_w;
  const void* conv_C_b;
  const float* dt_bias;
  const float* A;
  const float* D;
  const void* norm_w;
  const void* out_proj;
  float* conv_state_x;
  float* conv_state_B;
  float* conv_state_C;
  float* ssm_state;
  void* out;
  void* scratch;
} ssm_mamba2_decode_args;

int ssm_mamba2_decode_supported(int32_t batch, int32_t d_model, int32_t heads, int32_t headdim, int32_t nstate, int32_t groups, int32_t width,
                                int32_t io_dtype);
int64_t ssm_mamba2_decode_scratch_bytes(int32_t batch, int32_t heads, int32_t groups);
int ssm_mamba2_decode(const ssm_mamba2_decode_args* args, ssm_stream_t stream);

#ifdef __cplusplus
}
#endif
#endif /* SSM_B200_H_ */
