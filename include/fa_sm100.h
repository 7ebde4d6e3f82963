/*
 * C ABI of libfa_sm100.so: flash-attention forward and backward for NVIDIA B200
 * (sm_100a), with an optional (B,H,M,N) additive bias / bool mask and a bias
 * gradient written at full size.
 *
 * Every entry point takes plain pointers and sizes, enqueues work on the CUDA
 * stream it is given, never synchronises the device (except where noted), never
 * throws and never frees caller memory.  All tensors are owned by the caller.
 * A return value of 0 means "enqueued"; any other value is an fa_error code
 * (fa_status_string() turns it into text).
 *
 * The entry points replace, one for one, the host launchers of the reference
 * project's flash_attention.py (cited per function below as FA:<line>).
 */
#ifndef FA_SM100_H_
#define FA_SM100_H_

#include <stdint.h>

#ifdef __cplusplus
extern "C" {
#endif

#define FA_ABI_VERSION 2

enum fa_dtype { FA_F16 = 0, FA_BF16 = 1 };

/* What the `bias` pointer holds. */
enum fa_bias_kind {
  FA_BIAS_NONE = 0,
  FA_BIAS_SAME = 1, /* float bias in the same 16-bit dtype as q; added to q.k^T*scale      */
  FA_BIAS_BOOL = 2, /* one byte per element; 0 masks the score out, non-zero keeps it      */
  FA_BIAS_F32 = 3   /* fp32 bias with 16-bit q/k/v: streamed as fp32, never rounded to 16 bits;
                       the bias gradient, when asked for, is written in fp32 (FA:52, FA:292, FA:799) */
};

enum fa_error {
  FA_OK = 0,
  FA_ERR_ABI = 1,         /* struct_size does not match this library            */
  FA_ERR_NULL = 2,        /* a required pointer is null                         */
  FA_ERR_SHAPE = 3,       /* a dimension is < 1 or the head dim is unsupported  */
  FA_ERR_DTYPE = 4,       /* unknown dtype / bias kind, or unsupported mix      */
  FA_ERR_ALIGN = 5,       /* a base pointer or stride breaks the 16-byte rule   */
  FA_ERR_CUDA = 6,        /* a CUDA runtime/driver call failed                  */
  FA_ERR_DEVICE_WAIT = 7, /* a kernel gave up a bounded wait (see fa_last_device_status) */
  FA_ERR_UNSUPPORTED = 8, /* legal in the reference, not built in this library
                             (no input reaches it today: every head dim of FA:776 runs) */
  FA_ERR_TOO_LARGE = 9    /* a size exceeds a stated limit of the entry point   */
};

/*
 * One attention problem.  Layouts (element strides; the innermost stride of
 * every tensor must be 1):
 *   q, o, do, dq : (B, M, H, D)  strides {B, M, H}
 *   k, v, dk, dv : (B, N, H, D)  strides {B, N, H}
 *   bias, dbias  : (B, H, M, N)  strides {B, H, M}; a stride of 0 (an expanded
 *                  view) is accepted for B and H of `bias`.  dbias has the bias's
 *                  element type (16-bit for FA_BIAS_SAME, fp32 for FA_BIAS_F32).  With
 *                  FA_BIAS_F32 and causal = 1 the caller zero-fills dbias first: tiles
 *                  above the diagonal are not visited (with FA_BIAS_SAME the library
 *                  writes those zeros itself, except at D = 256, where the caller
 *                  zero-fills a causal dbias of either type)
 *   lse, delta   : (B, H, M) fp32, contiguous
 * Alignment: q/k/v/do base pointers and strides*2 bytes are multiples of 16; the
 * same holds for bias/dbias strides in bytes (the Python layer pads when a row
 * pitch does not qualify).
 */
typedef struct fa_params {
  uint32_t struct_size; /* sizeof(fa_params), checked against the library */
  int32_t device;       /* CUDA device ordinal all pointers live on       */
  int32_t B, H, M, N, D;
  int32_t dtype;       /* fa_dtype of q, k, v, o, do, dq, dk, dv          */
  int32_t bias_kind;   /* fa_bias_kind                                    */
  int32_t causal;      /* 1: key n is visible to query m iff n <= m       */
  int32_t write_dbias; /* backward only: 1 = store dS into dbias          */
  float sm_scale;      /* multiplies q.k^T (not the bias)                 */

  const void* q;
  const void* k;
  const void* v;
  void* o;         /* forward: out; backward: in                          */
  const void* d_o; /* backward in: gradient of o                          */
  void* dq;
  void* dk;
  void* dv;
  const void* bias;
  void* dbias;
  float* lse;   /* forward out / backward in: log2-domain log-sum-exp      */
  float* delta; /* backward scratch: rowsum(o * do), written by fa_bwd_pre and by whole backwards */

  int64_t q_stride[3];
  int64_t k_stride[3];
  int64_t v_stride[3];
  int64_t o_stride[3];
  int64_t do_stride[3];
  int64_t dq_stride[3];
  int64_t dk_stride[3];
  int64_t dv_stride[3];
  int64_t bias_stride[3];
  int64_t dbias_stride[3];

  /* Backward with FA_BIAS_F32, and every backward at D = 256 except the one that writes a
   * 16-bit dbias (FA_BIAS_SAME with write_dbias = 1): a (B,H,M,N) scratch tensor in q's 16-bit
   * dtype, required in those cases, ignored otherwise.  The dK/dV stage leaves dS there for
   * the dQ stage (which consumes dS as a 16-bit tensor-core operand, exactly as the reference
   * rounds dS before its dQ product, FA:517).  Same stride rules as dbias.  Contents
   * after fa_bwd_dkdv and, at any size, fa_bwd: dS rounded to 16 bits at and below the causal
   * diagonal, unspecified above it.  fa_bwd_workspace with a workspace and fa_small_bwd leave
   * it alone. */
  void* ds16;
  int64_t ds16_stride[3];
} fa_params;

/* Library / ABI version (FA_ABI_VERSION of the build). */
int fa_version(void);

/*
 * Number of kernels this library has launched since it was loaded (forward 1 per call; backward 3:
 * preprocess, dK/dV, dQ, with more parts two more each, or 1 where it is one launch (see fa_bwd); a row copy 1).  For
 * benchmarks and tests that must show the work ran here.  No counterpart in the reference.
 */
uint64_t fa_launch_count(void);

/* Text for an fa_error code; never null. */
const char* fa_status_string(int code);

/*
 * Forward: o = softmax(q.k^T * sm_scale + bias, masks) . v and the log2-domain
 * log-sum-exp of every row.  Replaces _flash_attn_fwd (FA:649-685) and the
 * _attn_fwd kernel (FA:88-194); the eager `bias * log2(e)` copy of FA:661-663 is
 * folded into the kernel.
 */
int fa_fwd(const fa_params* p, void* stream);

/*
 * Whether fa_fwd reads the bias of a problem with M query rows of head dim D element by element
 * (few rows: a decode step).  Such a bias needs a unit innermost stride and nothing else: any
 * naturally aligned address (else FA_ERR_ALIGN), any other strides, 0 for M included.
 */
int fa_fwd_takes_any_bias(int M, int D);

/*
 * Short sequences (fa_small_takes: M, N <= 64 and D <= 64).  fa_fwd, fa_bwd and fa_bwd_workspace use the same kernels
 * for them and ask of the bias, its gradient and ds16 what they ask at any size.  These two take the bias and write its
 * gradient at any naturally aligned address with any strides (the innermost is 1; those of the gradient are positive where
 * the extent is more than 1), use no ds16 and no scratch, and leave every element of a gradient of shape (B, H, M, N)
 * written.  Other sizes: FA_ERR_UNSUPPORTED.  An address or a stride that breaks this: FA_ERR_ALIGN.
 */
int fa_small_takes(int M, int N, int D);
int fa_small_fwd(const fa_params* p, void* stream);
int fa_small_bwd(const fa_params* p, void* stream);

/*
 * Copies for callers whose bias does not meet the 16-byte rule, in elements of elem_bytes (1, 2, 4; strides and pitch in
 * elements, the innermost is 1).  fa_pad_rows: a (B, H, M, N) tensor of any strides (0 included) into rows that start at
 * multiples of 16 bytes; the last 16-byte unit of each row is filled up with zeros.  fa_pack_rows (2 or 4 bytes): rows of
 * one pitch into a dense, 16-byte aligned tensor.  A row of more than 2^31 - 17 bytes is FA_ERR_TOO_LARGE, as are more than
 * 65535 (batch, head) pairs or 16 GiB a pair in fa_pad_rows.
 */
int fa_pad_rows(void* dst, const int64_t dst_stride[3], const void* src, const int64_t src_stride[3], int elem_bytes, int B, int H,
                int M, int N, int device, void* stream);
int fa_pack_rows(void* dst, const void* src, int64_t pitch, int elem_bytes, int64_t rows, int N, int device, void* stream);

/*
 * Backward on `stream`: the three stages below in order, or one launch that does the work of all of them, with `delta` and
 * `ds16` written as the stages do.  One launch take M, N, D <= 64 (the kernels for short sequences, whose gradients may
 * differ from the stages' in the last bits) and N <= 128, M <= 256, D <= 64 with an fp32 bias or with B * H of at most
 * twice the CTAs of a full grid (the same bits as the stages).  Replaces _flash_attn_bwd
 * (FA:688-763): the eager pre-scaled copies of k and bias (FA:699-704) and the
 * zero fill of dbias (FA:799) are folded into the kernels.
 */
int fa_bwd(const fa_params* p, void* stream);

/*
 * Backward with scratch: the same results as fa_bwd, faster wherever dS has no tensor of its own
 * (no bias, a mask, a bias without gradient, an fp32 bias, D = 256).  The dK/dV stage leaves
 * dS in `workspace` as 16-bit values and the dQ stage is one streamed product over it, where
 * fa_bwd computes the scores a second time; `ds16` is not needed then.  The (batch, head)
 * problems are worked through in parts that fit the workspace.
 *   workspace: 16-byte aligned device memory, contents unspecified before and after;
 *   bytes: any size; fa_bwd_workspace_bytes(p) is what the call works best with (0: it has no
 *     use for one: dS has its own tensor, or recomputing is faster than parts of so few problems).
 *     That is at most 1.5 GiB, except at D = 256 and with an fp32 bias, which have no other way to
 *     dQ: as many problems as fill the SMs, at the most all.  Less than the dS of one problem (M rows of N 16-bit values, rows padded
 *     to 16 bytes), or a null workspace: the call is fa_bwd.
 */
uint64_t fa_bwd_workspace_bytes(const fa_params* p);
int fa_bwd_workspace(const fa_params* p, void* workspace, uint64_t bytes, void* stream);

/*
 * Backward for callers that cannot allocate device memory (a plugin living inside a
 * host runtime with a frozen memory plan, a real-time loop, a foreign-language
 * binding without an allocator).  Same as fa_bwd, except that `p->delta` is ignored:
 * the row-sum scratch lives in a fixed 8 MiB device array inside the library.
 *   - limit: B * H * M <= 2,097,152, else FA_ERR_TOO_LARGE;
 *   - the first call on a device resolves the array's device address; make it before
 *     any stream capture starts;
 *   - all calls on a device share the array: calls that overlap on the GPU race,
 *     nothing in it has to be cleared between calls;
 *   - no cudaMalloc / cudaFree or other allocating call is made.
 * This entry point has no counterpart in the reference (its launcher allocates
 * `delta` with torch.empty_like on every call).
 */
int fa_bwd_static_scratch(const fa_params* p, void* stream);

/*
 * The three backward stages on their own, at any size (per-kernel timing and tests).  Order matters:
 * fa_bwd_pre writes `delta`, which the other two read; and when write_dbias is 1 with a
 * 16-bit bias, fa_bwd_dq READS `dbias` (it forms dQ from the dS tiles fa_bwd_dkdv has just
 * stored there), so fa_bwd_dkdv must have run on the same stream before it.
 */
int fa_bwd_pre(const fa_params* p, void* stream);  /* _attn_bwd_preprocess FA:197-233 */
int fa_bwd_dkdv(const fa_params* p, void* stream); /* _attn_bwd_dkdv       FA:330-454 */
int fa_bwd_dq(const fa_params* p, void* stream);   /* _attn_bwd_dq         FA:538-646 */

/*
 * Reads the device-side status word of `device` into out[0..7] (synchronises the
 * device).  out[0] != 0 means a kernel abandoned a bounded wait; out[1..5] hold
 * kernel id, block x, block y, wait site and loop iteration.  Returns FA_OK or
 * FA_ERR_DEVICE_WAIT / FA_ERR_CUDA.  No counterpart in the reference.
 */
int fa_last_device_status(int device, int32_t out[8]);

/* Clears the status word of `device` and its host copy (synchronises the device). */
int fa_reset_device_status(int device);

/*
 * Registers `host_words` (8 x int32 of page-locked host memory, e.g. from cudaHostAlloc;
 * NULL to unregister) as a host copy of the status word of `device`: a kernel that abandons
 * a wait writes words 0..5 there as well, so the host can notice the failure by reading
 * host_words[0] before its next call, without synchronising.  The memory stays owned by
 * the caller and must outlive the registration.  Synchronises the device once.  No
 * counterpart in the reference (its kernels have no waits of their own).
 */
int fa_set_status_mirror(int device, int32_t* host_words);

/*
 * Failure-path self-test: launches one CTA that waits, for at most `limit_us`
 * microseconds (1..100000), on a barrier nothing ever completes.  The wait gives up, the
 * kernel returns, and the status word reads {1, kernel 101, block 0, 0, site 7, limit_us}.
 * Every later kernel of the library on this device then does no work until
 * fa_reset_device_status() is called.  Nothing hangs or faults.  No counterpart in the
 * reference.
 */
int fa_selftest_wait_timeout(int device, uint32_t limit_us, void* stream);

/*
 * Self-test of the tensor-core building blocks on one 128x128x128 tile:
 *   mode 0: c = a . b^T            (both operands K-major in shared memory)
 *   mode 1: c = a . b              (b MN-major)
 *   mode 2: c = a^T . b            (both MN-major)
 *   mode 3: c = a . b              (a staged through tensor memory, b MN-major)
 *   mode 4: c16 = a                (shared-memory rewrite + bulk tensor store, 16-bit out)
 * a, b: [128][128] 16-bit row-major device buffers of `dtype`; c: [128][128] fp32
 * (mode 4: 16-bit).  Used by the test-suite to pin descriptor encodings; no
 * counterpart in the reference.
 */
int fa_selftest_umma(int mode, int dtype, const void* a, const void* b, void* c, int device,
                     void* stream);

#ifdef __cplusplus
}
#endif
#endif /* FA_SM100_H_ */
