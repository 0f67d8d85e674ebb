// Shared helpers for libi8linear (sm_100a only).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/i8linear.h"

namespace i8l {

// Records printf-style text for i8l_last_error() (thread local) and returns `code`.
int fail(int code, const char* fmt, ...);

// I8L_OK when the current device is compute capability 10.x.
int check_arch();

// Shared launch settings of the tensor-core kernels (defined next to the GEMM launcher): the poll limit of
// the bounded device-side waits (lowered only by the test hook) and the number of CTAs a persistent kernel
// launched by this host thread may use (i8l_set_cta_limit, else the SM count).
uint32_t gemm_wait_limit();
int gemm_cta_budget();
int sm_count();  // of the current device
int32_t* mirror_of(const int32_t* status_word);   // see i8l_status_mirror; null without one

// Both operands of a product, a [a_batch, a_rows, cols] (with its transpose if aqt) and b, in one launch: see quant.cu.
int quant_pair(const void* a, int64_t a_batch, int64_t a_rows, int a_gran, int8_t* aq, float* as, int8_t* aqt, float* ast, const void* b,
               int64_t b_batch, int64_t b_rows, int b_gran, int8_t* bq, float* bs, int64_t cols, int qmode, int hadamard,
               cudaStream_t st);
// i8l_col_sum; in a chain it runs beside its neighbours.
int col_sum(const void* x, int64_t rows, int64_t cols, void* out, cudaStream_t st);
// Clears n floats; in a chain the next kernel waits for it before anything else.
int clear(float* ptr, int64_t n, cudaStream_t st);
// Whether the next one keeps a column on chip, and needs no maxima in memory.
bool col_t_in_one_pass(int64_t rows, bool rot);
// i8l_quant_col_t (rot = false) or i8l_quant_col_t_rot; zeroed: colmax is zero already.
int quant_col_t(const char* name, const void* x, int64_t rows, int64_t cols, int qmode, bool rot, int8_t* qt, float* scale_t,
                float* colmax, bool zeroed, cudaStream_t st);

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

#define I8L_CUDA_OK(expr)                                                                  \
  do {                                                                                     \
    cudaError_t _e = (expr);                                                               \
    if (_e != cudaSuccess)                                                                 \
      return i8l::fail(I8L_ERR_CUDA, "%s failed: %s", #expr, cudaGetErrorString(_e));      \
  } while (0)

// ---------------------------------------------------------------- chains of launches
// The kernels of one composed call (compose.cu) follow one another on a stream and are launched with programmatic
// serialization: each starts as soon as every block of its predecessor has triggered it (or ended) and there is room, so
// that launch latency, prologues and the tails of small grids overlap (2-3 us a launch).  chain_wait() returns when the
// predecessor has completed and its writes are visible.
//   The first kernel of a chain waits before anything else and triggers its successor then: when the successor starts,
//   whatever was in the stream before the chain is done.  (The predecessor is any kernel of the caller's.)
//   Quantizers behind it read the caller's inputs and write memory that no kernel of the chain reads or writes before them.
//   They trigger first thing and wait at their end, so that "predecessor completed" covers the whole chain.
//   Passes that need a predecessor's result (scales from a column maximum) and GEMMs wait behind their set-up, and a GEMM
//   triggers only another GEMM, and none under a limit on its CTAs; the rest starts when its blocks have ended.  A kernel
//   that clears memory for a later pass and the one behind it wait like a first one.
// Outside a chain both instructions do nothing.
__device__ __forceinline__ void chain_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_start(int first) {
  if (first) chain_wait();
  chain_trigger();
}

// How the kernels of a chain read tensors and scales.  A kernel ahead in the stream may write that memory while this grid is
// resident already, so it is no read-only memory in PTX's sense (ld.global.nc, __ldg), whose loads may move ahead of the wait; an
// ordinary load is ordered by it.  volatile as the wait is, so that the compiler keeps the order too.
__device__ __forceinline__ uint4 chain_load(const uint4* ptr) {
  uint4 v;
  asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(ptr));
  return v;
}
__device__ __forceinline__ float chain_load(const float* ptr) {
  float v;
  asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(ptr));
  return v;
}

// This host thread's chain.
struct ChainState {
  bool active, attribute;   // a chain is being launched; its next kernel may start ahead of its predecessor's end
  int wait;                 // it waits before anything else
  int gemm_next;            // it is a GEMM and another one follows
};
extern thread_local ChainState chain_state;
struct LaunchChain {
  explicit LaunchChain(cudaStream_t st) {
    // while a stream is captured, the first kernel depends on whatever precedes it in full: the graph's edges into it
    // may come from other things than one kernel
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    const bool unknown = cudaStreamIsCapturing(st, &cap) != cudaSuccess;
    if (unknown) (void)cudaGetLastError();   // the legacy stream while another one is captured: the launches report it
    const bool plain = unknown || cap != cudaStreamCaptureStatusNone;
    chain_state = ChainState{true, !plain, 1, 0};
  }
  ~LaunchChain() { chain_state = ChainState{}; }
};
// The argument `first` of the kernel launched next.
inline int chain_first() {
  const int w = chain_state.wait;
  chain_state.wait = 0;
  return w;
}
// Adds the attribute to a launch of the chain; attrs has room for one more.
inline void chain_attribute(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attrs) {
  if (chain_state.attribute) {
    attrs[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[cfg.numAttrs].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attrs;
    ++cfg.numAttrs;
  }
  chain_state.attribute = chain_state.active;
}
template <typename... P, typename... A>
cudaError_t launch(void (*kernel)(P...), dim3 grid, unsigned block, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attrs[1];
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  chain_attribute(cfg, attrs);
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// ---------------------------------------------------------------- scale / rounding arithmetic
// All operations are spelled with explicit round-to-nearest intrinsics so that the compiler can
// neither contract x*s+0.5 into an FMA nor replace a division by a reciprocal: the int8 values
// and the stored scales must equal the reference's bit for bit.  The exception are packed products
// (__fmul2_rn), which may be fused with a packed addition behind them: see quant2.

template <int MODE>
__device__ __forceinline__ void make_scale(float amax, float& s, float& stored) {
  if (MODE == I8L_QMODE_TRITON || MODE == I8L_QMODE_TRITON_BF16S) {
    amax = amax > 1e-4f ? amax : 1e-4f;
    s = __fdiv_rn(127.0f, amax);
    stored = __fdiv_rn(1.0f, s);
    if (MODE == I8L_QMODE_TRITON_BF16S) stored = __bfloat162float(__float2bfloat16_rn(stored));
  } else if (MODE == I8L_QMODE_RNE) {
    amax = fmaxf(amax, 1e-4f);
    s = __fmul_rn(__frcp_rn(amax), 127.0f);
    stored = __frcp_rn(s);
  } else if (MODE == I8L_QMODE_FUSED) {
    s = __fdiv_rn(127.0f, __fadd_rn(amax, 1e-5f));
    stored = s;
  } else {  // I8L_QMODE_ROWRCP
    amax = fmaxf(amax, 1e-4f);
    s = __fmul_rn(__frcp_rn(amax), 127.0f);
    stored = __fdiv_rn(amax, 127.0f);
  }
}

// One value: y = x*s, then floor(y + 0.5) clamped to [-128, 127] (a single saturating
// round-toward-minus-infinity conversion), or rint(y) clamped to [-127, 127] for the RNE mode.
template <int MODE>
__device__ __forceinline__ int quant1(float v, float s) {
  const float y = __fmul_rn(v, s);
  int q;
  if (MODE == I8L_QMODE_RNE) {
    asm("cvt.rni.sat.s8.f32 %0, %1;" : "=r"(q) : "f"(y));
    q = max(q, -127);
  } else {
    asm("cvt.rmi.sat.s8.f32 %0, %1;" : "=r"(q) : "f"(__fadd_rn(y, 0.5f)));  // never saturates for FUSED: |x*s| < 127
  }
  return q;
}

// Four quantised values (sign-extended in 32-bit registers) -> four bytes, lowest address first.
__device__ __forceinline__ uint32_t pack4(int a, int b, int c, int d) {
  // cvt.pack puts its first operand in bits 8-15, the second in bits 0-7, and the low half of the
  // third operand in bits 16-31
  uint32_t hi, r;
  asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, 0;" : "=r"(hi) : "r"(d), "r"(c));            // c | d<<8
  asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(b), "r"(a), "r"(hi));   // a | b<<8 | c<<16 | d<<24
  return r;
}

// Packed fp32 pairs (one issue slot for two IEEE operations).  a - b is fma(b, -1, a): one rounding,
// the same result as a subtraction.
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }

// Two values at once.  The packed product may be fused with the +0.5 (one rounding instead of two).  That changes a byte only
// where the product lies just below -0.5 and its rounding moves it there, and for a scale that belongs to the bf16
// maximum of the group no bf16 value does (tests/test_half_up_products_cpu.py goes through all of them, in each mode).
// Nearest-even ties do part, so that mode keeps its product away from any addition.
template <int MODE>
__device__ __forceinline__ void quant2(float2 v, float2 s2, int& q0, int& q1) {
  float2 y = __fmul2_rn(v, s2);
  if (MODE == I8L_QMODE_RNE) {
    asm("cvt.rni.sat.s8.f32 %0, %1;" : "=r"(q0) : "f"(y.x));
    asm("cvt.rni.sat.s8.f32 %0, %1;" : "=r"(q1) : "f"(y.y));
    q0 = max(q0, -127);
    q1 = max(q1, -127);
  } else {
    y = __fadd2_rn(y, make_float2(0.5f, 0.5f));
    asm("cvt.rmi.sat.s8.f32 %0, %1;" : "=r"(q0) : "f"(y.x));
    asm("cvt.rmi.sat.s8.f32 %0, %1;" : "=r"(q1) : "f"(y.y));
  }
}

// Eight bf16 (a 16-byte piece) -> eight int8 in two words.
template <int MODE>
__device__ __forceinline__ uint2 quant_piece(const uint4& u, float s) {
  const float2 s2 = make_float2(s, s);
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
  int q[8];
#pragma unroll
  for (int k = 0; k < 4; ++k)
    quant2<MODE>(make_float2(__uint_as_float(w[k] << 16), __uint_as_float(w[k] & 0xffff0000u)), s2, q[2 * k], q[2 * k + 1]);
  return make_uint2(pack4(q[0], q[1], q[2], q[3]), pack4(q[4], q[5], q[6], q[7]));
}

// The same bytes for finite values whose |max| gave the scale: |v * s| < 127.5, so nothing saturates, and adding
// 1.5 * 2^23 with the rounding wanted (down after the +0.5, to nearest even for the RNE mode) leaves the integer in
// the low byte of the sum.  The saturating conversion runs on the slow conversion pipe, one value at a time.
// It also turns NaN into 0, which this does not: infinite or NaN inputs take quant_piece.
template <int MODE>
__device__ __forceinline__ uint32_t quant_pair_finite(uint32_t w, float s) {   // two bf16 -> two bytes
  const float2 s2 = make_float2(s, s), half2 = make_float2(0.5f, 0.5f), magic2 = make_float2(12582912.f, 12582912.f);
  const float2 v = make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
  float2 y;
  if (MODE == I8L_QMODE_RNE)   // scalar products: a packed one is fused with the addition, which turns ties over (see quant2)
    y = __fadd2_rn(make_float2(__fmul_rn(v.x, s), __fmul_rn(v.y, s)), magic2);
  else
    y = __fadd2_rd(__fadd2_rn(__fmul2_rn(v, s2), half2), magic2);
  return __byte_perm(__float_as_uint(y.x), __float_as_uint(y.y), 0x0040);
}
template <int MODE>
__device__ __forceinline__ uint2 quant_piece_finite(const uint4& u, float s) {
  return make_uint2(__byte_perm(quant_pair_finite<MODE>(u.x, s), quant_pair_finite<MODE>(u.y, s), 0x5410),
                    __byte_perm(quant_pair_finite<MODE>(u.z, s), quant_pair_finite<MODE>(u.w, s), 0x5410));
}

__device__ __forceinline__ float bf16_bits_to_float(uint32_t b) { return __uint_as_float(b << 16); }

__device__ __forceinline__ void unpack8(const uint4& u, float* v) {
  v[0] = bf16_bits_to_float(u.x & 0xffffu); v[1] = __uint_as_float(u.x & 0xffff0000u);
  v[2] = bf16_bits_to_float(u.y & 0xffffu); v[3] = __uint_as_float(u.y & 0xffff0000u);
  v[4] = bf16_bits_to_float(u.z & 0xffffu); v[5] = __uint_as_float(u.z & 0xffff0000u);
  v[6] = bf16_bits_to_float(u.w & 0xffffu); v[7] = __uint_as_float(u.w & 0xffff0000u);
}

__device__ __forceinline__ float round_to_bf16(float v) {
  return __bfloat162float(__float2bfloat16_rn(v));
}

// 128-point Walsh-Hadamard transform of a row segment held as 8 consecutive values in each of 16
// consecutive lanes (lane & 15 selects the 8-wide chunk).  Butterfly spans double from 1 to 64,
// the order the CPU oracle uses; fp32 adds commute, so the result is bit-equal to it.
__device__ __forceinline__ void fwht128_lanes16(float* v, int lane) {
#pragma unroll
  for (int h = 1; h < 8; h <<= 1) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if ((j & h) == 0) {
        float a = v[j], b = v[j | h];
        v[j] = __fadd_rn(a, b);
        v[j | h] = __fsub_rn(a, b);
      }
    }
  }
#pragma unroll
  for (int m = 1; m < 16; m <<= 1) {
    const bool upper = (lane & m) != 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float p = __shfl_xor_sync(0xffffffffu, v[j], m);
      v[j] = upper ? __fsub_rn(p, v[j]) : __fadd_rn(v[j], p);
    }
  }
}

}  // namespace i8l
