// bf16 -> int8 absmax quantizers: 128x128-tile kernels (plain, rotated, either or both orientations), 128x256 tiles,
// row kernels (rows on chip, rotated in 128-groups or whole, long rows in two sweeps), column-absmax kernel.
#include <atomic>
#include <cstdarg>
#include <cstdio>
#include <type_traits>

#include "common.cuh"
#include "ptx.cuh"

namespace i8l {

static thread_local char g_err[512] = "";
thread_local ChainState chain_state;

int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
  return code;
}

int check_arch() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return fail(I8L_ERR_CUDA, "cudaGetDevice failed");
  static std::atomic<int> cached_major[64];  // 0 = unknown
  int major = (dev >= 0 && dev < 64) ? cached_major[dev].load(std::memory_order_relaxed) : 0;
  if (major == 0) {
    if (cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev) != cudaSuccess)
      return fail(I8L_ERR_CUDA, "cudaDeviceGetAttribute failed");
    if (dev >= 0 && dev < 64) cached_major[dev].store(major, std::memory_order_relaxed);
  }
  if (major != 10)
    return fail(I8L_ERR_ARCH, "device %d has compute capability %d.x; this library is sm_100a only", dev, major);
  return I8L_OK;
}

// ------------------------------------------------------------------------------------------------
// Tile kernel.  One CTA of 256 threads owns one 128x128 tile of x.
// Thread mapping: warp w owns tile rows 16w..16w+15; pass it in {0,1}; lane = (half<<4)|cc;
// the thread holds rows 16w + 8it + 4half + i (i<4), columns 8cc..8cc+7: every global load is a
// 16-byte vector and 16 lanes cover one 256-byte row segment.
// ------------------------------------------------------------------------------------------------
constexpr int GRAN_COLFULL = 3;  // internal: per-column scale from a precomputed column absmax
constexpr int GRAN_COLMAX_PASS = 4;  // internal: only accumulate the column absmax of the rotated tile

// |x| maximum of the 8 bf16 values of a 16-byte vector, as two packed maxima (exact: bf16 compare).
__device__ __forceinline__ __nv_bfloat162 absmax8(const uint4& u, __nv_bfloat162 m) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int k = 0; k < 4; ++k) m = __hmax2(m, __habs2(h[k]));
  return m;
}
constexpr float BF16_LARGEST = 3.3895314e38f;
__device__ __forceinline__ float hmax_of(__nv_bfloat162 m) { return fmaxf(__low2float(m), __high2float(m)); }

template <int GRAN, int MODE, bool OUT_N, bool OUT_T>
__device__ __forceinline__ void
quant_tile_body(const dim3 block, const __nv_bfloat16* __restrict__ x, int64_t rows, int64_t cols,
                int8_t* __restrict__ q, float* __restrict__ scale, int8_t* __restrict__ qt,
                float* __restrict__ scale_t, const float* __restrict__ colmax, int first) {
  __shared__ float s_red[8];
  __shared__ float s_colred[(GRAN == I8L_GRAN_GROUP128 && OUT_T) ? 8 * 128 : 1];
  __shared__ float s_cols[(GRAN != I8L_GRAN_TILE128 && OUT_T) ? 128 : 1];
  __shared__ uint32_t s_t[OUT_T ? 128 * 32 : 1];

  const int tid = threadIdx.x, w = tid >> 5, l = tid & 31, cc = l & 15, half = l >> 4;
  const int64_t r_base = (int64_t)block.y * 128, c_base = (int64_t)block.x * 128;
  const int64_t boff = (int64_t)block.z * rows * cols;
  const __nv_bfloat16* xb = x + boff;
  chain_start(first);

  // The tile stays in registers as packed bf16 (32 registers per thread, 4 CTAs per SM).
  uint4 raw[2][4];
#pragma unroll
  for (int it = 0; it < 2; ++it)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = 16 * w + 8 * it + 4 * half + i;
      raw[it][i] = chain_load(reinterpret_cast<const uint4*>(xb + (r_base + r) * cols + c_base + 8 * cc));
    }

  // ---- scales
  const __nv_bfloat162 zero2 = __floats2bfloat162_rn(0.f, 0.f);
  float s_tile = 0.f;          // TILE128
  float s_row[2][4];           // GROUP128 natural
  float s_col[8];              // column scales (GROUP128 transposed / COLFULL)
  if (GRAN == I8L_GRAN_TILE128) {
    __nv_bfloat162 m2 = zero2;
#pragma unroll
    for (int it = 0; it < 2; ++it)
#pragma unroll
      for (int i = 0; i < 4; ++i) m2 = absmax8(raw[it][i], m2);
    float m = hmax_of(m2);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (l == 0) s_red[w] = m;
    __syncthreads();
    m = s_red[0];
#pragma unroll
    for (int k = 1; k < 8; ++k) m = fmaxf(m, s_red[k]);
    float stored;
    make_scale<MODE>(m, s_tile, stored);
    if (tid == 0) {
      const int64_t nrb = rows / 128, ncb = cols / 128;
      if (OUT_N) scale[((int64_t)block.z * nrb + block.y) * ncb + block.x] = stored;
      if (OUT_T) scale_t[((int64_t)block.z * ncb + block.x) * nrb + block.y] = stored;
    }
  } else if (GRAN == I8L_GRAN_GROUP128 && OUT_N) {
#pragma unroll
    for (int it = 0; it < 2; ++it)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float m = hmax_of(absmax8(raw[it][i], zero2));
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        float stored;
        make_scale<MODE>(m, s_row[it][i], stored);
        if (cc == 0) {
          const int r = 16 * w + 8 * it + 4 * half + i;
          scale[((int64_t)block.z * rows + r_base + r) * (cols / 128) + block.x] = stored;
        }
      }
  } else {  // column scales
    if (GRAN == I8L_GRAN_GROUP128) {
      __nv_bfloat162 cm[4] = {zero2, zero2, zero2, zero2};   // per-column maxima of this thread's 8 rows
#pragma unroll
      for (int it = 0; it < 2; ++it)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw[it][i]);
#pragma unroll
          for (int k = 0; k < 4; ++k) cm[k] = __hmax2(cm[k], __habs2(h[k]));
        }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float m = (j & 1) ? __high2float(cm[j >> 1]) : __low2float(cm[j >> 1]);
        m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 16));
        if (half == 0) s_colred[w * 128 + 8 * cc + j] = m;
      }
      __syncthreads();
    }
    if (tid < 128) {
      float m;
      if (GRAN == I8L_GRAN_GROUP128) {
        m = s_colred[tid];
#pragma unroll
        for (int k = 1; k < 8; ++k) m = fmaxf(m, s_colred[k * 128 + tid]);
      } else {
        chain_wait();
        m = chain_load(colmax + c_base + tid);
      }
      float s, stored;
      make_scale<MODE>(m, s, stored);
      s_cols[tid] = s;
      if (GRAN == I8L_GRAN_GROUP128)
        scale_t[((int64_t)block.z * cols + c_base + tid) * (rows / 128) + block.y] = stored;
      else if (block.y == 0)
        scale_t[c_base + tid] = stored;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 8; ++j) s_col[j] = s_cols[8 * cc + j];
  }

  // ---- quantise, write
#pragma unroll
  for (int it = 0; it < 2; ++it) {
    int b[4][8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float v[8];
      unpack8(raw[it][i], v);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float s;
        if (GRAN == I8L_GRAN_TILE128) s = s_tile;
        else if (GRAN == I8L_GRAN_GROUP128 && OUT_N) s = s_row[it][i];
        else s = s_col[j];
        b[i][j] = quant1<MODE>(v[j], s);
      }
    }
    if (OUT_N) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = 16 * w + 8 * it + 4 * half + i;
        uint2 o;
        o.x = pack4(b[i][0], b[i][1], b[i][2], b[i][3]);
        o.y = pack4(b[i][4], b[i][5], b[i][6], b[i][7]);
        *reinterpret_cast<uint2*>(q + boff + (r_base + r) * cols + c_base + 8 * cc) = o;
      }
    }
    if (OUT_T) {
      // word (4 consecutive rows of one column) goes to transposed row c = 8cc+j, word index
      // widx = 4w + 2it + half, XOR-swizzled with 2*(c>>3) so that the 32 lanes hit 32 banks.
      const int widx = 4 * w + 2 * it + half;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int c = 8 * cc + j;
        s_t[c * 32 + (widx ^ (2 * cc))] = pack4(b[0][j], b[1][j], b[2][j], b[3][j]);
      }
    }
  }
  if (OUT_T) {
    __syncthreads();
    int8_t* qtb = qt + boff;
#pragma unroll 4
    for (int t = 0; t < 16; ++t) {
      const int c = 16 * w + t;
      const uint32_t word = s_t[c * 32 + (l ^ (2 * (c >> 3)))];
      *reinterpret_cast<uint32_t*>(qtb + (c_base + c) * rows + r_base + 4 * l) = word;
    }
  }
  chain_wait();
}
template <int GRAN, int MODE, bool OUT_N, bool OUT_T>
__global__ void __launch_bounds__(256, 4)
quant_tile_kernel(const __nv_bfloat16* __restrict__ x, int64_t rows, int64_t cols,
                  int8_t* __restrict__ q, float* __restrict__ scale, int8_t* __restrict__ qt,
                  float* __restrict__ scale_t, const float* __restrict__ colmax, int first) {
  quant_tile_body<GRAN, MODE, OUT_N, OUT_T>(dim3(blockIdx.x, blockIdx.y, blockIdx.z), x, rows, cols, q, scale, qt, scale_t, colmax, first);
}

// ------------------------------------------------------------------------------------------------
// One scale per 128 rows x 256 columns (the activation grouping of the reference's TileLang forward).
// One CTA of 256 threads per group: warp w holds rows 16w..16w+15, one 16-byte piece per lane and row
// (32 lanes cover the 512-byte row segment), 64 registers of packed bf16 per thread.
// ------------------------------------------------------------------------------------------------
template <int MODE>
__global__ void __launch_bounds__(256, 3)
quant_tile256_kernel(const __nv_bfloat16* __restrict__ x, int64_t rows, int64_t cols, int8_t* __restrict__ q,
                     float* __restrict__ scale, int first) {
  __shared__ float s_red[8];
  const int tid = threadIdx.x, w = tid >> 5, l = tid & 31;
  const int64_t r_base = (int64_t)blockIdx.y * 128, c_base = (int64_t)blockIdx.x * 256;
  const int64_t boff = (int64_t)blockIdx.z * rows * cols;
  chain_start(first);
  uint4 raw[16];
  __nv_bfloat162 m2 = __floats2bfloat162_rn(0.f, 0.f);
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    raw[i] = chain_load(reinterpret_cast<const uint4*>(x + boff + (r_base + 16 * w + i) * cols + c_base + 8 * l));
    m2 = absmax8(raw[i], m2);
  }
  float m = hmax_of(m2);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (l == 0) s_red[w] = m;
  __syncthreads();
  m = s_red[0];
#pragma unroll
  for (int k = 1; k < 8; ++k) m = fmaxf(m, s_red[k]);
  float s, stored;
  make_scale<MODE>(m, s, stored);
  if (tid == 0) scale[((int64_t)blockIdx.z * (rows / 128) + blockIdx.y) * (cols / 256) + blockIdx.x] = stored;
#pragma unroll
  for (int i = 0; i < 16; ++i)
    *reinterpret_cast<uint2*>(q + boff + (r_base + 16 * w + i) * cols + c_base + 8 * l) = quant_piece<MODE>(raw[i], s);
  chain_wait();
}

// ------------------------------------------------------------------------------------------------
// Rotated tiles: q = the tile rotated along its columns (the contraction axis of the natural operand), qt =
// its transpose rotated along the rows (the contraction axis of the dW operands and of W^T), either or both
// from ONE read, each with scales of its own.  One CTA of 128 threads per 128x128 tile; the tile is staged
// in shared memory as bf16 and a thread owns a whole row, then a whole column, so that all seven butterfly
// stages run in its registers as packed pairs: no shuffles, which together with 16-bit shared-memory reads
// cost 4.2 load/store slots per element when four lanes shared a row and two a column.  The output rows leave the same
// way as in the GEMMs, through shared memory in whole lines' halves (quant_store128).  No unit is near its limit over a
// block's life, but each of its phases fills one (load/store, adds, conversions), with 12 warps per SM (150 registers;
// about 10 instructions per element and output).  [32768, 8192], two lanes a column -> a column a thread -> staged
// stores: both outputs 353 -> 294 -> 275 us, q 194 -> 171 -> 157, qt 284 -> 181 -> 166; W^T of [28672, 8192] in its two
// passes 404 -> 241 -> 236.  Slower: a persistent form that copies the next tile meanwhile (393 us with both outputs),
// fetching a later block's tile into L2 (315), two threads per row and column with half the registers and twice the warps
// (316), blocks started apart from one another (304).
// ------------------------------------------------------------------------------------------------
constexpr int ROT_LD = 272;  // bytes per staged row: 256 + 16, conflict-free for 16-byte row reads and for column reads

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

// Transform of p[k] = (x[k], x[k + N]) over 2N points but for the last span: spans 1..N/2 between the pairs, in the
// order of the CPU oracle; the caller adds and subtracts the halves of each pair (span N).
template <int N>
__device__ __forceinline__ void fwht_pairs(float2* p) {
#pragma unroll
  for (int span = 1; span < N; span <<= 1)
#pragma unroll
    for (int k = 0; k < N; ++k)
      if ((k & span) == 0) {
        const float2 a = p[k], b = p[k | span];
        p[k] = add2(a, b);
        p[k | span] = sub2(a, b);
      }
}

// 128 staged bf16 values of a row -> p[k] = (x[k], x[k + 64]).
__device__ __forceinline__ void load_row128(const uint8_t* row, float2* p) {
#pragma unroll
  for (int c = 0; c < 16; ++c) {
    float v[8];
    unpack8(*reinterpret_cast<const uint4*>(row + 16 * c), v);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if (c < 8) p[8 * c + j].x = v[j];
      else p[8 * (c - 8) + j].y = v[j];
    }
  }
}

// 128-point transform of p[k] = (x[k], x[k + 64]).  Returns the results rounded to bf16, h[i] = (y[2i], y[2i+1]), and their |max|, NaN
// if one of them is NaN.
__device__ __forceinline__ float rot128(float2* p, uint32_t* h) {
  fwht_pairs<64>(p);
  __nv_bfloat162 hm = __floats2bfloat162_rn(0.f, 0.f);
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    const float2 a = p[2 * i], b = p[2 * i + 1];
    const __nv_bfloat162 lo = __floats2bfloat162_rn(__fadd_rn(a.x, a.y), __fadd_rn(b.x, b.y));
    const __nv_bfloat162 hi = __floats2bfloat162_rn(__fsub_rn(a.x, a.y), __fsub_rn(b.x, b.y));
    hm = __hmax2_nan(hm, __hmax2_nan(__habs2(lo), __habs2(hi)));
    h[i] = *reinterpret_cast<const uint32_t*>(&lo);
    h[32 + i] = *reinterpret_cast<const uint32_t*>(&hi);
  }
  const __nv_bfloat16 m = __hmax_nan(__low2bfloat16(hm), __high2bfloat16(hm));
  return __bfloat162float(m);
}

__device__ __forceinline__ float max_without_nan(const uint32_t* h) {
  __nv_bfloat162 hm = __floats2bfloat162_rn(0.f, 0.f);
#pragma unroll
  for (int i = 0; i < 64; i += 4) hm = absmax8(make_uint4(h[i], h[i + 1], h[i + 2], h[i + 3]), hm);
  return hmax_of(hm);
}

// 128 rotated values per lane -> 128 bytes of row `lane` of the warp's rows, `pitch` bytes apart from `out` on; rows: how many
// there are.  A lane owns a row, so a plain store instruction touches 32 lines, and the stores took a quarter of the
// load/store unit's time.  The warp passes its rows through shared memory in halves (`stage`, 32 pieces of OUT_LD bytes), and an
// instruction stores 64 bytes of eight rows.  FINITE: quant_piece_finite instead of the saturating conversions.
constexpr int OUT_LD = 80;   // 64 + 16: conflict-free both ways
template <int MODE, bool FINITE>
__device__ __forceinline__ void quant_stage64(const uint32_t* h, float s, uint32_t dst) {
#pragma unroll
  for (int i = 0; i < 32; i += 8) {
    const uint2 a = FINITE ? quant_piece_finite<MODE>(make_uint4(h[i], h[i + 1], h[i + 2], h[i + 3]), s)
                           : quant_piece<MODE>(make_uint4(h[i], h[i + 1], h[i + 2], h[i + 3]), s);
    const uint2 b = FINITE ? quant_piece_finite<MODE>(make_uint4(h[i + 4], h[i + 5], h[i + 6], h[i + 7]), s)
                           : quant_piece<MODE>(make_uint4(h[i + 4], h[i + 5], h[i + 6], h[i + 7]), s);
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + 2 * i), "r"(a.x), "r"(a.y), "r"(b.x), "r"(b.y) : "memory");
  }
}
template <int MODE>
__device__ __forceinline__ void quant_store128(const uint32_t* h, float s, bool finite, uint32_t stage, int lane, int8_t* out, int64_t pitch,
                                               int rows) {
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    __syncwarp();   // what was staged before has been read
    if (finite) quant_stage64<MODE, true>(h + 32 * half, s, stage + lane * OUT_LD);
    else quant_stage64<MODE, false>(h + 32 * half, s, stage + lane * OUT_LD);
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = 8 * i + (lane >> 2);
      uint4 v;
      asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                   : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                   : "r"(stage + row * OUT_LD + 16 * (lane & 3))
                   : "memory");
      if (row < rows) *reinterpret_cast<uint4*>(out + row * pitch + 64 * half + 16 * (lane & 3)) = v;
    }
  }
}

// GRAN: TILE128, GROUP128 (one scale per output row and 128 contraction elements), or for qt alone
// GRAN_COLMAX_PASS / GRAN_COLFULL: the two passes of one scale per output row over all of its elements.
template <int GRAN, int MODE, bool OUT_N, bool OUT_T>
__global__ void __launch_bounds__(128, 3)
quant_tile_rot_kernel(const __nv_bfloat16* __restrict__ x, int64_t rows, int64_t cols, int8_t* __restrict__ q,
                      float* __restrict__ scale, int8_t* __restrict__ qt, float* __restrict__ scale_t,
                      float* __restrict__ colmax, int first) {
  __shared__ __align__(16) uint8_t s_raw[128 * ROT_LD];
  __shared__ __align__(16) uint8_t s_out[GRAN == GRAN_COLMAX_PASS ? 16 : 128 * OUT_LD];
  __shared__ float s_red[2][4];
  const int tid = threadIdx.x, w = tid >> 5, l = tid & 31;
  const int64_t r_base = (int64_t)blockIdx.y * 128, c_base = (int64_t)blockIdx.x * 128;
  const int64_t boff = (int64_t)blockIdx.z * rows * cols;
  chain_start(first);
  {
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(s_raw) + (tid >> 4) * ROT_LD + 16 * (tid & 15);
    const __nv_bfloat16* src = x + boff + (r_base + (tid >> 4)) * cols + c_base + 8 * (tid & 15);
#pragma unroll
    for (int i = 0; i < 16; ++i) cp_async16(dst + i * 8 * ROT_LD, src + (int64_t)i * 8 * cols);
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
  }
  __syncthreads();
  // Both orientations run through the same code, a row and then a column per thread (two unrolled copies of the
  // transform measured the same).
#pragma unroll 1
  for (int ph = OUT_N ? 0 : 1; ph < (OUT_T ? 2 : 1); ++ph) {
    float2 p[64];
    if (ph == 0) {
      load_row128(s_raw + tid * ROT_LD, p);
    } else {
      const uint8_t* col = s_raw + 2 * tid;
#pragma unroll
      for (int k = 0; k < 64; ++k) {
        p[k].x = bf16_bits_to_float(*reinterpret_cast<const uint16_t*>(col + k * ROT_LD));
        p[k].y = bf16_bits_to_float(*reinterpret_cast<const uint16_t*>(col + (k + 64) * ROT_LD));
      }
    }
    uint32_t h[64];
    float m = rot128(p, h), s, stored;
    const bool finite = m <= BF16_LARGEST;
    if (!finite) m = max_without_nan(h);
    if (GRAN == GRAN_COLMAX_PASS) {  // |x| >= 0: the bit patterns order like integers, so an integer maximum is exact
      atomicMax(reinterpret_cast<int*>(colmax + c_base + tid), __float_as_int(m));
      break;
    }
    if (GRAN == I8L_GRAN_TILE128) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
      if (l == 0) s_red[ph][w] = m;
      __syncthreads();
      m = fmaxf(fmaxf(s_red[ph][0], s_red[ph][1]), fmaxf(s_red[ph][2], s_red[ph][3]));
    }
    if (GRAN == GRAN_COLFULL) {
      chain_wait();
      m = chain_load(colmax + c_base + tid);
    }
    make_scale<MODE>(m, s, stored);
    const int64_t o_base = ph == 0 ? r_base : c_base, k_base = ph == 0 ? c_base : r_base;  // output row, contraction axis
    const int64_t o_n = ph == 0 ? rows : cols, k_n = ph == 0 ? cols : rows, kb = k_base / 128, nkb = k_n / 128;
    float* sc = ph == 0 ? scale : scale_t;
    if (GRAN == GRAN_COLFULL) { if (kb == 0) sc[o_base + tid] = stored; }
    else if (GRAN == I8L_GRAN_GROUP128) sc[(blockIdx.z * o_n + o_base + tid) * nkb + kb] = stored;
    else if (tid == 0) sc[(blockIdx.z * (o_n / 128) + o_base / 128) * nkb + kb] = stored;
    int8_t* out = ph == 0 ? q : qt;
    quant_store128<MODE>(h, s, finite, (uint32_t)__cvta_generic_to_shared(s_out) + w * 32 * OUT_LD, l,
                         out + boff + (o_base + 32 * w) * k_n + k_base, k_n, 32);
  }
  chain_wait();
}

// Column absmax of x [rows, cols] into colmax[cols] (pre-zeroed); |x| >= 0 so the float bit
// patterns order like integers and atomicMax on int is exact.
__global__ void __launch_bounds__(256)
col_absmax_kernel(const __nv_bfloat16* __restrict__ x, int64_t rows, int64_t cols, float* __restrict__ colmax, int first) {
  __shared__ float s_colred[8 * 128];
  const int tid = threadIdx.x, w = tid >> 5, l = tid & 31, cc = l & 15, half = l >> 4;
  const int64_t r_base = (int64_t)blockIdx.y * 128, c_base = (int64_t)blockIdx.x * 128;
  chain_start(first);
  float m[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) m[j] = 0.f;
#pragma unroll
  for (int it = 0; it < 2; ++it)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = 16 * w + 8 * it + 4 * half + i;
      const uint4 u = chain_load(reinterpret_cast<const uint4*>(x + (r_base + r) * cols + c_base + 8 * cc));
      float v[8];
      unpack8(u, v);
#pragma unroll
      for (int j = 0; j < 8; ++j) m[j] = fmaxf(m[j], fabsf(v[j]));
    }
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    m[j] = fmaxf(m[j], __shfl_xor_sync(0xffffffffu, m[j], 16));
    if (half == 0) s_colred[w * 128 + 8 * cc + j] = m[j];
  }
  __syncthreads();
  if (tid < 128) {
    float mm = s_colred[tid];
#pragma unroll
    for (int k = 1; k < 8; ++k) mm = fmaxf(mm, s_colred[k * 128 + tid]);
    atomicMax(reinterpret_cast<int*>(colmax + c_base + tid), __float_as_int(mm));
  }
  chain_wait();
}

// ------------------------------------------------------------------------------------------------
// x^T with one scale per column of x, in one pass: the CTAs of a cluster share a strip of 64 columns (a 128-byte line per
// row), each keeps up to BLOCKS blocks of 128 rows of it in registers, and they exchange the column maxima through distributed shared
// memory.  One read instead of two, one launch instead of three (clearing the maxima, taking them, quantizing), no
// atomics.  A thread holds four consecutive rows of eight columns per block, so that it packs words of the transposed
// rows by itself; these go through shared memory (16-byte pieces, XOR-swizzled: conflict-free both ways) and leave in
// runs of a CTA's rows.  Up to 32 blocks a strip: [1024, 1024] 10.8 -> 6.7 us, [2176, 1408] 12.8 -> 8.0, [4096, 4096] 19.0 -> 14.9,
// [4096, 11008] 46.6 -> 45.6 against the two passes.  With 64 blocks (eight a CTA, 190 registers, one CTA per SM) it is the
// slower way: [8192, 4096] 29 -> 43.
// ------------------------------------------------------------------------------------------------
constexpr int COLT_COLS = 64;
template <int BLOCKS> constexpr size_t COLT_SMEM = (size_t)BLOCKS * 128 * COLT_COLS;

// Two bf16 of neighbouring columns -> two bytes, as quant_pair_finite but with a scale each; or with the saturating conversions.
template <int MODE, bool FINITE>
__device__ __forceinline__ uint32_t quant_cols2(uint32_t w, float2 s2) {
  const float2 v = make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
  if (FINITE) {
    const float2 half2 = make_float2(0.5f, 0.5f), magic2 = make_float2(12582912.f, 12582912.f);
    float2 y;
    if (MODE == I8L_QMODE_RNE) y = __fadd2_rn(make_float2(__fmul_rn(v.x, s2.x), __fmul_rn(v.y, s2.y)), magic2);   // see quant_pair_finite
    else y = __fadd2_rd(__fadd2_rn(__fmul2_rn(v, s2), half2), magic2);
    return __byte_perm(__float_as_uint(y.x), __float_as_uint(y.y), 0x0040);
  }
  return __byte_perm((uint32_t)quant1<MODE>(v.x, s2.x), (uint32_t)quant1<MODE>(v.y, s2.y), 0x0040);
}

template <int MODE, int BLOCKS>
__global__ void __launch_bounds__(256, BLOCKS == 4 ? 2 : 4)
quant_col_strip_kernel(const __nv_bfloat16* __restrict__ x, int64_t rows, int64_t cols, int8_t* __restrict__ qt,
                       float* __restrict__ scale_t, int first) {
  extern __shared__ __align__(16) float s_f[];   // words [64 columns][32 BLOCKS], see below
  __shared__ float s_warp[8][COLT_COLS], s_max[COLT_COLS], s_scale[COLT_COLS];
  uint32_t* s_t = reinterpret_cast<uint32_t*>(s_f);
  constexpr int PITCH = 32 * BLOCKS;   // words per column
  const int tid = threadIdx.x, c = tid & 7, g = tid >> 3, w = tid >> 5, l = tid & 31;
  const int64_t nb = rows / 128, share = gridDim.y, b0 = nb * blockIdx.y / share;
  const int mine = (int)(nb * (blockIdx.y + 1) / share - b0);
  chain_start(first);
  const uint4* src = reinterpret_cast<const uint4*>(x + (b0 * 128 + 4 * g) * cols + (int64_t)blockIdx.x * COLT_COLS) + c;
  uint4 raw[BLOCKS][4];
#pragma unroll
  for (int b = 0; b < BLOCKS; ++b)
#pragma unroll
    for (int i = 0; i < 4; ++i) raw[b][i] = b < mine ? chain_load(src + (b * 128 + i) * (cols / 8)) : make_uint4(0, 0, 0, 0);
  // column maxima, with and without NaNs
  __nv_bfloat162 any = __floats2bfloat162_rn(0.f, 0.f), m[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    m[k] = __floats2bfloat162_rn(0.f, 0.f);
#pragma unroll
    for (int b = 0; b < BLOCKS; ++b)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t u = k == 0 ? raw[b][i].x : k == 1 ? raw[b][i].y : k == 2 ? raw[b][i].z : raw[b][i].w;
        const __nv_bfloat162 a = __habs2(*reinterpret_cast<const __nv_bfloat162*>(&u));
        m[k] = __hmax2(m[k], a);
        any = __hmax2_nan(any, a);
      }
#pragma unroll
    for (int o = 8; o < 32; o <<= 1) m[k] = __hmax2(m[k], __shfl_xor_sync(0xffffffffu, m[k], o));
    if (l < 8) {
      s_warp[w][8 * c + 2 * k] = __low2float(m[k]);
      s_warp[w][8 * c + 2 * k + 1] = __high2float(m[k]);
    }
  }
  const bool finite = __bfloat162float(__hmax_nan(__low2bfloat16(any), __high2bfloat16(any))) <= BF16_LARGEST;
  __syncthreads();
  if (tid < COLT_COLS) {
    float v = s_warp[0][tid];
#pragma unroll
    for (int k = 1; k < 8; ++k) v = fmaxf(v, s_warp[k][tid]);
    s_max[tid] = v;
  }
  if (share > 1) cluster_sync_all();
  if (tid < COLT_COLS) {
    float v = s_max[tid], s, stored;
    for (uint32_t k = 0; k < share; ++k) {
      float o;
      asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(o) : "r"(map_to_cta((uint32_t)__cvta_generic_to_shared(&s_max[tid]), k)) : "memory");
      v = fmaxf(v, o);
    }
    make_scale<MODE>(v, s, stored);
    s_scale[tid] = s;
    if (blockIdx.y == 0) scale_t[(int64_t)blockIdx.x * COLT_COLS + tid] = stored;
  }
  __syncthreads();
  float2 s2[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) s2[k] = *reinterpret_cast<const float2*>(&s_scale[8 * c + 2 * k]);
  // word g + 32 b of column 8 c + j = rows 4 g .. 4 g + 3 of block b, at 16-byte piece (word / 4) ^ c
  auto pack = [&](auto finite_c) {
    constexpr bool FINITE = decltype(finite_c)::value;
#pragma unroll
    for (int b = 0; b < BLOCKS; ++b) {
      if (b >= mine) break;
      uint32_t* dst = s_t + 8 * c * PITCH + ((g + 32 * b) ^ (4 * c));
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        uint32_t p[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
          p[i] = quant_cols2<MODE, FINITE>(k == 0 ? raw[b][i].x : k == 1 ? raw[b][i].y : k == 2 ? raw[b][i].z : raw[b][i].w, s2[k]);
        const uint32_t t01 = __byte_perm(p[0], p[1], 0x5140), t23 = __byte_perm(p[2], p[3], 0x5140);
        dst[2 * k * PITCH] = __byte_perm(t01, t23, 0x5410);
        dst[(2 * k + 1) * PITCH] = __byte_perm(t01, t23, 0x7632);
      }
    }
  };
  if (finite) pack(std::true_type{});
  else pack(std::false_type{});
  __syncthreads();
  // 8 pieces of 16 bytes per block and column; consecutive threads store consecutive pieces of a column
  const int pieces = 8 * mine;
  for (int i = tid; i < COLT_COLS * pieces; i += 256) {
    const int col = i / pieces, piece = i - col * pieces;
    const uint4 v = *reinterpret_cast<const uint4*>(s_t + col * PITCH + 4 * (piece ^ (col >> 3)));
    *reinterpret_cast<uint4*>(qt + ((int64_t)blockIdx.x * COLT_COLS + col) * rows + b0 * 128 + 16 * piece) = v;
  }
  if (share > 1) cluster_sync_all();   // the others have read this CTA's maxima
  chain_wait();
}

// ------------------------------------------------------------------------------------------------
// Column sums of x [rows, cols] in bf16, the bias gradient.  A CTA of 256 threads sums a strip of 64 columns (a 128-byte
// line per row) over its share of the rows, the CTAs of a cluster share a strip and add up through distributed shared
// memory: one launch, no atomics, always the same order.  At most 128 values are added in a row in fp32, the rest in
// fp64.  Bound by memory (L2, when its neighbours read the same tensor).  Against
// torch's sum: [512, 1024] 8.9 -> 3.3 us, [4096, 4096] 15.7 -> 6.6, [32768, 8192] 98 -> 80 (6.7 TB/s), [32768, 256] 40 -> 11.5; the error
// against float64 is the rounding to bf16 in both.
// ------------------------------------------------------------------------------------------------
constexpr int SUM_COLS = 64;
__global__ void __launch_bounds__(256)
col_sum_kernel(const __nv_bfloat16* __restrict__ x, int64_t rows, int64_t cols, __nv_bfloat16* __restrict__ out, int first) {
  __shared__ float s_part[32][SUM_COLS + 8];   // rows of 72 floats: 16-byte aligned, conflict-free in both directions
  __shared__ double s_sum[SUM_COLS];
  const int tid = threadIdx.x, c = tid & 7, r = tid >> 3;
  const int64_t blocks = rows / 128, share = gridDim.y;
  const int64_t begin = blocks * blockIdx.y / share * 128, end = blocks * (blockIdx.y + 1) / share * 128;
  chain_start(first);
  const uint4* src = reinterpret_cast<const uint4*>(x + (int64_t)blockIdx.x * SUM_COLS) + c;
  double total[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) total[j] = 0.;
  for (int64_t r0 = begin; r0 < end;) {
    const int64_t stop = end - r0 > 4096 ? r0 + 4096 : end;   // 128 rows per thread
    float sum[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) sum[j] = 0.f;
#pragma unroll 2
    for (; r0 < stop; r0 += 128) {
      float v[4][8];
#pragma unroll
      for (int i = 0; i < 4; ++i) unpack8(chain_load(src + (r0 + 32 * i + r) * (cols / 8)), v[i]);
#pragma unroll
      for (int j = 0; j < 8; ++j) sum[j] += (v[0][j] + v[1][j]) + (v[2][j] + v[3][j]);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) total[j] += (double)sum[j];
  }
  // the 32 threads of a column: fp32 is enough to hand a sum of fewer than 4096 rows on, more go in two parts
#pragma unroll
  for (int part = 0; part < 2; ++part) {
    float* dst = &s_part[r][8 * c];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float hi = (float)total[j];
      dst[j] = hi;
      total[j] = isfinite(hi) ? total[j] - (double)hi : 0.;
    }
    __syncthreads();
    if (tid < SUM_COLS) {
      double t = part ? s_sum[tid] : 0.;
#pragma unroll 8
      for (int k = 0; k < 32; ++k) t += (double)s_part[k][tid];
      s_sum[tid] = t;
    }
    __syncthreads();
    if (end - begin <= 4096) break;   // the sums were fp32
  }
  if (share > 1) cluster_sync_all();
  if (blockIdx.y == 0 && tid < SUM_COLS) {
    double t = s_sum[tid];
    for (uint32_t k = 1; k < share; ++k) {
      double o;
      asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(o) : "r"(map_to_cta((uint32_t)__cvta_generic_to_shared(&s_sum[tid]), k)) : "memory");
      t += o;
    }
    out[(int64_t)blockIdx.x * SUM_COLS + tid] = __float2bfloat16_rn((float)t);
  }
  if (share > 1) cluster_sync_all();   // the others' shared memory stays until it has been read
  chain_wait();
}

// ------------------------------------------------------------------------------------------------
// Row kernel for rows of more than 16384 elements: one CTA per row, two sweeps (the second one hits L1/L2).
// HAD128: the 16 lanes that hold one 128-wide group rotate it with shuffles in both sweeps.
// ------------------------------------------------------------------------------------------------
template <int MODE, bool HAD128>
__global__ void __launch_bounds__(256)
quant_row_kernel(const __nv_bfloat16* __restrict__ x, int64_t cols, int8_t* __restrict__ q,
                 float* __restrict__ scale, int first) {
  __shared__ float s_red[8];
  const int tid = threadIdx.x, l = tid & 31;
  const int64_t row = blockIdx.x;
  const uint4* xr = reinterpret_cast<const uint4*>(x + row * cols);
  const int nchunks = (int)(cols / 8);
  chain_start(first);

  float m = 0.f;
  for (int base = 0; base < nchunks; base += 256) {
    const int ch = base + tid;
    float v[8];
    if (ch < nchunks) unpack8(chain_load(xr + ch), v);
    else {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = 0.f;
    }
    if (HAD128) {
      fwht128_lanes16(v, l);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = round_to_bf16(v[j]);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) m = fmaxf(m, fabsf(v[j]));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (l == 0) s_red[tid >> 5] = m;
  __syncthreads();
  m = s_red[0];
#pragma unroll
  for (int k = 1; k < 8; ++k) m = fmaxf(m, s_red[k]);
  float s, stored;
  make_scale<MODE>(m, s, stored);
  if (tid == 0) scale[row] = stored;

  uint2* qr = reinterpret_cast<uint2*>(q + row * cols);
  for (int base = 0; base < nchunks; base += 256) {
    const int ch = base + tid;
    float v[8];
    if (ch < nchunks) unpack8(chain_load(xr + ch), v);
    else {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = 0.f;
    }
    if (HAD128) {
      fwht128_lanes16(v, l);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = round_to_bf16(v[j]);
    }
    if (ch < nchunks) {
      uint2 o;
      o.x = pack4(quant1<MODE>(v[0], s), quant1<MODE>(v[1], s), quant1<MODE>(v[2], s), quant1<MODE>(v[3], s));
      o.y = pack4(quant1<MODE>(v[4], s), quant1<MODE>(v[5], s), quant1<MODE>(v[6], s), quant1<MODE>(v[7], s));
      qr[ch] = o;
    }
  }
  chain_wait();
}

// Rows of at most 16384 elements: T threads per row (256/T rows per CTA) keep the row in registers, up to
// eight 16-byte pieces each, between the maximum and the quantization: one read, no second sweep through the
// caches, and rows of 4096 elements do not leave half of a CTA idle.  Bound by HBM.  [11008, 4096] 39 -> 29 us,
// [4096, 4096] 19.5 -> 15.4, [28672, 8192] 115.6 -> 109.4 (6.4 TB/s) against two sweeps by one CTA per row.
template <int MODE, int T>
__device__ __forceinline__ void
quant_row_cached_body(unsigned block, const __nv_bfloat16* __restrict__ x, int64_t rows, int64_t cols, int8_t* __restrict__ q,
                        float* __restrict__ scale, int first) {
  __shared__ float s_red[8];
  const int tid = threadIdx.x, l = tid & 31, t = tid & (T - 1);
  const int64_t row = (int64_t)block * (256 / T) + tid / T;
  const bool live = row < rows;
  const uint4* xr = reinterpret_cast<const uint4*>(x + row * cols);
  const int nchunks = live ? (int)(cols / 8) : 0;
  chain_start(first);
  uint4 cache[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) cache[i] = i * T + t < nchunks ? chain_load(xr + i * T + t) : make_uint4(0, 0, 0, 0);
  __nv_bfloat162 hm = __floats2bfloat162_rn(0.f, 0.f);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&cache[i]);
#pragma unroll
    for (int k = 0; k < 4; ++k) hm = __hmax2_nan(hm, __habs2(h[k]));
  }
  float m = __bfloat162float(__hmax_nan(__low2bfloat16(hm), __high2bfloat16(hm)));
  const bool finite = m <= BF16_LARGEST;
  if (!finite) {   // the maximum leaves NaNs out
    hm = __floats2bfloat162_rn(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 8; ++i) hm = absmax8(cache[i], hm);
    m = hmax_of(hm);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (T > 32) {
    if (l == 0) s_red[tid >> 5] = m;
    __syncthreads();
    const float* r = s_red + (tid / T) * (T / 32);
    m = r[0];
#pragma unroll
    for (int k = 1; k < T / 32; ++k) m = fmaxf(m, r[k]);
  }
  float s, stored;
  make_scale<MODE>(m, s, stored);
  if (live && t == 0) scale[row] = stored;
  uint2* qr = reinterpret_cast<uint2*>(q + row * cols);
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if (i * T + t < nchunks) qr[i * T + t] = finite ? quant_piece_finite<MODE>(cache[i], s) : quant_piece<MODE>(cache[i], s);
  chain_wait();
}
template <int MODE, int T>
__global__ void __launch_bounds__(256)
quant_row_cached_kernel(const __nv_bfloat16* __restrict__ x, int64_t rows, int64_t cols, int8_t* __restrict__ q,
                        float* __restrict__ scale, int first) {
  quant_row_cached_body<MODE, T>(blockIdx.x, x, rows, cols, q, scale, first);
}

// The same with the 128-point rotation.  A CTA takes as many whole rows as fit into 128 groups of 128 elements,
// staged like the tiles above, and a thread owns a group: no shuffles, and each group is rotated once.  Bound by
// issue next to HBM.  [11008, 4096] 69 -> 33 us, [28672, 8192] 183 -> 142, [8192, 256] 47 -> 9 against one CTA per
// row with a group in 16 lanes.
template <int MODE>
__global__ void __launch_bounds__(128, 3)
quant_row_rot_kernel(const __nv_bfloat16* __restrict__ x, int64_t rows, int groups, int rows_per_cta, int8_t* __restrict__ q,
                     float* __restrict__ scale, int first) {
  __shared__ __align__(16) uint8_t s_raw[128 * ROT_LD];
  __shared__ __align__(16) uint8_t s_out[128 * OUT_LD];
  __shared__ int s_max[128];
  const int tid = threadIdx.x, my_row = tid / groups;
  const int64_t row0 = (int64_t)blockIdx.x * rows_per_cta;
  const int n_rows = (int)(rows - row0 < rows_per_cta ? rows - row0 : rows_per_cta), n = n_rows * groups;
  chain_start(first);
  const __nv_bfloat16* src = x + row0 * groups * 128 + 8 * tid;   // whole rows are contiguous
  const uint32_t dst = (uint32_t)__cvta_generic_to_shared(s_raw) + (tid >> 4) * ROT_LD + 16 * (tid & 15);
#pragma unroll
  for (int i = 0; i < 16; ++i)
    if (i * 8 + (tid >> 4) < n) cp_async16(dst + i * 8 * ROT_LD, src + i * 1024);
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
  s_max[tid] = 0;
  __syncthreads();
  const bool live = tid < n;
  uint32_t h[64];
  float m = 0.f;
  bool finite = true;
  if (live) {
    float2 p[64];
    load_row128(s_raw + tid * ROT_LD, p);
    m = rot128(p, h);
    finite = m <= BF16_LARGEST;
    if (!finite) m = max_without_nan(h);
    atomicMax(&s_max[my_row], __float_as_int(m));   // |x| >= 0: the bit patterns order like integers
  }
  __syncthreads();
  const int w = tid >> 5, left = n - 32 * w;   // groups of this warp
  if (left > 0) {
    float s, stored;
    make_scale<MODE>(__int_as_float(s_max[live ? my_row : 0]), s, stored);
    if (live && tid == my_row * groups) scale[row0 + my_row] = stored;
    if (!live) {
#pragma unroll
      for (int i = 0; i < 64; ++i) h[i] = 0;   // staged with the rest, not stored
    }
    quant_store128<MODE>(h, s, finite, (uint32_t)__cvta_generic_to_shared(s_out) + w * 32 * OUT_LD, tid & 31,
                         q + (row0 * groups + 32 * w) * 128, 128, left);
  }
  chain_wait();
}

// ------------------------------------------------------------------------------------------------
// Two quantizers in one launch, for operands so small that the launch itself counts (quant_pair): blocks below `split` run the
// first, the others the second.
// ------------------------------------------------------------------------------------------------
struct PairArgs {
  const __nv_bfloat16* x;
  int64_t batch, rows, cols;
  int8_t *q, *qt;
  float *scale, *scale_t;
};
template <int GRAN, int MODE, bool OUT_T> struct TileQuant {
  static unsigned blocks(const PairArgs& a) { return (unsigned)(a.batch * (a.rows / 128) * (a.cols / 128)); }
  static __device__ __forceinline__ void run(const PairArgs& a, unsigned id, int first) {
    const unsigned nx = (unsigned)(a.cols / 128), ny = (unsigned)(a.rows / 128);
    const dim3 block(id % nx, id / nx % ny, id / nx / ny);
    quant_tile_body<GRAN, MODE, true, OUT_T>(block, a.x, a.rows, a.cols, a.q, a.scale, a.qt, a.scale_t, nullptr, first);
  }
};
template <int MODE, int T> struct RowQuant {   // rows of at most 64 T elements
  static unsigned blocks(const PairArgs& a) { return (unsigned)((a.batch * a.rows + 256 / T - 1) / (256 / T)); }
  static __device__ __forceinline__ void run(const PairArgs& a, unsigned id, int first) {
    quant_row_cached_body<MODE, T>(id, a.x, a.batch * a.rows, a.cols, a.q, a.scale, first);
  }
};
template <typename A, typename B>
__global__ void __launch_bounds__(256, 4)
quant_pair_kernel(const PairArgs a, const PairArgs b, unsigned split, int first) {
  if (blockIdx.x < split) A::run(a, blockIdx.x, first);
  else B::run(b, blockIdx.x - split, first);
}

// Whole-row rotation of rows of G groups of 128 (G = 2..128).  A CTA takes 128/G whole rows.  Spans 1..64 run in
// the registers of the thread that owns the group; one exchange through shared memory then gives thread i the
// elements i, i + 128, ... of every row, where the remaining spans run in registers too.  Bytes of four neighbouring
// positions are gathered by two shuffles per word, so that every store fills whole sectors.  Bound by issue and
// latency (20 instructions per element, 12 warps per SM).  Against one CTA per row with a shared-memory pass per
// span: [8192, 4096] 92 -> 45 us, [8192, 8192] 187 -> 80, [8192, 1024] 37 -> 21, [2048, 16384] 116 -> 46.
template <int MODE, bool FINITE>
__device__ __forceinline__ uint32_t quant_word(uint32_t h0, uint32_t h1, float s0, float s1) {
  if (FINITE) return __byte_perm(quant_pair_finite<MODE>(h0, s0), quant_pair_finite<MODE>(h1, s1), 0x5410);
  int q[4];
  quant2<MODE>(make_float2(__uint_as_float(h0 << 16), __uint_as_float(h0 & 0xffff0000u)), make_float2(s0, s0), q[0], q[1]);
  quant2<MODE>(make_float2(__uint_as_float(h1 << 16), __uint_as_float(h1 & 0xffff0000u)), make_float2(s1, s1), q[2], q[3]);
  return pack4(q[0], q[1], q[2], q[3]);
}

constexpr int FULL_LD = 132;   // floats per staged group: 16-byte aligned, conflict-free both ways
constexpr size_t FULL_SMEM = 128 * FULL_LD * sizeof(float);

template <int MODE, int G>
__global__ void __launch_bounds__(128, 3)
quant_row_rotfull_kernel(const __nv_bfloat16* __restrict__ x, int64_t rows, int8_t* __restrict__ q, float* __restrict__ scale,
                         int first) {
  constexpr int R = 128 / G;   // rows per CTA
  extern __shared__ __align__(16) float s_f[];   // [128][FULL_LD]; the bf16 input lies in it first
  __shared__ __nv_bfloat16 s_red[R][4];
  __shared__ float s_scale[R];
  uint8_t* s_raw = reinterpret_cast<uint8_t*>(s_f);
  const int tid = threadIdx.x, w = tid >> 5, l = tid & 31;
  const int64_t row0 = (int64_t)blockIdx.x * R;
  const int n_rows = (int)(rows - row0 < R ? rows - row0 : R), n = n_rows * G;
  chain_start(first);
  {
    const __nv_bfloat16* src = x + row0 * G * 128 + 8 * tid;   // whole rows are contiguous
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(s_raw) + (tid >> 4) * ROT_LD + 16 * (tid & 15);
#pragma unroll
    for (int i = 0; i < 16; ++i)
      if (i * 8 + (tid >> 4) < n) cp_async16(dst + i * 8 * ROT_LD, src + i * 1024);
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
  }
  __syncthreads();
  {
    float2 p[64];
    if (tid < n) {
      load_row128(s_raw + tid * ROT_LD, p);
    } else {   // rows past the end
#pragma unroll
      for (int k = 0; k < 64; ++k) p[k] = make_float2(0.f, 0.f);
    }
    __syncthreads();
    fwht_pairs<64>(p);
    float* out = s_f + tid * FULL_LD;
#pragma unroll
    for (int k = 0; k < 64; k += 4) {
      *reinterpret_cast<float4*>(out + k) = make_float4(__fadd_rn(p[k].x, p[k].y), __fadd_rn(p[k + 1].x, p[k + 1].y),
                                                        __fadd_rn(p[k + 2].x, p[k + 2].y), __fadd_rn(p[k + 3].x, p[k + 3].y));
      *reinterpret_cast<float4*>(out + 64 + k) = make_float4(__fsub_rn(p[k].x, p[k].y), __fsub_rn(p[k + 1].x, p[k + 1].y),
                                                             __fsub_rn(p[k + 2].x, p[k + 2].y), __fsub_rn(p[k + 3].x, p[k + 3].y));
    }
    __syncthreads();
  }
  // h[e / 2] = elements tid of groups e, e + 1 (e counts the groups of all rows), rounded to bf16
  uint32_t h[64];
  __nv_bfloat16 m[R];
  __nv_bfloat162 any = __floats2bfloat162_rn(0.f, 0.f);
  bool finite = true;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    float2 p[G / 2];
#pragma unroll
    for (int g = 0; g < G / 2; ++g) {
      p[g].x = s_f[(r * G + g) * FULL_LD + tid];
      p[g].y = s_f[(r * G + g + G / 2) * FULL_LD + tid];
    }
    fwht_pairs<G / 2>(p);
    __nv_bfloat162 hm = __floats2bfloat162_rn(0.f, 0.f);
    if constexpr (G == 2) {
      // 64 maxima: taken without NaNs at once, the NaNs seen by a second one (replacing them all below spills 144 bytes)
      const __nv_bfloat162 v = __floats2bfloat162_rn(__fadd_rn(p[0].x, p[0].y), __fsub_rn(p[0].x, p[0].y)), a = __habs2(v);
      hm = __hmax2(hm, a);
      any = __hmax2_nan(any, a);
      h[r] = *reinterpret_cast<const uint32_t*>(&v);
      m[r] = __hmax(__low2bfloat16(hm), __high2bfloat16(hm));
    } else {
#pragma unroll
      for (int g = 0; g < G / 2; g += 2) {
        const __nv_bfloat162 lo = __floats2bfloat162_rn(__fadd_rn(p[g].x, p[g].y), __fadd_rn(p[g + 1].x, p[g + 1].y));
        const __nv_bfloat162 hi = __floats2bfloat162_rn(__fsub_rn(p[g].x, p[g].y), __fsub_rn(p[g + 1].x, p[g + 1].y));
        hm = __hmax2_nan(hm, __hmax2_nan(__habs2(lo), __habs2(hi)));
        h[(r * G + g) / 2] = *reinterpret_cast<const uint32_t*>(&lo);
        h[(r * G + g) / 2 + G / 4] = *reinterpret_cast<const uint32_t*>(&hi);
      }
      m[r] = __hmax_nan(__low2bfloat16(hm), __high2bfloat16(hm));
      finite = finite && __bfloat162float(m[r]) <= BF16_LARGEST;
    }
  }
  if constexpr (G == 2) {
    finite = __bfloat162float(__hmax_nan(__low2bfloat16(any), __high2bfloat16(any))) <= BF16_LARGEST;
  } else if (!finite) {   // the maximum leaves NaNs out
#pragma unroll
    for (int r = 0; r < R; ++r) {
      __nv_bfloat162 hm = __floats2bfloat162_rn(0.f, 0.f);
#pragma unroll
      for (int i = 0; i < G / 2; ++i) hm = __hmax2(hm, __habs2(*reinterpret_cast<const __nv_bfloat162*>(&h[r * G / 2 + i])));
      m[r] = __hmax(__low2bfloat16(hm), __high2bfloat16(hm));
    }
  }
#pragma unroll
  for (int r = 0; r < R; r += 2) {   // two rows per shuffle
    __nv_bfloat162 v = __halves2bfloat162(m[r], m[r + 1 < R ? r + 1 : r]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = __hmax2(v, __shfl_xor_sync(0xffffffffu, v, o));
    if (l == 0) {
      s_red[r][w] = __low2bfloat16(v);
      if (r + 1 < R) s_red[r + 1][w] = __high2bfloat16(v);
    }
  }
  __syncthreads();
  if (tid < R) {
    float s, stored;
    const float mm = fmaxf(fmaxf(__bfloat162float(s_red[tid][0]), __bfloat162float(s_red[tid][1])),
                           fmaxf(__bfloat162float(s_red[tid][2]), __bfloat162float(s_red[tid][3])));
    make_scale<MODE>(mm, s, stored);
    s_scale[tid] = s;
    if (tid < n_rows) scale[row0 + tid] = stored;
  }
  __syncthreads();
  int8_t* out = q + row0 * G * 128 + (tid & 3) * 128 + 4 * (tid >> 2);
  auto write = [&](auto finite_c) {
    constexpr bool FINITE = decltype(finite_c)::value;
#pragma unroll
    for (int k = 0; k < 32; ++k) {   // groups 4k..4k+3: one byte each of position tid -> four positions of group 4k + lane % 4
      const uint32_t a = quant_word<MODE, FINITE>(h[2 * k], h[2 * k + 1], s_scale[4 * k / G], s_scale[(4 * k + 2) / G]);
      const uint32_t b = __shfl_xor_sync(0xffffffffu, a, 1);
      const uint32_t c = __byte_perm(a, b, (l & 1) ? 0x3715 : 0x6240);
      const uint32_t d = __shfl_xor_sync(0xffffffffu, c, 2);
      if (4 * k + (tid & 3) < n)
        *reinterpret_cast<uint32_t*>(out + 4 * k * 128) = __byte_perm(c, d, (l & 2) ? 0x3276 : 0x5410);
    }
  };
  if (__all_sync(0xffffffffu, finite)) write(std::true_type{});   // one branch per warp: the shuffles need all lanes
  else write(std::false_type{});
  chain_wait();
}

// Whole-row Hadamard, one CTA per row (few rows, or rows of 32768 elements): the row lives in shared memory as fp32.
// Spans 1..64 run in registers/shuffles, spans >= 128 as shared-memory passes.
template <int MODE>
__global__ void __launch_bounds__(256)
quant_row_hadfull_kernel(const __nv_bfloat16* __restrict__ x, int64_t cols, int8_t* __restrict__ q,
                         float* __restrict__ scale, int first) {
  extern __shared__ float s_row[];
  __shared__ float s_red[8];
  const int tid = threadIdx.x, l = tid & 31;
  const int64_t row = blockIdx.x;
  const uint4* xr = reinterpret_cast<const uint4*>(x + row * cols);
  const int n = (int)cols, nchunks = n / 8;
  chain_start(first);

  for (int base = 0; base < nchunks; base += 256) {
    const int ch = base + tid;
    float v[8];
    if (ch < nchunks) unpack8(chain_load(xr + ch), v);
    else {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = 0.f;
    }
    fwht128_lanes16(v, l);
    if (ch < nchunks) {
      *reinterpret_cast<float4*>(s_row + 8 * ch) = make_float4(v[0], v[1], v[2], v[3]);
      *reinterpret_cast<float4*>(s_row + 8 * ch + 4) = make_float4(v[4], v[5], v[6], v[7]);
    }
  }
  __syncthreads();
  for (int h = 128; h < n; h <<= 1) {
    for (int p = tid; p < n / 2; p += 256) {
      const int i = ((p & ~(h - 1)) << 1) | (p & (h - 1));
      const float a = s_row[i], b = s_row[i + h];
      s_row[i] = __fadd_rn(a, b);
      s_row[i + h] = __fsub_rn(a, b);
    }
    __syncthreads();
  }
  float m = 0.f;
  for (int i = tid; i < n; i += 256) {
    const float r = round_to_bf16(s_row[i]);
    s_row[i] = r;
    m = fmaxf(m, fabsf(r));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (l == 0) s_red[tid >> 5] = m;
  __syncthreads();
  m = s_red[0];
#pragma unroll
  for (int k = 1; k < 8; ++k) m = fmaxf(m, s_red[k]);
  float s, stored;
  make_scale<MODE>(m, s, stored);
  if (tid == 0) scale[row] = stored;
  uint32_t* qr = reinterpret_cast<uint32_t*>(q + row * cols);
  for (int i = tid; i < n / 4; i += 256) {
    const float4 f = *reinterpret_cast<const float4*>(s_row + 4 * i);
    qr[i] = pack4(quant1<MODE>(f.x, s), quant1<MODE>(f.y, s), quant1<MODE>(f.z, s), quant1<MODE>(f.w, s));
  }
  chain_wait();
}

// ------------------------------------------------------------------------------------------------ host
constexpr int MAX_DEVICES = 64;
static int device_ordinal() {
  int dev = 0;
  cudaGetDevice(&dev);
  return (dev < 0 || dev >= MAX_DEVICES) ? 0 : dev;
}
// Raises a kernel's dynamic shared-memory limit once per device (function attributes are per device;
// the call is idempotent, so two threads racing here only repeat it).
template <typename Kernel>
static cudaError_t ensure_smem(Kernel kernel, std::atomic<bool>* done_per_device, size_t bytes) {
  std::atomic<bool>& done = done_per_device[device_ordinal()];
  if (done.load(std::memory_order_acquire)) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess) done.store(true, std::memory_order_release);
  return e;
}

template <int MODE, int G>
static int launch_rotfull(const __nv_bfloat16* x, int64_t rows, int8_t* q, float* scale, cudaStream_t st) {
  static std::atomic<bool> attr_done[MAX_DEVICES];
  I8L_CUDA_OK(ensure_smem(quant_row_rotfull_kernel<MODE, G>, attr_done, FULL_SMEM));
  constexpr int R = 128 / G;
  I8L_CUDA_OK(launch(quant_row_rotfull_kernel<MODE, G>, dim3((unsigned)((rows + R - 1) / R)), 128, FULL_SMEM, st, x, rows, q, scale, chain_first()));
  return I8L_OK;
}
template <int MODE>
static int launch_hadfull(const __nv_bfloat16* x, int64_t rows, int64_t cols, int8_t* q, float* scale, cudaStream_t st) {
  // Few rows do not fill the chip with 128 groups per CTA, and a group per thread is the longer chain: below 3/4 M
  // elements one CTA per row is faster ([512, 256] 7 against 10 us, [1000, 512] 9.4 / 10.2, [1000, 1024] 10.6 / 10.2,
  // [512, 4096] 14.3 / 11.8), and it takes rows of 32768, more groups than a CTA of the other has threads.
  if (rows * cols >= 3ll << 18) switch (cols / 128) {
    case 2: return launch_rotfull<MODE, 2>(x, rows, q, scale, st);
    case 4: return launch_rotfull<MODE, 4>(x, rows, q, scale, st);
    case 8: return launch_rotfull<MODE, 8>(x, rows, q, scale, st);
    case 16: return launch_rotfull<MODE, 16>(x, rows, q, scale, st);
    case 32: return launch_rotfull<MODE, 32>(x, rows, q, scale, st);
    case 64: return launch_rotfull<MODE, 64>(x, rows, q, scale, st);
    case 128: return launch_rotfull<MODE, 128>(x, rows, q, scale, st);
    default: break;
  }
  static std::atomic<bool> attr_done[MAX_DEVICES];
  const size_t smem = (size_t)cols * sizeof(float);
  I8L_CUDA_OK(ensure_smem(quant_row_hadfull_kernel<MODE>, attr_done, 32768 * sizeof(float)));
  I8L_CUDA_OK(launch(quant_row_hadfull_kernel<MODE>, dim3((unsigned)rows), 256, smem, st, x, cols, q, scale, chain_first()));
  return I8L_OK;
}

static int check_dims(int64_t batch, int64_t rows, int64_t cols) {
  if (batch <= 0 || rows <= 0 || cols <= 0 || rows % 128 || cols % 128)
    return fail(I8L_ERR_SHAPE, "batch=%lld rows=%lld cols=%lld: all must be positive and rows, cols multiples of 128",
                (long long)batch, (long long)rows, (long long)cols);
  if (batch > 65535 || rows / 128 > 65535 || rows * cols >= (1ll << 40))
    return fail(I8L_ERR_SHAPE, "shape too large for the launch grid");
  return I8L_OK;
}

template <int GRAN, int MODE, bool OUT_N, bool OUT_T>
static cudaError_t launch_tile(const void* x, int64_t batch, int64_t rows, int64_t cols, int8_t* q, float* scale,
                        int8_t* qt, float* scale_t, const float* colmax, cudaStream_t st) {
  dim3 grid((unsigned)(cols / 128), (unsigned)(rows / 128), (unsigned)batch);
  return launch(quant_tile_kernel<GRAN, MODE, OUT_N, OUT_T>, grid, 256, 0, st, static_cast<const __nv_bfloat16*>(x), rows, cols, q,
                scale, qt, scale_t, colmax, chain_first());
}

template <int GRAN, int MODE>
static int dispatch_tile(const void* x, int64_t batch, int64_t rows, int64_t cols, bool had, int8_t* q,
                         float* scale, int8_t* qt, float* scale_t, const float* colmax, cudaStream_t st) {
  const bool n = q != nullptr, t = qt != nullptr;
  if (had) {  // whatever is wanted of the two orientations, from one read of the tile
    const dim3 grid((unsigned)(cols / 128), (unsigned)(rows / 128), (unsigned)batch);
    const __nv_bfloat16* xp = static_cast<const __nv_bfloat16*>(x);
    if (n && t) I8L_CUDA_OK(launch(quant_tile_rot_kernel<GRAN, MODE, true, true>, grid, 128, 0, st, xp, rows, cols, q, scale, qt, scale_t, nullptr, chain_first()));
    else if (n) I8L_CUDA_OK(launch(quant_tile_rot_kernel<GRAN, MODE, true, false>, grid, 128, 0, st, xp, rows, cols, q, scale, nullptr, nullptr, nullptr, chain_first()));
    else I8L_CUDA_OK(launch(quant_tile_rot_kernel<GRAN, MODE, false, true>, grid, 128, 0, st, xp, rows, cols, nullptr, nullptr, qt, scale_t, nullptr, chain_first()));
  } else if (GRAN == I8L_GRAN_TILE128) {
    if (n && t) I8L_CUDA_OK((launch_tile<GRAN, MODE, true, true>(x, batch, rows, cols, q, scale, qt, scale_t, colmax, st)));
    else if (n) I8L_CUDA_OK((launch_tile<GRAN, MODE, true, false>(x, batch, rows, cols, q, scale, qt, scale_t, colmax, st)));
    else I8L_CUDA_OK((launch_tile<GRAN, MODE, false, true>(x, batch, rows, cols, q, scale, qt, scale_t, colmax, st)));
  } else {  // grouped scales differ between the two orientations: one launch each
    if (n) I8L_CUDA_OK((launch_tile<GRAN, MODE, true, false>(x, batch, rows, cols, q, scale, nullptr, nullptr, colmax, st)));
    if (t) I8L_CUDA_OK((launch_tile<GRAN, MODE, false, true>(x, batch, rows, cols, nullptr, nullptr, qt, scale_t, colmax, st)));
  }
  return I8L_OK;
}

}  // namespace i8l

using namespace i8l;

namespace i8l {
template <typename A, typename B>
static int launch_pair(const PairArgs& a, const PairArgs& b, cudaStream_t st) {
  const unsigned split = A::blocks(a);
  const cudaError_t e = launch(quant_pair_kernel<A, B>, dim3(split + B::blocks(b)), 256, 0, st, a, b, split, chain_first());
  return e == cudaSuccess ? 1 : fail(I8L_ERR_CUDA, "quant_pair: %s", cudaGetErrorString(e));
}

// Both operands of a product in one launch.  1: done, 0: not a pair that this takes, < 0: an error.  It pays where a call is
// bound by its launches: M, N, K 128, 1024, 1024 forward 15.5 -> 13.0 us, 512, 1024, 1024 11.3 -> 9.4, 1024, 2048, 1024
// 11.4 -> 10.3 a call; 1024, 1024, 2048 12.0 -> 11.8; 2048, 2048, 1024 12.7 -> 12.9; 1024, 1024, 3072 14.8 -> 15.2; 2048,
// 1536, 2048 16.7 -> 17.3.  The line lies at 1.5 M elements of either operand, which is on the safe side: of these shapes it leaves
// the two launches to 1024, 2048, 1024 too.  A line on the sum of both has not been measured at few tokens and wide weights.
int quant_pair(const void* a, int64_t a_batch, int64_t a_rows, int a_gran, int8_t* aq, float* as, int8_t* aqt, float* ast, const void* b,
               int64_t b_batch, int64_t b_rows, int b_gran, int8_t* bq, float* bs, int64_t cols, int qmode, int hadamard,
               cudaStream_t st) {
  constexpr int64_t MOST = 3ll << 19;
  if (hadamard != I8L_HAD_NONE || cols > 4096 || a_batch * a_rows * cols > MOST || b_batch * b_rows * cols > MOST || !a || !b || !aligned16(a) || !aligned16(b) ||
      !aligned16(aqt))
    return 0;
  if (int e = check_arch()) return e;
  const PairArgs pa{static_cast<const __nv_bfloat16*>(a), a_batch, a_rows, cols, aq, aqt, as, ast};
  const PairArgs pb{static_cast<const __nv_bfloat16*>(b), b_batch, b_rows, cols, bq, nullptr, bs, nullptr};
  const bool t = aqt != nullptr;
#define I8L_PAIR(...) return launch_pair<__VA_ARGS__>(pa, pb, st)
#define I8L_TILE_ROW(G, Mo, TT)                                                               \
  if (a_gran == G && b_gran == I8L_GRAN_ROW && qmode == Mo && t == TT) {                      \
    if (cols <= 2048) I8L_PAIR(TileQuant<G, Mo, TT>, RowQuant<Mo, 32>);                \
    I8L_PAIR(TileQuant<G, Mo, TT>, RowQuant<Mo, 64>);                                  \
  }
  I8L_TILE_ROW(I8L_GRAN_TILE128, I8L_QMODE_TRITON, false)
  I8L_TILE_ROW(I8L_GRAN_TILE128, I8L_QMODE_TRITON, true)
  I8L_TILE_ROW(I8L_GRAN_GROUP128, I8L_QMODE_RNE, false)
  if (t) return 0;
  if (a_gran == I8L_GRAN_ROW && b_gran == I8L_GRAN_ROW && qmode == I8L_QMODE_ROWRCP) {
    if (cols <= 2048) I8L_PAIR(RowQuant<I8L_QMODE_ROWRCP, 32>, RowQuant<I8L_QMODE_ROWRCP, 32>);
    I8L_PAIR(RowQuant<I8L_QMODE_ROWRCP, 64>, RowQuant<I8L_QMODE_ROWRCP, 64>);
  }
#define I8L_TILE_TILE(G, H, Mo) \
  if (a_gran == G && b_gran == H && qmode == Mo) I8L_PAIR(TileQuant<G, Mo, false>, TileQuant<H, Mo, false>);
  I8L_TILE_TILE(I8L_GRAN_TILE128, I8L_GRAN_TILE128, I8L_QMODE_TRITON)
  I8L_TILE_TILE(I8L_GRAN_TILE128, I8L_GRAN_TILE128, I8L_QMODE_FUSED)
  I8L_TILE_TILE(I8L_GRAN_TILE128, I8L_GRAN_GROUP128, I8L_QMODE_FUSED)
#undef I8L_TILE_TILE
#undef I8L_TILE_ROW
#undef I8L_PAIR
  return 0;
}
}  // namespace i8l

extern "C" const char* i8l_last_error(void) { return g_err; }
extern "C" int i8l_version(void) { return 100; }

extern "C" int i8l_quant_tile(const void* x, int64_t batch, int64_t rows, int64_t cols, int gran, int qmode,
                              int hadamard, int8_t* q, float* scale, int8_t* qt, float* scale_t, void* stream) {
  if (int e = check_dims(batch, rows, cols)) return e;
  if (!x || (!q && !qt) || (q && !scale) || (qt && !scale_t)) return fail(I8L_ERR_ARG, "null pointer");
  if (!aligned16(x) || !aligned16(q) || !aligned16(qt)) return fail(I8L_ERR_ALIGN, "x, q, qt must be 16-byte aligned");
  if (hadamard != I8L_HAD_NONE && hadamard != I8L_HAD_128)
    return fail(I8L_ERR_ARG, "i8l_quant_tile: hadamard must be NONE or 128");
  if (int e = check_arch()) return e;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool had = hadamard == I8L_HAD_128;
  if (gran == I8L_GRAN_TILE128X256) {
    if (cols % 256 || had || qt || !q) return fail(I8L_ERR_ARG, "i8l_quant_tile: 128x256 groups need cols %% 256 == 0, no rotation, q only");
    const dim3 grid((unsigned)(cols / 256), (unsigned)(rows / 128), (unsigned)batch);
    const __nv_bfloat16* xp = static_cast<const __nv_bfloat16*>(x);
    if (qmode == I8L_QMODE_TRITON) I8L_CUDA_OK(launch(quant_tile256_kernel<I8L_QMODE_TRITON>, grid, 256, 0, st, xp, rows, cols, q, scale, chain_first()));
    else if (qmode == I8L_QMODE_TRITON_BF16S) I8L_CUDA_OK(launch(quant_tile256_kernel<I8L_QMODE_TRITON_BF16S>, grid, 256, 0, st, xp, rows, cols, q, scale, chain_first()));
    else return fail(I8L_ERR_ARG, "i8l_quant_tile: 128x256 groups support qmode TRITON and TRITON_BF16S");
    return I8L_OK;
  }
#define I8L_TILE_CASE(G, Mo) \
  if (gran == G && qmode == Mo) return dispatch_tile<G, Mo>(x, batch, rows, cols, had, q, scale, qt, scale_t, nullptr, st);
  I8L_TILE_CASE(I8L_GRAN_TILE128, I8L_QMODE_TRITON)
  I8L_TILE_CASE(I8L_GRAN_TILE128, I8L_QMODE_RNE)
  I8L_TILE_CASE(I8L_GRAN_TILE128, I8L_QMODE_FUSED)
  I8L_TILE_CASE(I8L_GRAN_GROUP128, I8L_QMODE_TRITON)
  I8L_TILE_CASE(I8L_GRAN_GROUP128, I8L_QMODE_RNE)
  I8L_TILE_CASE(I8L_GRAN_GROUP128, I8L_QMODE_FUSED)
#undef I8L_TILE_CASE
  return fail(I8L_ERR_ARG, "i8l_quant_tile: unsupported gran=%d qmode=%d", gran, qmode);
}

extern "C" int i8l_quant_row(const void* x, int64_t rows, int64_t cols, int qmode, int hadamard, int8_t* q,
                             float* scale, void* stream) {
  if (rows <= 0 || cols <= 0 || cols % 128 || rows > 0x7fffffffll || cols > (1 << 20))
    return fail(I8L_ERR_SHAPE, "rows=%lld cols=%lld: need rows>0, cols a positive multiple of 128",
                (long long)rows, (long long)cols);
  if (!x || !q || !scale) return fail(I8L_ERR_ARG, "null pointer");
  if (!aligned16(x) || !aligned16(q)) return fail(I8L_ERR_ALIGN, "x, q must be 16-byte aligned");
  if (int e = check_arch()) return e;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const __nv_bfloat16* xp = static_cast<const __nv_bfloat16*>(x);
  if (hadamard == I8L_HAD_FULL) {
    if ((cols & (cols - 1)) || cols > 32768)
      return fail(I8L_ERR_SHAPE, "full Hadamard needs cols a power of two <= 32768, got %lld", (long long)cols);
    if (cols > 128) {
      if (qmode == I8L_QMODE_TRITON) return launch_hadfull<I8L_QMODE_TRITON>(xp, rows, cols, q, scale, st);
      if (qmode == I8L_QMODE_RNE) return launch_hadfull<I8L_QMODE_RNE>(xp, rows, cols, q, scale, st);
      if (qmode == I8L_QMODE_ROWRCP) return launch_hadfull<I8L_QMODE_ROWRCP>(xp, rows, cols, q, scale, st);
      return fail(I8L_ERR_ARG, "i8l_quant_row: unsupported qmode=%d", qmode);
    }
    if (qmode != I8L_QMODE_TRITON && qmode != I8L_QMODE_RNE && qmode != I8L_QMODE_ROWRCP)
      return fail(I8L_ERR_ARG, "i8l_quant_row: unsupported qmode=%d", qmode);
    hadamard = I8L_HAD_128;   // a row of 128 is one group
  }
  if (hadamard != I8L_HAD_NONE && hadamard != I8L_HAD_128) return fail(I8L_ERR_ARG, "bad hadamard=%d", hadamard);
  // Rows of up to 16384 elements stay on chip; longer ones are swept twice.  Threads per row: the fewest that hold
  // it in eight pieces each.
  const int groups = (int)(cols / 128), rpc = 128 / groups;
#define I8L_ROW_T(Mo, T) \
  launch(quant_row_cached_kernel<Mo, T>, dim3((unsigned)((rows + 256 / T - 1) / (256 / T))), 256, 0, st, xp, rows, cols, q, scale, chain_first())
#define I8L_ROW_CASE(Mo)                                                                                      \
  if (qmode == Mo) {                                                                                          \
    I8L_CUDA_OK(                                                                                              \
        hadamard && rpc ? launch(quant_row_rot_kernel<Mo>, dim3((unsigned)((rows + rpc - 1) / rpc)), 128, 0, st, xp, rows, groups, \
                                 rpc, q, scale, chain_first())                                                \
        : hadamard      ? launch(quant_row_kernel<Mo, true>, dim3((unsigned)rows), 256, 0, st, xp, cols, q, scale, chain_first()) \
        : cols <= 2048  ? I8L_ROW_T(Mo, 32)                                                                   \
        : cols <= 4096  ? I8L_ROW_T(Mo, 64)                                                                   \
        : cols <= 8192  ? I8L_ROW_T(Mo, 128)                                                                  \
        : cols <= 16384 ? I8L_ROW_T(Mo, 256)                                                                  \
                        : launch(quant_row_kernel<Mo, false>, dim3((unsigned)rows), 256, 0, st, xp, cols, q, scale, chain_first())); \
    return I8L_OK;                                                                                            \
  }
  I8L_ROW_CASE(I8L_QMODE_TRITON)
  I8L_ROW_CASE(I8L_QMODE_RNE)
  I8L_ROW_CASE(I8L_QMODE_ROWRCP)
  I8L_ROW_CASE(I8L_QMODE_TRITON_BF16S)
#undef I8L_ROW_CASE
#undef I8L_ROW_T
  return fail(I8L_ERR_ARG, "i8l_quant_row: unsupported qmode=%d", qmode);
}

__global__ void __launch_bounds__(1024) clear_kernel(float* __restrict__ ptr, int64_t n) {
  chain_start(1);   // a kernel ahead of it may still read what it clears
  const int64_t i = (int64_t)blockIdx.x * 1024 + threadIdx.x;
  if (i < n) ptr[i] = 0.f;
}

// CTAs that share a strip of `blocks` blocks of 128 rows.
static int col_strip_share(int64_t blocks) { return blocks >= 8 ? 8 : blocks >= 4 ? 4 : blocks >= 2 ? 2 : 1; }
template <int MODE, int BLOCKS>
static int launch_col_strip(const __nv_bfloat16* x, int64_t rows, int64_t cols, int8_t* qt, float* scale_t, cudaStream_t st) {
  static std::atomic<bool> attr_done[MAX_DEVICES];
  I8L_CUDA_OK(ensure_smem(quant_col_strip_kernel<MODE, BLOCKS>, attr_done, COLT_SMEM<BLOCKS>));
  const unsigned share = (unsigned)col_strip_share(rows / 128);
  if (rows / 128 > (int64_t)share * BLOCKS) return fail(I8L_ERR_SHAPE, "a column of %lld elements does not fit on chip", (long long)rows);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attrs[2];
  cfg.gridDim = dim3((unsigned)(cols / COLT_COLS), share, 1);
  cfg.blockDim = dim3(256, 1, 1);
  cfg.dynamicSmemBytes = COLT_SMEM<BLOCKS>;
  cfg.stream = st;
  attrs[0].id = cudaLaunchAttributeClusterDimension;
  attrs[0].val.clusterDim.x = 1;
  attrs[0].val.clusterDim.y = share;
  attrs[0].val.clusterDim.z = 1;
  cfg.attrs = attrs;
  cfg.numAttrs = 1;
  chain_attribute(cfg, attrs);
  I8L_CUDA_OK(cudaLaunchKernelEx(&cfg, quant_col_strip_kernel<MODE, BLOCKS>, x, rows, cols, qt, scale_t, chain_first()));
  return I8L_OK;
}

// One scale per column: in one pass (col_t_in_one_pass), or a pass for the maxima, from a colmax of zeros, and one to quantize.
template <int MODE>
static int launch_col_t(const void* x, int64_t rows, int64_t cols, bool rot, int8_t* qt, float* scale_t, float* colmax,
                        cudaStream_t st) {
  const __nv_bfloat16* xp = static_cast<const __nv_bfloat16*>(x);
  const dim3 grid((unsigned)(cols / 128), (unsigned)(rows / 128), 1);
  if (rot) {
    I8L_CUDA_OK(launch(quant_tile_rot_kernel<GRAN_COLMAX_PASS, MODE, false, true>, grid, 128, 0, st, xp, rows, cols, nullptr, nullptr,
                       nullptr, nullptr, colmax, chain_first()));
    I8L_CUDA_OK(launch(quant_tile_rot_kernel<GRAN_COLFULL, MODE, false, true>, grid, 128, 0, st, xp, rows, cols, nullptr, nullptr, qt,
                       scale_t, colmax, chain_first()));
  } else if (i8l::col_t_in_one_pass(rows, rot)) {
    const int64_t blocks = rows / 128;
    return blocks == col_strip_share(blocks) ? launch_col_strip<MODE, 1>(xp, rows, cols, qt, scale_t, st)
                                             : launch_col_strip<MODE, 4>(xp, rows, cols, qt, scale_t, st);
  } else {
    I8L_CUDA_OK(launch(col_absmax_kernel, grid, 256, 0, st, xp, rows, cols, colmax, chain_first()));
    I8L_CUDA_OK((launch_tile<GRAN_COLFULL, MODE, false, true>(x, 1, rows, cols, nullptr, nullptr, qt, scale_t, colmax, st)));
  }
  return I8L_OK;
}

namespace i8l {
bool col_t_in_one_pass(int64_t rows, bool rot) { return !rot && rows <= 8 * 4 * 128; }
int col_sum(const void* x, int64_t rows, int64_t cols, void* out, cudaStream_t st) {
  if (rows <= 0 || cols <= 0 || rows % 128 || cols % 128 || cols / SUM_COLS > 0x7fffffffll)
    return fail(I8L_ERR_SHAPE, "rows=%lld cols=%lld: positive multiples of 128", (long long)rows, (long long)cols);
  if (!x || !out) return fail(I8L_ERR_ARG, "null pointer");
  if (!aligned16(x)) return fail(I8L_ERR_ALIGN, "x must be 16-byte aligned");
  if (int e = check_arch()) return e;
  // a strip of 64 columns on 1 to 8 CTAs, for two on each SM, but no fewer than 512 rows each
  const int64_t strips = cols / SUM_COLS;
  int share = 1;
  while (share < 8 && strips * share < 2 * sm_count() && rows >= 1024 * share) share *= 2;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attrs[2];
  cfg.gridDim = dim3((unsigned)strips, (unsigned)share, 1);
  cfg.blockDim = dim3(256, 1, 1);
  cfg.stream = st;
  attrs[0].id = cudaLaunchAttributeClusterDimension;
  attrs[0].val.clusterDim.x = 1;
  attrs[0].val.clusterDim.y = (unsigned)share;
  attrs[0].val.clusterDim.z = 1;
  cfg.attrs = attrs;
  cfg.numAttrs = 1;
  chain_attribute(cfg, attrs);
  I8L_CUDA_OK(cudaLaunchKernelEx(&cfg, col_sum_kernel, static_cast<const __nv_bfloat16*>(x), rows, cols, static_cast<__nv_bfloat16*>(out), chain_first()));
  return I8L_OK;
}
int clear(float* ptr, int64_t n, cudaStream_t st) {   // a kernel and not a memset, which would break the chain
  I8L_CUDA_OK(launch(clear_kernel, dim3((unsigned)((n + 1023) / 1024)), 1024, 0, st, ptr, n));
  chain_state.wait = 1;
  return I8L_OK;
}
int quant_col_t(const char* name, const void* x, int64_t rows, int64_t cols, int qmode, bool rot, int8_t* qt, float* scale_t,
                float* colmax, bool zeroed, cudaStream_t st) {
  if (int e = check_dims(1, rows, cols)) return e;
  if (!x || !qt || !scale_t || !colmax) return fail(I8L_ERR_ARG, "null pointer");
  if (!aligned16(x) || !aligned16(qt)) return fail(I8L_ERR_ALIGN, "x, qt must be 16-byte aligned");
  if (int e = check_arch()) return e;
  if (!zeroed && !col_t_in_one_pass(rows, rot))
    if (int e = clear(colmax, cols, st)) return e;
  if (qmode == I8L_QMODE_TRITON) return launch_col_t<I8L_QMODE_TRITON>(x, rows, cols, rot, qt, scale_t, colmax, st);
  if (qmode == I8L_QMODE_RNE) return launch_col_t<I8L_QMODE_RNE>(x, rows, cols, rot, qt, scale_t, colmax, st);
  if (qmode == I8L_QMODE_ROWRCP) return launch_col_t<I8L_QMODE_ROWRCP>(x, rows, cols, rot, qt, scale_t, colmax, st);
  return fail(I8L_ERR_ARG, "%s: unsupported qmode=%d", name, qmode);
}
}  // namespace i8l

extern "C" int i8l_col_sum(const void* x, int64_t rows, int64_t cols, void* out, void* stream) {
  return col_sum(x, rows, cols, out, static_cast<cudaStream_t>(stream));
}

extern "C" int i8l_quant_col_t(const void* x, int64_t rows, int64_t cols, int qmode, int8_t* qt, float* scale_t,
                               float* colmax_scratch, void* stream) {
  return quant_col_t("i8l_quant_col_t", x, rows, cols, qmode, false, qt, scale_t, colmax_scratch, false, static_cast<cudaStream_t>(stream));
}

extern "C" int i8l_quant_col_t_rot(const void* x, int64_t rows, int64_t cols, int qmode, int8_t* qt, float* scale_t,
                                   float* colmax_scratch, void* stream) {
  return quant_col_t("i8l_quant_col_t_rot", x, rows, cols, qmode, true, qt, scale_t, colmax_scratch, false, static_cast<cudaStream_t>(stream));
}

// ------------------------------------------------------------------------------------------------
// Allocation-free variant of i8l_quant_col_t: the column-absmax scratch lives in a file-scope device
// array instead of caller memory.  In host code `g_colmax_static` is only a stand-in symbol, not a
// device address; the real address is looked up once per device with cudaGetSymbolAddress (with
// that device current) and cached.
// ------------------------------------------------------------------------------------------------
static __device__ __align__(256) float g_colmax_static[I8L_STATIC_SCRATCH_MAX_COLS];
static std::atomic<float*> g_colmax_static_addr[MAX_DEVICES];  // per device ordinal, nullptr = not looked up yet

extern "C" int i8l_quant_col_t_static(const void* x, int64_t rows, int64_t cols, int qmode, int8_t* qt,
                                      float* scale_t, void* stream) {
  if (cols > I8L_STATIC_SCRATCH_MAX_COLS)
    return fail(I8L_ERR_SHAPE, "i8l_quant_col_t_static: cols=%lld exceeds the built-in scratch of %d columns; "
                "use i8l_quant_col_t with caller-provided scratch", (long long)cols, I8L_STATIC_SCRATCH_MAX_COLS);
  // the same argument and device checks as i8l_quant_col_t, before the symbol query
  if (int e = check_dims(1, rows, cols)) return e;
  if (!x || !qt || !scale_t) return fail(I8L_ERR_ARG, "null pointer");
  if (!aligned16(x) || !aligned16(qt)) return fail(I8L_ERR_ALIGN, "x, qt must be 16-byte aligned");
  if (int e = check_arch()) return e;
  int dev = 0;
  I8L_CUDA_OK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= MAX_DEVICES) return fail(I8L_ERR_ARG, "device ordinal %d out of range", dev);
  float* ptr = g_colmax_static_addr[dev].load(std::memory_order_acquire);
  if (!ptr) {
    I8L_CUDA_OK(cudaGetSymbolAddress(reinterpret_cast<void**>(&ptr), g_colmax_static));
    g_colmax_static_addr[dev].store(ptr, std::memory_order_release);
  }
  return i8l_quant_col_t(x, rows, cols, qmode, qt, scale_t, ptr, stream);
}
