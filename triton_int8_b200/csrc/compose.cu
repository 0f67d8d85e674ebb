// Whole products of the library behind one call: quantize both operands into a caller-provided workspace and
// multiply.  Host code only; every step is the entry point of the same name, with its checks and launches.  One call
// from Python instead of three, and one allocation instead of four, is what small problems are bound by.
#include "common.cuh"

using namespace i8l;

namespace {

constexpr int64_t ALIGN = 256;
int64_t padded(int64_t bytes) { return (bytes + ALIGN - 1) / ALIGN * ALIGN; }

// Carves 256-byte aligned pieces out of the workspace.
struct Carver {
  char* p;
  char* end;
  bool short_of_space = false;
  template <typename T> T* take(int64_t count) {
    const int64_t bytes = padded(count * (int64_t)sizeof(T));
    if (bytes > end - p) { short_of_space = true; return nullptr; }
    T* r = reinterpret_cast<T*>(p);
    p += bytes;
    return r;
  }
};

int64_t scale_count(int gran, int64_t batch, int64_t rows, int64_t cols) {
  switch (gran) {
    case I8L_GRAN_TILE128: return batch * (rows / 128) * (cols / 128);
    case I8L_GRAN_TILE128X256: return batch * (rows / 128) * (cols / 256);
    case I8L_GRAN_GROUP128: return batch * rows * (cols / 128);
    default: return batch * rows;
  }
}
int a_kind_of(int gran) {
  return gran == I8L_GRAN_TILE128 ? I8L_ASCALE_TILE : (gran == I8L_GRAN_TILE128X256 ? I8L_ASCALE_TILE256 : I8L_ASCALE_GROUP);
}
int b_kind_of(int gran) {
  return gran == I8L_GRAN_ROW ? I8L_BSCALE_CHANNEL : (gran == I8L_GRAN_TILE128 ? I8L_BSCALE_TILE : I8L_BSCALE_GROUP);
}
int quant(const void* x, int64_t batch, int64_t rows, int64_t cols, int gran, int qmode, int had, int8_t* q, float* s,
          void* stream) {
  if (gran == I8L_GRAN_ROW) return i8l_quant_row(x, batch * rows, cols, qmode, had, q, s, stream);
  return i8l_quant_tile(x, batch, rows, cols, gran, qmode, had, q, s, nullptr, nullptr, stream);
}
int quant_col_t(const void* x, int64_t rows, int64_t cols, int qmode, int had, int8_t* qt, float* st, float* scratch,
                bool zeroed, void* stream) {
  if (had != I8L_HAD_128 && had != I8L_HAD_NONE)
    return fail(I8L_ERR_ARG, "a transposed operand is rotated in 128-wide groups or not at all");
  return i8l::quant_col_t("quant_col_t", x, rows, cols, qmode, had == I8L_HAD_128, qt, st, scratch, zeroed,
                          static_cast<cudaStream_t>(stream));
}
// Before sizes are multiplied (batch * rows * K must fit 64 bits): the entry points below check the rest, with the limits
// of their own grids.  batch * M and batch * N fit 31 bits wherever a GEMM accepts them.
int check_extents(int64_t batch, int64_t M, int64_t N, int64_t K) {
  constexpr int64_t LIM = 1ll << 31;
  if (batch <= 0 || M <= 0 || N <= 0 || K <= 0 || M % 128 || N % 128 || K % 128 || batch >= LIM || M >= LIM || N >= LIM ||
      K >= LIM || batch * M >= LIM || batch * N >= LIM)
    return fail(I8L_ERR_SHAPE, "batch=%lld M=%lld N=%lld K=%lld: all positive, M, N, K multiples of 128", (long long)batch,
                (long long)M, (long long)N, (long long)K);
  return I8L_OK;
}

}  // namespace

extern "C" int i8l_quant_gemm(const void* a, const void* b, const void* bias, void* c, int8_t* a_qt, float* a_st,
                              int64_t batch, int64_t M, int64_t N, int64_t K, int b_batched, int a_gran, int b_gran,
                              int qmode, int hadamard, float post_scale, int flags, void* workspace,
                              int64_t workspace_bytes, int32_t* status, void* stream) {
  if (int e = check_extents(batch, M, N, K)) return e;
  if ((a_gran == I8L_GRAN_ROW && b_gran != I8L_GRAN_ROW) || b_gran == I8L_GRAN_TILE128X256)
    return fail(I8L_ERR_ARG, "i8l_quant_gemm: per-row scales of A need per-row scales of B, 128x256 groups are for A");
  if (!workspace || (a_qt && (!a_st || batch != 1))) return fail(I8L_ERR_ARG, "i8l_quant_gemm: bad pointers");
  const int64_t b_n = b_batched ? batch : 1;
  Carver ws{static_cast<char*>(workspace), static_cast<char*>(workspace) + workspace_bytes};
  int8_t* aq = ws.take<int8_t>(batch * M * K);
  int8_t* bq = ws.take<int8_t>(b_n * N * K);
  float* as = ws.take<float>(scale_count(a_gran, batch, M, K));
  float* bs = ws.take<float>(scale_count(b_gran, b_n, N, K));
  float* colmax = a_qt && a_gran == I8L_GRAN_ROW ? ws.take<float>(K) : nullptr;
  if (ws.short_of_space) return fail(I8L_ERR_ARG, "i8l_quant_gemm: workspace of %lld bytes is too small", (long long)workspace_bytes);
  if (!aligned16(workspace)) return fail(I8L_ERR_ALIGN, "i8l_quant_gemm: the workspace must be aligned");   // every piece then is
  const LaunchChain chain(static_cast<cudaStream_t>(stream));
  if (colmax) {   // ahead of the GEMM, while A is in L2
    if (int e = quant_col_t(a, M, K, qmode, hadamard, a_qt, a_st, colmax, false, stream)) return e;
  }
  const bool grouped_t = a_qt && a_gran == I8L_GRAN_GROUP128;   // needs launches of its own
  const int paired = grouped_t ? 0
                               : quant_pair(a, batch, M, a_gran, aq, as, colmax ? nullptr : a_qt, a_st, b, b_n, N, b_gran, bq, bs, K, qmode,
                                            hadamard, static_cast<cudaStream_t>(stream));
  if (paired < 0) return paired;
  if (paired) {
  } else if (a_qt && a_gran != I8L_GRAN_ROW) {   // both orientations of A from one call
    if (int e = i8l_quant_tile(a, batch, M, K, a_gran, qmode, hadamard, aq, as, a_qt, a_st, stream)) return e;
  } else {
    if (int e = quant(a, batch, M, K, a_gran, qmode, hadamard, aq, as, stream)) return e;
  }
  if (!paired)
    if (int e = quant(b, b_n, N, K, b_gran, qmode, hadamard, bq, bs, stream)) return e;
  if (a_gran == I8L_GRAN_ROW)
    return i8l_gemm_rowcol(aq, bq, as, bs, b_batched, bias, post_scale, c, batch, M, N, K, flags, status, stream);
  return i8l_gemm_block(aq, bq, as, bs, a_kind_of(a_gran), b_kind_of(b_gran), b_batched, bias, post_scale, c, batch, M, N, K,
                        flags, status, stream);
}

extern "C" int i8l_linear_backward(const void* dy, const void* w, const int8_t* x_qt, const float* x_st, void* dx, void* dw,
                                   int64_t M, int64_t N, int64_t K, int gran, int qmode, int hadamard, float post_dx,
                                   float post_dw, int flags, void* workspace, int64_t workspace_bytes, int32_t* status,
                                   void* stream) {
  return i8l_linear_backward_bias(dy, w, x_qt, x_st, dx, dw, nullptr, M, N, K, gran, qmode, hadamard, post_dx, post_dw, flags,
                                  workspace, workspace_bytes, status, stream);
}

extern "C" int i8l_linear_backward_bias(const void* dy, const void* w, const int8_t* x_qt, const float* x_st, void* dx, void* dw,
                                        void* db, int64_t M, int64_t N, int64_t K, int gran, int qmode, int hadamard,
                                        float post_dx, float post_dw, int flags, void* workspace, int64_t workspace_bytes,
                                        int32_t* status, void* stream) {
  if (int e = check_extents(1, M, N, K)) return e;
  if (!workspace || (dw && (!x_qt || !x_st))) return fail(I8L_ERR_ARG, "i8l_linear_backward: bad pointers");
  if (gran == I8L_GRAN_TILE128X256) return fail(I8L_ERR_ARG, "i8l_linear_backward: unsupported gran=%d", gran);
  const bool whole_k = gran == I8L_GRAN_ROW;
  Carver ws{static_cast<char*>(workspace), static_cast<char*>(workspace) + workspace_bytes};
  int8_t *dyq = nullptr, *dyqt = nullptr, *wqt = nullptr;
  float *dys = nullptr, *dyst = nullptr, *wst = nullptr;
  if (dx) {
    dyq = ws.take<int8_t>(M * N);
    dys = ws.take<float>(scale_count(gran, 1, M, N));
    // dw [N, K] is written after dx has used w^T: its memory holds w^T meanwhile, and the peak is not above that of
    // separate calls, which free w^T ahead of dw (32768 x 8192 x 28672: 0.24 GB)
    wqt = dw ? static_cast<int8_t*>(dw) : ws.take<int8_t>(K * N);
    wst = ws.take<float>(K);
  }
  if (dw) {
    dyqt = ws.take<int8_t>(N * M);
    dyst = ws.take<float>(scale_count(gran, 1, N, M));
  }
  float* colmax = ws.take<float>(K > N ? K : N);
  if (ws.short_of_space) return fail(I8L_ERR_ARG, "i8l_linear_backward: workspace of %lld bytes is too small", (long long)workspace_bytes);
  if ((dx || dw) && !aligned16(workspace)) return fail(I8L_ERR_ALIGN, "i8l_linear_backward: the workspace must be aligned");
  const LaunchChain chain(static_cast<cudaStream_t>(stream));
  // The column maxima of W start from zeros; cleared up front, where no other pass needs the scratch, the first maximum
  // pass does not have to wait for it.
  const bool zeroed = dx && !whole_k && !col_t_in_one_pass(N, hadamard == I8L_HAD_128);
  if (zeroed) {
    if (int e = check_arch()) return e;
    if (int e = clear(colmax, K, static_cast<cudaStream_t>(stream))) return e;
  }
  if (db)
    if (int e = col_sum(dy, M, N, db, static_cast<cudaStream_t>(stream))) return e;
  if (whole_k) {
    if (dx)
      if (int e = i8l_quant_row(dy, M, N, qmode, hadamard, dyq, dys, stream)) return e;
    if (dw)
      if (int e = quant_col_t(dy, M, N, qmode, hadamard, dyqt, dyst, colmax, false, stream)) return e;
  } else if (dx || dw) {
    if (int e = i8l_quant_tile(dy, 1, M, N, gran, qmode, hadamard, dyq, dys, dyqt, dyst, stream)) return e;
  }
  if (dx) {   // dX = dY W, contraction over N
    if (int e = quant_col_t(w, N, K, qmode, hadamard, wqt, wst, colmax, zeroed, stream)) return e;
    chain_state.gemm_next = dw != nullptr;
    const int e = whole_k ? i8l_gemm_rowcol(dyq, wqt, dys, wst, 0, nullptr, post_dx, dx, 1, M, K, N, flags, status, stream)
                          : i8l_gemm_block(dyq, wqt, dys, wst, a_kind_of(gran), I8L_BSCALE_CHANNEL, 0, nullptr, post_dx, dx, 1, M,
                                           K, N, flags, status, stream);
    if (e) return e;
  }
  if (dw) {   // dW = dY^T X, contraction over M
    const int e = whole_k ? i8l_gemm_rowcol(dyqt, x_qt, dyst, x_st, 1, nullptr, post_dw, dw, 1, N, K, M, flags, status, stream)
                          : i8l_gemm_block(dyqt, x_qt, dyst, x_st, a_kind_of(gran), b_kind_of(gran), 1, nullptr, post_dw, dw, 1, N,
                                           K, M, flags, status, stream);
    if (e) return e;
  }
  return I8L_OK;
}
