// INT8 GEMMs on the 5th-generation tensor cores: tcgen05.mma kind::i8 with int32 accumulators in
// tensor memory, operands staged by TMA into a 128B-swizzled shared-memory ring.
//
// One persistent CTA per SM, 384 threads, or 640 in the generic kind:
//   warp 0      TMA producer (one elected lane)
//   warp 1      tensor-memory allocator + MMA issuer (one elected lane, see elect_one)
//   warp 2      factor warp (fast block-scaled kind): prepares, one tile ahead, the per-K-block
//               factors, corrections and column scales the epilogue needs; idle in the other kinds
//   warp 3      idle (completes the first warpgroup so register budgets can be rebalanced)
//   warps 4-    epilogue: warp%4 selects the 32 accumulator lanes (rows) a warp may read, the group of
//               four warps a share of the columns of the 128x256 tile.  Sixteen warps with 64 columns
//               each in the generic kind, whose per-K-block drain is bound by instruction latency (more resident
//               warps hide it).  The shifted kinds have one or two packed FMAs per two elements left and want long
//               runs of tensor-memory loads instead: eight warps with 128 columns each and up to 208 registers, 32
//               columns in flight per wait (fast kind, 8192^3: 16 warps 508 us, 8 warps 501, 8 warps and 32 columns 489).
//               Eight warps in the row x column kind as well, which take their whole share into registers at once.
// Tensor memory holds two 128x256 int32 accumulators (all 512 columns), or four of the narrow tiles' 128x128.  In block-scaled mode the
// MMA warp alternates between them every 128-wide K block while the epilogue drains the other one
// into fp32 registers (acc += float(P) * scale; in the shifted kinds a fifth MMA per K block moves P into the
// non-negative range, where its bits ARE a float, and the shift is taken out again); in
// row x column mode a buffer holds a whole tile and the epilogue of tile i overlaps the main loop of tile i+1.
//
// Every wait on an mbarrier is bounded (a poll count worth about two seconds); on expiry the CTA raises
// a shared abort flag and reports through the status word.  The producer and the MMA issuer then leave
// their loops; the epilogue warps run through their remaining tiles without waiting, computing or
// storing; copies in flight are awaited, so the kernel always terminates and frees its tensor memory.
//
// Scatter mode (i8l_gemm_block_scatter): the epilogue writes each 128-row block into a slot of a
// buffer owned by another GPU (plain stores to peer-mapped memory), for a reduce-scatter without a
// separate collective kernel.
#include <cuda.h>

#include <atomic>
#include <cstddef>
#include <cstring>
#include <mutex>
#include <new>
#include <type_traits>

#include "common.cuh"
#include "ptx.cuh"

namespace i8l {

constexpr int BM = 128, BK = 128;
constexpr int WIDE = 256, NARROW = 128;   // columns of a tile (BN below), see narrow_tiles
constexpr int A_STAGE = BM * BK;  // bytes
// One CTA per tile: 128x256 tile, 3 stages of 16 KB (A) + 32 KB (B), or 128x128, 5 stages of 16 + 16 KB.
// CTA pair per tile (cta_group::2): 256x256 tile, each CTA stages its own 128 rows of A and 128 of the
// 256 rows of B (16 KB + 16 KB), 5 stages: half the B traffic through each SM's shared memory.
// One stage less than fits leaves the 64 KB that a bf16 output tile is staged in (store_tile).
template <bool TWO, int BN> struct Cfg {
  static constexpr int STAGES = TWO || BN == NARROW ? 5 : 3;
  static constexpr int B_STAGE = TWO ? BM * BK : BN * BK;
  static constexpr uint32_t STAGE_TX = TWO ? 2u * (A_STAGE + BM * BK) : (uint32_t)(A_STAGE + BN * BK);
  static constexpr int OUT_STAGE = BM * BN * 2;   // the bf16 output tile
  static constexpr int SMEM_DYN = STAGES * (A_STAGE + B_STAGE) + OUT_STAGE + 1024;
};
constexpr int MAX_STAGES = 5;
// the kinds whose partial products are shifted by an extra MMA (K_BLOCK_FAST and the row and column factor kinds)
template <int KIND> constexpr bool SHIFTED_OF = KIND >= 2;
template <int KIND> constexpr int EPI_WARPS_OF = KIND == 1 ? 16 : 8;   // 1: K_BLOCK_GEN
constexpr int FAC_MAX = 192;                  // K blocks whose factors are staged in shared memory at a time (a multiple of 4)
constexpr int TMEM_COLS = 512;

// Division of 0 <= n < 2^31 by a number known at launch: n * mul >> shift with mul = ceil(2^shift / d) and shift = 31 + ceil(log2 d),
// so that mul fits 32 bits and the rounding of mul stays below one part in 2^31.  Dividing costs an epilogue warp about
// 500 cycles for the coordinates of a tile, which it needs at its start and at its end, this about 100.
struct FastDiv {
  uint32_t mul, shift;
  int d;
  __device__ __forceinline__ int div(int n) const { return (int)((uint64_t)(uint32_t)n * mul >> shift); }
  void set(int divisor) {
    int log = 0;
    while ((1ll << log) < divisor) ++log;
    d = divisor;
    shift = 31 + log;
    mul = (uint32_t)(((1ull << shift) + divisor - 1) / divisor);
  }
};

struct GemmParams {
  const float* a_scale;
  const float* b_scale;
  const __nv_bfloat16* bias;
  void* c;
  int32_t* status;
  int32_t* mirror;   // pinned host memory that follows the status word (i8l_status_mirror), or null
  int m_blocks;  // batch*M/128
  int mpb;       // M/128 (m-blocks per batch)
  int n_tiles;   // ceil(N / columns of a tile)
  int M, N, KB;  // KB = K/128
  int a_kind, b_kind, b_batched;
  int exact, divide, out_f32, dump;  // dump: 0 none, 1 whole-K int32, 2 per-K-block int32
  int a_kshift;       // an A tile scale serves 2^a_kshift consecutive K blocks (1 for 128x256 groups)
  int product_first;  // exact order only: float(P) * (a_s*b_s) instead of (float(P)*a_s)*b_s
  int raster;     // M-units per group of the tile order
  FastDiv per_group, full_group, last_group, per_batch;   // tiles of a group, M-units of a group (all but the last; the last), mpb
  int c_align32;  // the output pointer is 32-byte aligned: 256-bit stores
  // scatter mode (rs_rows > 0): rows [o*rs_rows, (o+1)*rs_rows) of the product go to c_slots[o], a
  // [world, rs_rows, N] bf16 buffer of rank o (peer memory), at slot rs_rank
  void* c_slots[I8L_MAX_RANKS];
  int rs_rows, rs_rank;
  int m_rot;  // 128-row blocks by which the tile order is rotated (0 unless scattering)
  float post_scale;
  uint32_t max_polls;  // limit of every mbarrier wait, in polls (WAIT_MAX_POLLS unless a test lowers it)
  int early;           // the kernel behind this one in a chain is a GEMM
  int withhold;        // test hook: the producer leaves out the last operand load of its first tile
};

// Instruction descriptor: D=s32, A and B s8 or (the MMA that shifts a partial product) u8, both K-major, dense, no
// saturation.  m: 128, or 256 for the CTA-pair instruction (128 rows per CTA).
__host__ __device__ constexpr uint32_t idesc(bool s8, int m, int n) {
  return (2u << 4) | (s8 ? (1u << 7) | (1u << 10) : 0u) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

struct TileCoord {
  int m_blk, n_tile;
};
__device__ __forceinline__ TileCoord tile_coord(int t, int m_units, const GemmParams& p) {
  const int g = p.per_group.div(t), local = t - g * p.per_group.d, first = g * p.raster;
  const FastDiv& size = first + p.raster <= m_units ? p.full_group : p.last_group;
  TileCoord tc;
  tc.n_tile = size.div(local);
  tc.m_blk = first + local - tc.n_tile * size.d;
  return tc;
}

// Epilogue kinds.  Everything but K_ROWCOL drains the accumulator every 128-wide K block.
constexpr int K_ROWCOL = 0;      // one drain per tile, (float(acc)*a_s[m])*b_s[n]
constexpr int K_BLOCK_GEN = 1;   // block-scaled, any scale layout, reference operation order, dumps
constexpr int K_BLOCK_FAST = 2;  // block-scaled, one scalar factor per (tile, K block) and 128-column half
constexpr int K_BLOCK_COLFAC = 3;  // block-scaled, per-tile A scale x per-(column, K block) B scale (fused forward)
constexpr int K_BLOCK_ROWFAC = 4;  // block-scaled, per-(row, K block) A scale x per-tile or per-channel B scale
constexpr int K_BLOCK_TILEDIV = 6; // block-scaled, per-tile scales on both sides as divisors (fused backward)
constexpr int K_BLOCK_OUTER = 5;   // block-scaled, per-(row, K block) A scale x per-(column, K block) B scale

template <int KIND, int BN> struct __align__(256) SharedCtl {   // tempty must directly follow tfull (the fast epilogue addresses both from one base)
  // shifted kinds: BN rows x 32 bytes of 0xFF, both operands of the shifting MMA (32-byte swizzle atoms)
  __align__(256) uint8_t ones[SHIFTED_OF<KIND> ? BN * 32 : 1];
  uint64_t full[MAX_STAGES], empty[MAX_STAGES], tfull[TMEM_COLS / BN], tempty[TMEM_COLS / BN], done;
  // fast block kind: factors written (factor warp), what the tile end needs written, all consumed (every epilogue thread)
  uint64_t fready[2], eready[2], ffree[2];
  uint32_t tmem_base;
  int abort_flag;
  union __align__(16) {   // scales are read four at a time
    struct {
      float bscale[BN];     // per-tile column scales (CHANNEL)
      __nv_bfloat16 bias[BN];
      float bstep[KIND == K_ROWCOL ? 1 : 2][KIND == K_ROWCOL ? 1 : BN];   // per-K-block column scales or factors (GROUP), double buffered
    };
    // K_BLOCK_FAST, written by the factor warp one unit (tile, or FAC_MAX-K-block chunk of a tile) ahead, two
    // buffers; each 128-column half (one epilogue group) has its factors (both share the first with per-channel B scales):
    struct {
      float2 fac[KIND == K_BLOCK_FAST ? 2 : 1][2][KIND == K_BLOCK_FAST ? FAC_MAX : 1];   // per K block: scaled factor, and the correction due at it (or 0)
      float fbscale[KIND == K_BLOCK_FAST ? 2 : 1][KIND == K_BLOCK_FAST ? BN : 1];        // what the sums are multiplied by at the end: per-channel column scale times post_scale, or 1
      __nv_bfloat16 fbias[KIND == K_BLOCK_FAST ? 2 : 1][KIND == K_BLOCK_FAST ? BN : 1];
      float2 fend[2][2];           // in front of that: times .x plus .y (undoes the scaling of the factors, takes out what is left of the shift)
    };
  };
};

// Shifted kinds: 32 products 255 * 255.  A partial product of 128 int8 pairs lies in [-128*128*127, 128*128*128],
// so P + SHIFT lies in [32, 4177952]: never negative and below 2^23, where the bits of an int32, read as a
// float, are the (denormal) number (P + SHIFT) * 2^-149 exactly.
constexpr float SHIFT_F = 2080800.f;
constexpr int FAC_EXP = 100;   // factors are scaled by a power of two that puts the tile's largest one near 2^100
constexpr int REPEATED = 4;    // a factor that this many of 32 K blocks share is divided out of the tile (see the factor warp)
__device__ __forceinline__ float pow2f(int e) { return __uint_as_float((uint32_t)(e + 127) << 23); }   // -126 <= e <= 127

// Two shifted partial products as they come from tensor memory -> P * 2^-23, exactly, by one packed FMA.
constexpr float FROM_SHIFTED = 8388608.f;   // 2^23, multiplied in at the tile end: factors of any size stay finite
__device__ __forceinline__ float2 from_shifted(uint32_t r0, uint32_t r1) {
  const float up = 0x1p126f, off = -SHIFT_F * 0x1p-23f;
  return __ffma2_rn(make_float2(__uint_as_float(r0), __uint_as_float(r1)), make_float2(up, up), make_float2(off, off));
}

__device__ __forceinline__ uint32_t pack_bf16x2(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}

__device__ __forceinline__ void st_global_256(void* ptr, const uint32_t* w) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"l"(ptr), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
               : "memory");
}

// 16 fp32 results of one row, straight to memory (32-byte stores where the output pointer allows them).
__device__ __forceinline__ void store16_f32(const GemmParams& p, const float* v, void* cbase, int64_t row, int col) {
  float* o = static_cast<float*>(cbase) + row * p.N + col;
  if (p.c_align32) {
    st_global_256(o, reinterpret_cast<const uint32_t*>(v));
    st_global_256(o + 8, reinterpret_cast<const uint32_t*>(v + 8));
  } else {
#pragma unroll
    for (int j = 0; j < 16; j += 4) *reinterpret_cast<float4*>(o + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
  }
}

// bf16 results leave through shared memory: a lane owns one row of the tile, so a plain store instruction touches 32
// lines (about 45 cycles of the load/store unit each, 1.6 us a tile that nothing overlaps).  Each warp writes its 32 rows in
// pieces of 64 columns (32 x 128 bytes, 128-byte swizzle: conflict-free) and one lane hands them to the TMA, which
// stores whole rows while the warp goes on with the next tile.  Against stores from registers: fast block kind 4096^3
// 71.4 -> 67.6 us, 8192^3 442 -> 434; row x channel 4096^3 100 -> 96.8; whole-K 384x11008x4096 20.5 -> 16.4, 4096^3
// 49.3 -> 48.0 (the tile end overlaps the next main loop there, but the last one).  The stage of operands given up for
// the staging memory costs nothing (4096^3 70.9 -> 70.4 us with 3 stages and stores from registers).
__device__ __forceinline__ void stage_wait(int lane) {   // the warp's previous pieces have left shared memory
  if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
  __syncwarp();
}
__device__ __forceinline__ void stage16(uint32_t piece, int lane, int chunk, const float* v) {   // chunk: 16-byte unit, 0..7
  uint32_t w[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) w[j] = pack_bf16x2(v[2 * j], v[2 * j + 1]);
  const uint32_t row = piece + lane * 128;
#pragma unroll
  for (int k = 0; k < 2; ++k)
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};"
                 ::"r"(row + (((chunk + k) ^ (lane & 7)) << 4)), "r"(w[4 * k]), "r"(w[4 * k + 1]), "r"(w[4 * k + 2]), "r"(w[4 * k + 3])
                 : "memory");
}
template <int PIECES>
__device__ __forceinline__ void stage_send(const CUtensorMap* map_c, uint32_t stage, int lane, int col, int row) {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncwarp();
  if (lane == 0) {
#pragma unroll
    for (int h = 0; h < PIECES; ++h) tma_store_2d(map_c, stage + h * 4096, col + 64 * h, row);
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
  }
}

// Bias, cast and store of one thread's EPI_COLS consecutive columns.  value(j) gives columns j .. j + 3 but for the bias,
// bias points to this group's in shared memory.  Each case is a loop of its own without branches: with them in the loop
// every 16 columns waited for their own loads, 2500 cycles a tile instead of 1600 (both with the store to the staging memory, which the MMAs share).
template <int EPI_COLS, typename Value>
__device__ __forceinline__ void store_tile(const GemmParams& p, const CUtensorMap* map_c, uint32_t stage, int lane, int64_t row, int col0,
                                           void* cbase, const __nv_bfloat16* bias, Value value) {
  auto columns16 = [&](int j0, float* v, auto with_bias) {
#pragma unroll
    for (int j = 0; j < 16; j += 4) {
      const float4 o = value(j0 + j);
      v[j] = o.x;
      v[j + 1] = o.y;
      v[j + 2] = o.z;
      v[j + 3] = o.w;
      if (decltype(with_bias)::value) {
        const uint2 b = *reinterpret_cast<const uint2*>(bias + j0 + j);
        v[j] = __fadd_rn(v[j], __uint_as_float(b.x << 16));
        v[j + 1] = __fadd_rn(v[j + 1], __uint_as_float(b.x & 0xffff0000u));
        v[j + 2] = __fadd_rn(v[j + 2], __uint_as_float(b.y << 16));
        v[j + 3] = __fadd_rn(v[j + 3], __uint_as_float(b.y & 0xffff0000u));
      }
    }
  };
  auto columns = [&](auto with_bias) {
    if (p.out_f32) {
#pragma unroll
      for (int j0 = 0; j0 < EPI_COLS; j0 += 16) {
        float v[16];
        columns16(j0, v, with_bias);
        store16_f32(p, v, cbase, row, col0 + j0);
      }
    } else {
      stage_wait(lane);
#pragma unroll
      for (int j0 = 0; j0 < EPI_COLS; j0 += 16) {
        float v[16];
        columns16(j0, v, with_bias);
        stage16(stage + j0 / 64 * 4096, lane, j0 % 64 / 8, v);
      }
      stage_send<EPI_COLS / 64>(map_c, stage, lane, col0, (int)row - lane);
    }
  };
  if (p.bias) columns(std::true_type{});
  else columns(std::false_type{});
}

template <int KIND, bool TWO, int BN>
__global__ void __launch_bounds__(128 + 32 * EPI_WARPS_OF<KIND>, 1)
gemm_i8_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
               const __grid_constant__ CUtensorMap map_c, const GemmParams p) {
  constexpr bool BLOCK = KIND != K_ROWCOL, SHIFTED = SHIFTED_OF<KIND>;
  constexpr int EPI_WARPS = EPI_WARPS_OF<KIND>, EPI_COLS = BN / (EPI_WARPS / 4), THREADS = 128 + 32 * EPI_WARPS;
  constexpr int STAGES = Cfg<TWO, BN>::STAGES, B_STAGE = Cfg<TWO, BN>::B_STAGE, OUT_STAGE = Cfg<TWO, BN>::OUT_STAGE;
  constexpr uint32_t STAGE_TX = Cfg<TWO, BN>::STAGE_TX;
  constexpr int BUFS = TMEM_COLS / BN;   // accumulators
  extern __shared__ uint8_t smem_raw[];
  using Ctl = SharedCtl<KIND, BN>;
  static_assert(offsetof(Ctl, bscale) % 16 == 0 && offsetof(Ctl, bias) % 8 == 0 && offsetof(Ctl, bstep) % 16 == 0 &&
                    (KIND != K_BLOCK_FAST || (offsetof(Ctl, fbscale) % 16 == 0 && offsetof(Ctl, fbias) % 8 == 0)) &&
                    offsetof(Ctl, tempty) == offsetof(Ctl, tfull) + BUFS * sizeof(uint64_t),
                "vector reads, and the barriers that share a base register");
  __shared__ Ctl ctl;
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t smem_a = smem_base, smem_b = smem_base + STAGES * A_STAGE;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  volatile int* abort_flag = &ctl.abort_flag;
  // CTA pair: rank 0 (the leader) owns the operand-ready and accumulator-free barriers and issues the MMAs
  const uint32_t rank = TWO ? cluster_ctarank() : 0u;
  const bool leader = rank == 0;
  // tile-processing unit (CTA or pair) and their count: read from the special registers at each use
  // instead of being kept live (the epilogue runs at its register budget)
#define I8L_UNIT (TWO ? (int)(blockIdx.x >> 1) : (int)blockIdx.x)
#define I8L_N_UNITS (TWO ? (int)(gridDim.x >> 1) : (int)gridDim.x)

  if constexpr (SHIFTED) {
    for (int i = threadIdx.x; i < (int)sizeof(ctl.ones) / 16; i += THREADS)
      reinterpret_cast<uint4*>(ctl.ones)[i] = make_uint4(~0u, ~0u, ~0u, ~0u);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (threadIdx.x == 0) {
    prefetch_tensormap(&map_a);
    prefetch_tensormap(&map_b);
    prefetch_tensormap(&map_c);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(&ctl.full[s]), 1);
      mbar_init(smem_u32(&ctl.empty[s]), 1);
    }
    for (int b = 0; b < BUFS; ++b) {
      mbar_init(smem_u32(&ctl.tfull[b]), 1);
      // arrivals that free an accumulator buffer: one per epilogue warp (of both CTAs of a pair); the shifted
      // kinds let every epilogue thread arrive for itself (no warp sync, no branch in their loop)
      mbar_init(smem_u32(&ctl.tempty[b]), SHIFTED ? EPI_WARPS * 32 : (TWO ? 2 : 1) * EPI_WARPS);
    }
    mbar_init(smem_u32(&ctl.done), 1);
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&ctl.fready[b]), 1);
      mbar_init(smem_u32(&ctl.eready[b]), 1);
      mbar_init(smem_u32(&ctl.ffree[b]), EPI_WARPS * 32);
    }
    ctl.abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    if (TWO) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctl.tmem_base)),
                   "r"(TMEM_COLS)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctl.tmem_base)),
                   "r"(TMEM_COLS)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  tc_fence_before();
  __syncthreads();
  if (TWO) cluster_sync_all();  // the peer's barriers are initialised before anything arrives on them
  tc_fence_after();
  // Only another GEMM is let in early, a CTA per SM as these become free.  Quantizer blocks that start while most SMs are
  // taken crowd onto the free ones and stay there (fused forward 2x1024x2048x1536, 96 tiles: 22.2 -> 23.7 us a call).
  if (p.early) chain_trigger();
  chain_wait();   // operands, scales and whatever still uses the output's memory
  const uint32_t tmem_base = ctl.tmem_base;
  // tiles of this unit: m_blocks counts 128-row blocks; a pair takes two consecutive ones
  const int total_tiles = (TWO ? p.m_blocks / 2 : p.m_blocks) * p.n_tiles;
  auto unit_tile = [&](int t) {  // 128-row block of THIS CTA and 256-column tile
    if constexpr (TWO) {
      TileCoord tc = tile_coord(t, p.m_blocks / 2, p);
      tc.m_blk = 2 * tc.m_blk + (int)cluster_ctarank();
      return tc;
    } else {
      TileCoord tc = tile_coord(t, p.m_blocks, p);
      tc.m_blk += p.m_rot;  // scatter mode: every rank starts at a different owner's rows (no incast)
      if (tc.m_blk >= p.m_blocks) tc.m_blk -= p.m_blocks;
      return tc;
    }
  };
  const int KB = p.KB;

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
    if (warp == 0) {
      // ------------------------------------------------------------------ TMA producer
      int s = 0;
      uint32_t ph = 0;
      uint32_t issued = 0, issued_ph = 0;  // bit s: a load into stage s is (or was) in flight, with parity
      bool ok = true;
      for (int t = I8L_UNIT; t < total_tiles && ok; t += I8L_N_UNITS) {
        const TileCoord tc = unit_tile(t);
        const int a_row = tc.m_blk * BM;
        const int b_row = (p.b_batched ? p.per_batch.div(tc.m_blk) * p.N : 0) + tc.n_tile * BN + (TWO ? (int)rank * BM : 0);
        for (int kb = 0; kb < KB; ++kb) {
          if (!(ok = mbar_wait<!BLOCK>(smem_u32(&ctl.empty[s]), ph ^ 1u, abort_flag, p.max_polls))) break;
          if (p.withhold && t == I8L_UNIT && kb == KB - 1) {
            // test hook: this stage is never filled, so the waits that depend on it run into their limit
            if (++s == STAGES) { s = 0; ph ^= 1u; }
            continue;
          }
          if (lane == 0) {
            const uint32_t bar = smem_u32(&ctl.full[s]);
            if (TWO) {  // both CTAs' copies complete on the leader's barrier, which expects the bytes of both
              if (leader) mbar_expect_tx(bar, STAGE_TX);
              const uint32_t lbar = map_to_cta(bar, 0);
              tma_load_2d_pair(smem_a + s * A_STAGE, &map_a, lbar, kb * BK, a_row);
              tma_load_2d_pair(smem_b + s * B_STAGE, &map_b, lbar, kb * BK, b_row);
            } else {
              mbar_expect_tx(bar, STAGE_TX);
              tma_load_2d(smem_a + s * A_STAGE, &map_a, bar, kb * BK, a_row);
              tma_load_2d(smem_b + s * B_STAGE, &map_b, bar, kb * BK, b_row);
            }
          }
          issued |= 1u << s;
          issued_ph = (issued_ph & ~(1u << s)) | (ph << s);
          if (++s == STAGES) { s = 0; ph ^= 1u; }
        }
      }
      if (!ok && leader) {
        // let copies already in flight land before the CTA's shared memory is released
        for (int k = 0; k < STAGES; ++k)
          if (issued & (1u << k)) {
            int dummy = 0;
            mbar_wait(smem_u32(&ctl.full[k]), (issued_ph >> k) & 1u, &dummy, 1u << 15);
          }
      }
    } else if (warp == 1 && leader) {
      // ------------------------------------------------------------------ MMA issuer
      const uint64_t ones_desc = smem_desc_sw32(smem_u32(ctl.ones));
      const bool elected = elect_one();
      int s = 0, ab = 0;
      uint32_t ph = 0, aph = 0;
      bool ok = true;
      for (int t = I8L_UNIT; t < total_tiles && ok; t += I8L_N_UNITS) {
        for (int kb = 0; kb < KB; ++kb) {
          const bool drain_start = BLOCK || kb == 0, drain_end = BLOCK || kb == KB - 1;
          // the generic block kind waits for the accumulator buffer last; the whole-K kinds measured 0.7 % faster the
          // other way round, the shifted kinds 1 % (8192^3 458 -> 454 us) with their first MMA in between
          if (!BLOCK && drain_start) {
            if (!(ok = mbar_wait<!BLOCK>(smem_u32(&ctl.tempty[ab]), aph ^ 1u, abort_flag, p.max_polls))) break;
          }
          if (SHIFTED) {   // D = SHIFT (see the epilogue) needs the buffer only: it goes out ahead of the operands' wait
            if (!(ok = mbar_wait<!BLOCK>(smem_u32(&ctl.tempty[ab]), aph ^ 1u, abort_flag, p.max_polls))) break;
            tc_fence_after();
            if (elected) tc_mma_i8(tmem_base + ab * BN, ones_desc, ones_desc, idesc(false, BM, BN), 0u);
          }
          if (!(ok = mbar_wait<!BLOCK>(smem_u32(&ctl.full[s]), ph, abort_flag, p.max_polls))) break;
          if (BLOCK && !SHIFTED) {
            if (!(ok = mbar_wait<!BLOCK>(smem_u32(&ctl.tempty[ab]), aph ^ 1u, abort_flag, p.max_polls))) break;
          }
          tc_fence_after();
          if (elected) {
            const uint64_t da = smem_desc(smem_a + s * A_STAGE), db = smem_desc(smem_b + s * B_STAGE);
            const uint32_t d = tmem_base + ab * BN;
#pragma unroll
            for (int k4 = 0; k4 < BK / 32; ++k4) {
              if (TWO) tc_mma_i8_pair(d, da + 2 * k4, db + 2 * k4, idesc(true, 2 * BM, BN), (k4 > 0 || !drain_start) ? 1u : 0u);
              else tc_mma_i8(d, da + 2 * k4, db + 2 * k4, idesc(true, BM, BN), (SHIFTED || k4 > 0 || !drain_start) ? 1u : 0u);
            }
            if (TWO) {  // both CTAs' producers and epilogues wait on their own copies of these barriers
              tc_commit_pair(smem_u32(&ctl.empty[s]));
              if (drain_end) tc_commit_pair(smem_u32(&ctl.tfull[ab]));
            } else {
              tc_commit(smem_u32(&ctl.empty[s]));
              if (drain_end) tc_commit(smem_u32(&ctl.tfull[ab]));
            }
          }
          __syncwarp();
          if (drain_end && ++ab == BUFS) {
            ab = 0;
            aph ^= 1u;
          }
          if (++s == STAGES) { s = 0; ph ^= 1u; }
        }
      }
      // all MMAs issued by this thread must have retired before tensor memory is freed
      if (elected) {
        if (TWO) tc_commit_pair_local(smem_u32(&ctl.done));
        else tc_commit(smem_u32(&ctl.done));
      }
      __syncwarp();
      int dummy = 0;
      mbar_wait(smem_u32(&ctl.done), 0, &dummy);
    } else if (KIND == K_BLOCK_FAST && warp == 2) {
      // ------------------------------------------------------------------ factor warp (fast block kind)
      // Prepares, one unit ahead of the epilogue, what the epilogue needs besides the accumulators: the factor
      // of every K block, the corrections and the column scales.  K block d contributes F_d * (P_d + SHIFT) * 2^-149
      // with F_d = f_d * 2^e, e common to the tile and chosen so that the largest |F_d| is near 2^FAC_EXP: nothing
      // over- or underflows whatever the scales are.  SHIFT * F_d is taken out four K blocks at a time, after the
      // second of them: the accumulators then stay within two K blocks' shift (4.2e6 f) of the true sum, an ulp of
      // which is at most f/2.  What the rounded corrections leave over is summed in fp64 and goes out at the tile end.
      // These roundings are as good as random while the factors differ.  Equal ones round the same way every time and
      // the error grows with K: an all-zero 128-row block, whose scales all sit on the quantizers' floor, came out at up
      // to 8 f (K = 32768).  So a factor that repeats is divided out of the whole tile and multiplied back at its end:
      // it becomes a power of two, SHIFT times it a float, and its K blocks add nothing but P.
      // Hand-over through mbarrier pairs (factors written, tile-end values written / buffer consumed), waits bounded like
      // all others.  The factors go out first: a kernel of one tile per CTA waits for them (3.2 us after its start when
      // everything was handed over at once).
      const bool chan = p.b_kind == I8L_BSCALE_CHANNEL;
      constexpr double SHIFT_D = (double)SHIFT_F * 0x1p-149;
      uint32_t u = 0;
      for (int t = I8L_UNIT; t < total_tiles; t += I8L_N_UNITS) {
        const TileCoord tc = unit_tile(t);
        const int64_t bcol0 = (int64_t)(p.b_batched ? p.per_batch.div(tc.m_blk) : 0) * p.N + tc.n_tile * BN;
        const float* as_ptr = p.a_scale + (int64_t)tc.m_blk * (KB >> p.a_kshift);
        const int halves = chan || BN == NARROW ? 1 : 2;   // with per-channel B scales a factor is the A scale alone
        int e[2];                                   // factors are scaled by 2^e, the sums by 2^(149 - e)
        float unit[2];                              // the factor that is divided out, or 1
        double left[2] = {0., 0.};                  // per lane, over the chunks of the tile
        for (int k0 = 0; k0 < KB; k0 += FAC_MAX, ++u) {
          const int dn = KB - k0 < FAC_MAX ? KB - k0 : FAC_MAX;
          const int buf = u & 1;
          if (u >= 2 && !mbar_wait(smem_u32(&ctl.ffree[buf]), ((u >> 1) - 1) & 1u, abort_flag, p.max_polls)) {
            t = total_tiles;   // gave up (or another warp did): leave both loops
            break;
          }
          auto factor = [&](int h, int d) {
            const float a = chain_load(as_ptr + (d >> p.a_kshift));
            if (chan || tc.n_tile * BN + h * 128 >= p.N) return a;   // no second half: a number that does no harm
            return a * (chain_load(p.b_scale + ((bcol0 >> 7) + h) * KB + d) * p.post_scale);
          };
          if (k0 == 0) {
            float m[2] = {0.f, 0.f};
            // one factor per lane, spread over K (lanes past K: a pattern of their own), to see which one repeats
            const int pick = lane + 32 * ((lane * (KB >> 5)) >> 5);
            uint32_t seen[2] = {0x7fc00000u | lane, 0x7fc00000u | lane};
            for (int i = lane; i < KB; i += 32)
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                if (h < halves) {
                  const float f = factor(h, i);
                  if (i < dn) ctl.fac[buf][h][i].x = f;
                  if (i == pick) seen[h] = __float_as_uint(f);
                  m[h] = fmaxf(m[h], fabsf(f));
                }
              }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              unit[h] = 1.f;
              if (h >= halves) continue;
#pragma unroll
              for (int o = 16; o > 0; o >>= 1) m[h] = fmaxf(m[h], __shfl_xor_sync(0xffffffffu, m[h], o));
              const uint32_t peers = __match_any_sync(0xffffffffu, seen[h]);
              const uint32_t most = __reduce_max_sync(0xffffffffu, lane < KB ? (uint32_t)__popc(peers) << 5 | lane : 0u);
              const float c = __uint_as_float(__shfl_sync(0xffffffffu, seen[h], most & 31));
              // normal, and no factor overflows when divided by it
              const int ec = (int)(__float_as_uint(c) >> 23 & 0xffu), em = (int)(__float_as_uint(m[h]) >> 23);
              if ((int)(most >> 5) >= (KB < REPEATED ? KB : REPEATED) && ec > 0 && ec < 255 && em - ec < 64) {
                unit[h] = c;
                m[h] = __fdiv_rn(m[h], fabsf(c));
              }
              e[h] = FAC_EXP + 127 - (int)(__float_as_uint(m[h]) >> 23);
            }
          } else {
            for (int i = lane; i < dn; i += 32)
#pragma unroll
              for (int h = 0; h < 2; ++h)
                if (h < halves) ctl.fac[buf][h][i].x = factor(h, k0 + i);
          }
          __syncwarp();
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if (h >= halves) continue;
            float2* fac = ctl.fac[buf][h];
            const float up0 = pow2f(e[h] >> 1), up1 = pow2f(e[h] - (e[h] >> 1));   // 2^e may be too large for one float
            for (int i = lane; i < (dn + 3) / 4; i += 32) {   // one lane per four K blocks
              float f4[4];
              double sum = 0.;
#pragma unroll
              for (int j = 0; j < 4; ++j) f4[j] = 4 * i + j < dn ? fac[4 * i + j].x : 0.f;
              if (unit[h] != 1.f) {
#pragma unroll
                for (int j = 0; j < 4; ++j) f4[j] = __fdiv_rn(f4[j], unit[h]);
              }
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                f4[j] = f4[j] * up0 * up1;
                sum += (double)f4[j];
              }
              const float corr = 4 * i + 2 < dn ? -(float)(SHIFT_D * sum) : 0.f;
              left[h] += SHIFT_D * sum + (double)corr;
#pragma unroll
              for (int j = 0; j < 4; ++j)
                if (4 * i + j < dn) fac[4 * i + j] = make_float2(f4[j], j == 2 ? corr : 0.f);
            }
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&ctl.fready[buf]));   // the K blocks may start; the rest is due at the tile end
          if (k0 + dn == KB) {
            // 2^(149 - e) as two factors: the sums are far below 1, so the first may take all of it, up to the largest
            // power there is; the rest goes with the column scale
            for (int i = lane; i < BN; i += 32) {
              const int h = (chan || i < 128) ? 0 : 1, back = 149 - (h ? e[1] : e[0]);
              const float d = pow2f(back < 127 ? 0 : back - 127) * (h ? unit[1] : unit[0]);
              ctl.fbscale[buf][i] = chan && tc.n_tile * BN + i < p.N ? chain_load(p.b_scale + bcol0 + i) * p.post_scale * d : d;
              if (p.bias) ctl.fbias[buf][i] = tc.n_tile * BN + i < p.N ? p.bias[tc.n_tile * BN + i] : __float2bfloat16_rn(0.f);
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              double all = left[h < halves ? h : 0];
#pragma unroll
              for (int o = 16; o > 0; o >>= 1) all += __shfl_xor_sync(0xffffffffu, all, o);
              const int back = 149 - e[h < halves ? h : 0];
              const float d = pow2f(back < 127 ? back : 127);
              if (lane == 0) ctl.fend[buf][h] = make_float2(d, -(float)all * d);
            }
            __syncwarp();
          }
          if (lane == 0) mbar_arrive(smem_u32(&ctl.eready[buf]));   // every chunk, so that one count gives all parities
        }
      }
    }
  } else {
    // -------------------------------------------------------------------- epilogue
    // 128 x 64 + 256 x 208 of the 384 x 168 registers of the launch; 128 x 64 + 512 x 104 of 640 x 96
    if (EPI_WARPS == 8) asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
    else asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
    const int q = warp & 3, wg = (warp - 4) >> 2;  // lane quarter, column group
    const int tix = q * 32 + lane;                 // row within the tile == thread index within the group
    const uint32_t lane_addr = (uint32_t)(q * 32) << 16;
    // this warp's 32 rows x EPI_COLS bf16 of the output tile; from the special register at each use, not kept live
    auto out_stage = [&]() {
      uint32_t tid;
      asm volatile("mov.u32 %0, %%tid.x;" : "=r"(tid));
      return ((smem_u32(smem_raw) + 1023u) & ~1023u) + STAGES * (A_STAGE + B_STAGE) + ((tid >> 5) - 4) * (OUT_STAGE / EPI_WARPS);
    };
    int ab = 0;
    uint32_t aph = 0;
    bool ok = true;
    auto release_accumulator = [&]() {  // all of this warp's tensor-memory loads of the buffer have completed
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (TWO) mbar_arrive_cluster(map_to_cta(smem_u32(&ctl.tempty[ab]), 0));  // the leader's barrier
        else mbar_arrive(smem_u32(&ctl.tempty[ab]));
      }
    };
    if constexpr (KIND == K_BLOCK_FAST) {
      // One scalar factor per (tile, K block) and column group: a per-tile A scale times a per-tile or
      // per-channel B scale.  The K-block loop keeps only the accumulators, one chunk of tensor-memory
      // data and a few scalars live: the factors of the tile are staged in shared memory first, and
      // what the final store needs is recomputed from the tile index afterwards.
      const uint32_t tfull0 = smem_u32(&ctl.tfull[0]);
      constexpr uint32_t TEMPTY_OFF = BUFS * sizeof(uint64_t);   // tempty[] follows tfull[] in SharedCtl: one base register serves both
      // Values derived from the thread index pass through an empty asm statement: the compiler then
      // keeps them in registers instead of recomputing them from the special register at every use
      // inside the K-block loop (which cost about 35 ALU instructions per warp and K block).
      uint32_t taddr0 = tmem_base + lane_addr + wg * EPI_COLS, fac_base = smem_u32(&ctl.fac[0][p.b_kind == I8L_BSCALE_CHANNEL || BN == NARROW ? 0 : wg][0]);
      asm volatile("" : "+r"(taddr0), "+r"(fac_base));
      constexpr int CH = 32;
      uint32_t gstep = 0, unit = 0;
      // The loops below never exit early (one exit and nothing to carry but the accumulators compiles to the
      // leanest code): after a wait timeout a warp runs through the remaining tiles without waiting or storing.
      for (int t = I8L_UNIT; t < total_tiles; t += I8L_N_UNITS) {
        float2 acc[EPI_COLS / 2];
#pragma unroll
        for (int j = 0; j < EPI_COLS / 2; ++j) acc[j] = make_float2(0.f, 0.f);
        const bool active = unit_tile(t).n_tile * BN + wg * EPI_COLS < p.N;
        for (int k0 = 0; k0 < KB; k0 += FAC_MAX) {
          const int dn = KB - k0 < FAC_MAX ? KB - k0 : FAC_MAX;
          if (k0) {   // the previous chunk's factors are no longer needed
            mbar_arrive(smem_u32(&ctl.ffree[unit & 1]));
            ++unit;
          }
          mbar_wait_or_flag(smem_u32(&ctl.fready[unit & 1]), (unit >> 1) & 1u, abort_flag, p.max_polls);   // written by the factor warp
          const uint32_t fac0 = fac_base + (unit & 1) * (uint32_t)sizeof(ctl.fac[0]);
          for (int d = 0; d < dn; ++d) {
            float f, corr;
            asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(f), "=f"(corr) : "r"(fac0 + 8 * d));
            // No early exit and no success flag: a loop with one exit and nothing to carry but the
            // accumulators compiles to the leanest code.  After a timeout the abort flag is set, the status
            // word reports it, and the remaining K blocks run on whatever tensor memory holds.
            mbar_spin_or_flag(tfull0 + 8 * ab, aph, abort_flag, p.max_polls);
            tc_fence_after();
            auto release = [&]() {  // all of this warp's tensor-memory loads of the buffer have completed
              tc_fence_before();
              mbar_arrive(tfull0 + TEMPTY_OFF + 8 * ab);   // every thread arrives for itself: no warp sync, no branch
            };
            if (active) {
              // int32 -> fp32 without any conversion: an extra K step of the tensor core has added SHIFT to P, so
              // the bits are the float (P + SHIFT) * 2^-149, which the FMA multiplies exactly.  One packed FMA per
              // two elements is all that is left; the shift is taken out every fourth K block.
              // A fifth MMA (+25 % tensor work) for half of the drain's instructions took 8192^3 from 560 us (an integer
              // add per element, sixteen warps; the drain was the bound) to 489 us, the error against fp64 from 2.1e-5 to
              // 0.7e-5.  With the MMAs issued by an elected lane the tensor pipe is the bound: 640 of 813 cycles per K block,
              // 426-455 us.
              const uint32_t taddr = taddr0 + ab * BN;
              const float2 f2 = make_float2(f, f);
              if (corr != 0.f) {
                const float2 c2 = make_float2(corr, corr);
#pragma unroll
                for (int j = 0; j < EPI_COLS / 2; ++j) acc[j] = __fadd2_rn(acc[j], c2);
              }
#pragma unroll
              for (int c = 0; c < EPI_COLS / CH; ++c) {
                uint32_t r[CH];
                tc_ld16(taddr + c * CH, r);   // two loads of 16: one of 32 makes the compiler spill (489 -> 513 us at 8192^3)
                tc_ld16(taddr + c * CH + 16, r + 16);
                tc_ld_wait();
                if (c == EPI_COLS / CH - 1) release();
#pragma unroll
                for (int j = 0; j < CH / 2; ++j)
                  acc[c * (CH / 2) + j] = __ffma2_rn(make_float2(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1])), f2,
                                                     acc[c * (CH / 2) + j]);
              }
            } else {
              release();
            }
            ++gstep;  // buffer and phase from one running count of K blocks
            ab = gstep % BUFS;
            aph = gstep / BUFS & 1u;
          }
        }
        // after a timeout the accumulators are not a product: nothing is stored (decided per warp: the store
        // path below synchronises the warp)
        mbar_wait_or_flag(smem_u32(&ctl.eready[unit & 1]), (unit >> 1) & 1u, abort_flag, p.max_polls);
        if (active && __all_sync(0xffffffffu, !*abort_flag)) {
          int t2 = t;
          asm volatile("" : "+r"(t2));  // keeps the tile's coordinates out of the K-block loop's live registers
          const TileCoord tc = unit_tile(t2);
          int64_t row = (int64_t)tc.m_blk * BM + tix;
          void* cbase = p.c;
          if (p.rs_rows) {  // scatter mode: this 128-row block belongs to rank `owner`; write into our slot of its buffer
            const int owner = (tc.m_blk * BM) / p.rs_rows;
            cbase = p.c_slots[owner];
            row += (int64_t)(p.rs_rank - owner) * p.rs_rows;
          }
          const float2 fe = ctl.fend[unit & 1][wg];
          const float2 fe_mul = make_float2(fe.x, fe.x), fe_add = make_float2(fe.y, fe.y);
          const float4* bsc4 = reinterpret_cast<const float4*>(ctl.fbscale[unit & 1] + wg * EPI_COLS);
          auto value = [&](int j) {
            const float4 bs = bsc4[j / 4];
            const float2 lo = __fmul2_rn(__ffma2_rn(acc[j / 2], fe_mul, fe_add), make_float2(bs.x, bs.y));
            const float2 hi = __fmul2_rn(__ffma2_rn(acc[j / 2 + 1], fe_mul, fe_add), make_float2(bs.z, bs.w));
            return make_float4(lo.x, lo.y, hi.x, hi.y);
          };
          const int col0 = tc.n_tile * BN + wg * EPI_COLS;
          if (p.rs_rows && !p.out_f32 && !p.bias) {
            // Peer stores.  A lane owns one row, so a plain store instruction would send 32 separate 32-byte
            // pieces over NVLink; here the warp passes four rows at a time through shared memory (16-byte
            // slots, XOR-swizzled so that writers and readers are conflict-free) and every store instruction
            // then covers four rows x 128 contiguous bytes.  Same values as store_tile.
            uint4* xp = reinterpret_cast<uint4*>(smem_raw + (out_stage() - smem_u32(smem_raw)));
            const int wr = lane & 3, rr = lane >> 3, rc = lane & 7;
            __nv_bfloat16* obase = static_cast<__nv_bfloat16*>(cbase) + (row - lane) * p.N + col0 + rc * 8;
#pragma unroll
            for (int h = 0; h < EPI_COLS; h += 64) {
              uint32_t w[32];
#pragma unroll
              for (int j = 0; j < 32; j += 2) {
                const float4 v = value(h + 2 * j);
                w[j] = pack_bf16x2(v.x, v.y);
                w[j + 1] = pack_bf16x2(v.z, v.w);
              }
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                if ((lane >> 2) == j) {
#pragma unroll
                  for (int c = 0; c < 8; ++c)
                    xp[wr * 8 + (c ^ (wr << 1))] = make_uint4(w[4 * c], w[4 * c + 1], w[4 * c + 2], w[4 * c + 3]);
                }
                __syncwarp();
                const uint4 v = xp[rr * 8 + (rc ^ (rr << 1))];
                *reinterpret_cast<uint4*>(obase + (int64_t)(4 * j + rr) * p.N + h) = v;
                __syncwarp();
              }
            }
          } else {
            store_tile<EPI_COLS>(p, &map_c, out_stage(), lane, row, col0, cbase, ctl.fbias[unit & 1] + wg * EPI_COLS, value);
          }
        }
        mbar_arrive(smem_u32(&ctl.ffree[unit & 1]));   // this tile's factors and column scales are no longer needed
        ++unit;
      }
    } else
    for (int t = I8L_UNIT; t < total_tiles; t += I8L_N_UNITS) {  // no early exit either (named barriers inside)
      const TileCoord tc = unit_tile(t);
      const int batch = p.per_batch.div(tc.m_blk);
      const int64_t row = (int64_t)tc.m_blk * BM + tix;  // row in the folded [batch*M] space
      const int col0 = tc.n_tile * BN + wg * EPI_COLS;
      const bool active = col0 < p.N;
      const int64_t bcol0 = (int64_t)(p.b_batched ? batch : 0) * p.N + col0;  // first b_scale column index
      const bool chan = p.b_kind == I8L_BSCALE_CHANNEL && !p.dump;
      if (chan || p.bias) {  // K-invariant column scales and bias of this group -> shared memory
        named_sync(1 + wg, 128);
        if (tix < EPI_COLS) {
          if (chan) ctl.bscale[wg * EPI_COLS + tix] = active ? chain_load(p.b_scale + bcol0 + tix) : 0.f;
          if (p.bias) ctl.bias[wg * EPI_COLS + tix] = active ? p.bias[col0 + tix] : __float2bfloat16_rn(0.f);
        }
        named_sync(1 + wg, 128);
      }
      const __nv_bfloat16* bias = ctl.bias + wg * EPI_COLS;

      if constexpr (SHIFTED) {
        // Before, with sixteen warps converting on two pipes, and now, 8192^3: row x channel 787 -> 607-620 us, column
        // 1051 -> 843-940 (box to box); row x column took the generic path: 4020 -> 871-920.
        // A factor per row, per column or both for every K block.  Two packed FMAs per two elements (the first
        // brings P back from its shift), a packed product more for row x column factors.  Row factors live in the
        // thread that owns the row; column factors (a_s * b_s or its reciprocal when the scales are multipliers, the
        // fused forward: acc += P / (s_a * s_b)) are published through shared memory, one column per thread.
        constexpr bool ROWF = KIND != K_BLOCK_COLFAC, COLF = KIND == K_BLOCK_COLFAC || KIND == K_BLOCK_OUTER;
        constexpr int CH = 32;
        static_assert(EPI_COLS <= 128, "a thread of the group publishes one column");
        const float* as_ptr = p.a_scale + (ROWF && KIND != K_BLOCK_TILEDIV ? row : (int64_t)tc.m_blk) * KB;
        const bool publish = tix < EPI_COLS && active;
        const float* bc_ptr = p.b_scale + (bcol0 + (publish ? tix : 0)) * KB;   // COLF: one scale per column and K block
        const float* bt_ptr = p.b_scale + (bcol0 >> 7) * KB;       // per-tile B scales
        // The scales of the next K block are loaded a whole block ahead and multiplied when it starts: multiplied at once
        // they held every warp up for the load (400 of 1200 cycles per K block with per-tile B scales, 900 of 1775 in the
        // column kind).  4096^3: row x channel 97.5 -> 92.3 us, row x tile 96.2 -> 88.8, column 129.6 -> 114.1, divisors 93.5 -> 90.7.
        float a_next, b_next = 1.f;
        auto load_scales = [&](int d) {
          a_next = chain_load(as_ptr + d);
          if (COLF) b_next = publish ? chain_load(bc_ptr + d) : 1.f;
          else if (!chan && active) b_next = chain_load(bt_ptr + d);
        };
        asm volatile("" : "+l"(bc_ptr));   // kept in registers: recomputed in every K block otherwise (column kind 877 -> 851 us)
        float2 acc[EPI_COLS / 2];
#pragma unroll
        for (int j = 0; j < EPI_COLS / 2; ++j) acc[j] = make_float2(0.f, 0.f);
        load_scales(0);
        // Column factors of K block d go to bstep[d & 1], with one barrier per K block: whoever writes a buffer has passed the
        // barrier of the block in between, which the readers of its previous contents reach when they are done.  With
        // an odd number of blocks a tile starts with the buffer that the last one ended with, hence a barrier per tile.
        // (One running count over all tiles needs none, but makes the K-block loops 2 % slower, the generic one 15 %;
        // the same barrier behind the tile's stores is 1 % slower.)
        if (COLF) named_sync(1 + wg, 128);
        for (int d = 0; d < KB; ++d) {   // single exit, see K_BLOCK_FAST
          float f = COLF && ROWF ? a_next : a_next * b_next;   // with both the column factor is the B scale alone
          if (KIND == K_BLOCK_TILEDIV || (KIND == K_BLOCK_COLFAC && p.divide)) f = __frcp_rn(f);
          const float2 fr = make_float2(f, f);
          if (COLF) {
            if (EPI_COLS == 128 || tix < EPI_COLS) ctl.bstep[d & 1][wg * EPI_COLS + tix] = ROWF ? b_next : f;
            named_sync(1 + wg, 128);
          }
          if (d + 1 < KB) load_scales(d + 1);
          mbar_spin_or_flag(smem_u32(&ctl.tfull[ab]), aph, abort_flag, p.max_polls);
          tc_fence_after();
          auto release = [&]() {
            tc_fence_before();
            mbar_arrive(smem_u32(&ctl.tempty[ab]));
          };
          if (active) {
            const uint32_t taddr = tmem_base + lane_addr + ab * BN + wg * EPI_COLS;
            const float4* fcol = reinterpret_cast<const float4*>(ctl.bstep[d & 1] + wg * EPI_COLS);
#pragma unroll
            for (int c = 0; c < EPI_COLS / CH; ++c) {
              uint32_t r[CH];
#pragma unroll
              for (int h = 0; h < CH; h += 16) tc_ld16(taddr + c * CH + h, r + h);
              tc_ld_wait();
              if (c == EPI_COLS / CH - 1) release();
#pragma unroll
              for (int j = 0; j < CH / 2; j += 2) {
                float2 f0 = fr, f1 = fr;
                if (COLF) {
                  const float4 fc = fcol[(c * CH + 2 * j) / 4];
                  f0 = make_float2(fc.x, fc.y);
                  f1 = make_float2(fc.z, fc.w);
                  if (ROWF) {
                    f0 = __fmul2_rn(f0, fr);
                    f1 = __fmul2_rn(f1, fr);
                  }
                }
                float2* o = acc + c * (CH / 2) + j;
                o[0] = __ffma2_rn(from_shifted(r[2 * j], r[2 * j + 1]), f0, o[0]);
                o[1] = __ffma2_rn(from_shifted(r[2 * j + 2], r[2 * j + 3]), f1, o[1]);
              }
            }
          } else {
            release();
          }
          if (++ab == BUFS) {
            ab = 0;
            aph ^= 1u;
          }
        }
        if (active && __all_sync(0xffffffffu, !*abort_flag)) {
          const float2 up = make_float2(FROM_SHIFTED, FROM_SHIFTED), post = make_float2(p.post_scale, p.post_scale);
          auto store = [&](auto with_scale) {
            store_tile<EPI_COLS>(p, &map_c, out_stage(), lane, row, col0, p.c, bias, [&](int j) {
              float2 lo = __fmul2_rn(acc[j / 2], up), hi = __fmul2_rn(acc[j / 2 + 1], up);
              if (decltype(with_scale)::value) {
                const float4 bs = *reinterpret_cast<const float4*>(ctl.bscale + wg * EPI_COLS + j);
                lo = __fmul2_rn(lo, make_float2(bs.x, bs.y));
                hi = __fmul2_rn(hi, make_float2(bs.z, bs.w));
              }
              lo = __fmul2_rn(lo, post);
              hi = __fmul2_rn(hi, post);
              return make_float4(lo.x, lo.y, hi.x, hi.y);
            });
          };
          if (!COLF && chan) store(std::true_type{});
          else store(std::false_type{});
        }
      } else {
        // ---- generic paths: reference operation order, per-column / per-step scales, dumps, row x column
        float acc[BLOCK ? EPI_COLS : 1];
        if (BLOCK) {
#pragma unroll
          for (int j = 0; j < EPI_COLS; ++j) acc[j] = 0.f;
        }
        const int ndrain = BLOCK ? KB : 1;
        for (int d = 0; d < ndrain; ++d) {
          float sa = 1.f, sb = 1.f;
          if (BLOCK && !p.dump) {
            sa = p.a_kind == I8L_ASCALE_GROUP ? chain_load(p.a_scale + row * KB + d)
                                              : chain_load(p.a_scale + (int64_t)tc.m_blk * (KB >> p.a_kshift) + (d >> p.a_kshift));
            if (p.b_kind == I8L_BSCALE_TILE && active) sb = chain_load(p.b_scale + (bcol0 >> 7) * KB + d);
            if (p.b_kind == I8L_BSCALE_GROUP) {
              if (tix < EPI_COLS) ctl.bstep[d & 1][wg * EPI_COLS + tix] = active ? chain_load(p.b_scale + (bcol0 + tix) * KB + d) : 0.f;
              named_sync(1 + wg, 128);
            }
          }
          const float sar = !BLOCK && !p.dump ? chain_load(p.a_scale + row) : 0.f;
          ok = ok && __all_sync(0xffffffffu, mbar_wait<!BLOCK>(smem_u32(&ctl.tfull[ab]), aph, abort_flag, p.max_polls));   // per warp: what follows synchronises it
          tc_fence_after();
          const bool live = ok && active;
          const uint32_t taddr = tmem_base + lane_addr + ab * BN + wg * EPI_COLS;
          if (!BLOCK && !p.dump) {
            // row x column: the whole share of the tile into registers, the buffer back, then scale and store
            uint32_t r[EPI_COLS];
            if (live) {
#pragma unroll
              for (int c = 0; c < EPI_COLS; c += 16) tc_ld16(taddr + c, r + c);
              tc_ld_wait();
            }
            release_accumulator();
            if (live) {
              const float2 sar2 = make_float2(sar, sar);
              auto store = [&](auto in_two_steps) {
                store_tile<EPI_COLS>(p, &map_c, out_stage(), lane, row, col0, p.c, bias, [&](int j) {
                  const float4 bs = *reinterpret_cast<const float4*>(ctl.bscale + wg * EPI_COLS + j);
                  const float2 lo = __fmul2_rn(__fmul2_rn(make_float2(__int2float_rn((int)r[j]), __int2float_rn((int)r[j + 1])), sar2), make_float2(bs.x, bs.y));
                  const float2 hi = __fmul2_rn(__fmul2_rn(make_float2(__int2float_rn((int)r[j + 2]), __int2float_rn((int)r[j + 3])), sar2), make_float2(bs.z, bs.w));
                  float4 v = make_float4(lo.x, lo.y, hi.x, hi.y);
                  if (decltype(in_two_steps)::value) {
                    // the reference stores the GEMM result in the output type before its 1/K pass: a bf16
                    // rounding for bf16 outputs, none for fp32 ones
                    if (!p.out_f32) v = make_float4(round_to_bf16(v.x), round_to_bf16(v.y), round_to_bf16(v.z), round_to_bf16(v.w));
                    v = make_float4(__fmul_rn(v.x, p.post_scale), __fmul_rn(v.y, p.post_scale), __fmul_rn(v.z, p.post_scale), __fmul_rn(v.w, p.post_scale));
                  }
                  return v;
                });
              };
              if (p.post_scale != 1.f || p.bias) store(std::true_type{});
              else store(std::false_type{});
            }
          } else
#pragma unroll
          for (int c = 0; c < EPI_COLS / 16; ++c) {
            uint32_t r[16];
            if (live) {
              tc_ld16(taddr + c * 16, r);
              tc_ld_wait();
            }
            if (c == EPI_COLS / 16 - 1) release_accumulator();
            if (!live) continue;
            if (BLOCK) {
              if (p.dump) {
                int32_t* o = static_cast<int32_t*>(p.c) +
                             (((int64_t)batch * KB + d) * p.M + (row - (int64_t)batch * p.M)) * p.N + col0 + c * 16;
#pragma unroll
                for (int j = 0; j < 16; j += 4)
                  *reinterpret_cast<uint4*>(o + j) = make_uint4(r[j], r[j + 1], r[j + 2], r[j + 3]);
              } else {
                const float* sbv = p.b_kind == I8L_BSCALE_CHANNEL ? ctl.bscale + wg * EPI_COLS
                                   : p.b_kind == I8L_BSCALE_GROUP ? ctl.bstep[d & 1] + wg * EPI_COLS
                                                                  : nullptr;
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                  const float pf = __int2float_rn((int)r[j]);
                  const float sbj = sbv ? sbv[c * 16 + j] : sb;
                  float term;
                  if (p.divide) term = __fdiv_rn(pf, __fmul_rn(sa, sbj));
                  else if (p.product_first) term = __fmul_rn(pf, __fmul_rn(sa, sbj));
                  else term = __fmul_rn(__fmul_rn(pf, sa), sbj);
                  acc[c * 16 + j] = __fadd_rn(acc[c * 16 + j], term);
                }
              }
            } else {
              int32_t* o = static_cast<int32_t*>(p.c) + row * p.N + col0 + c * 16;
#pragma unroll
              for (int j = 0; j < 16; j += 4)
                *reinterpret_cast<uint4*>(o + j) = make_uint4(r[j], r[j + 1], r[j + 2], r[j + 3]);
            }
          }
          if (++ab == BUFS) {
            ab = 0;
            aph ^= 1u;
          }
        }
        if constexpr (BLOCK) {
          if (ok && active && !p.dump)
            store_tile<EPI_COLS>(p, &map_c, out_stage(), lane, row, col0, p.c, bias, [&](int j) {
              return make_float4(__fmul_rn(acc[j], p.post_scale), __fmul_rn(acc[j + 1], p.post_scale),
                                 __fmul_rn(acc[j + 2], p.post_scale), __fmul_rn(acc[j + 3], p.post_scale));
            });
          if (p.b_kind == I8L_BSCALE_GROUP) named_sync(1 + wg, 128);   // bstep is free for the next tile (see the column factors above)
        }
      }
    }
  }

  if (warp >= 4 && lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // shared memory outlives the copies out of it
#undef I8L_UNIT
#undef I8L_N_UNITS
  tc_fence_before();
  __syncthreads();
  if (TWO) cluster_sync_all();  // no remote arrival or tensor-memory write of the pair is still pending
  if (threadIdx.x == 0 && ctl.abort_flag && p.status) {
    atomicExch(p.status, I8L_ERR_TIMEOUT);
    if (p.mirror) {
      __threadfence_system();   // who sees the mirror finds the word set
      *static_cast<volatile int32_t*>(p.mirror) = I8L_ERR_TIMEOUT;
    }
  }
  if (warp == 1) {
    tc_fence_after();
    if (TWO) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

// out[r, c] = sum over the `world` slots of slots[w, r, c], added in slot order in fp32 and rounded once:
// the local half of the reduce-scatter whose other half is the scatter-mode GEMM epilogue.
__global__ void __launch_bounds__(256) sum_slots_kernel(const uint4* __restrict__ slots, uint4* __restrict__ out,
                                                        int world, int64_t n16) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n16; i += (int64_t)gridDim.x * blockDim.x) {
    float acc[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = 0.f;
    for (int w = 0; w < world; ++w) {
      float v[8];
      unpack8(__ldg(slots + (int64_t)w * n16 + i), v);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] = __fadd_rn(acc[j], v[j]);
    }
    out[i] = make_uint4(pack_bf16x2(acc[0], acc[1]), pack_bf16x2(acc[2], acc[3]), pack_bf16x2(acc[4], acc[5]),
                        pack_bf16x2(acc[6], acc[7]));
  }
}

// ------------------------------------------------------------------------------------------ host
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode() {
  static std::atomic<EncodeTiledFn> cached{nullptr};
  EncodeTiledFn fn = cached.load(std::memory_order_acquire);
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
    cached.store(fn, std::memory_order_release);
  }
  return fn;
}

// int8 [rows, K] row-major -> boxes of box_rows x 128 bytes, 128B swizzle.  A tensor map depends only
// on (pointer, rows, K, box rows); a training loop calls with the same few operands step after step, so
// the last maps of each host thread are kept (no lock: the cache is thread local) and the driver's
// encode call leaves the launch path.
// bf16_out: an output [rows, K] in boxes of box_rows x 64 elements instead (128 bytes as well).
struct MapKey {
  const void* ptr;
  int64_t rows, K;
  int box_rows;
  bool bf16_out;
};
static int make_map(CUtensorMap* map, const void* ptr, int64_t rows, int64_t K, int box_rows, bool bf16_out = false) {
  constexpr int SLOTS = 16;
  thread_local MapKey keys[SLOTS] = {};
  thread_local CUtensorMap maps[SLOTS];
  thread_local int next_slot = 0;
  for (int i = 0; i < SLOTS; ++i)
    if (keys[i].ptr == ptr && keys[i].rows == rows && keys[i].K == K && keys[i].box_rows == box_rows &&
        keys[i].bf16_out == bf16_out) {
      *map = maps[i];
      return I8L_OK;
    }
  EncodeTiledFn enc = get_encode();
  if (!enc) return fail(I8L_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
  cuuint64_t gdim[2] = {(cuuint64_t)K, (cuuint64_t)rows};
  cuuint64_t gstr[1] = {(cuuint64_t)K * (bf16_out ? 2 : 1)};
  cuuint32_t box[2] = {(cuuint32_t)(bf16_out ? 64 : BK), (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(map, bf16_out ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(ptr), gdim, gstr, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(I8L_ERR_CUDA, "cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
  keys[next_slot] = MapKey{ptr, rows, K, box_rows, bf16_out};
  maps[next_slot] = *map;
  next_slot = (next_slot + 1) % SLOTS;
  return I8L_OK;
}

// bf16 [rows, K] row-major -> boxes of 128 rows x 128 elements (256-byte rows in shared memory, no swizzle):
// the staging tiles of the single-kernel fused GEMM.
int make_tile_map_bf16(CUtensorMap* map, const void* ptr, int64_t rows, int64_t K) {
  EncodeTiledFn enc = get_encode();
  if (!enc) return fail(I8L_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
  cuuint64_t gdim[2] = {(cuuint64_t)K, (cuuint64_t)rows};
  cuuint64_t gstr[1] = {(cuuint64_t)K * 2};
  cuuint32_t box[2] = {128, 128};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), gdim, gstr, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(I8L_ERR_CUDA, "cuTensorMapEncodeTiled (bf16) failed with CUresult %d", (int)r);
  return I8L_OK;
}

constexpr int MAX_DEVICES = 64;
static int current_device() {
  int dev = 0;
  cudaGetDevice(&dev);
  return (dev < 0 || dev >= MAX_DEVICES) ? 0 : dev;
}

int sm_count() {
  static std::atomic<int> cached[MAX_DEVICES];
  const int dev = current_device();
  int n = cached[dev].load(std::memory_order_relaxed);
  if (!n) {
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    cached[dev].store(n, std::memory_order_relaxed);
  }
  return n;
}

// i8l_set_cta_limit: CTAs a persistent GEMM launched by this host thread may occupy (0 = every SM).
static thread_local int g_cta_limit = 0;

// Test hooks (i8l_test_set_wait_limit): 0 = production values.
static std::atomic<uint32_t> g_test_max_polls{0};
static std::atomic<int> g_test_withhold{0};

uint32_t gemm_wait_limit() {
  const uint32_t lim = g_test_max_polls.load(std::memory_order_relaxed);
  return lim ? lim : WAIT_MAX_POLLS;
}
int gemm_cta_budget() {
  const int sms = sm_count();
  return (g_cta_limit > 0 && g_cta_limit < sms) ? g_cta_limit : sms;
}

// Status words with a mirror: a few per process, written when a poller is set up and read by every launch.
struct Mirror {
  std::atomic<const int32_t*> word{nullptr};
  int32_t* device_ptr = nullptr;
};
static Mirror g_mirrors[MAX_DEVICES];
static std::mutex g_mirror_lock;
int32_t* mirror_of(const int32_t* word) {
  for (const Mirror& m : g_mirrors) {
    const int32_t* w = m.word.load(std::memory_order_acquire);
    if (!w) return nullptr;
    if (w == word) return m.device_ptr;
  }
  return nullptr;
}

template <int KIND, bool TWO, int BN>
static int launch_kind(const CUtensorMap& ma, const CUtensorMap& mb, const CUtensorMap& mc, const GemmParams& p, int64_t tiles, cudaStream_t st) {
  // per-device set-up, done by whichever thread comes first (idempotent, so a race only repeats it)
  static std::atomic<int> max_units[MAX_DEVICES];   // 0 = not set up yet
  const int dev = current_device();
  auto kernel = gemm_i8_kernel<KIND, TWO, BN>;
  constexpr int SMEM_DYN = Cfg<TWO, BN>::SMEM_DYN;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  cfg.blockDim = dim3(128 + 32 * EPI_WARPS_OF<KIND>, 1, 1);
  cfg.dynamicSmemBytes = SMEM_DYN;
  cfg.stream = st;
  if (TWO) {
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
  }
  int units = max_units[dev].load(std::memory_order_acquire);
  if (!units) {
    I8L_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_DYN));
    units = sm_count();
    if (TWO) {  // how many CTA pairs can be co-resident (GPCs with an odd SM count leave one SM unpaired)
      cfg.gridDim = dim3(2 * sm_count(), 1, 1);
      int n = 0;
      I8L_CUDA_OK(cudaOccupancyMaxActiveClusters(&n, kernel, &cfg));
      units = n > 0 ? n : 1;
    }
    max_units[dev].store(units, std::memory_order_release);
  }
  if (g_cta_limit > 0) {   // leave SMs free for a kernel that runs beside this one
    const int lim = TWO ? g_cta_limit / 2 : g_cta_limit;
    units = units < lim ? units : (lim > 0 ? lim : 1);
  }
  const int grid_units = (int)(tiles < units ? tiles : units);
  cfg.gridDim = dim3(TWO ? 2 * grid_units : grid_units, 1, 1);
  chain_attribute(cfg, attr);
  I8L_CUDA_OK(cudaLaunchKernelEx(&cfg, kernel, ma, mb, mc, p));
  return I8L_OK;
}

// Tiles of 128 columns (a CTA each) or of 256?  A grid that fills no SM twice finishes with its slowest CTA, and a narrow tile takes
// 0.62 of a wide one's time (0.67 with row x column factors; 0.8 in the whole-K kind, whose wide tiles run two tensor pipes
// on one): half the columns to drain and store, four accumulators instead of two to hide the hand-off in, but as many MMAs of
// nearly the same duration.  So narrow ones pay where they need fewer than 1 / 0.62 times as many waves.  Kernel time, wide
// and narrow: 128x1024x1024 fast kind 9.3 / 7.3 us, row x channel 10.1 / 6.9; 1024x1024x4096 19.1 / 13.7, 24.9 / 15.5, whole-K
// 15.9 / 13.2; 12544x384x2048 (2 waves and 2) 22.2 / 16.1; 6400x1024x4096 (2 and 3) 36.3 / 34.4, row x column factors 69.6 /
// 70.7, whole-K 26.9 / 32.0; 2048^3 (1 and 2) 14.3 / 16.0; 4096^3 (4 and 7) 67.8 / 72.2.
static bool narrow_tiles(int64_t wide, int64_t narrow, int sms, int percent) {
  return (narrow + sms - 1) / sms * percent < (wide + sms - 1) / sms * 100;
}

static int launch_gemm(bool block, const int8_t* a_q, const int8_t* b_q, GemmParams p, int64_t batch, int64_t M,
                       int64_t N, int64_t K, cudaStream_t st) {
  if (batch <= 0 || M <= 0 || N <= 0 || K <= 0 || M % 128 || N % 128 || K % 128)
    return fail(I8L_ERR_SHAPE, "batch=%lld M=%lld N=%lld K=%lld: all positive, M, N, K multiples of 128",
                (long long)batch, (long long)M, (long long)N, (long long)K);
  if (batch * M >= (1ll << 31) || batch * N >= (1ll << 31) || K >= (1ll << 31) ||
      (batch * M / 128) * (N / 128) >= (1ll << 31))
    return fail(I8L_ERR_SHAPE, "problem too large for 32-bit tile coordinates");
  if (!a_q || !b_q || !p.c) return fail(I8L_ERR_ARG, "null pointer");
  if (!aligned16(a_q) || !aligned16(b_q) || !aligned16(p.c)) return fail(I8L_ERR_ALIGN, "a_q, b_q, c must be 16-byte aligned");
  if (int e = check_arch()) return e;
  // One factor per (row or tile, K block) and 128 columns.  Divisors (fused backward, per-tile A scales only) take the
  // exact conversion of the row kind: the fast kind's running shift rounds to about 7e-6, the fused variants are held
  // to 1e-6.
  const bool a_group = p.a_kind == I8L_ASCALE_GROUP, b_group = p.b_kind == I8L_BSCALE_GROUP;
  const bool factors = block && !p.exact && !p.dump;
  const bool scalar_factor = factors && !b_group && (!p.divide || !a_group);
  const bool column_factor = factors && !a_group && b_group;
  const bool outer_factor = factors && !p.divide && a_group && b_group;
  const bool generic = block && !scalar_factor && !column_factor && !outer_factor;   // this kind has wide tiles only
  const int64_t m_blocks = batch * M / 128, wide_tiles = (N + WIDE - 1) / WIDE;
  const int percent = !block ? 80 : outer_factor ? 67 : 62;
  const bool narrow = !generic && narrow_tiles(m_blocks * wide_tiles, m_blocks * (N / NARROW), gemm_cta_budget(), percent);
  // CTA pairs (cta_group::2) need two 128-row blocks of the same batch per tile.  They pay off for the
  // whole-K accumulation (half the B traffic per SM: +2.5 % sustained at the power cap); the per-K-block
  // hand-off of the block-scaled kinds is slower across two CTAs (990 vs 1510 TOP/s), so those stay 1-CTA.
  const bool two = !block && !narrow && (M % 256 == 0);
  const int BN = narrow ? NARROW : WIDE;
  (void)chain_first();   // GEMMs always wait
  // Not under a limit on the CTAs: those of the next GEMM would wait on the very SMs that the limit keeps free.
  p.early = chain_state.gemm_next && gemm_cta_budget() == sm_count();
  chain_state.gemm_next = 0;
  CUtensorMap ma, mb, mc;
  if (int e = make_map(&ma, a_q, batch * M, K, BM)) return e;
  if (int e = make_map(&mb, b_q, p.b_batched ? batch * N : N, K, two ? BM : BN)) return e;
  mc = ma;   // read by nobody when the output is not bf16, or leaves for the owners of its rows
  if (!p.out_f32 && !p.dump && !p.rs_rows)
    if (int e = make_map(&mc, p.c, batch * M, N, 32, true)) return e;
  p.m_blocks = (int)m_blocks;
  p.mpb = (int)(M / 128);
  p.n_tiles = (int)(narrow ? N / NARROW : wide_tiles);
  p.M = (int)M;
  p.N = (int)N;
  p.KB = (int)(K / 128);
  {
    p.mirror = p.status ? mirror_of(p.status) : nullptr;
    p.max_polls = gemm_wait_limit();
    p.withhold = g_test_withhold.load(std::memory_order_relaxed);
  }
  p.c_align32 = (reinterpret_cast<uintptr_t>(p.c) & 31u) == 0;
  for (int r = 0; r < I8L_MAX_RANKS; ++r)
    if (p.rs_rows && p.c_slots[r] && (reinterpret_cast<uintptr_t>(p.c_slots[r]) & 31u)) p.c_align32 = 0;
  // M-units (128-row blocks, or 256-row pair blocks) per raster group: the group's A panel should stay
  // L2-resident while the N tiles are swept (measured best: 4096 rows at K = 8192, flat for deeper K).
  {
    const int64_t fit = (32ll << 20) / (128 * K);
    const int blocks = (int)(fit < 16 ? 16 : (fit > 32 ? 32 : fit));  // below 16 the B re-reads double (ncu: 17.6 vs 9.4 GB)
    p.raster = two ? blocks / 2 : blocks;
  }
  {
    const int m_units = two ? p.m_blocks / 2 : p.m_blocks, last = m_units % p.raster;
    p.per_group.set(p.raster * p.n_tiles);
    p.full_group.set(p.raster);
    p.last_group.set(last ? last : p.raster);
    p.per_batch.set(p.mpb);
  }
  const int64_t tiles = (int64_t)(two ? p.m_blocks / 2 : p.m_blocks) * p.n_tiles;
#define I8L_KIND(K) \
  (narrow ? launch_kind<K, false, NARROW>(ma, mb, mc, p, tiles, st) : launch_kind<K, false, WIDE>(ma, mb, mc, p, tiles, st))
  if (!block) return two ? launch_kind<K_ROWCOL, true, WIDE>(ma, mb, mc, p, tiles, st) : I8L_KIND(K_ROWCOL);
  if (generic) return launch_kind<K_BLOCK_GEN, false, WIDE>(ma, mb, mc, p, tiles, st);
  if (scalar_factor && !a_group && !p.divide) return I8L_KIND(K_BLOCK_FAST);
  if (scalar_factor && p.divide) return I8L_KIND(K_BLOCK_TILEDIV);
  if (scalar_factor) return I8L_KIND(K_BLOCK_ROWFAC);
  if (outer_factor) return I8L_KIND(K_BLOCK_OUTER);
  return I8L_KIND(K_BLOCK_COLFAC);
#undef I8L_KIND
}

}  // namespace i8l

using namespace i8l;

extern "C" int i8l_gemm_block(const int8_t* a_q, const int8_t* b_q, const float* a_scale, const float* b_scale,
                              int a_scale_kind, int b_scale_kind, int b_batched, const void* bias, float post_scale,
                              void* c, int64_t batch, int64_t M, int64_t N, int64_t K, int flags, int32_t* status,
                              void* stream) {
  if (!a_scale || !b_scale) return fail(I8L_ERR_ARG, "null scale pointer");
  if (a_scale_kind != I8L_ASCALE_TILE && a_scale_kind != I8L_ASCALE_GROUP && a_scale_kind != I8L_ASCALE_TILE256)
    return fail(I8L_ERR_ARG, "bad a_scale_kind");
  if (a_scale_kind == I8L_ASCALE_TILE256 && (K % 256 || b_scale_kind != I8L_BSCALE_CHANNEL || (flags & I8L_GEMM_DIVIDE)))
    return fail(I8L_ERR_ARG, "I8L_ASCALE_TILE256 needs K %% 256 == 0 and per-channel b scales");
  if ((flags & I8L_GEMM_PRODUCT_FIRST) && !(flags & I8L_GEMM_EXACT_ORDER))
    return fail(I8L_ERR_ARG, "I8L_GEMM_PRODUCT_FIRST selects an operation order: it needs I8L_GEMM_EXACT_ORDER");
  if (b_scale_kind < I8L_BSCALE_CHANNEL || b_scale_kind > I8L_BSCALE_GROUP) return fail(I8L_ERR_ARG, "bad b_scale_kind");
  if ((flags & I8L_GEMM_DIVIDE) && b_scale_kind == I8L_BSCALE_CHANNEL)
    return fail(I8L_ERR_ARG, "I8L_GEMM_DIVIDE needs per-K-block b scales");
  GemmParams p{};
  p.a_scale = a_scale; p.b_scale = b_scale; p.bias = static_cast<const __nv_bfloat16*>(bias); p.c = c;
  p.status = status; p.b_kind = b_scale_kind; p.b_batched = b_batched ? 1 : 0;
  // 128x256 groups are per-tile scales indexed with a halved K-block number
  p.a_kind = a_scale_kind == I8L_ASCALE_TILE256 ? I8L_ASCALE_TILE : a_scale_kind;
  p.a_kshift = a_scale_kind == I8L_ASCALE_TILE256 ? 1 : 0;
  p.product_first = (flags & I8L_GEMM_PRODUCT_FIRST) ? 1 : 0;
  p.exact = (flags & I8L_GEMM_EXACT_ORDER) ? 1 : 0;
  p.divide = (flags & I8L_GEMM_DIVIDE) ? 1 : 0;
  p.out_f32 = (flags & I8L_GEMM_OUT_F32) ? 1 : 0;
  p.post_scale = post_scale;
  return launch_gemm(true, a_q, b_q, p, batch, M, N, K, static_cast<cudaStream_t>(stream));
}

extern "C" int i8l_gemm_rowcol(const int8_t* a_q, const int8_t* b_q, const float* a_scale, const float* b_scale,
                               int b_batched, const void* bias, float post_scale, void* c, int64_t batch, int64_t M,
                               int64_t N, int64_t K, int flags, int32_t* status, void* stream) {
  if (!a_scale || !b_scale) return fail(I8L_ERR_ARG, "null scale pointer");
  GemmParams p{};
  p.a_scale = a_scale; p.b_scale = b_scale; p.bias = static_cast<const __nv_bfloat16*>(bias); p.c = c;
  p.status = status; p.b_batched = b_batched ? 1 : 0; p.b_kind = I8L_BSCALE_CHANNEL;
  p.out_f32 = (flags & I8L_GEMM_OUT_F32) ? 1 : 0;
  p.post_scale = post_scale;
  return launch_gemm(false, a_q, b_q, p, batch, M, N, K, static_cast<cudaStream_t>(stream));
}

extern "C" int i8l_gemm_dump_i32(const int8_t* a_q, const int8_t* b_q, int b_batched, int32_t* out, int64_t batch,
                                 int64_t M, int64_t N, int64_t K, int per_block, int32_t* status, void* stream) {
  GemmParams p{};
  p.c = out; p.status = status; p.b_batched = b_batched ? 1 : 0; p.dump = per_block ? 2 : 1; p.post_scale = 1.f;
  return launch_gemm(per_block != 0, a_q, b_q, p, batch, M, N, K, static_cast<cudaStream_t>(stream));
}

extern "C" int i8l_gemm_block_scatter(const int8_t* a_q, const int8_t* b_q, const float* a_scale, const float* b_scale,
                                      int b_scale_kind, float post_scale, void* const* c_slots, int world, int rank,
                                      int64_t M, int64_t N, int64_t K, int32_t* status, void* stream) {
  if (!a_scale || !b_scale || !c_slots) return fail(I8L_ERR_ARG, "null pointer");
  if (b_scale_kind != I8L_BSCALE_CHANNEL && b_scale_kind != I8L_BSCALE_TILE) return fail(I8L_ERR_ARG, "bad b_scale_kind");
  if (world < 1 || world > I8L_MAX_RANKS || rank < 0 || rank >= world)
    return fail(I8L_ERR_ARG, "rank %d of %d: at most %d ranks", rank, world, I8L_MAX_RANKS);
  if (M <= 0 || M % ((int64_t)world * 128))
    return fail(I8L_ERR_SHAPE, "M=%lld must split into %d row blocks that are multiples of 128", (long long)M, world);
  GemmParams p{};
  p.a_scale = a_scale; p.b_scale = b_scale; p.status = status;
  p.a_kind = I8L_ASCALE_TILE; p.b_kind = b_scale_kind; p.post_scale = post_scale;
  for (int r = 0; r < world; ++r) {
    if (!c_slots[r] || !aligned16(c_slots[r])) return fail(I8L_ERR_ALIGN, "c_slots[%d] must be a 16-byte aligned device pointer", r);
    p.c_slots[r] = c_slots[r];
  }
  p.c = c_slots[rank];
  p.rs_rows = (int)(M / world);
  p.rs_rank = rank;
  // All ranks walk the row blocks in the same order; starting rank r at the rows of rank r+1 keeps the
  // ranks on different owners at any time (with eight ranks all writing to the same owner the dX GEMM
  // took 5.3 ms instead of 2.5 ms).
  p.m_rot = (int)(((rank + 1) % world) * (M / world / 128));
  return launch_gemm(true, a_q, b_q, p, 1, M, N, K, static_cast<cudaStream_t>(stream));
}

extern "C" int i8l_sum_slots(const void* slots, void* out, int world, int64_t rows, int64_t cols, void* stream) {
  if (!slots || !out) return fail(I8L_ERR_ARG, "null pointer");
  if (world < 1 || rows <= 0 || cols <= 0 || cols % 8) return fail(I8L_ERR_SHAPE, "world >= 1, rows > 0, cols a positive multiple of 8");
  if (!aligned16(slots) || !aligned16(out)) return fail(I8L_ERR_ALIGN, "slots and out must be 16-byte aligned");
  if (int e = check_arch()) return e;
  const int64_t n16 = rows * cols / 8;
  const int64_t want = (n16 + 255) / 256;
  const int64_t cap = (int64_t)sm_count() * 8;
  const int grid = (int)(want < cap ? want : cap);
  sum_slots_kernel<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<const uint4*>(slots),
                                                                        static_cast<uint4*>(out), world, n16);
  I8L_CUDA_OK(cudaGetLastError());
  return I8L_OK;
}

// One device's status word with its pinned host copy: see i8l_status_poll.
struct StatusPoller {
  const int32_t* word;
  volatile int32_t* host;
  volatile int32_t* mirror;   // or null
  cudaStream_t side;
  cudaEvent_t event;
  bool pending;
  std::mutex lock;
};

extern "C" void* i8l_status_open(const int32_t* word, int32_t* host) {
  if (!word || !host) { fail(I8L_ERR_ARG, "null pointer"); return nullptr; }
  StatusPoller* s = new (std::nothrow) StatusPoller;
  if (!s) { fail(I8L_ERR_CUDA, "out of host memory"); return nullptr; }
  s->word = word;
  s->host = host;
  s->mirror = nullptr;
  s->pending = false;
  cudaError_t e = cudaEventCreateWithFlags(&s->event, cudaEventDisableTiming);
  s->side = nullptr;
  if (e != cudaSuccess) {
    fail(I8L_ERR_CUDA, "cudaEventCreateWithFlags failed: %s", cudaGetErrorString(e));
    delete s;
    return nullptr;
  }
  return s;
}

extern "C" int i8l_status_poll(void* poller, void* stream) {
  if (!poller) return fail(I8L_ERR_ARG, "null pointer");
  StatusPoller* s = static_cast<StatusPoller*>(poller);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  I8L_CUDA_OK(cudaStreamIsCapturing(st, &cap));
  if (cap != cudaStreamCaptureStatusNone) return I8L_OK;
  const std::unique_lock<std::mutex> hold(s->lock, std::try_to_lock);
  if (!hold.owns_lock()) return I8L_OK;   // another thread is polling this device
  if (s->pending) {
    const cudaError_t e = cudaEventQuery(s->event);
    if (e == cudaErrorNotReady) {
      (void)cudaGetLastError();   // not an error: leave no trace for the launches that check
      return I8L_OK;
    }
    I8L_CUDA_OK(e);
    s->pending = false;
    if (*s->host) return fail(I8L_ERR_TIMEOUT, "a bounded device-side wait gave up");
  }
  // On a stream of its own: in the caller's stream the copy held up what followed by 3.5 us, and the word may be sampled
  // at any time.
  if (!s->side) I8L_CUDA_OK(cudaStreamCreateWithFlags(&s->side, cudaStreamNonBlocking));
  I8L_CUDA_OK(cudaMemcpyAsync(const_cast<int32_t*>(s->host), s->word, sizeof(int32_t), cudaMemcpyDeviceToHost, s->side));
  I8L_CUDA_OK(cudaEventRecord(s->event, s->side));
  s->pending = true;
  return I8L_OK;
}

extern "C" int i8l_status_reset(void* poller) {
  if (!poller) return fail(I8L_ERR_ARG, "null pointer");
  StatusPoller* s = static_cast<StatusPoller*>(poller);
  const std::lock_guard<std::mutex> hold(s->lock);
  if (s->pending) I8L_CUDA_OK(cudaEventSynchronize(s->event));
  s->pending = false;
  *s->host = 0;
  if (s->mirror) *s->mirror = 0;
  return I8L_OK;
}

extern "C" int i8l_status_mirror(void* poller, int32_t* pinned) {
  if (!poller || !pinned) return fail(I8L_ERR_ARG, "null pointer");
  StatusPoller* s = static_cast<StatusPoller*>(poller);
  void* dev = nullptr;
  I8L_CUDA_OK(cudaHostGetDevicePointer(&dev, pinned, 0));
  const std::lock_guard<std::mutex> hold(g_mirror_lock);
  for (Mirror& m : g_mirrors) {
    const int32_t* w = m.word.load(std::memory_order_relaxed);
    if (w == s->word) return fail(I8L_ERR_ARG, "the status word has a mirror");
    if (w) continue;
    m.device_ptr = static_cast<int32_t*>(dev);
    s->mirror = pinned;
    m.word.store(s->word, std::memory_order_release);
    return I8L_OK;
  }
  return fail(I8L_ERR_ARG, "too many mirrored status words");
}

extern "C" int i8l_status_peek(void* poller) {
  const StatusPoller* s = static_cast<const StatusPoller*>(poller);
  if (s && s->mirror && *s->mirror) return fail(I8L_ERR_TIMEOUT, "a bounded device-side wait gave up");
  return I8L_OK;
}

extern "C" int i8l_set_cta_limit(int max_ctas) {
  if (max_ctas < 0) return fail(I8L_ERR_ARG, "i8l_set_cta_limit: max_ctas must be >= 0");
  g_cta_limit = max_ctas;
  return I8L_OK;
}

extern "C" int i8l_test_set_wait_limit(uint32_t max_polls, int withhold_one_load) {
  g_test_max_polls.store(max_polls, std::memory_order_relaxed);
  g_test_withhold.store(withhold_one_load ? 1 : 0, std::memory_order_relaxed);
  return I8L_OK;
}
