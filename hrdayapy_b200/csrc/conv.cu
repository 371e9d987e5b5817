// tcgen05 3x3x3 convolution kernels (see tc_conv.cuh for the design) and
// their C entry points.
#include "hp_common.cuh"
#include "tc_conv.cuh"

#include <cudaTypedefs.h>

#include <algorithm>
#include <mutex>

namespace hp {
namespace tc {

// One input line (130 voxels: a tile and its halo) in shared memory as the
// forward kernels' K-major A operand: a row of 32, 64 or 128 bytes a voxel in
// the swizzle of that width; 48 and 96 channels are three sub-lines of 32 and
// 64 bytes a voxel.  A TMA box of 8 channels, the unswizzled core matrices,
// fetches the same line as CIN / 8 rows of 16 bytes a voxel: 48 -> 16 at
// 64 x 56 x 128 64 us against 58, 96 -> 32 at 32 x 28 x 128 56.5 against 55.5.
// The swizzle permutes 16-byte columns by address bits, so moving the
// descriptor's start by a voxel row (dx) or by 32 bytes (the next 16 channels)
// needs no other change.
template <int CIN>
struct ALine {
  static constexpr int RB = CIN % 64 == 0 ? 128 : (CIN % 32 == 0 ? 64 : 32);  // bytes a row
  static constexpr int CH = RB / 2;                     // channels a sub-line
  static constexpr int SUB = CIN / CH;                  // sub-lines
  static constexpr int ALIGN = 8 * RB;                  // the swizzle pattern's period
  static constexpr int SUB_BYTES = (LINE + 7) / 8 * ALIGN;
  static constexpr int BYTES = SUB * SUB_BYTES;
  static constexpr int TX = SUB * LINE * RB;
  // byte offset of 16-channel group k
  __host__ __device__ static constexpr int k_off(int k) {
    return 32 * k / RB * SUB_BYTES + 32 * k % RB;
  }
};

template <int CIN, int COUT>
struct ConvCfg {
  using A = ALine<CIN>;
  static constexpr int G = CIN / 8;
  static constexpr int A_BYTES = A::BYTES;
  static constexpr int A_TX = A::TX;
  static constexpr int B_BYTES = 3 * CIN * COUT * 2;
  static constexpr int STAGE = A_BYTES + B_BYTES;
  static constexpr int SMEM = 2 * STAGE + A::ALIGN;
  static constexpr uint32_t COLS = TmemCols<COUT>::value;
  static constexpr uint32_t IDESC = idesc_bf16(TILE_M, COUT);
  static_assert(CIN % 16 == 0 && COUT % 16 == 0 && COUT <= 256, "channel counts");
  static_assert(STAGE % A::ALIGN == 0, "stage alignment");
};

template <int CIN, int COUT>
__global__ void __launch_bounds__(128)
conv3_tc_kernel(const __grid_constant__ CUtensorMap tmX, const __nv_bfloat16* __restrict__ Wp,
                const float* __restrict__ bias, void* __restrict__ Yv,
                const __nv_bfloat16* __restrict__ mask, int D, int H, int W, int epi, int* err) {
  using C = ConvCfg<CIN, COUT>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem =
      (uint8_t*)(((uintptr_t)smem_raw + C::A::ALIGN - 1) & ~(uintptr_t)(C::A::ALIGN - 1));
  __shared__ __align__(8) uint64_t full[2];
  __shared__ __align__(8) uint64_t empty[2];
  __shared__ __align__(8) uint64_t done;
  __shared__ uint32_t tmem_base;
  __shared__ int failed;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int w0 = blockIdx.x * TILE_M, h = blockIdx.y, d = blockIdx.z;

  if (tid == 0) {
    mbar_init(&full[0], 1);
    mbar_init(&full[1], 1);
    mbar_init(&empty[0], 1);
    mbar_init(&empty[1], 1);
    mbar_init(&done, 1);
    failed = 0;
    fence_barrier_init();
  }
  if (warp == 0) tmem_alloc(&tmem_base, C::COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base, 0);

  if (warp == 0) {
    // the warp stays converged; one elected lane issues copies and products
    auto issue = [&](int s, int buf) {
      const int dz = s / 3 - 1, dy = s % 3 - 1;
      uint8_t* A = smem + buf * C::STAGE;
      uint8_t* B = A + C::A_BYTES;
      mbar_expect_tx(&full[buf], C::A_TX + C::B_BYTES);
#pragma unroll
      for (int g = 0; g < C::A::SUB; ++g)
        tma_load_4d(A + g * C::A::SUB_BYTES, &tmX, g * C::A::CH, w0 - 1, h + dy, d + dz,
                    &full[buf]);
      const int tap0 = 9 * (dz + 1) + 3 * (dy + 1);
      bulk_load(B, Wp + (size_t)tap0 * CIN * COUT, C::B_BYTES, &full[buf]);
    };
    if (elect_one()) {
      issue(0, 0);
      issue(1, 1);
    }
    __syncwarp();
    int issued = 2, consumed = 0, code = 0;
    for (int s = 0; s < 9; ++s) {
      const int buf = s & 1;
      const uint32_t par = (s >> 1) & 1;
      if (!mbar_wait_warp(&full[buf], par)) {
        code = 1;
        break;
      }
      tc_fence_after();
      const uint32_t a0 = smem_u32(smem + buf * C::STAGE);
      const uint64_t a_d = smem_desc_sw<C::A::RB>(a0);
      const uint64_t b_d = smem_desc(a0 + C::A_BYTES, COUT * 16, 128);
      if (elect_one()) {
#pragma unroll
        for (int dx = 0; dx < 3; ++dx)
#pragma unroll
          for (int k = 0; k < CIN / 16; ++k)
            mma_bf16(tmem, desc_add(a_d, C::A::k_off(k) + dx * C::A::RB),
                     desc_add(b_d, (dx * C::G + 2 * k) * COUT * 16), C::IDESC,
                     (s | dx | k) != 0);
        mma_commit(&empty[buf]);
      }
      __syncwarp();
      consumed = s + 1;
      if (s + 2 < 9) {
        if (!mbar_wait_warp(&empty[buf], par)) {
          code = 2;
          break;
        }
        if (elect_one()) issue(s + 2, buf);
        __syncwarp();
        ++issued;
      }
    }
    if (code) {
      // let the copies already issued land before the CTA releases smem
      for (int s = consumed; s < issued; ++s) (void)mbar_wait_warp(&full[s & 1], (s >> 1) & 1);
    }
    if (elect_one()) {
      if (code) {
        atomicOr(err, code);
        failed = 1;
      }
      mma_commit(&done);
    }
  }
  __syncthreads();
  const bool ok = mbar_wait(&done, 0) && !failed;
  if (!ok && tid == 0) atomicOr(err, 4);
  tc_fence_after();
  if (ok) {
    // epilogue: this thread owns output voxel w0 + tid, TMEM lane tid
    const uint32_t trow = tmem + ((uint32_t)(warp * 32) << 16);
    const int64_t vox = ((int64_t)d * H + h) * W + w0 + tid;
    if (epi == EPI_F32_C0) {
      float v[16];
      tmem_ld16(trow, v);
      ((float*)Yv)[vox] = v[0] + bias[0];
    } else {
      __nv_bfloat16* Y = (__nv_bfloat16*)Yv;
#pragma unroll
      for (int c0 = 0; c0 < COUT; c0 += 16) {
        float v[16];
        tmem_ld16(trow + c0, v);
        __align__(16) __nv_bfloat16 o[16];
        if (epi == EPI_MASK) {
          const uint4* mp = (const uint4*)(mask + vox * COUT + c0);
          __align__(16) __nv_bfloat16 m[16];
          *(uint4*)&m[0] = mp[0];
          *(uint4*)&m[8] = mp[1];
#pragma unroll
          for (int q = 0; q < 16; ++q)
            o[q] = __float2bfloat16(__bfloat162float(m[q]) > 0.0f ? v[q] : 0.0f);
        } else {
#pragma unroll
          for (int q = 0; q < 16; ++q) {
            float y = v[q] + bias[c0 + q];
            if (epi == EPI_RELU) y = fmaxf(y, 0.0f);
            o[q] = __float2bfloat16(y);
          }
        }
        uint4* yp = (uint4*)(Y + vox * COUT + c0);
        yp[0] = *(uint4*)&o[0];
        yp[1] = *(uint4*)&o[8];
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, C::COLS);
}

// The products of input line ri (h0 - 1 + ri) of a depth slice.  It feeds the
// output lines r within one row of it, by tap row dy = ri - 1 - r.  The tap
// rows are neighbours in the weight block ([dx][CIN/8][dy][COUT][8]) and
// output line r accumulates in columns (R - 1 - r) COUT.., so one product with
// N = 3 COUT does all three (as many as fit N = 256).  A product of 128 rows
// by 16 channels takes about 50 clocks of an SM at N = 16 and hardly more at
// 48 -- reading A, not the arithmetic --, so a narrow layer wants few and wide
// ones: 16 -> 16 at 64 x 56 x 128 20.6 us against 25.1 with a product for each
// tap row, 48 -> 16 39.3 against 57.5, 96 -> 32 at 32 x 28 x 128 34.9 against
// 39.6.
// Within each output line the order of the taps is (dz, dy, dx, channels).
// `first` marks the first depth slice, whose first product into a line (dy -1,
// dx 0, channel group 0) overwrites the accumulator.
template <int CIN, int COUT, int R>
__device__ __forceinline__ void issue_line(uint32_t acc0, uint64_t a_d, uint64_t b_d, int ri,
                                           bool first) {
  using A = ALine<CIN>;
  constexpr int NT = 256 / COUT < 3 ? 256 / COUT : 3;   // tap rows a product
  const int r_hi = ri < R ? ri : R - 1, r_lo = ri > 2 ? ri - 2 : 0;
  const int dy_lo = ri - 1 - r_hi, n_dy = r_hi - r_lo + 1;
#pragma unroll
  for (int q0 = 0; q0 < 3; q0 += NT) {
    if (q0 >= n_dy) continue;
    const int n = n_dy - q0 < NT ? n_dy - q0 : NT;
    const uint32_t td = acc0 + (uint32_t)((R - 1 - r_hi + q0) * COUT);
#pragma unroll
    for (int dx = 0; dx < 3; ++dx)
#pragma unroll
      for (int k = 0; k < CIN / 16; ++k) {
        const uint64_t ad = desc_add(a_d, A::k_off(k) + dx * A::RB);
        const uint64_t bd =
            desc_add(b_d, ((dx * (CIN / 8) + 2 * k) * 3 + dy_lo + 1 + q0) * COUT * 16);
        if (first && dy_lo + q0 == -1 && dx == 0 && k == 0) {
          mma_bf16(td, ad, bd, idesc_bf16(TILE_M, COUT), 0u);
          if (n > 1)
            mma_bf16(td + COUT, ad, desc_add(bd, COUT * 16), idesc_bf16(TILE_M, (n - 1) * COUT),
                     1u);
        } else {
          mma_bf16(td, ad, bd, idesc_bf16(TILE_M, n * COUT), 1u);
        }
      }
  }
}

// The nine taps of depth slice zi to dst as [dx][CIN/8][dy][COUT][8].
template <int CIN, int COUT>
__device__ __forceinline__ void load_taps(uint8_t* dst, const CUtensorMap* tmB, int zi,
                                          uint64_t* bar) {
#pragma unroll
  for (int q = 0; q < 3 * (CIN / 8); ++q)
    tma_load_5d(dst + q * 3 * COUT * 16, tmB, 0, 0, q % (CIN / 8), 9 * zi + q / (CIN / 8), 0, bar);
}

// -------------------------------------------------------------------------
// Row-blocked variant: one CTA computes R output lines (h0 .. h0+R-1 at the
// same (d, w0..w0+127)), one TMEM accumulator of COUT FP32 columns per line.
// One thread issues the copies up to NS stages ahead, one lane of warp 0 the
// products (copy latency does not serialise with the products' completion).
// The K loop runs over dz and the R+2 input lines h0-1 .. h0+R of that
// depth slice: each input line is loaded once and feeds every output line
// within one row of it (up to three), and the 9 (dy, dx) taps of a depth
// slice arrive once per slice -- against one line tile per CTA,
// which loads every input line three times per depth slice and the weights
// nine times.  Two weight buffers (slice zi uses buffer zi & 1; a buffer is
// rewritten only after the MMAs of every stage that read it have completed,
// which the line-stage "empty" wait already guarantees because stages
// complete in order).
template <int CIN, int COUT, int R>
struct RowsCfg {
  using A = ALine<CIN>;
  static constexpr int G = CIN / 8;
  static constexpr int A_BYTES = A::BYTES;
  static constexpr int A_TX = A::TX;
  static constexpr int B_BYTES = 9 * CIN * COUT * 2;
  static constexpr int ACC = COUT;                    // TMEM columns per output line
  static constexpr uint32_t COLS = R * ACC <= 32 ? 32 : (R * ACC <= 64 ? 64 : (R * ACC <= 128 ? 128 : (R * ACC <= 256 ? 256 : 512)));
  // line stages in flight: four where that keeps the CTA's shared memory
  // small (48 KB), else two (more CTAs per SM measured faster there)
  static constexpr int NS = 4 * A_BYTES + 2 * B_BYTES + A::ALIGN <= 48 * 1024 ? 4 : 2;
  static constexpr int SMEM = NS * A_BYTES + 2 * B_BYTES + A::ALIGN;
  static constexpr int NSTG = 3 * (R + 2);
  static_assert(CIN % 16 == 0 && COUT % 16 == 0 && COUT <= 256, "channel counts");
  static_assert(R * ACC <= 512, "TMEM columns");
  static_assert(B_BYTES % 128 == 0 && A_BYTES % A::ALIGN == 0, "stage alignment");
};

constexpr int CONV_ROWS = 4;

template <int CIN, int COUT, int R>
__global__ void __launch_bounds__(128)
conv3_tc_rows_kernel(const __grid_constant__ CUtensorMap tmX,
                     const __grid_constant__ CUtensorMap tmB, const float* __restrict__ bias,
                     void* __restrict__ Yv,
                     const __nv_bfloat16* __restrict__ mask, int D, int H, int W, int epi,
                     int* err) {
  using C = RowsCfg<CIN, COUT, R>;
  constexpr int NS = C::NS;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem =
      (uint8_t*)(((uintptr_t)smem_raw + C::A::ALIGN - 1) & ~(uintptr_t)(C::A::ALIGN - 1));
  __shared__ __align__(8) uint64_t full[NS];
  __shared__ __align__(8) uint64_t empty[NS];
  __shared__ __align__(8) uint64_t done;
  __shared__ uint32_t tmem_base;
  __shared__ volatile int failed;
  __shared__ int issued_s, consumed_s;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int w0 = blockIdx.x * TILE_M, h0 = blockIdx.y * R, d = blockIdx.z;

  if (tid == 0) {
    for (int b = 0; b < NS; ++b) {
      mbar_init(&full[b], 1);
      mbar_init(&empty[b], 1);
    }
    mbar_init(&done, 1);
    failed = 0;
    issued_s = 0;
    consumed_s = 0;
    fence_barrier_init();
  }
  if (warp == 0) tmem_alloc(&tmem_base, C::COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base, 0);
  uint8_t* const Bbase = smem + NS * C::A_BYTES;

  // Producer (thread 32): line stage s goes to buffer s % NS; it is
  // refilled once the products of the stage that last used it completed
  // (its "empty" barrier), so the copies run up to NS stages ahead of the
  // products.  A weight buffer is rewritten (first stage of slice 2) only
  // after the products of every stage of slice 0 completed: stages complete
  // in order and slice 0 ends at least NS stages earlier.
  if (tid == 32) {
    int s = 0;
    for (; s < C::NSTG && !failed; ++s) {
      const int buf = s % NS;
      if (s >= NS && !mbar_wait(&empty[buf], ((s / NS) - 1) & 1)) {
        atomicOr(err, 2);
        failed = 1;
        break;
      }
      const int zi = s / (R + 2), ri = s % (R + 2);
      uint8_t* A = smem + buf * C::A_BYTES;
      const bool new_slice = ri == 0;
      mbar_expect_tx(&full[buf], C::A_TX + (new_slice ? C::B_BYTES : 0));
#pragma unroll
      for (int g = 0; g < C::A::SUB; ++g)
        tma_load_4d(A + g * C::A::SUB_BYTES, &tmX, g * C::A::CH, w0 - 1, h0 - 1 + ri, d + zi - 1,
                    &full[buf]);
      if (new_slice)
        load_taps<CIN, COUT>(Bbase + (zi & 1) * C::B_BYTES, &tmB, zi, &full[buf]);
    }
    issued_s = s;
  }
  // MMA issuer (warp 0, one elected lane).  The line index is unrolled, so a
  // product's operands are a base and a constant.
  if (warp == 0) {
    int s = 0;
    bool ok = true;
    for (int zi = 0; zi < 3 && ok; ++zi) {
      const uint64_t b_d = smem_desc(smem_u32(Bbase + (zi & 1) * C::B_BYTES), 3 * COUT * 16, 128);
#pragma unroll
      for (int ri = 0; ri < R + 2; ++ri) {
        const int buf = s % NS;
        if (!mbar_wait_warp(&full[buf], (s / NS) & 1)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint64_t a_d = smem_desc_sw<C::A::RB>(smem_u32(smem + buf * C::A_BYTES));
        if (elect_one()) {
          issue_line<CIN, COUT, R>(tmem, a_d, b_d, ri, zi == 0);
          mma_commit(&empty[buf]);
        }
        __syncwarp();
        ++s;
      }
    }
    if (elect_one()) {
      if (!ok) {
        atomicOr(err, 1);
        failed = 1;
      }
      consumed_s = s;
      mma_commit(&done);
    }
  }
  __syncthreads();
  if (tid == 32 && failed) {
    // let the copies already issued land before the CTA releases smem
    for (int s = consumed_s; s < issued_s; ++s) (void)mbar_wait(&full[s % NS], (s / NS) & 1);
  }
  __syncthreads();
  const bool ok = mbar_wait(&done, 0) && !failed;
  if (!ok && tid == 0) atomicOr(err, 4);
  tc_fence_after();
  if (ok) {
    // epilogue: this thread owns voxel w0 + tid of every output line, TMEM lane tid
    const uint32_t trow = tmem + ((uint32_t)(warp * 32) << 16);
#pragma unroll 1
    for (int r = 0; r < R; ++r) {
      if (h0 + r >= H) break;
      const uint32_t tl = trow + (uint32_t)((R - 1 - r) * C::ACC);
      const int64_t vox = ((int64_t)d * H + h0 + r) * W + w0 + tid;
      if (epi == EPI_F32_C0) {
        float v[16];
        tmem_ld16(tl, v);
        ((float*)Yv)[vox] = v[0] + bias[0];
      } else {
        __nv_bfloat16* Y = (__nv_bfloat16*)Yv;
#pragma unroll
        for (int c0 = 0; c0 < COUT; c0 += 16) {
          float v[16];
          tmem_ld16(tl + c0, v);
          __align__(16) __nv_bfloat16 o[16];
          if (epi == EPI_MASK) {
            const uint4* mp = (const uint4*)(mask + vox * COUT + c0);
            __align__(16) __nv_bfloat16 m[16];
            *(uint4*)&m[0] = mp[0];
            *(uint4*)&m[8] = mp[1];
#pragma unroll
            for (int q = 0; q < 16; ++q)
              o[q] = __float2bfloat16(__bfloat162float(m[q]) > 0.0f ? v[q] : 0.0f);
          } else {
#pragma unroll
            for (int q = 0; q < 16; ++q) {
              float y = v[q] + bias[c0 + q];
              if (epi == EPI_RELU) y = fmaxf(y, 0.0f);
              o[q] = __float2bfloat16(y);
            }
          }
          uint4* yp = (uint4*)(Y + vox * COUT + c0);
          yp[0] = *(uint4*)&o[0];
          yp[1] = *(uint4*)&o[8];
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, C::COLS);
}

// -------------------------------------------------------------------------
// Persistent warp-specialised variant.  One CTA per SM walks the tiles
// (128 voxels along W x R output lines x one depth) t = blockIdx.x,
// blockIdx.x + gridDim.x, ... with three roles:
//   warp 0, lane 0: producer -- the line stages of every tile in one
//     continuous sequence (dz-major, R + 2 input lines per depth slice,
//     TMA line loads plus the slice's 9-tap weight block on the slice's
//     first line) into an NS-stage ring, refilling a stage once the
//     products that read it completed;
//   warp 1, lane 0: MMA issuer -- the products of tile j into one of two
//     TMEM accumulator sets (R lines x ACC columns each, set j & 1), then a
//     commit that hands the set to the epilogue;
//   warps 2-5: epilogue -- each thread owns TMEM lane (warp & 3) * 32 +
//     lane, i.e. one voxel of the tile: it reads the R lines' accumulators,
//     applies the epilogue, stores, and releases the set, while the products
//     of the next tile run in the other set.
// The weight block of a depth slice is double-buffered by global slice
// index; a buffer is rewritten at the first stage of the slice two later,
// whose ring wait (NS <= R + 2 stages back) already covers every product of
// the slice that read it.  Every wait is bounded; on a timeout the role
// records the location in *err and sets a shared flag that makes the other
// roles stop, the CTA waits (bounded) for its copies and products in
// flight, frees its TMEM and returns.
template <int CIN, int COUT, int RR>
struct PersistCfg {
  using A = ALine<CIN>;
  static constexpr int G = CIN / 8;
  static constexpr int A_BYTES = A::BYTES;
  static constexpr int A_TX = A::TX;
  static constexpr int B_BYTES = 9 * CIN * COUT * 2;
  static constexpr int ACC = COUT;                           // TMEM columns per output line
  static constexpr int R = RR;                                // output lines per tile
  static constexpr int NSTG = 3 * (R + 2);                   // line stages per tile
  static constexpr uint32_t COLS = 2 * R * ACC <= 128 ? 128 : (2 * R * ACC <= 256 ? 256 : 512);
  static constexpr int NS_FIT = (200 * 1024 - 2 * B_BYTES - A::ALIGN) / A_BYTES;
  static constexpr int NS = NS_FIT > R + 2 ? R + 2 : NS_FIT;
  static constexpr int SMEM = NS * A_BYTES + 2 * B_BYTES + A::ALIGN;
  static_assert(CIN % 16 == 0 && COUT % 16 == 0 && COUT <= 256, "channel counts");
  static_assert(NS >= 2 && NS <= R + 2, "ring depth (the weight-buffer reuse needs NS <= R + 2)");
  static_assert(2 * R * ACC <= 512, "TMEM columns");
  static_assert(B_BYTES % 128 == 0 && A_BYTES % A::ALIGN == 0, "stage alignment");
};

constexpr int PERSIST_THREADS = 192;

template <int CIN, int COUT, int RR>
__global__ void __launch_bounds__(PERSIST_THREADS, 1)
conv3_tc_persist_kernel(const __grid_constant__ CUtensorMap tmX,
                        const __grid_constant__ CUtensorMap tmB, const float* __restrict__ bias,
                        void* __restrict__ Yv, const __nv_bfloat16* __restrict__ mask, int D,
                        int H, int W, int epi, int* err) {
  using C = PersistCfg<CIN, COUT, RR>;
  constexpr int NS = C::NS, R = C::R, NSTG = C::NSTG, ACC = C::ACC;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem =
      (uint8_t*)(((uintptr_t)smem_raw + C::A::ALIGN - 1) & ~(uintptr_t)(C::A::ALIGN - 1));
  __shared__ __align__(8) uint64_t full[NS];
  __shared__ __align__(8) uint64_t empty[NS];
  __shared__ __align__(8) uint64_t acc_full[2];
  __shared__ __align__(8) uint64_t acc_empty[2];
  __shared__ __align__(8) uint64_t done;
  __shared__ uint32_t tmem_base;
  __shared__ volatile int failed;
  __shared__ int issued_s, consumed_s;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int n_wt = W / TILE_M, n_hb = (H + R - 1) / R;
  const int n_tiles = n_wt * n_hb * D;

  if (tid == 0) {
    for (int b = 0; b < NS; ++b) {
      mbar_init(&full[b], 1);
      mbar_init(&empty[b], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 128);
    }
    mbar_init(&done, 1);
    failed = 0;
    issued_s = 0;
    consumed_s = 0;
    fence_barrier_init();
  }
  if (warp == 0) tmem_alloc(&tmem_base, C::COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base, 0);
  uint8_t* const Bbase = smem + NS * C::A_BYTES;
  auto fail = [&](int code) {
    atomicOr(err, code);
    failed = 1;
  };

  if (warp == 0) {
    if (lane == 0) {  // producer
      int s = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x) {
        const int w0 = (t % n_wt) * TILE_M, q = t / n_wt;
        const int h0 = (q % n_hb) * R, d = q / n_hb;
        for (int st = 0; st < NSTG; ++st, ++s) {
          const int buf = s % NS;
          if (s >= NS && !mbar_wait_f(&empty[buf], ((s / NS) - 1) & 1, &failed)) {
            fail(2);
            ok = false;
            break;
          }
          const int zi = st / (R + 2), ri = st % (R + 2);
          uint8_t* A = smem + buf * C::A_BYTES;
          const bool new_slice = ri == 0;
          mbar_expect_tx(&full[buf], C::A_TX + (new_slice ? C::B_BYTES : 0));
#pragma unroll
          for (int g = 0; g < C::A::SUB; ++g)
            tma_load_4d(A + g * C::A::SUB_BYTES, &tmX, g * C::A::CH, w0 - 1, h0 - 1 + ri,
                        d + zi - 1, &full[buf]);
          if (new_slice)
            load_taps<CIN, COUT>(Bbase + ((s / (R + 2)) & 1) * C::B_BYTES, &tmB, zi, &full[buf]);
        }
      }
      issued_s = s;
    }
  } else if (warp == 1) {
    // MMA issuer: the warp stays converged, one elected lane issues
    int s = 0, j = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x, ++j) {
      const int b = j & 1;
      if (j >= 2 && !__all_sync(0xffffffffu,
                                mbar_wait_f(&acc_empty[b], ((j >> 1) - 1) & 1, &failed))) {
        if (lane == 0) fail(8);
        break;
      }
      tc_fence_after();
      const uint32_t accb = tmem + (uint32_t)(b * R * ACC);
      for (int zi = 0; zi < 3 && ok; ++zi) {
        const uint64_t b_d =
            smem_desc(smem_u32(Bbase + ((s / (R + 2)) & 1) * C::B_BYTES), 3 * COUT * 16, 128);
#pragma unroll
        for (int ri = 0; ri < R + 2; ++ri) {
          const int buf = s % NS;
          if (!__all_sync(0xffffffffu, mbar_wait_f(&full[buf], (s / NS) & 1, &failed))) {
            if (lane == 0) fail(1);
            ok = false;
            break;
          }
          tc_fence_after();
          const uint64_t a_d = smem_desc_sw<C::A::RB>(smem_u32(smem + buf * C::A_BYTES));
          if (elect_one()) {
            issue_line<CIN, COUT, R>(accb, a_d, b_d, ri, zi == 0);
            mma_commit(&empty[buf]);
          }
          __syncwarp();
          ++s;
        }
      }
      if (!ok) break;
      if (elect_one()) mma_commit(&acc_full[b]);
      __syncwarp();
    }
    // every product issued has completed before the CTA releases TMEM
    if (elect_one()) {
      consumed_s = s;
      mma_commit(&done);
      if (!mbar_wait(&done, 0)) atomicOr(err, 4);
    }
  } else {  // epilogue: warps 2-5, TMEM lane quarter warp & 3
    const int row = (warp & 3) * 32 + lane;
    const uint32_t tlane = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    int j = 0;
    for (int t = blockIdx.x; t < n_tiles; t += gridDim.x, ++j) {
      const int b = j & 1;
      if (!mbar_wait_sleep(&acc_full[b], (j >> 1) & 1, &failed)) {
        if (lane == 0) fail(16);
        break;
      }
      tc_fence_after();
      const int w0 = (t % n_wt) * TILE_M, q = t / n_wt;
      const int h0 = (q % n_hb) * R, d = q / n_hb;
#pragma unroll 1
      for (int r = 0; r < R; ++r) {
        if (h0 + r >= H) break;
        const uint32_t tl = tlane + (uint32_t)((b * R + R - 1 - r) * ACC);
        const int64_t vox = ((int64_t)d * H + h0 + r) * W + w0 + row;
        if (epi == EPI_F32_C0) {
          float v[16];
          tmem_ld16(tl, v);
          ((float*)Yv)[vox] = v[0] + bias[0];
        } else {
          __nv_bfloat16* Y = (__nv_bfloat16*)Yv;
#pragma unroll
          for (int c0 = 0; c0 < COUT; c0 += 16) {
            float v[16];
            tmem_ld16(tl + c0, v);
            __align__(16) __nv_bfloat16 o[16];
            if (epi == EPI_MASK) {
              const uint4* mp = (const uint4*)(mask + vox * COUT + c0);
              __align__(16) __nv_bfloat16 m[16];
              *(uint4*)&m[0] = mp[0];
              *(uint4*)&m[8] = mp[1];
#pragma unroll
              for (int qq = 0; qq < 16; ++qq)
                o[qq] = __float2bfloat16(__bfloat162float(m[qq]) > 0.0f ? v[qq] : 0.0f);
            } else {
#pragma unroll
              for (int qq = 0; qq < 16; ++qq) {
                float y = v[qq] + bias[c0 + qq];
                if (epi == EPI_RELU) y = fmaxf(y, 0.0f);
                o[qq] = __float2bfloat16(y);
              }
            }
            uint4* yp = (uint4*)(Y + vox * COUT + c0);
            yp[0] = *(uint4*)&o[0];
            yp[1] = *(uint4*)&o[8];
          }
        }
      }
      tc_fence_before();
      mbar_arrive(&acc_empty[b]);
    }
  }
  __syncthreads();
  if (tid == 0 && failed) {
    // let the copies already issued land before the CTA releases its smem
    for (int s = consumed_s; s < issued_s; ++s) (void)mbar_wait(&full[s % NS], (s / NS) & 1);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, C::COLS);
}

// -------------------------------------------------------------------------
// host side: tensor maps and dispatch

static PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;

static hp_status get_encode() {
  static std::once_flag once;
  static cudaError_t st = cudaSuccess;
  std::call_once(once, [] {
    cudaDriverEntryPointQueryResult q;
    void* fn = nullptr;
    st = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q);
    if (st == cudaSuccess && q == cudaDriverEntryPointSuccess) g_encode = (PFN_cuTensorMapEncodeTiled_v12000)fn;
  });
  if (!g_encode) {
    hp::set_error("cuTensorMapEncodeTiled is not available");
    return HP_ERR_CUDA;
  }
  return HP_OK;
}

// Tensor map over X[D][H][W][C] (bf16) with box (box_c ch, box_w voxels, 1, 1);
// boxes of 16, 32 and 64 channels land in the swizzle of their row's width.
hp_status make_line_map(CUtensorMap* map, const void* X, int D, int H, int W, int Cch,
                        int box_w = LINE, int box_c = 8) {
  hp_status s = get_encode();
  if (s != HP_OK) return s;
  if (((uintptr_t)X & 15) != 0) {
    hp::set_error("conv input must be 16-byte aligned");
    return HP_ERR_INVALID;
  }
  cuuint64_t dims[4] = {(cuuint64_t)Cch, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)D};
  cuuint64_t strides[3] = {(cuuint64_t)Cch * 2, (cuuint64_t)W * Cch * 2,
                           (cuuint64_t)H * W * Cch * 2};
  cuuint32_t box[4] = {(cuuint32_t)box_c, (cuuint32_t)box_w, 1, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  const CUtensorMapSwizzle swizzle = box_c == 64   ? CU_TENSOR_MAP_SWIZZLE_128B
                                     : box_c == 32 ? CU_TENSOR_MAP_SWIZZLE_64B
                                     : box_c == 16 ? CU_TENSOR_MAP_SWIZZLE_32B
                                                   : CU_TENSOR_MAP_SWIZZLE_NONE;
  CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, (void*)X, dims, strides, box,
                        estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    hp::set_error("cuTensorMapEncodeTiled failed (%d)", (int)r);
    return HP_ERR_CUDA;
  }
  return HP_OK;
}

// Tensor map over the packed weights [27][cin/8][cout][8] whose box is the
// three dy taps of one (dz, dx, channel group) as [dy][cout][8].
hp_status make_tap_map(CUtensorMap* map, const void* Wp, int cin, int cout) {
  hp_status s = get_encode();
  if (s != HP_OK) return s;
  const cuuint64_t row = (cuuint64_t)cout * 16, tap = row * (cin / 8);
  cuuint64_t dims[5] = {128, (cuuint64_t)cout / 16, (cuuint64_t)cin / 8, 21, 3};
  cuuint64_t strides[4] = {256, row, tap, 3 * tap};
  cuuint32_t box[5] = {128, (cuuint32_t)cout / 16, 1, 1, 3};
  cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, (void*)Wp, dims, strides, box,
                        estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    hp::set_error("cuTensorMapEncodeTiled failed (%d)", (int)r);
    return HP_ERR_CUDA;
  }
  return HP_OK;
}

typedef void (*ConvFn)(CUtensorMap, const __nv_bfloat16*, const float*, void*,
                       const __nv_bfloat16*, int, int, int, int, int*);
typedef void (*ConvLinesFn)(CUtensorMap, CUtensorMap, const float*, void*, const __nv_bfloat16*,
                            int, int, int, int, int*);

struct ConvEntry {
  int cin, cout, box_c, smem;
  ConvFn fn;
  int rows_smem;
  ConvLinesFn rows_fn;   // CONV_ROWS output lines per CTA
  int persist_smem;
  ConvLinesFn persist_fn;   // persistent warp-specialised kernel, or null
  int persist_rows;
  uint32_t persist_cols;
};

// Kernel per layer shape, from timings of hp_conv3_forward (cold L2, CUDA
// events) at 32 x 28 x 128 and 64 x 56 x 128: with few input channels a
// product chain is short and row-blocked CTAs, several on an SM, hide its
// waits (16 -> 16 22.6 us against 38.4 for the persistent kernel, 48 -> 16
// 49.2 against 52.2, 16 -> 32 17.4 against 18.4, 32 -> 32 20.0 against 20.5);
// with many, or with COUT 96, the weights leave room for one or two CTAs and
// the persistent kernel's second accumulator set hides the epilogue.
#define HP_CONV(ci, co)                                                                     \
  {ci, co, ALine<ci>::CH, ConvCfg<ci, co>::SMEM, conv3_tc_kernel<ci, co>,                   \
   RowsCfg<ci, co, CONV_ROWS>::SMEM, conv3_tc_rows_kernel<ci, co, CONV_ROWS>, 0, nullptr, 0, 0}
#define HP_CONV_P(ci, co)                                                                   \
  {ci, co, ALine<ci>::CH, ConvCfg<ci, co>::SMEM, conv3_tc_kernel<ci, co>,                   \
   RowsCfg<ci, co, CONV_ROWS>::SMEM, conv3_tc_rows_kernel<ci, co, CONV_ROWS>,               \
   PersistCfg<ci, co, 2>::SMEM, conv3_tc_persist_kernel<ci, co, 2>, 2, PersistCfg<ci, co, 2>::COLS}
static const ConvEntry kConv[] = {
    HP_CONV(16, 16),   HP_CONV(16, 32),   HP_CONV(32, 16),   HP_CONV(32, 32), HP_CONV(32, 64),
    HP_CONV_P(64, 32), HP_CONV_P(64, 64), HP_CONV(48, 16),   HP_CONV_P(96, 32), HP_CONV(16, 48),
    HP_CONV_P(32, 96),
};
#undef HP_CONV
#undef HP_CONV_P

hp_status conv3_launch(const void* X, const void* Wp, const float* bias, void* Y,
                       const void* mask, int D, int H, int W, int cin, int cout, int epi,
                       int* err, cudaStream_t s) {
  const ConvEntry* e = nullptr;
  for (const auto& c : kConv)
    if (c.cin == cin && c.cout == cout) e = &c;
  if (!e) {
    hp::set_error("conv %d->%d is not compiled", cin, cout);
    return HP_ERR_UNSUPPORTED;
  }
  if (W % TILE_M != 0 || D < 1 || H < 1) {
    hp::set_error("conv grid W=%d must be a multiple of %d", W, TILE_M);
    return HP_ERR_INVALID;
  }
  if (((uintptr_t)Wp & 15) || ((uintptr_t)Y & 15) || (mask && ((uintptr_t)mask & 15))) {
    hp::set_error("conv buffers must be 16-byte aligned");
    return HP_ERR_INVALID;
  }
  CUtensorMap map;
  hp_status st = make_line_map(&map, X, D, H, W, cin, LINE, e->box_c);
  if (st != HP_OK) return st;
  CUtensorMap taps;
  st = make_tap_map(&taps, Wp, cin, cout);
  if (st != HP_OK) return st;
  static bool attr_set[sizeof(kConv) / sizeof(kConv[0])] = {false};
  static int persist_grid[sizeof(kConv) / sizeof(kConv[0])] = {0};
  const int idx = (int)(e - kConv);
  if (!attr_set[idx]) {
    HP_CUDA_TRY(cudaFuncSetAttribute((const void*)e->fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     e->smem));
    HP_CUDA_TRY(cudaFuncSetAttribute((const void*)e->rows_fn,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, e->rows_smem));
    if (e->persist_fn) {
      HP_CUDA_TRY(cudaFuncSetAttribute((const void*)e->persist_fn,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       e->persist_smem));
      // resident CTAs of the persistent kernel: shared memory and TMEM columns
      int dev = 0, n_sm = 0, per_sm = 0;
      HP_CUDA_TRY(cudaGetDevice(&dev));
      HP_CUDA_TRY(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev));
      HP_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
          &per_sm, (const void*)e->persist_fn, PERSIST_THREADS, e->persist_smem));
      per_sm = std::min(per_sm, (int)(512 / e->persist_cols));
      persist_grid[idx] = std::max(1, per_sm) * n_sm;
    }
    attr_set[idx] = true;
  }
  if (e->persist_fn) {
    const int n_tiles = (W / TILE_M) * ((H + e->persist_rows - 1) / e->persist_rows) * D;
    const int grid = std::min(n_tiles, persist_grid[idx]);
    e->persist_fn<<<grid, PERSIST_THREADS, e->persist_smem, s>>>(
        map, taps, bias, Y, (const __nv_bfloat16*)mask, D, H, W, epi, err);
    HP_CUDA_TRY(cudaGetLastError());
    return HP_OK;
  }
  // Row-blocked CTAs where their two line stages and two weight slices stay
  // small enough for several CTAs per SM; else (32 -> 64) one line per CTA:
  // 15.3 us at 16 x 14 x 128, as the persistent kernel takes, and 19.5 against
  // 20.5 at 24 x 20 x 128.
  if (e->rows_smem <= 64 * 1024) {
    dim3 grid(W / TILE_M, (H + CONV_ROWS - 1) / CONV_ROWS, D);
    e->rows_fn<<<grid, 128, e->rows_smem, s>>>(map, taps, bias, Y, (const __nv_bfloat16*)mask, D,
                                               H, W, epi, err);
  } else {
    dim3 grid(W / TILE_M, H, D);
    e->fn<<<grid, 128, e->smem, s>>>(map, (const __nv_bfloat16*)Wp, bias, Y,
                                     (const __nv_bfloat16*)mask, D, H, W, epi, err);
  }
  HP_CUDA_TRY(cudaGetLastError());
  return HP_OK;
}


// -------------------------------------------------------------------------
// Weight gradient of a 3x3x3 layer on the tensor cores:
//   gw[co][ci][t] = sum_v G[v][co] X[v + off(t)][ci],  gb[co] = sum_v G[v][co]
// as GEMMs with K = voxels.  The [voxel][8-channel] line tiles that TMA
// brings in for the forward pass are, read transposed, MN-major UMMA
// operands: a core matrix is 8 voxel rows (K) of 16 bytes (8 channels), K
// groups 128 bytes apart, channel groups one tile chunk apart.  A CTA owns
// one dz and a range of output lines (d, h, 128 voxels along W); per line
// it loads the three input lines (d+dz, h-1..h+1) of X (130 voxels with the
// halo, zero-filled outside the grid) as 3 CIN/8 chunk slots and the G line
// as N/8 chunks.  The slots form M tiles of 128 rows (16 slots; rows past
// the last slot read zeroed slots), and the three dx taps are the same tile
// with the descriptor start moved by one voxel row (16 bytes), as in the
// forward kernel.  Each (M tile, dx) accumulates over the CTA's lines in
// its own TMEM columns (M = 128 rows, N = padded COUT, FP32).  The CTAs'
// partial sums go to a workspace and a second kernel adds them in a fixed
// order: the result does not depend on scheduling (no atomics).
template <int CIN, int N>
struct WgCfg {
  static constexpr int G = CIN / 8;              // chunks per input line
  static constexpr int S = 3 * G;                // loaded slots per line (dy = -1, 0, 1)
  static constexpr int T = (S + 15) / 16;        // M tiles of 128 rows
  static constexpr int A_BYTES = 16 * T * CHUNK;
  static constexpr int A_TX = S * LINE * 16;
  static constexpr int B_BYTES = (N / 8) * TILE_M * 16;
  static constexpr int STAGE = A_BYTES + B_BYTES;
  static constexpr int SMEM = 2 * STAGE + 128;
  static constexpr int ACC = 3 * T * N;          // TMEM columns of the accumulators
  static constexpr uint32_t COLS =
      ACC <= 32 ? 32 : (ACC <= 64 ? 64 : (ACC <= 128 ? 128 : (ACC <= 256 ? 256 : 512)));
  // BF16 x BF16 -> FP32, M = 128, both operands MN-major (bits 15 and 16)
  static constexpr uint32_t IDESC = idesc_bf16(TILE_M, N) | (1u << 15) | (1u << 16);
  static_assert(CIN % 8 == 0 && N % 16 == 0 && N <= 256, "channel counts");
  static_assert(ACC <= 512, "TMEM columns");
  static_assert(SMEM <= 227 * 1024, "shared memory");
  static_assert(A_BYTES % 128 == 0 && B_BYTES % 128 == 0, "stage alignment");
};

template <int CIN, int N>
__global__ void __launch_bounds__(128)
wgrad3_tc_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmG,
                 int D, int H, int WT, int lines_per_cta, float* __restrict__ part, int* err) {
  using C = WgCfg<CIN, N>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 127) & ~(uintptr_t)127);
  __shared__ __align__(8) uint64_t full[2];
  __shared__ __align__(8) uint64_t empty[2];
  __shared__ __align__(8) uint64_t done;
  __shared__ uint32_t tmem_base;
  __shared__ int failed;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int dz = (int)blockIdx.y - 1;
  const int nl = D * H * WT;
  const int l0 = blockIdx.x * lines_per_cta;
  const int l1 = min(nl, l0 + lines_per_cta);

  // the slots past the loaded ones are read by the last M tile: zero them
  // in both stages (the TMA never writes them)
  for (int buf = 0; buf < 2; ++buf) {
    uint4* z = (uint4*)(smem + buf * C::STAGE + C::S * CHUNK);
    const int n16 = (16 * C::T - C::S) * CHUNK / 16;
    for (int q = tid; q < n16; q += 128) z[q] = make_uint4(0u, 0u, 0u, 0u);
  }
  fence_proxy_async();
  if (tid == 0) {
    mbar_init(&full[0], 1);
    mbar_init(&full[1], 1);
    mbar_init(&empty[0], 1);
    mbar_init(&empty[1], 1);
    mbar_init(&done, 1);
    failed = 0;
    fence_barrier_init();
  }
  if (warp == 0) tmem_alloc(&tmem_base, C::COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base, 0);
  const int nmine = max(0, l1 - l0);

  if (warp == 0) {
    // the warp stays converged; one elected lane issues copies and products
    auto issue = [&](int li, int buf) {
      const int wt = li % WT, h = (li / WT) % H, d = li / (WT * H);
      uint8_t* A = smem + buf * C::STAGE;
      uint8_t* B = A + C::A_BYTES;
      mbar_expect_tx(&full[buf], C::A_TX + C::B_BYTES);
#pragma unroll
      for (int dy = 0; dy < 3; ++dy)
#pragma unroll
        for (int g = 0; g < C::G; ++g)
          tma_load_4d(A + (dy * C::G + g) * CHUNK, &tmX, g * 8, wt * TILE_M - 1, h + dy - 1,
                      d + dz, &full[buf]);
#pragma unroll
      for (int g = 0; g < N / 8; ++g)
        tma_load_4d(B + g * TILE_M * 16, &tmG, g * 8, wt * TILE_M, h, d, &full[buf]);
    };
    int issued = min(nmine, 2), consumed = 0, code = 0;
    if (elect_one()) {
      for (int s = 0; s < issued; ++s) issue(l0 + s, s);
    }
    __syncwarp();
    for (int s = 0; s < nmine; ++s) {
      const int buf = s & 1;
      const uint32_t par = (s >> 1) & 1;
      if (!mbar_wait_warp(&full[buf], par)) {
        code = 8;
        break;
      }
      tc_fence_after();
      const uint32_t a0 = smem_u32(smem + buf * C::STAGE);
      const uint64_t a_d = smem_desc(a0, 128, CHUNK);
      const uint64_t b_d = smem_desc(a0 + C::A_BYTES, 128, TILE_M * 16);
      if (elect_one()) {
#pragma unroll
        for (int t = 0; t < C::T; ++t)
#pragma unroll
          for (int dx = 0; dx < 3; ++dx)
#pragma unroll
            for (int k = 0; k < TILE_M / 16; ++k)
              mma_bf16(tmem + (uint32_t)((t * 3 + dx) * N),
                       desc_add(a_d, 16 * t * CHUNK + dx * 16 + k * 256), desc_add(b_d, k * 256),
                       C::IDESC, (s | k) != 0);
        mma_commit(&empty[buf]);
      }
      __syncwarp();
      consumed = s + 1;
      if (s + 2 < nmine) {
        if (!mbar_wait_warp(&empty[buf], par)) {
          code = 16;
          break;
        }
        if (elect_one()) issue(l0 + s + 2, buf);
        __syncwarp();
        ++issued;
      }
    }
    if (code) {
      for (int s = consumed; s < issued; ++s) (void)mbar_wait_warp(&full[s & 1], (s >> 1) & 1);
    }
    if (elect_one()) {
      if (code) {
        atomicOr(err, code);
        failed = 1;
      }
      mma_commit(&done);
    }
  }
  __syncthreads();
  const bool ok = mbar_wait(&done, 0) && !failed;
  if (!ok && tid == 0) atomicOr(err, 32);
  tc_fence_after();
  // epilogue: TMEM lane tid = GEMM row tid of every (M tile, dx)
  const uint32_t trow = tmem + ((uint32_t)(warp * 32) << 16);
  const int64_t base = ((int64_t)blockIdx.y * gridDim.x + blockIdx.x) * (C::T * 3);
#pragma unroll 1
  for (int q = 0; q < C::T * 3; ++q) {
    float* dst = part + ((base + q) * TILE_M + tid) * N;
#pragma unroll
    for (int c0 = 0; c0 < N; c0 += 16) {
      float v[16];
      if (ok && nmine > 0) {
        tmem_ld16(trow + (uint32_t)(q * N + c0), v);
      } else {
#pragma unroll
        for (int u = 0; u < 16; ++u) v[u] = 0.0f;
      }
#pragma unroll
      for (int u = 0; u < 16; u += 4) *(float4*)(dst + c0 + u) = make_float4(v[u], v[u + 1], v[u + 2], v[u + 3]);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, C::COLS);
}

// Per-block partial sums of G over voxels (bias gradient), fixed order:
// thread (r, co) sums voxels r, r + R, ... of the block's range, then the
// block adds its R rows in order.
constexpr int GS_BLOCKS = 256;
__global__ void __launch_bounds__(256)
gsum_partial_kernel(const __nv_bfloat16* __restrict__ G, int64_t n, int coP, float* __restrict__ part) {
  __shared__ float sh[256];
  const int R = 256 / coP;
  const int r = threadIdx.x / coP, co = threadIdx.x % coP;
  const int64_t chunk = (n + gridDim.x - 1) / gridDim.x;
  const int64_t v0 = blockIdx.x * chunk, v1 = min(n, v0 + chunk);
  float acc = 0.0f;
  if (r < R)
    for (int64_t v = v0 + r; v < v1; v += R) acc += __bfloat162float(G[v * coP + co]);
  sh[threadIdx.x] = r < R ? acc : 0.0f;
  __syncthreads();
  if (threadIdx.x < coP) {
    float s = 0.0f;
    for (int q = 0; q < R; ++q) s += sh[q * coP + threadIdx.x];
    part[(int64_t)blockIdx.x * coP + threadIdx.x] = s;
  }
}

// gw[co][ci][t] and gb[co] from the partials, each summed in CTA order.  A
// warp's lanes take consecutive output channels of one (dz, M tile, dx, row),
// so every read is a row segment of the partial tiles, RED_BATCH chunks in
// flight (threads in gw's own order read one float a sector).  The bias blocks,
// 16 channels each, bring their GS_BLOCKS rows to shared memory at once and add
// them there.
constexpr int RED_BATCH = 25;
template <int CIN, int N>
__global__ void __launch_bounds__(256)
wgrad_reduce_kernel(const float* __restrict__ part, int nchunk, const float* __restrict__ gpart,
                    int cout, float* __restrict__ gw, float* __restrict__ gb) {
  using C = WgCfg<CIN, N>;
  constexpr int ROWS = 8 * C::S;  // loaded rows over the M tiles
  constexpr int W_BLOCKS = (9 * ROWS * N + 255) / 256;
  if (blockIdx.x >= W_BLOCKS) {
    __shared__ float sh[GS_BLOCKS][17];
    const int c0 = (blockIdx.x - W_BLOCKS) * 16, c = threadIdx.x % 16;
    float v[GS_BLOCKS / 16];
#pragma unroll
    for (int u = 0; u < GS_BLOCKS / 16; ++u)
      v[u] = __ldg(gpart + (int64_t)(threadIdx.x / 16 + 16 * u) * N + c0 + c);
#pragma unroll
    for (int u = 0; u < GS_BLOCKS / 16; ++u) sh[threadIdx.x / 16 + 16 * u][c] = v[u];
    __syncthreads();
    if (threadIdx.x < 16 && c0 + c < cout) {
      float s = 0.0f;
#pragma unroll 16
      for (int b = 0; b < GS_BLOCKS; ++b) s += sh[b][c];
      gb[c0 + c] = s;
    }
    return;
  }
  const int e = blockIdx.x * 256 + threadIdx.x;
  const int co = e % N, slot_row = (e / N) % ROWS, q = e / (N * ROWS);  // q = 3 dz + dx
  if (q >= 9 || co >= cout) return;
  const int dzi = q / 3, dx = q % 3, slot = slot_row / 8;
  const int dy = slot / C::G, ci = slot % C::G * 8 + slot_row % 8;
  constexpr int64_t step = (int64_t)(C::T * 3) * TILE_M * N;
  const float* src = part + (int64_t)dzi * nchunk * step +
                     ((int64_t)(slot / 16 * 3 + dx) * TILE_M + slot % 16 * 8 + slot_row % 8) * N + co;
  float s = 0.0f;
  int k = 0;
  for (; k + RED_BATCH <= nchunk; k += RED_BATCH) {
    float v[RED_BATCH];
#pragma unroll
    for (int u = 0; u < RED_BATCH; ++u) v[u] = __ldg(src + (k + u) * step);
#pragma unroll
    for (int u = 0; u < RED_BATCH; ++u) s += v[u];
  }
#pragma unroll 4
  for (; k < nchunk; ++k) s += __ldg(src + k * step);
  gw[((int64_t)co * CIN + ci) * 27 + dzi * 9 + dy * 3 + dx] = s;
}

static int wg_chunks(int nl) {
  // about two CTAs per SM over the three dz slices, at least one line each
  const int target = 100;
  const int per = std::max(1, (nl + target - 1) / target);
  return (nl + per - 1) / per;
}

int64_t wgrad3_workspace(int D, int H, int W, int cin, int cout) {
  const int N = cout < 16 ? 16 : cout;
  const int T = (3 * (cin / 8) + 15) / 16;
  const int nl = D * H * std::max(1, W / TILE_M);
  return (int64_t)3 * wg_chunks(nl) * T * 3 * TILE_M * N * 4 + (int64_t)GS_BLOCKS * N * 4;
}

typedef void (*WgFn)(CUtensorMap, CUtensorMap, int, int, int, int, float*, int*);
typedef void (*WgRedFn)(const float*, int, const float*, int, float*, float*);
struct WgEntry {
  int cin, n, smem;
  WgFn fn;
  WgRedFn red;
};
#define HP_WG(ci, n) {ci, n, WgCfg<ci, n>::SMEM, wgrad3_tc_kernel<ci, n>, wgrad_reduce_kernel<ci, n>}
static const WgEntry kWg[] = {
    HP_WG(16, 16), HP_WG(16, 32), HP_WG(32, 32), HP_WG(32, 64), HP_WG(64, 64), HP_WG(96, 32),
    HP_WG(48, 16), HP_WG(32, 16), HP_WG(64, 32),
};
#undef HP_WG

hp_status wgrad3_launch(const void* X, const void* G, int D, int H, int W, int cin, int cout,
                        float* gw, float* gb, void* work, int64_t work_bytes, int* err,
                        cudaStream_t s) {
  const int N = cout < 16 ? 16 : cout;
  const WgEntry* e = nullptr;
  for (const auto& c : kWg)
    if (c.cin == cin && c.n == N) e = &c;
  if (!e) {
    hp::set_error("weight gradient %d->%d is not compiled", cin, cout);
    return HP_ERR_UNSUPPORTED;
  }
  if (W % TILE_M != 0 || D < 1 || H < 1) {
    hp::set_error("weight gradient grid W=%d must be a multiple of %d", W, TILE_M);
    return HP_ERR_INVALID;
  }
  if (((uintptr_t)G & 15) || ((uintptr_t)work & 15)) {
    hp::set_error("weight gradient buffers must be 16-byte aligned");
    return HP_ERR_INVALID;
  }
  const int64_t need = wgrad3_workspace(D, H, W, cin, cout);
  if (work_bytes < need) {
    hp::set_error("weight gradient workspace of %lld bytes is below the %lld needed",
                  (long long)work_bytes, (long long)need);
    return HP_ERR_INVALID;
  }
  CUtensorMap mx, mg;
  hp_status st = make_line_map(&mx, X, D, H, W, cin, LINE);
  if (st != HP_OK) return st;
  st = make_line_map(&mg, G, D, H, W, N, TILE_M);
  if (st != HP_OK) return st;
  static bool attr_set[sizeof(kWg) / sizeof(kWg[0])] = {false};
  const int idx = (int)(e - kWg);
  if (!attr_set[idx]) {
    HP_CUDA_TRY(cudaFuncSetAttribute((const void*)e->fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     e->smem));
    attr_set[idx] = true;
  }
  const int WT = W / TILE_M;
  const int nl = D * H * WT;
  const int nchunk = wg_chunks(nl);
  const int per = (nl + nchunk - 1) / nchunk;
  float* part = (float*)work;
  const int T = (3 * (cin / 8) + 15) / 16;
  float* gpart = part + (int64_t)3 * nchunk * T * 3 * TILE_M * N;
  e->fn<<<dim3(nchunk, 3), 128, e->smem, s>>>(mx, mg, D, H, WT, per, part, err);
  HP_CUDA_TRY(cudaGetLastError());
  gsum_partial_kernel<<<GS_BLOCKS, 256, 0, s>>>((const __nv_bfloat16*)G, (int64_t)D * H * W, N,
                                                gpart);
  HP_CUDA_TRY(cudaGetLastError());
  const int red_blocks = (27 * cin * N + 255) / 256 + (cout + 15) / 16;  // weights, then biases
  e->red<<<red_blocks, 256, 0, s>>>(part, nchunk, gpart, cout, gw, gb);
  HP_CUDA_TRY(cudaGetLastError());
  return HP_OK;
}

}  // namespace tc
}  // namespace hp

// Test / building-block entry point: one 3x3x3 convolution (zero padding 1).
extern "C" hp_status hp_conv3_forward(const void* X, const void* Wp, const float* bias, void* Y,
                                      const void* mask, int32_t D, int32_t H, int32_t W,
                                      int32_t cin, int32_t cout, int32_t epi, int32_t* err,
                                      void* stream) {
  HP_REQUIRE(X && Wp && Y && err && (bias || epi == hp::tc::EPI_MASK),
             "hp_conv3_forward: null argument");
  HP_REQUIRE(epi >= 0 && epi <= 3, "hp_conv3_forward: bad epilogue %d", epi);
  HP_REQUIRE(epi != hp::tc::EPI_MASK || mask, "hp_conv3_forward: mask epilogue needs mask");
  return hp::tc::conv3_launch(X, Wp, bias, Y, mask, D, H, W, cin, cout, epi, err,
                              (cudaStream_t)stream);
}

extern "C" int64_t hp_conv3_wgrad_workspace(int32_t D, int32_t H, int32_t W, int32_t cin,
                                            int32_t cout) {
  if (D < 1 || H < 1 || W < 1 || cin < 8 || cout < 1) return -1;
  return hp::tc::wgrad3_workspace(D, H, W, cin, cout);
}

extern "C" hp_status hp_conv3_wgrad(const void* X, const void* G, int32_t D, int32_t H, int32_t W,
                                    int32_t cin, int32_t cout, float* gw, float* gb, void* work,
                                    int64_t work_bytes, int32_t* err, void* stream) {
  HP_REQUIRE(X && G && gw && gb && work && err, "hp_conv3_wgrad: null argument");
  return hp::tc::wgrad3_launch(X, G, D, H, W, cin, cout, gw, gb, work, work_bytes, err,
                               (cudaStream_t)stream);
}
