// Per-frame torso Poisson solve (ECG forward problem) for sm_100a.
//
// Replaces make_gpu_solver / solve_frame / _pcg_gpu of the reference
// (ecg/functions/compute_bspm.py:164-436) over the sharp-boundary 7-point
// operator of _assemble_stiffness (ecg/functions/build_torso_grid.py:276-397):
//   A_kk = sum_faces g_f,  A_kn = -g_f,  g_f = harm(sigma_k, sigma_n) / h^2,
// air faces skipped (Neumann), one pinned row fixed to 0.
//
// The operator is never assembled.  Conductivity is piecewise constant by
// material label, so a face conductance is a lookup in an M x M table; the
// solver keeps one byte per voxel of operator data instead of 7 CSR entries.
// Grid arrays are dense over the torso box padded by one air voxel on every
// side (no bounds tests in the stencil); k is the fastest axis, so a warp's
// accesses and its +/-k neighbours are contiguous and the +/-j, +/-i
// neighbours are rows / planes that the previous warps just brought into L2.
//
// Precision: vectors r, p, Ap and the SpMV run in FP32; the solution x and
// every dot product / norm are FP64; the convergence decision for the
// relative rule is taken on the FP64 true residual b - A x evaluated with the
// FP64 conductance table (the reference operator's own coefficients).  If the
// recursive FP32 residual claims convergence but the true residual does not,
// r is replaced by the true residual and CG restarts (residual replacement).
//
// The Jacobi-PCG iterations run in one cooperative launch per solve
// (pcg_resident.cuh); the flexible-CG passes walk tissue lines, one launch
// each.  Reductions are deterministic (partials added in block order).
#include "hp_common.cuh"
#include "precond_apply.cuh"

#include <math.h>
#include <thread>
#include <stdint.h>

#include <algorithm>
#include <vector>

namespace hp {

constexpr int TB = 256;            // threads per block
constexpr int NPART = 4;           // partial sums per block
constexpr int FCG_SPMV_BLOCKS = 4; // blocks a multiprocessor of the flexible CG's A p (fixes its sums' order)

enum Scal : int {
  SC_RZ = 0, SC_PAP, SC_ALPHA, SC_BETA, SC_ZZ, SC_ZMAX, SC_RR, SC_BB,
  SC_TRUE_RR, SC_SRC_MEAN, SC_STAT, SC_TOL, SC_HIST0, N_SCAL = SC_HIST0 + 8
};
enum IScal : int {
  IS_DONE = 0, IS_ITER, IS_RULE, IS_MAXIT, IS_BREAKDOWN, IS_NONFINITE, IS_STAGNANT, IS_NH,
  IS_STAG_ON, N_ISCAL
};

struct TorsoArgs {
  int64_t ng;          // padded grid cells
  int32_t pj, pk;      // padded dims j, k (i stride = pj * pk)
  const uint8_t* label;
  const float* invd;
  float* r;
  float* p0;
  float* Ap;
  double* x;
  float* b;
  int64_t pin;         // padded grid index of the pinned voxel
  int64_t n_rows;
  double* scal;
  int32_t* iscal;
  double* part;        // gridDim x NPART
  unsigned int* ticket;
  // tissue lines: the k-run from the first to the last tissue cell of every
  // (i, j) line that has one (air inside a run is allowed)
  int32_t n_lines;
  const int4* line;    // row of the padded grid, unpadded k of its first and past its last cell,
                       // unpadded i
  // smoothed-boundary domain function per padded cell (0 off the rows), or
  // null for the sharp boundary
  const float* psi;
  // this handle's FP64 conductance table of the true residual (harmonic-mean
  // face conductance / h^2, HP_MAX_MATERIALS x HP_MAX_MATERIALS): per handle,
  // so that handles with different conductivities can live side by side
  const double* T64;
};

// flags over the host copy of the labels: all six neighbours carry the cell's
// own label (and, with a smoothed boundary, psi is 1 at the cell and all six);
// the pinned voxel
constexpr int LAB_UNIFORM = 0x80;
constexpr int LAB_PIN = 0x40;
constexpr int LAB_MASK = 0x3F;  // the material label (< HP_MAX_MATERIALS)
static_assert(HP_MAX_MATERIALS <= LAB_MASK + 1, "material labels must fit under the flag bits");

// Smoothed-boundary factor of a face: the harmonic mean of the two cells'
// domain function, 0 when both are 0 (build_torso_grid.py:350-375).
__host__ __device__ inline double psi_face64(double pa, double pb) {
  const double s = pa + pb;
  return s < 1e-30 ? 0.0 : (2.0 * pa * pb) / s;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_down_sync(0xffffffffu, v, o));
  return v;
}

// Block-reduces NV values into part[blockIdx] -- slot q is a sum, or a max
// where bit q of max_mask is set (identity -inf) -- then returns true in the
// one block that arrived last, after which `tot` holds the grid totals in
// every thread of that block.
template <int NV>
__device__ bool block_reduce_last(double (&v)[NV], uint32_t max_mask, double* part,
                                  unsigned int* ticket, double (&tot)[NV]) {
  __shared__ double sh[TB / 32][NV];
  __shared__ bool am_last;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < NV; ++q) {
    const bool mx = (max_mask >> q) & 1u;
    double w = mx ? (double)warp_max((float)v[q]) : warp_sum(v[q]);
    if (lane == 0) sh[wid][q] = w;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      const bool mx = (max_mask >> q) & 1u;
      double s = sh[0][q];
      for (int w = 1; w < TB / 32; ++w) s = mx ? fmax(s, sh[w][q]) : s + sh[w][q];
      part[(int64_t)blockIdx.x * NPART + q] = s;
    }
    __threadfence();
    const unsigned int t = atomicAdd(ticket, 1u);
    am_last = (t == gridDim.x - 1);
  }
  __syncthreads();
  if (!am_last) return false;
  __threadfence();
  // the last block sums all partials in block order (deterministic)
#pragma unroll
  for (int q = 0; q < NV; ++q) v[q] = ((max_mask >> q) & 1u) ? -INFINITY : 0.0;
  for (int blk = threadIdx.x; blk < (int)gridDim.x; blk += TB) {
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      const double pv = ((volatile double*)part)[(int64_t)blk * NPART + q];
      v[q] = ((max_mask >> q) & 1u) ? fmax(v[q], pv) : v[q] + pv;
    }
  }
  // fixed-order tree over the block
  __shared__ double sh2[TB][NV];
#pragma unroll
  for (int q = 0; q < NV; ++q) sh2[threadIdx.x][q] = v[q];
  __syncthreads();
  for (int s = TB / 2; s > 0; s >>= 1) {
    if ((int)threadIdx.x < s) {
#pragma unroll
      for (int q = 0; q < NV; ++q)
        sh2[threadIdx.x][q] = ((max_mask >> q) & 1u)
                                  ? fmax(sh2[threadIdx.x][q], sh2[threadIdx.x + s][q])
                                  : sh2[threadIdx.x][q] + sh2[threadIdx.x + s][q];
    }
    __syncthreads();
  }
#pragma unroll
  for (int q = 0; q < NV; ++q) tot[q] = sh2[0][q];
  if (threadIdx.x == 0) *ticket = 0u;
  return true;
}

__device__ __forceinline__ bool is_row(const TorsoArgs& a, int64_t g) {
  return a.label[g] != 0 && g != a.pin;
}

}  // namespace hp
#include "pcg_resident.cuh"
namespace hp {

// What a residual pass starts: the iteration budget, stopping rule and
// tolerance of the recursion that follows.
struct SolveInit {
  int32_t rule, max_iter, stag_on, iter;
  double tol;
};

// FP64 true residual r = b - A x (written to r in FP32), and ||r||^2,
// ||b||^2, r.M^-1 r.  reset = 1 starts a CG recursion (beta = 0, the flags and
// limits of `init`), done at once where b = 0 or the relative rule already
// holds; 2 checks a finished one, leaving its flags (r is replaced under the
// relative rule only); 0 evaluates the norms alone.
__global__ void __launch_bounds__(TB) true_residual(TorsoArgs a, int reset, SolveInit init) {
  const int64_t SJ = a.pk, SI = (int64_t)a.pj * a.pk;
  double acc[3] = {0.0, 0.0, 0.0};
  for (int64_t g = blockIdx.x * (int64_t)TB + threadIdx.x; g < a.ng;
       g += (int64_t)gridDim.x * TB) {
    if (!is_row(a, g)) continue;
    const int l = a.label[g];
    const int64_t nb[6] = {g + SI, g - SI, g + SJ, g - SJ, g + 1, g - 1};
    const double xg = a.x[g];
    double ax = 0.0;
#pragma unroll
    for (int f = 0; f < 6; ++f) {
      double t = a.T64[l * HP_MAX_MATERIALS + a.label[nb[f]]];
      if (a.psi) t *= psi_face64(a.psi[g], a.psi[nb[f]]);
      ax += t * (xg - a.x[nb[f]]);   // x is 0 on air and at the pinned voxel
    }
    const double bb = (double)a.b[g];
    const double rr = bb - ax;
    const float rf = (float)rr;
    if (reset == 1 || (reset == 2 && init.rule == HP_STOP_REL)) a.r[g] = rf;
    acc[0] += rr * rr;
    acc[1] += bb * bb;
    acc[2] += (double)rf * ((double)a.invd[g] * rf);
  }
  double tot[3];
  if (block_reduce_last<3>(acc, 0u, a.part, a.ticket, tot) && threadIdx.x == 0) {
    a.scal[SC_TRUE_RR] = tot[0];
    a.scal[SC_BB] = tot[1];
    if (reset == 1) {
      a.scal[SC_RZ] = tot[2];
      a.scal[SC_BETA] = 0.0;
      a.scal[SC_TOL] = init.tol;
      const bool zero = tot[1] == 0.0;
      const double rel = zero ? 0.0 : sqrt(tot[0] / tot[1]);
      a.iscal[IS_DONE] = init.rule == HP_STOP_REL && (zero || rel <= init.tol) ? 1 : 0;
      a.iscal[IS_ITER] = init.iter;
      a.iscal[IS_RULE] = init.rule;
      a.iscal[IS_MAXIT] = init.max_iter;
      a.iscal[IS_BREAKDOWN] = a.iscal[IS_NONFINITE] = a.iscal[IS_STAGNANT] = a.iscal[IS_NH] = 0;
      a.iscal[IS_STAG_ON] = init.stag_on;
    }
  }
}

// ---------------------------------------------------------------- sources

struct SrcArgs {
  int32_t n_heart;
  const int32_t* nbr;      // n_heart x 6
  const int32_t* proj;     // n_heart (coarse row or -1)
  const float* vm;         // n_heart, mV
  float* iv;               // n_heart: (sigma_i/h^2) K Vm (V) on projected voxels
  double coeff;
  double* part;
  unsigned int* ticket;
  double* scal;
  int64_t* mean_count;     // [1] number of projected voxels
};

// iv_i = coeff * sum_n (V_n - V_i) with V = Vm * 1e-3 volts (compute_bspm.py:381-387)
__global__ void __launch_bounds__(TB) src_laplacian(SrcArgs s) {
  double acc[1] = {0.0};
  for (int64_t i = blockIdx.x * (int64_t)TB + threadIdx.x; i < s.n_heart;
       i += (int64_t)gridDim.x * TB) {
    if (s.proj[i] < 0) continue;
    // differences of the mV values first (exact for equal neighbours), then
    // one scaling by 1e-3 * sigma_i / h^2
    const float vi = s.vm[i];
    float lap = 0.0f;
#pragma unroll
    for (int f = 0; f < 6; ++f) {
      const int32_t n = s.nbr[i * 6 + f];
      if (n >= 0) lap += __fsub_rn(s.vm[n], vi);
    }
    const float iv = lap * (float)(s.coeff * 1e-3);
    s.iv[i] = iv;
    acc[0] += (double)iv;
  }
  double tot[1];
  if (block_reduce_last<1>(acc, 0u, s.part, s.ticket, tot) && threadIdx.x == 0)
    s.scal[SC_SRC_MEAN] = tot[0] / (double)fmax(1.0, (double)*s.mean_count);
}

// b[row] = (sum of iv over the heart voxels of row - count * mean) / n_expected,
// one thread per receiving row (rows listed in seg order, deterministic).
__global__ void __launch_bounds__(TB) src_scatter(const float* iv, const int32_t* seg_ptr,
                                                  const int32_t* seg_vox, const int64_t* seg_grid,
                                                  int32_t n_seg, const double* scal,
                                                  double inv_nexp, float* b, int64_t pin,
                                                  const float* psi) {
  const int q = blockIdx.x * TB + threadIdx.x;
  if (q >= n_seg) return;
  const float mean = (float)scal[SC_SRC_MEAN];
  float s = 0.0f;
  for (int t = seg_ptr[q]; t < seg_ptr[q + 1]; ++t) s += iv[seg_vox[t]] - mean;
  const int64_t g = seg_grid[q];
  float bg = (float)(s * inv_nexp);
  if (psi) bg *= psi[g];   // smoothed boundary: psi b (compute_bspm.py:413-414)
  b[g] = g == pin ? 0.0f : bg;
}

__global__ void gather_out(const double* x, const int64_t* grid_of_read, int32_t n, float* out) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q < n) out[q] = (float)(x[grid_of_read[q]] * 1e3);
}

__global__ void gather_rows(const double* x, const int64_t* grid_of_row, int64_t n, double* out) {
  const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (q < n) out[q] = x[grid_of_row[q]];
}

__global__ void gather_rows_f(const float* b, const int64_t* grid_of_row, int64_t n, float* out) {
  const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (q < n) out[q] = b[grid_of_row[q]];
}

// flexible-CG passes (defined with the FCG driver below)
__global__ void __launch_bounds__(TB, 4) fcg_spmv(TorsoArgs a, PcgArgs c);
__global__ void __launch_bounds__(TB) fcg_update(TorsoArgs a, pc::SegArgs seg);
__global__ void __launch_bounds__(TB) fcg_beta(TorsoArgs a, pc::ZArgs z);
__global__ void __launch_bounds__(TB) fcg_p(TorsoArgs a, pc::ZArgs z, int first);

}  // namespace hp

using namespace hp;

// kernels that stride over the tissue lines, in the order of HpTorso::nblk_k
enum LineKernel : int { K_FCG_SPMV = 0, K_FCG_UPDATE, K_FCG_BETA, K_FCG_P, N_LINE_KERNELS };

struct HpTorso {
  TorsoArgs a;
  SrcArgs s;
  int nblk;
  int nblk_k[N_LINE_KERNELS];  // line kernels: each one's resident grid
  bool pairs;                  // stencil on cell pairs (even padded row)
  int ni, nj, nk;
  int64_t n_rows;
  std::vector<void*> allocs;
  int32_t n_read;
  int64_t* grid_of_read;
  int64_t* grid_of_row;
  int32_t* seg_ptr;
  int32_t* seg_vox;
  int64_t* seg_grid;
  int32_t n_seg;
  double inv_nexp;
  float* vm_dev;
  float* out_dev;
  double* h_scal;   // pinned host mirrors
  int32_t* h_iscal;
  bool have_x;
  PcgArgs pcg;
  int pcg_grid;
  size_t pcg_smem;
  void (*pcg_fn[2])(TorsoArgs, PcgArgs);   // [1]: the p99 rule
  int fail_in;   // launches until one counts as timed out (hp_torso_inject_timeout), or 0
  cudaGraphExec_t fcg_graph[4];   // FCG chunk without the network / net every 1, 2, 4
  // serial number of the preconditioner handle the FCG graphs hold (not its
  // address: a destroyed handle's address can come back for a new one, whose
  // buffers the old graphs do not point to)
  uint64_t fcg_graph_pc;
  cudaStream_t fcg_graph_stream;
};

template <typename T>
static hp_status tup(HpTorso* h, T** dst, const T* src, size_t n, cudaStream_t s) {
  hp_status st = dev_upload(dst, src, n, s);
  if (st == HP_OK && *dst) h->allocs.push_back((void*)*dst);
  return st;
}
template <typename T>
static hp_status tal(HpTorso* h, T** dst, size_t n) {
  hp_status st = dev_alloc(dst, n);
  if (st == HP_OK && *dst) h->allocs.push_back((void*)*dst);
  return st;
}

#define HP_TRY_T(x)              \
  do {                           \
    hp_status _s = (x);          \
    if (_s != HP_OK) return _s;  \
  } while (0)

#define TT_TRY(x)                \
  do {                           \
    hp_status _s = (x);          \
    if (_s != HP_OK) {           \
      hp_torso_destroy(h);       \
      return _s;                 \
    }                            \
  } while (0)

template <int MODE>
static void pcg_kernels(HpTorso* h) {
  h->pcg_fn[0] = h->pairs ? pcg_resident<MODE, true, false> : pcg_resident<MODE, false, false>;
  h->pcg_fn[1] = h->pairs ? pcg_resident<MODE, true, true> : pcg_resident<MODE, false, true>;
}

// f(0) .. f(n - 1) on host threads; where one cannot be started, here.  f must
// not throw.
template <typename F>
static void host_parts(int n, F f) {
  std::vector<std::thread> ts;
  ts.reserve(n);
  int t = 1;
  try {
    for (; t < n; ++t) ts.emplace_back(f, t);
  } catch (...) {
  }
  for (; t < n; ++t) f(t);
  f(0);
  for (auto& x : ts) x.join();
}

// The resident PCG's tables (pcg_resident.cuh) from the tissue lines, and
// where a block keeps its vectors: all in shared memory where 36 bytes a pair
// fit (up to about 1.7 M cells), else r alone (8 bytes, up to about 7.5 M),
// else none; the lines' records too stay in memory from about 1.3 M on.
static hp_status setup_pcg(HpTorso* h, const std::vector<int64_t>& line_g0,
                           const std::vector<int32_t>& line_len, const std::vector<uint8_t>& lab_u,
                           const std::vector<float>& psi, const std::vector<float>& invd,
                           const float* T32, int nsm, cudaStream_t s) {
  const TorsoArgs& a = h->a;
  PcgArgs& c = h->pcg;
  memset(&c, 0, sizeof(c));
  const int64_t PK = a.pk, PJ = a.pj, PK2 = (PK + 1) / 2;  // pairs a row of p
  const int64_t SJ = PK, SI = PJ * PK;
  const int64_t nbr[6] = {SI, -SI, SJ, -SJ, 1, -1};
  HP_REQUIRE(a.ng / PK * PK2 < ((int64_t)1 << 31), "hp_torso_create: the grid is too large");
  const int n_lines = (int)line_g0.size();
  h->pcg_grid = std::max(1, std::min(nsm, PCG_MAX_BLOCKS));
  std::vector<PcgLine> lines(n_lines);
  std::vector<int32_t> used(h->pcg_grid, 0);
  int64_t n_pairs = 0;
  for (int l = 0; l < n_lines; ++l) {
    const int64_t row = line_g0[l] / PK, k0 = line_g0[l] % PK, k1 = k0 + line_len[l];
    PcgLine& L = lines[l];
    int32_t& at = used[(l / PCG_WARPS) % h->pcg_grid];  // lines go round by warps
    L.p2 = (uint32_t)(row * PK2 + k0 / 2);
    L.n2 = (int32_t)((k1 + 1) / 2 - k0 / 2);
    L.c2 = (int32_t)n_pairs;
    L.s2 = at;
    L.first = (int32_t)(k0 & 1);
    L.len = line_len[l];
    at += L.n2;
    n_pairs += L.n2;
  }
  // The pairs' words and the mixed pairs' coefficients, by host threads over
  // ranges of lines: mixed pairs are counted within a range first, then moved
  // by the counts of the ranges before it.
  struct Part {
    uint32_t mixed, base;
    float tu[HP_MAX_MATERIALS], inv[HP_MAX_MATERIALS];
    bool has[HP_MAX_MATERIALS];
  };
  const int n_range = n_lines < 2048
                         ? 1
                         : (int)std::min(16u, std::max(1u, std::thread::hardware_concurrency()));
  std::vector<Part> ranges(n_range);
  std::vector<uint32_t> meta(n_pairs);
  std::vector<float> mixed;
  // each pair of the range's lines: f(word, first cell, cells of the pair on the line)
  auto walk = [&](int t, auto f) {
    for (int l = (int)((int64_t)n_lines * t / n_range); l < (int64_t)n_lines * (t + 1) / n_range; ++l) {
      const int64_t row = line_g0[l] / PK, k0 = line_g0[l] % PK, k1 = k0 + line_len[l];
      uint32_t* m = &meta[lines[l].c2];
      for (int64_t k = k0 / 2 * 2; k < k1; k += 2, ++m)
        f(*m, row * PK + k, k >= k0, k + 1 < k1);
    }
  };
  host_parts(n_range, [&](int t) {
    Part& P = ranges[t];
    memset(&P, 0, sizeof(P));
    walk(t, [&](uint32_t& m, int64_t g, bool on0, bool on1) {
      const int u0 = on0 ? lab_u[g] : 0, u1 = on1 ? lab_u[g + 1] : 0;
      if ((u0 & u1 & LAB_UNIFORM) && !((u0 | u1) & LAB_PIN)) {  // then both are one material
        const int mat = u0 & LAB_MASK;
        P.has[mat] = true;
        P.tu[mat] = T32[mat * (HP_MAX_MATERIALS + 1)];
        P.inv[mat] = invd[g];
        m = (uint32_t)mat;
      } else {
        m = PQ_MIXED | P.mixed++;
      }
    });
  });
  size_t n_mixed = 0;
  for (Part& P : ranges) {
    P.base = (uint32_t)n_mixed;
    n_mixed += P.mixed;
    for (int mat = 0; mat < HP_MAX_MATERIALS; ++mat)
      if (P.has[mat]) {
        c.tu[mat] = P.tu[mat];
        c.inv[mat] = P.inv[mat];
      }
  }
  mixed.resize(14 * n_mixed, 0.0f);
  host_parts(n_range, [&](int t) {
    walk(t, [&](uint32_t& m, int64_t g0, bool on0, bool on1) {
      if (!(m & PQ_MIXED)) return;
      m += ranges[t].base;
      const size_t x = m & ~PQ_MIXED;
      for (int e = 0; e < 2; ++e) {
        if (!(e ? on1 : on0)) continue;
        const int64_t g = g0 + e;
        const int l = lab_u[g] & LAB_MASK;
        const bool row = l != 0 && !(lab_u[g] & LAB_PIN);
        for (int f = 0; f < 6 && row; ++f) {
          const int64_t n = g + nbr[f];
          float t = T32[l * HP_MAX_MATERIALS + (lab_u[n] & LAB_MASK)];
          if (!psi.empty()) {
            const float pa = psi[g], pb = psi[n], sum = pa + pb;
            t *= sum < 1e-30f ? 0.0f : 2.0f * pa * pb / sum;
          }
          mixed[((size_t)f * n_mixed + x) * 2 + e] = t;
        }
        mixed[((size_t)6 * n_mixed + x) * 2 + e] = invd[g];
      }
    });
  });
  c.n_lines = n_lines;
  c.n_pairs = (int32_t)meta.size();
  c.n_mixed = (int32_t)n_mixed;
  c.sj = (uint32_t)PK2;
  c.si = (uint32_t)(PJ * PK2);
  const size_t np = (size_t)(a.ng / PK * PK2) * 2;
  HP_TRY_T(tup(h, (PcgLine**)&c.line, lines.data(), lines.size(), s));
  HP_TRY_T(tup(h, (uint32_t**)&c.meta, meta.data(), meta.size(), s));
  if (c.n_mixed) HP_TRY_T(tup(h, (float**)&c.mixed, mixed.data(), mixed.size(), s));
  HP_CUDA_TRY(cudaStreamSynchronize(s));  // the host vectors are temporaries
  HP_TRY_T(tal(h, (float**)&c.p, np));
  HP_CUDA_TRY(cudaMemsetAsync(c.p, 0, np * 4, s));
  int dev = 0, most = 0;
  HP_CUDA_TRY(cudaGetDevice(&dev));
  HP_CUDA_TRY(cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  const size_t all_lines =
      (size_t)(n_lines + PCG_WARPS * h->pcg_grid - 1) / (PCG_WARPS * h->pcg_grid) * PCG_WARPS *
      sizeof(PcgLine);
  const size_t fixed = 14 * 1024;  // the reductions' static share
  const bool lines_fit = fixed + all_lines <= (size_t)most;
  const size_t line_bytes = lines_fit ? all_lines : 0;
  const size_t room = (size_t)most - fixed - line_bytes;
  const size_t per = ((size_t)*std::max_element(used.begin(), used.end()) + 3) / 4 * 4;
  const int mode = !lines_fit                              ? PCG_MEM
                   : per * pcg_pair_bytes(PCG_ALL) <= room ? PCG_ALL
                   : per * pcg_pair_bytes(PCG_R) <= room   ? PCG_R
                                                           : PCG_NONE;
  c.room = mode == PCG_ALL || mode == PCG_R ? (int32_t)per : 0;
  h->pcg_smem = per * pcg_pair_bytes(mode) + line_bytes;
  if (mode == PCG_ALL) pcg_kernels<PCG_ALL>(h);
  else if (mode == PCG_R) pcg_kernels<PCG_R>(h);
  else if (mode == PCG_NONE) pcg_kernels<PCG_NONE>(h);
  else pcg_kernels<PCG_MEM>(h);
  for (auto fn : h->pcg_fn) HP_TRY_T(allow_dynamic_smem((const void*)fn));
  if (mode != PCG_ALL) {
    HP_TRY_T(tal(h, &c.Ap, c.n_pairs));
    HP_TRY_T(tal(h, &c.x, c.n_pairs));
  }
  if (mode == PCG_NONE || mode == PCG_MEM) HP_TRY_T(tal(h, &c.r, c.n_pairs));
  const size_t n_part = (size_t)2 * PCG_GROUPS * 4;
  HP_TRY_T(tal(h, &c.part, n_part + GRID_SYNC_WORDS));
  HP_CUDA_TRY(cudaMemsetAsync(c.part, 0, (n_part + GRID_SYNC_WORDS) * sizeof(double), s));
  c.sync = grid_sync_at(c.part + n_part);
  c.sync.err = a.iscal + N_ISCAL;
  return HP_OK;
}

extern "C" hp_status hp_torso_destroy(HpTorso* h);

extern "C" hp_status hp_torso_create(const HpTorsoDesc* d, HpTorso** out, void* stream) {
  HP_REQUIRE(d && out, "hp_torso_create: null argument");
  *out = nullptr;
  HP_REQUIRE(d->ni > 0 && d->nj > 0 && d->nk > 0 && d->label, "hp_torso_create: empty grid");
  HP_REQUIRE(d->n_materials >= 1 && d->n_materials <= HP_MAX_MATERIALS && d->sigma,
             "hp_torso_create: n_materials must be 1..%d", HP_MAX_MATERIALS);
  HP_REQUIRE(d->h_m > 0.0, "hp_torso_create: h_m must be positive");
  HP_REQUIRE(d->n_heart >= 0 && (d->n_heart == 0 || (d->heart_nbr && d->proj)),
             "hp_torso_create: missing heart arrays");
  HP_REQUIRE(d->n_read >= 0 && (d->n_read == 0 || d->read_rows), "hp_torso_create: missing read_rows");
  cudaStream_t s = (cudaStream_t)stream;
  const int ni = d->ni, nj = d->nj, nk = d->nk;
  const int PI = ni + 2, PJ = nj + 2, PK = nk + 2;
  const int64_t ng = (int64_t)PI * PJ * PK;
  // padded labels (and smoothed-boundary psi), row <-> grid maps (rows in
  // flat active order)
  std::vector<uint8_t> lab(ng, 0);
  std::vector<float> psi(d->psi ? ng : 0, 0.0f);
  std::vector<int64_t> grid_of_row;
  grid_of_row.reserve((size_t)ni * nj * nk);
  for (int i = 0; i < ni; ++i)
    for (int j = 0; j < nj; ++j)
      for (int k = 0; k < nk; ++k) {
        const uint8_t l = d->label[((int64_t)i * nj + j) * nk + k];
        if (l >= d->n_materials) {
          hp::set_error("hp_torso_create: label %d at (%d,%d,%d) >= n_materials", l, i, j, k);
          return HP_ERR_INVALID;
        }
        const int64_t g = ((int64_t)(i + 1) * PJ + (j + 1)) * PK + (k + 1);
        lab[g] = l;
        if (l != 0) grid_of_row.push_back(g);
        if (d->psi) {
          const float pv = d->psi[((int64_t)i * nj + j) * nk + k];
          if (!(pv >= 0.0f && pv <= 1.0f) || (pv > 0.0f) != (l != 0)) {
            hp::set_error("hp_torso_create: psi %g at (%d,%d,%d) must be in (0, 1] exactly where "
                          "the label is non-zero (label %d)", (double)pv, i, j, k, l);
            return HP_ERR_INVALID;
          }
          psi[g] = pv;
        }
      }
  const int64_t n_rows = (int64_t)grid_of_row.size();
  HP_REQUIRE(d->pin_row >= 0 && d->pin_row < n_rows, "hp_torso_create: pin_row out of range");
  for (int m = 0; m < d->n_read; ++m)
    HP_REQUIRE(d->read_rows[m] >= 0 && d->read_rows[m] < n_rows,
               "hp_torso_create: read_rows[%d] out of range", m);
  // conductance tables (harmonic mean / h^2; both-zero pairs -> 0)
  float T32[HP_MAX_MATERIALS * HP_MAX_MATERIALS] = {0};
  double T64[HP_MAX_MATERIALS * HP_MAX_MATERIALS] = {0};
  const double h2 = d->h_m * d->h_m;
  for (int u = 0; u < d->n_materials; ++u)
    for (int v = 0; v < d->n_materials; ++v) {
      const double su = d->sigma[u], sv = d->sigma[v];
      if (u == 0 || v == 0 || su + sv < 1e-30) continue;   // air never couples
      const double g = (2.0 * su * sv) / (su + sv) / h2;
      T64[u * HP_MAX_MATERIALS + v] = g;
      T32[u * HP_MAX_MATERIALS + v] = (float)g;
    }
  // Jacobi inverse diagonal (FP32 of the FP64 diagonal), 0 on the pin
  const int64_t SJ = PK, SI = (int64_t)PJ * PK;
  std::vector<float> invd(ng, 0.0f);
  const int64_t pin_g = grid_of_row[d->pin_row];
  for (int64_t r = 0; r < n_rows; ++r) {
    const int64_t g = grid_of_row[r];
    if (g == pin_g) continue;
    const int l = lab[g];
    const int64_t nb[6] = {g + SI, g - SI, g + SJ, g - SJ, g + 1, g - 1};
    double dg = 0.0;
    for (int f = 0; f < 6; ++f)
      dg += T64[l * HP_MAX_MATERIALS + lab[nb[f]]] *
            (d->psi ? psi_face64(psi[g], psi[nb[f]]) : 1.0);
    invd[g] = dg > 1e-30 ? (float)(1.0 / dg) : 1.0f;
  }
  HpTorso* h = new HpTorso();
  memset(&h->a, 0, sizeof(h->a));
  memset(&h->s, 0, sizeof(h->s));
  for (int k = 0; k < 4; ++k) h->fcg_graph[k] = nullptr;
  h->fcg_graph_pc = 0;
  h->fcg_graph_stream = nullptr;
  h->fail_in = 0;
  h->ni = ni; h->nj = nj; h->nk = nk;
  h->n_rows = n_rows;
  h->have_x = false;
  TorsoArgs& a = h->a;
  TT_TRY(tup(h, (double**)&a.T64, T64, HP_MAX_MATERIALS * HP_MAX_MATERIALS, s));
  a.ng = ng; a.pj = PJ; a.pk = PK; a.pin = pin_g; a.n_rows = n_rows;
  TT_TRY(tup(h, (uint8_t**)&a.label, lab.data(), ng, s));
  TT_TRY(tup(h, (float**)&a.invd, invd.data(), ng, s));
  a.psi = nullptr;
  if (d->psi) TT_TRY(tup(h, (float**)&a.psi, psi.data(), ng, s));
  // the flexible CG's own vectors, where a preconditioner can be made at all
  if (!d->psi && ni % 8 == 0 && nj % 8 == 0 && nk % 256 == 0)
    for (float** v : {&a.p0, &a.Ap}) {
      TT_TRY(tal(h, v, ng));
      HP_CUDA_TRY(cudaMemsetAsync(*v, 0, ng * 4, s));
    }
  TT_TRY(tal(h, &a.r, ng));
  TT_TRY(tal(h, &a.x, ng));
  TT_TRY(tal(h, &a.b, ng));
  HP_CUDA_TRY(cudaMemsetAsync(a.r, 0, ng * 4, s));
  HP_CUDA_TRY(cudaMemsetAsync(a.x, 0, ng * 8, s));
  HP_CUDA_TRY(cudaMemsetAsync(a.b, 0, ng * 4, s));
  int nsm = 148;
  {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  }
  h->nblk = nsm * 8;
  {
    // the line loops stride over the grid, so a grid larger than what is
    // resident would leave a tail wave: each kernel gets its resident grid
    int o = 0;
    // cell pairs need even padded strides (an even padded row)
    h->pairs = (PK % 2) == 0;
    const void* fs[N_LINE_KERNELS] = {(const void*)fcg_spmv, (const void*)fcg_update,
                                      (const void*)fcg_beta, (const void*)fcg_p};
    for (int q = 0; q < N_LINE_KERNELS; ++q) {
      HP_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, fs[q], TB, 0));
      h->nblk_k[q] = nsm * std::min(8, std::max(o, 1));
    }
    h->nblk_k[K_FCG_SPMV] = nsm * FCG_SPMV_BLOCKS;
  }
  // the scalars, the integer scalars and the barrier's error flag lie in one
  // piece: one copy brings them to the host
  TT_TRY(tal(h, &a.scal, N_SCAL + N_ISCAL / 2 + 1));
  a.iscal = (int32_t*)(a.scal + N_SCAL);
  TT_TRY(tal(h, &a.part, (size_t)h->nblk * NPART));
  TT_TRY(tal(h, &a.ticket, 1));
  HP_CUDA_TRY(cudaMemsetAsync(a.scal, 0, N_SCAL * 8 + (N_ISCAL + 1) * 4, s));
  HP_CUDA_TRY(cudaMemsetAsync(a.ticket, 0, 4, s));
  TT_TRY(tup(h, &h->grid_of_row, grid_of_row.data(), n_rows, s));
  {
    // tissue lines of the padded grid: first .. last tissue cell in k
    std::vector<int64_t> g0;
    std::vector<int32_t> len;
    for (int i = 1; i <= ni; ++i)
      for (int j = 1; j <= nj; ++j) {
        const int64_t base = ((int64_t)i * PJ + j) * PK;
        int k0 = -1, k1 = -1;
        for (int k = 1; k <= nk; ++k)
          if (lab[base + k] != 0) {
            if (k0 < 0) k0 = k;
            k1 = k;
          }
        if (k0 >= 0) {
          g0.push_back(base + k0);
          len.push_back(k1 - k0 + 1);
        }
      }
    a.n_lines = (int32_t)g0.size();
    std::vector<uint8_t> lab_u(lab);
    for (int64_t r = 0; r < n_rows; ++r) {
      const int64_t g = grid_of_row[r];
      const int64_t nb[6] = {g + SI, g - SI, g + SJ, g - SJ, g + 1, g - 1};
      bool uni = !d->psi || psi[g] == 1.0f;
      for (int f = 0; f < 6; ++f)
        uni = uni && lab[nb[f]] == lab[g] && (!d->psi || psi[nb[f]] == 1.0f);
      if (uni) lab_u[g] |= (uint8_t)LAB_UNIFORM;
    }
    lab_u[pin_g] |= (uint8_t)LAB_PIN;

    std::vector<int4> line(g0.size());
    for (size_t L = 0; L < g0.size(); ++L) {
      const int row = (int)(g0[L] / PK), k0 = (int)(g0[L] % PK) - 1;
      line[L] = make_int4(row, k0, k0 + len[L], row / PJ - 1);
    }
    TT_TRY(tup(h, (int4**)&a.line, line.data(), line.size(), s));
    HP_CUDA_TRY(cudaStreamSynchronize(s));  // line is a stack temporary
    TT_TRY(setup_pcg(h, g0, len, lab_u, psi, invd, T32, nsm, s));
  }
  // heart sources: segments of heart voxels per receiving row
  SrcArgs& sa = h->s;
  sa.n_heart = d->n_heart;
  sa.coeff = d->coeff;
  sa.part = a.part;
  sa.ticket = a.ticket;
  sa.scal = a.scal;
  h->inv_nexp = 1.0 / d->n_expected;
  std::vector<int32_t> order;
  int64_t n_valid = 0;
  for (int32_t i = 0; i < d->n_heart; ++i) {
    if (d->proj[i] >= n_rows) {
      hp::set_error("hp_torso_create: proj[%d]=%d out of range", i, d->proj[i]);
      hp_torso_destroy(h);
      return HP_ERR_INVALID;
    }
    for (int f = 0; f < 6; ++f) {
      const int32_t nbv = d->heart_nbr[(int64_t)i * 6 + f];
      if (nbv >= d->n_heart) {
        hp::set_error("hp_torso_create: heart_nbr out of range at %d", i);
        hp_torso_destroy(h);
        return HP_ERR_INVALID;
      }
    }
    if (d->proj[i] >= 0) { order.push_back(i); ++n_valid; }
  }
  std::stable_sort(order.begin(), order.end(),
                   [&](int32_t u, int32_t v) { return d->proj[u] < d->proj[v]; });
  std::vector<int32_t> seg_ptr(1, 0), seg_vox;
  std::vector<int64_t> seg_grid;
  for (size_t t = 0; t < order.size(); ++t) {
    if (t > 0 && d->proj[order[t]] != d->proj[order[t - 1]]) {
      seg_ptr.push_back((int32_t)t);
    }
    if (t == 0 || d->proj[order[t]] != d->proj[order[t - 1]])
      seg_grid.push_back(grid_of_row[d->proj[order[t]]]);
    seg_vox.push_back(order[t]);
  }
  seg_ptr.push_back((int32_t)order.size());
  if (order.empty()) seg_ptr.assign(1, 0);
  h->n_seg = (int32_t)seg_grid.size();
  TT_TRY(tup(h, &h->seg_ptr, seg_ptr.data(), seg_ptr.size(), s));
  TT_TRY(tup(h, &h->seg_vox, seg_vox.data(), seg_vox.size(), s));
  TT_TRY(tup(h, &h->seg_grid, seg_grid.data(), seg_grid.size(), s));
  TT_TRY(tup(h, (int32_t**)&sa.nbr, d->heart_nbr, (size_t)d->n_heart * 6, s));
  TT_TRY(tup(h, (int32_t**)&sa.proj, d->proj, d->n_heart, s));
  TT_TRY(tal(h, &h->vm_dev, d->n_heart));
  TT_TRY(tal(h, &sa.iv, d->n_heart));
  if (d->n_heart) HP_CUDA_TRY(cudaMemsetAsync(sa.iv, 0, d->n_heart * 4, s));
  TT_TRY(tup(h, &sa.mean_count, &n_valid, 1, s));
  sa.vm = h->vm_dev;
  // read-out rows
  h->n_read = d->n_read;
  std::vector<int64_t> gr(d->n_read);
  for (int m = 0; m < d->n_read; ++m) gr[m] = grid_of_row[d->read_rows[m]];
  TT_TRY(tup(h, &h->grid_of_read, gr.data(), gr.size(), s));
  TT_TRY(tal(h, &h->out_dev, d->n_read));
  HP_CUDA_TRY(cudaMallocHost((void**)&h->h_scal, N_SCAL * 8 + (N_ISCAL + 1) * 4));
  h->h_iscal = (int32_t*)(h->h_scal + N_SCAL);
  HP_CUDA_TRY(cudaStreamSynchronize(s));
  *out = h;
  return HP_OK;
}

extern "C" int64_t hp_torso_rows(const HpTorso* h) { return h ? h->n_rows : -1; }

// CG iterations from the state that true_residual (or the last launch) left,
// until the done flag: one cooperative launch.
static hp_status run_iterations(HpTorso* h, bool p99, cudaStream_t s) {
  void* args[] = {&h->a, &h->pcg};
  HP_CUDA_TRY(cudaLaunchCooperativeKernel((const void*)h->pcg_fn[p99 ? 1 : 0], dim3(h->pcg_grid),
                                          dim3(32 * PCG_WARPS), args, h->pcg_smem, s));
  if (h->fail_in > 0 && --h->fail_in == 0)
    HP_CUDA_TRY(cudaMemsetAsync(h->pcg.sync.err, 1, sizeof(int32_t), s));
  return HP_OK;
}

extern "C" hp_status hp_torso_inject_timeout(HpTorso* h, int32_t launch) {
  HP_REQUIRE(h && launch >= 1, "hp_torso_inject_timeout: null handle or launch < 1");
  h->fail_in = launch;
  return HP_OK;
}

namespace hp {

// b <- per-frame source (compute_bspm.py:381-419)
static hp_status build_rhs(HpTorso* h, const float* vm, int vm_on_device, cudaStream_t s) {
  TorsoArgs& a = h->a;
  SrcArgs& sa = h->s;
  if (sa.n_heart > 0) {
    HP_REQUIRE(vm, "torso solve: vm is null");
    HP_CUDA_TRY(cudaMemcpyAsync(h->vm_dev, vm, (size_t)sa.n_heart * 4,
                                vm_on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice, s));
  }
  HP_CUDA_TRY(cudaMemsetAsync(a.b, 0, a.ng * 4, s));
  if (sa.n_heart > 0) {
    src_laplacian<<<h->nblk, TB, 0, s>>>(sa);
    if (h->n_seg > 0)
      src_scatter<<<(h->n_seg + TB - 1) / TB, TB, 0, s>>>(sa.iv, h->seg_ptr, h->seg_vox,
                                                           h->seg_grid, h->n_seg, a.scal,
                                                           h->inv_nexp, a.b, a.pin, a.psi);
  }
  HP_CUDA_TRY(cudaGetLastError());
  return HP_OK;
}

// Enqueues the read-out of the current x (read-out potentials in mV).
static hp_status readout(HpTorso* h, float* out, int out_on_device, cudaStream_t s) {
  if (h->n_read > 0 && out) {
    gather_out<<<(h->n_read + 255) / 256, 256, 0, s>>>(h->a.x, h->grid_of_read, h->n_read,
                                                        out_on_device ? out : h->out_dev);
    HP_CUDA_TRY(cudaGetLastError());
    if (!out_on_device)
      HP_CUDA_TRY(cudaMemcpyAsync(out, h->out_dev, h->n_read * 4, cudaMemcpyDeviceToHost, s));
  }
  return HP_OK;
}

// The device scalars on the host; out (may be null) receives the read-out of
// the current x in the same wait.
static hp_status read_scalars(HpTorso* h, cudaStream_t s, float* out = nullptr,
                              int out_on_device = 0) {
  HP_CUDA_TRY(cudaMemcpyAsync(h->h_scal, h->a.scal, N_SCAL * 8 + (N_ISCAL + 1) * 4,
                              cudaMemcpyDeviceToHost, s));
  const hp_status st = readout(h, out, out_on_device, s);
  if (st != HP_OK) return st;
  HP_CUDA_TRY(cudaStreamSynchronize(s));
  if (h->h_iscal[N_ISCAL]) {
    hp::set_error("torso solve: a grid barrier timed out");
    return HP_ERR_TIMEOUT;
  }
  return HP_OK;
}

// Jacobi-PCG from the current x on the current b.  *result receives the
// outcome (HP_OK, NOT_CONVERGED, STAGNATED, NONFINITE).  Residual, iterations
// and the check of the result are enqueued together; the host reads the
// scalars once per recursion and only repeats where the true residual of the
// relative rule missed.  out (may be null) receives the read-out.
static hp_status pcg_solve(HpTorso* h, double tol, int rule, int max_iter, HpSolveStats* stats,
                           hp_status* result_out, float* out, int out_on_device,
                           cudaStream_t s) {
  TorsoArgs& a = h->a;
  const double tol_dev = rule == HP_STOP_REL ? tol : tol * 1e-3;   // mV -> V for the mV rules
  // r = b - A x0 (warm start; x = 0 for the first frame), beta = 0
  SolveInit init{rule, max_iter, 0, 0, tol_dev};
  true_residual<<<h->nblk, TB, 0, s>>>(a, 1, init);
  HP_CUDA_TRY(cudaGetLastError());
  int restarts = 0;
  int total_it = 0;
  hp_status result = HP_OK;
  double rel = 0.0;
  for (;;) {
    hp_status st = run_iterations(h, rule == HP_STOP_P99, s);
    if (st != HP_OK) return st;
    // the relative rule restarts from the replaced residual where it missed
    init.max_iter = max_iter;
    true_residual<<<h->nblk, TB, 0, s>>>(a, 2, init);
    HP_CUDA_TRY(cudaGetLastError());
    st = read_scalars(h, s, out, out_on_device);
    if (st != HP_OK) return st;
    const double bb = h->h_scal[SC_BB];
    rel = bb > 0.0 ? sqrt(h->h_scal[SC_TRUE_RR] / bb) : 0.0;
    const int its = h->h_iscal[IS_ITER];
    total_it += its;
    if (bb == 0.0 && rule == HP_STOP_REL) {   // zero source: the pinned solution is 0
      HP_CUDA_TRY(cudaMemsetAsync(a.x, 0, a.ng * 8, s));
      st = read_scalars(h, s, out, out_on_device);
      if (st != HP_OK) return st;
      rel = 0.0;
      break;
    }
    if (h->h_iscal[IS_NONFINITE]) { result = HP_ERR_NONFINITE; break; }
    if (rule != HP_STOP_REL) {
      // reference mV rules: the recursive statistic decides
      if (!(h->h_scal[SC_STAT] < tol_dev)) result = HP_ERR_NOT_CONVERGED;
      if (h->h_iscal[IS_BREAKDOWN]) result = HP_OK;   // reference: break, return x
      break;
    }
    if (its > 0 || rel > tol) ++restarts;   // a recursion ran (or broke down at once)
    if (rel <= tol) break;
    if (total_it >= max_iter) { result = HP_ERR_NOT_CONVERGED; break; }
    if (restarts > 50) { result = HP_ERR_STAGNATED; break; }
    init.max_iter = max_iter - total_it;
    true_residual<<<h->nblk, TB, 0, s>>>(a, 1, init);
    HP_CUDA_TRY(cudaGetLastError());
  }
  if (rule == HP_STOP_REL && restarts > 0) --restarts;   // the final check is not a restart
  if (stats) {
    stats->iterations = total_it;
    stats->status = result;
    stats->rel_residual = rel;
    stats->stat = h->h_scal[SC_STAT];
    stats->restarts = restarts;
  }
  *result_out = result;
  return HP_OK;
}

static hp_status finish(hp_status result, const char* what) {
  if (result == HP_ERR_NOT_CONVERGED || result == HP_ERR_STAGNATED) return HP_OK;  // in stats
  if (result != HP_OK) {
    hp::set_error("%s: non-finite values in the solve", what);
    return result;
  }
  return HP_OK;
}

}  // namespace hp

extern "C" hp_status hp_torso_solve_frame(HpTorso* h, const float* vm, int32_t vm_on_device,
                                          float* out, int32_t out_on_device, double tol,
                                          int32_t rule, int32_t max_iter, HpSolveStats* stats,
                                          void* stream) {
  HP_REQUIRE(h, "hp_torso_solve_frame: null handle");
  HP_REQUIRE(rule >= 0 && rule <= 3, "hp_torso_solve_frame: unknown rule %d", rule);
  HP_REQUIRE(max_iter >= 1, "hp_torso_solve_frame: max_iter must be >= 1");
  HP_REQUIRE(tol > 0.0, "hp_torso_solve_frame: tol must be positive");
  cudaStream_t s = (cudaStream_t)stream;
  hp_status st = build_rhs(h, vm, vm_on_device, s);
  if (st != HP_OK) return st;
  hp_status result = HP_OK;
  st = pcg_solve(h, tol, rule, max_iter, stats, &result, out, out_on_device, s);
  if (st != HP_OK) return st;
  h->have_x = true;
  return finish(result, "hp_torso_solve_frame");
}

extern "C" hp_status hp_torso_arrays(HpTorso* h, HpTorsoArrays* o) {
  HP_REQUIRE(h && o, "hp_torso_arrays: null argument");
  o->ni = h->ni; o->nj = h->nj; o->nk = h->nk;
  o->n_cells = h->a.ng;
  o->pin_cell = h->a.pin;
  o->label = h->a.label;
  o->invd = h->a.invd;
  o->r = h->a.r;
  o->x = h->a.x;
  o->b = h->a.b;
  return HP_OK;
}

// ------------------------------------------------------------ flexible CG

namespace hp {

// q = A p (p in p0), partial p.q and p.r; last block: alpha = p.r / p.q.  On
// the resident PCG's pair tables (41 us on the full torso where every cell
// decoded its label, 31 here), one warp per tissue line; the order of the
// two sums is fixed like the PCG's (see pcg_resident.cuh), so the grid is.
// (The preconditioners need an even padded row, so pairs are aligned.)
__global__ void __launch_bounds__(TB, 4) fcg_spmv(TorsoArgs a, PcgArgs c) {
  __shared__ float s_t[HP_MAX_MATERIALS];
  if (a.iscal[IS_DONE]) return;
  if (threadIdx.x < HP_MAX_MATERIALS) s_t[threadIdx.x] = c.tu[threadIdx.x];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int n_warps = gridDim.x * (TB / 32);
  const int64_t sj = a.pk / 2, si = (int64_t)a.pj * sj;
  double acc[2] = {0.0, 0.0};
  for (int l = blockIdx.x * (TB / 32) + (threadIdx.x >> 5); l < c.n_lines; l += n_warps) {
    const PcgLine L = c.line[l];
    const int64_t g2 = (int64_t)(L.p2 / c.sj) * sj + L.p2 % c.sj;  // first pair in the padded grid
    const float2* __restrict__ p = (const float2*)a.p0 + g2;
    const float2* __restrict__ rv = (const float2*)a.r + g2;
    float2* __restrict__ Ap = (float2*)a.Ap + g2;
    const uint32_t* __restrict__ m = c.meta + L.c2;
    for (int q = lane; q < L.n2; q += 32) {
      const uint32_t mq = m[q];
      const float2 pc = p[q], ip = p[q + si], im = p[q - si], jp = p[q + sj], jm = p[q - sj];
      const float km = ((const float*)p)[2 * q - 1], kp = ((const float*)p)[2 * q + 2];
      const float2 rq = rv[q];
      const float pv[2] = {pc.x, pc.y};
      const float nb[6][2] = {{ip.x, ip.y}, {im.x, im.y}, {jp.x, jp.y},
                              {jm.x, jm.y}, {pc.y, kp},   {km, pc.x}};
      float ap[2] = {0.0f, 0.0f};
      if (mq & PQ_MIXED) {
        const float2* __restrict__ W = c.mixed + (mq & ~PQ_MIXED);
#pragma unroll
        for (int f = 0; f < 6; ++f) {
          const float2 w = W[f * (int64_t)c.n_mixed];
          ap[0] = __fmaf_rn(w.x, __fsub_rn(pv[0], nb[f][0]), ap[0]);
          ap[1] = __fmaf_rn(w.y, __fsub_rn(pv[1], nb[f][1]), ap[1]);
        }
      } else {
        const float w = s_t[mq];
#pragma unroll
        for (int f = 0; f < 6; ++f)
#pragma unroll
          for (int e = 0; e < 2; ++e) ap[e] = __fmaf_rn(w, __fsub_rn(pv[e], nb[f][e]), ap[e]);
      }
      Ap[q] = make_float2(ap[0], ap[1]);
      acc[0] += (double)pv[0] * (double)ap[0];
      acc[1] += (double)pv[0] * (double)rq.x;
      acc[0] += (double)pv[1] * (double)ap[1];
      acc[1] += (double)pv[1] * (double)rq.y;
    }
  }
  double tot[2];
  if (block_reduce_last<2>(acc, 0u, a.part, a.ticket, tot) && threadIdx.x == 0) {
    a.scal[SC_PAP] = tot[0];
    if (!(fabs(tot[0]) >= 1e-30) || !isfinite(tot[0])) {
      a.iscal[IS_BREAKDOWN] = isfinite(tot[0]) ? 1 : 0;
      a.iscal[IS_NONFINITE] = isfinite(tot[0]) ? 0 : 1;
      a.iscal[IS_DONE] = 1;
      a.scal[SC_ALPHA] = 0.0;
    } else {
      a.scal[SC_ALPHA] = tot[1] / tot[0];
    }
  }
}

// The flexible-CG vector passes below take pieces of 32 LB cells of a tissue
// line that start on a multiple of 32 LB of the unpadded k, one warp per piece
// (whole lines left the last of 5 rounds of the full torso's warps a tenth
// full), all loads of a piece issued before any arithmetic: load(u, g) on the
// line's cells, apply(u, g, on) by all lanes (on: a cell of the line), then
// done(i, j, k) with the unpadded line and the piece's first k.
template <int LB, class Load, class Apply, class Done>
__device__ __forceinline__ void for_aligned_lines(const TorsoArgs& a, Load&& load, Apply&& apply,
                                                  Done&& done) {
  const int lane = threadIdx.x & 31;
  const int n_warps = gridDim.x * (TB / 32);
  const int per = (a.pk + 32 * LB - 3) / (32 * LB);  // pieces of a row of pk - 2 cells
  const int n = a.n_lines * per;
  int w = blockIdx.x * (TB / 32) + (threadIdx.x >> 5);
  int4 next = w < n ? a.line[w / per] : make_int4(0, 0, 0, 0);  // one piece ahead
  for (; w < n; w += n_warps) {
    const int4 line = next;
    if (w + n_warps < n) next = a.line[(w + n_warps) / per];
    const int k0 = w % per * 32 * LB, first = line.y, end = line.z;
    if (k0 >= end || k0 + 32 * LB <= first) continue;
    const int64_t base = (int64_t)line.x * a.pk + 1;
#pragma unroll
    for (int u = 0; u < LB; ++u) {
      const int k = k0 + 32 * u + lane;
      if (k >= first && k < end) load(u, base + k);
    }
#pragma unroll
    for (int u = 0; u < LB; ++u) {
      const int k = k0 + 32 * u + lane;
      apply(u, base + k, k >= first && k < end);
    }
    done(line.w, line.x - (line.w + 1) * a.pj - 1, k0);
  }
}

// x += alpha p, r -= alpha q, partial r.r, and the sums of r over the coarse
// level's line segments (while r is in registers: a pass over r of its own
// took 35 us on the full torso); last block: recursive stat, done test.
// Bound by memory: 32 bytes a cell, 43 us cold on the full torso (29 us at the
// copy bandwidth).
__global__ void __launch_bounds__(TB) fcg_update(TorsoArgs a, pc::SegArgs seg) {
  if (a.iscal[IS_DONE]) return;
  const double alpha = a.scal[SC_ALPHA];
  const float af = (float)alpha;
  const float* __restrict__ p = a.p0;
  const float* __restrict__ Ap = a.Ap;
  float* __restrict__ rv = a.r;
  double* __restrict__ x = a.x;
  double acc[1] = {0.0};
  constexpr int LB = 4;
  const int lane = threadIdx.x & 31;
  float pb[LB], rb[LB];
  double xb[LB], sb[LB];
  for_aligned_lines<LB>(
      a,
      [&](int u, int64_t g) {
        pb[u] = p[g];
        xb[u] = x[g];
        rb[u] = rv[g] - af * Ap[g];
      },
      [&](int u, int64_t g, bool on) {
        sb[u] = 0.0;
        if (on) {
          x[g] = xb[u] + alpha * (double)pb[u];
          rv[g] = rb[u];
          sb[u] = (double)rb[u];
          acc[0] += sb[u] * sb[u];
        }
      },
      [&](int i, int j, int k) {
        if (!seg.seg) return;
        // four steps' sums at once: lanes exchange two, then one of them, so
        // that lane l goes on with step l % 4; then over the segment
        const bool b0 = lane & 1, b1 = lane & 2;
        double t0 = (b0 ? sb[1] : sb[0]) + __shfl_xor_sync(0xffffffffu, b0 ? sb[0] : sb[1], 1);
        double t1 = (b0 ? sb[3] : sb[2]) + __shfl_xor_sync(0xffffffffu, b0 ? sb[2] : sb[3], 1);
        double s = (b1 ? t1 : t0) + __shfl_xor_sync(0xffffffffu, b1 ? t0 : t1, 2);
        for (int o = 4; o < seg.len; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        const int ks = (k + 32 * (lane & 3) + (lane & ~3)) / seg.len;
        if ((lane & (seg.len - 1)) < 4 && ks < seg.n_seg)
          seg.seg[((int64_t)i * seg.nj + j) * seg.n_seg + ks] = s;
      });
  double tot[1];
  if (block_reduce_last<1>(acc, 0u, a.part, a.ticket, tot) && threadIdx.x == 0) {
    a.scal[SC_RR] = tot[0];
    const double stat = sqrt(tot[0] / fmax(a.scal[SC_BB], 1e-300));
    a.scal[SC_STAT] = stat;
    const int it = ++a.iscal[IS_ITER];
    // stagnation: less than 3 % progress over the last 5 iterations
    const int nh = ++a.iscal[IS_NH];
    a.scal[SC_HIST0 + (nh - 1) % 8] = stat;
    const bool stagnant =
        a.iscal[IS_STAG_ON] && nh > 6 && stat > 0.97 * a.scal[SC_HIST0 + (nh - 6) % 8];
    if (!isfinite(tot[0])) { a.iscal[IS_NONFINITE] = 1; a.iscal[IS_DONE] = 1; }
    else if (stat < 0.5 * a.scal[SC_TOL] || it >= a.iscal[IS_MAXIT]) a.iscal[IS_DONE] = 1;
    else if (stagnant) { a.iscal[IS_STAGNANT] = 1; a.iscal[IS_DONE] = 1; }
  }
}

// partial z.q with z = M(r) formed on the fly (zero on air and at the pin,
// where invd is zero); last block: beta = -z.q / p.q.  Forming z here and
// again in fcg_p reads r and invd twice but saves its store and two loads and
// the pass that made it (47 + 16 + 15 us on the full torso; 24 + 20 now).
__global__ void __launch_bounds__(TB) fcg_beta(TorsoArgs a, pc::ZArgs z) {
  if (a.iscal[IS_DONE]) return;
  const float* __restrict__ Ap = a.Ap;
  const float* __restrict__ rv = a.r;
  const float* __restrict__ invd = a.invd;
  double acc[1] = {0.0};
  constexpr int LB = 4;
  const int lane = threadIdx.x & 31;
  float qb[LB], rb[LB], ib[LB];
  for_aligned_lines<LB>(
      a, [&](int u, int64_t g) { qb[u] = Ap[g]; rb[u] = rv[g]; ib[u] = invd[g]; },
      [&](int u, int64_t, bool on) { if (!on) ib[u] = 0.0f; },
      [&](int i, int j, int k) {
#pragma unroll
        for (int u = 0; u < LB; ++u)
          if (ib[u] != 0.0f)
            acc[0] += (double)pc::z_value(z, ib[u], rb[u], i, j, k + 32 * u + lane) * qb[u];
      });
  double tot[1];
  if (block_reduce_last<1>(acc, 0u, a.part, a.ticket, tot) && threadIdx.x == 0)
    a.scal[SC_BETA] = -tot[0] / a.scal[SC_PAP];
}

// p = z + beta p, z = M(r) formed on the fly again; `first` starts a recursion
// without reading p, which may hold what a non-finite solve left
__global__ void __launch_bounds__(TB) fcg_p(TorsoArgs a, pc::ZArgs z, int first) {
  if (a.iscal[IS_DONE]) return;
  const float beta = first ? 0.0f : (float)a.scal[SC_BETA];
  const float* __restrict__ rv = a.r;
  const float* __restrict__ invd = a.invd;
  float* __restrict__ p = a.p0;
  constexpr int LB = 4;
  const int lane = threadIdx.x & 31;
  float pb[LB], rb[LB], ib[LB];
  int64_t gb[LB];
  for_aligned_lines<LB>(
      a, [&](int u, int64_t g) { pb[u] = first ? 0.0f : p[g]; rb[u] = rv[g]; ib[u] = invd[g]; },
      [&](int u, int64_t g, bool on) { gb[u] = g; if (!on) ib[u] = 0.0f; },
      [&](int i, int j, int k) {
#pragma unroll
        for (int u = 0; u < LB; ++u)
          if (ib[u] != 0.0f)
            p[gb[u]] = __fmaf_rn(beta, pb[u],
                                 pc::z_value(z, ib[u], rb[u], i, j, k + 32 * u + lane));
      });
}

__global__ void error_kernel(TorsoArgs a, const double* __restrict__ xstar, float* __restrict__ e) {
  for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < a.ng;
       g += (int64_t)gridDim.x * blockDim.x)
    e[g] = is_row(a, g) ? (float)(xstar[g] - a.x[g]) : 0.0f;
}

constexpr int FCG_CHUNK = 4;

// The FCG iteration body (A p, x / r update and stopping tests, z = M(r),
// beta, p) for FCG_CHUNK iterations, captured once per network period,
// stream and preconditioner handle.  use_net = k > 0 applies the network
// term on every k-th iteration of the chunk (k divides FCG_CHUNK) and the
// Jacobi + coarse terms alone on the others: flexible CG admits a
// preconditioner that changes from one iteration to the next.
static hp_status fcg_graph(HpTorso* h, HpPrecond* p, int use_net, cudaStream_t s) {
  const int q = use_net == 0 ? 0 : (use_net == 1 ? 1 : (use_net == 2 ? 2 : 3));
  const uint64_t serial = pc::precond_serial(p);
  if (h->fcg_graph[q] && h->fcg_graph_stream == s && h->fcg_graph_pc == serial)
    return HP_OK;
  if (h->fcg_graph_stream != s || h->fcg_graph_pc != serial) {
    for (int k = 0; k < 4; ++k)
      if (h->fcg_graph[k]) { cudaGraphExecDestroy(h->fcg_graph[k]); h->fcg_graph[k] = nullptr; }
  }
  TorsoArgs& a = h->a;
  cudaGraph_t g;
  HP_CUDA_TRY(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
  hp_status st = HP_OK;
  for (int it = 0; it < FCG_CHUNK && st == HP_OK; ++it) {
    fcg_spmv<<<h->nblk_k[K_FCG_SPMV], TB, 0, s>>>(a, h->pcg);
    fcg_update<<<h->nblk_k[K_FCG_UPDATE], TB, 0, s>>>(a, pc::precond_segments(p));
    const int net = use_net > 0 && it % use_net == 0;
    st = pc::precond_update(p, a.label, a.invd, a.r, net, s);
    if (st != HP_OK) break;
    const pc::ZArgs z = pc::precond_z(p, net);
    fcg_beta<<<h->nblk_k[K_FCG_BETA], TB, 0, s>>>(a, z);
    fcg_p<<<h->nblk_k[K_FCG_P], TB, 0, s>>>(a, z, 0);
  }
  cudaError_t ce = cudaStreamEndCapture(s, &g);
  if (st != HP_OK) return st;
  HP_CUDA_TRY(ce);
  HP_CUDA_TRY(cudaGraphInstantiate(&h->fcg_graph[q], g, 0));
  cudaGraphDestroy(g);
  h->fcg_graph_stream = s;
  h->fcg_graph_pc = serial;
  return HP_OK;
}

// One flexible-CG run with M (use_net selects the network term) from the
// current x; returns with *fallback set when it did not converge within
// fallback_iter iterations, stagnated or broke down.
static hp_status fcg_run(HpTorso* h, HpPrecond* p, double tol, int fallback_iter, int use_net,
                         int* it_out, int* restarts_out, double* rel_out, bool* fallback,
                         cudaStream_t s) {
  TorsoArgs& a = h->a;
  *fallback = false;
  // the stagnation test guards the runs with the network; the method
  // without it runs until convergence or the iteration budget
  SolveInit init{HP_STOP_REL, fallback_iter, use_net ? 1 : 0, 0, tol};
  true_residual<<<h->nblk, TB, 0, s>>>(a, 1, init);
  HP_CUDA_TRY(cudaGetLastError());
  hp_status st = read_scalars(h, s);
  if (st != HP_OK) return st;
  const double bb = h->h_scal[SC_BB];
  double rel = bb > 0.0 ? sqrt(h->h_scal[SC_TRUE_RR] / bb) : 0.0;
  int it = 0;
  if (bb == 0.0) {
    HP_CUDA_TRY(cudaMemsetAsync(a.x, 0, a.ng * 8, s));
    *rel_out = 0.0;
    *it_out = 0;
    return HP_OK;
  }
  if (!isfinite(bb) || !isfinite(h->h_scal[SC_TRUE_RR])) {  // rel says nothing; the plain PCG reports it
    *rel_out = rel;
    *it_out = 0;
    *fallback = true;
    return HP_OK;
  }
  // chunks of FCG_CHUNK iterations replayed from a CUDA graph; kernels of a
  // chunk after the device-side done flag return at once (the
  // preconditioner's then only writes its own scratch and z)
  // z = M(r0), p = z (this first application also sets up anything the
  // preconditioner initialises lazily, before the capture)
  const pc::ZArgs z0 = pc::precond_z(p, use_net);
  st = pc::precond_begin(p, a.label, a.invd, a.r, use_net, s);
  if (st != HP_OK) return st;
  fcg_p<<<h->nblk_k[K_FCG_P], TB, 0, s>>>(a, z0, 1);
  st = fcg_graph(h, p, use_net, s);
  if (st != HP_OK) return st;
  bool restart = false;
  while (rel > tol) {
    if (restart) {
      st = pc::precond_begin(p, a.label, a.invd, a.r, use_net, s);
      if (st != HP_OK) return st;
      fcg_p<<<h->nblk_k[K_FCG_P], TB, 0, s>>>(a, z0, 1);
      restart = false;
    }
    HP_CUDA_TRY(cudaGraphLaunch(h->fcg_graph[use_net == 0 ? 0 : (use_net == 1 ? 1 : (use_net == 2 ? 2 : 3))], s));
    st = read_scalars(h, s);
    if (st != HP_OK) return st;
    it = h->h_iscal[IS_ITER];
    if (h->h_iscal[IS_NONFINITE] || h->h_iscal[IS_BREAKDOWN] || h->h_iscal[IS_STAGNANT]) {
      *fallback = true;
      break;
    }
    if (h->h_iscal[IS_DONE]) {
      if (h->h_scal[SC_STAT] >= 0.5 * tol) { *fallback = true; break; }   // iteration budget
      // recursive residual below tol / 2: the FP64 true residual decides
      init.iter = it;
      true_residual<<<h->nblk, TB, 0, s>>>(a, 1, init);
      st = read_scalars(h, s);
      if (st != HP_OK) return st;
      rel = sqrt(h->h_scal[SC_TRUE_RR] / h->h_scal[SC_BB]);
      if (rel <= tol) break;
      ++*restarts_out;
      restart = true;
    }
  }
  *it_out = it;
  *rel_out = rel;
  return HP_OK;
}

// Flexible CG with the learned preconditioner.  Safeguards, in order: when
// the run with the network fails (no convergence within fallback_iter,
// stagnation or breakdown), FCG restarts from the current iterate without
// the network (the two-level method, restarts += 100; no stagnation test,
// up to max(fallback_iter, 1000) iterations); when that fails too, plain
// Jacobi-PCG finishes the frame (restarts += 1000).
static hp_status fcg_solve(HpTorso* h, HpPrecond* p, double tol, int max_iter, int fallback_iter,
                           int use_net, HpSolveStats* stats, hp_status* result_out, cudaStream_t s) {
  int it_total = 0, restarts = 0;
  double rel = 0.0;
  bool fallback = false;
  hp_status result = HP_OK;
  // the run with the network (use_net = its period) for at most
  // fallback_iter iterations, then without it (the two-level method, which
  // converges on its own: up to 1000 iterations, or fallback_iter if more)
  for (int net = use_net; net >= 0; net = net > 0 ? 0 : -1) {
    int it = 0;
    const int cap = net > 0 ? fallback_iter : std::max(fallback_iter, 1000);
    const int budget = std::max(1, std::min(cap, max_iter - it_total));
    hp_status st = fcg_run(h, p, tol, budget, net, &it, &restarts, &rel, &fallback, s);
    if (st != HP_OK) return st;
    it_total += it;
    if (!fallback) break;
    if (net > 0) restarts += 100;
  }
  if (fallback) {
    HpSolveStats st2;
    hp_status r2 = HP_OK;
    hp_status st = pcg_solve(h, tol, HP_STOP_REL, std::max(1, max_iter - it_total), &st2, &r2,
                             nullptr, 0, s);
    if (st != HP_OK) return st;
    it_total += st2.iterations;
    rel = st2.rel_residual;
    result = r2;
    restarts += 1000;
  }
  if (stats) {
    stats->iterations = it_total;
    stats->status = result;
    stats->rel_residual = rel;
    stats->stat = rel;
    stats->restarts = restarts;
  }
  *result_out = result;
  return HP_OK;
}

}  // namespace hp

extern "C" hp_status hp_torso_solve_frame_fcg(HpTorso* h, HpPrecond* p, const float* vm,
                                              int32_t vm_on_device, float* out,
                                              int32_t out_on_device, double tol, int32_t max_iter,
                                              int32_t fallback_iter, int32_t use_net,
                                              HpSolveStats* stats, void* stream) {
  HP_REQUIRE(h, "hp_torso_solve_frame_fcg: null torso handle");
  HP_REQUIRE(!h->a.psi, "hp_torso_solve_frame_fcg: the flexible-CG preconditioners are built for "
                        "the sharp-boundary operator; a smoothed-boundary (psi) handle solves "
                        "with hp_torso_solve_frame");
  HP_REQUIRE(p, "hp_torso_solve_frame_fcg: null preconditioner");
  HP_REQUIRE(h->a.p0, "hp_torso_solve_frame_fcg: the torso's dims must be multiples of (8, 8, 256)");
  HP_REQUIRE(max_iter >= 1 && fallback_iter >= 1, "hp_torso_solve_frame_fcg: bad iteration limits");
  HP_REQUIRE(use_net == 0 || use_net == 1 || use_net == 2 || use_net == 4,
             "hp_torso_solve_frame_fcg: use_net must be 0, 1, 2 or 4");
  HP_REQUIRE(tol > 0.0, "hp_torso_solve_frame_fcg: tol must be positive");
  cudaStream_t s = (cudaStream_t)stream;
  hp_status st = build_rhs(h, vm, vm_on_device, s);
  if (st != HP_OK) return st;
  hp_status result = HP_OK;
  st = fcg_solve(h, p, tol, max_iter, fallback_iter, use_net, stats, &result, s);
  if (st != HP_OK) return st;
  st = readout(h, out, out_on_device, s);
  if (st != HP_OK) return st;
  HP_CUDA_TRY(cudaStreamSynchronize(s));
  h->have_x = true;
  return finish(result, "hp_torso_solve_frame_fcg");
}

namespace hp {
// n more iterations of the current CG recursion (no restart, no stopping
// test): x is the n-th iterate.
static hp_status pcg_continue(HpTorso* h, int n, cudaStream_t s) {
  TorsoArgs& a = h->a;
  const double never = 0.0;     // relative rule with tolerance 0: runs all n
  HP_CUDA_TRY(cudaMemcpyAsync(a.scal + SC_TOL, &never, 8, cudaMemcpyHostToDevice, s));
  int32_t is_run[N_ISCAL] = {0, 0, HP_STOP_REL, n, 0, 0};
  HP_CUDA_TRY(cudaMemcpyAsync(a.iscal, is_run, sizeof(is_run), cudaMemcpyHostToDevice, s));
  hp_status st = run_iterations(h, false, s);
  if (st != HP_OK) return st;
  return read_scalars(h, s);   // waits: the host scalars above are stack temporaries
}
}  // namespace hp

extern "C" hp_status hp_torso_train_precond(HpTorso* h, HpPrecond* p, const float* vm_frames,
                                            int64_t frame_stride, int32_t n_frames,
                                            const int32_t* ks, int32_t n_ks, int32_t repeats,
                                            float lr, double tol_exact, float* loss_hist,
                                            void* stream) {
  HP_REQUIRE(h && !h->a.psi, "hp_torso_train_precond: the preconditioners are built for the "
                            "sharp-boundary operator (this handle has psi)");
  HP_REQUIRE(h && p && vm_frames && ks && n_frames >= 1 && n_ks >= 1 && repeats >= 1,
             "hp_torso_train_precond: bad arguments");
  for (int q = 0; q < n_ks; ++q)
    HP_REQUIRE(ks[q] >= 0 && (q == 0 || ks[q] >= ks[q - 1]),
               "hp_torso_train_precond: ks must be non-negative and ascending");
  cudaStream_t s = (cudaStream_t)stream;
  TorsoArgs& a = h->a;
  double *xstar = nullptr, *x0 = nullptr;
  float* e = nullptr;
  HP_CUDA_TRY(cudaMalloc((void**)&xstar, a.ng * 8));
  HP_CUDA_TRY(cudaMalloc((void**)&x0, a.ng * 8));
  HP_CUDA_TRY(cudaMalloc((void**)&e, a.ng * 4));
  hp_status ret = HP_OK;
  int64_t q = 0;
  for (int f = 0; f < n_frames && ret == HP_OK; ++f) {
    ret = build_rhs(h, vm_frames + (int64_t)f * frame_stride, 1, s);
    if (ret != HP_OK) break;
    if (cudaMemcpyAsync(x0, a.x, a.ng * 8, cudaMemcpyDeviceToDevice, s) != cudaSuccess) { ret = HP_ERR_CUDA; break; }
    hp_status res = HP_OK;
    ret = pcg_solve(h, tol_exact, HP_STOP_REL, 20000, nullptr, &res, nullptr, 0, s);
    if (ret != HP_OK) break;
    if (cudaMemcpyAsync(xstar, a.x, a.ng * 8, cudaMemcpyDeviceToDevice, s) != cudaSuccess) { ret = HP_ERR_CUDA; break; }
    // one plain-PCG trajectory from the warm start; pairs at iterations ks
    // (ascending): r_k (the recursion's residual) and e_k = x* - x_k
    if (cudaMemcpyAsync(a.x, x0, a.ng * 8, cudaMemcpyDeviceToDevice, s) != cudaSuccess) { ret = HP_ERR_CUDA; break; }
    // r = b - A x0, fresh recursion
    true_residual<<<h->nblk, TB, 0, s>>>(a, 1, SolveInit{HP_STOP_REL, 0, 0, 0, 0.0});
    int done = 0;
    for (int kq = 0; kq < n_ks && ret == HP_OK; ++kq) {
      if (ks[kq] > done) {
        ret = pcg_continue(h, ks[kq] - done, s);
        if (ret != HP_OK) break;
        done = ks[kq];
      }
      error_kernel<<<h->nblk, TB, 0, s>>>(a, xstar, e);
      for (int rp = 0; rp < repeats && ret == HP_OK; ++rp) {
        float loss = 0.0f;
        ret = hp_precond_train_step(p, a.label, a.invd, a.r, e, lr, &loss, s);
        if (loss_hist) loss_hist[q] = loss;
        ++q;
      }
    }
    if (ret == HP_OK && cudaMemcpyAsync(a.x, xstar, a.ng * 8, cudaMemcpyDeviceToDevice, s) != cudaSuccess)
      ret = HP_ERR_CUDA;
  }
  cudaStreamSynchronize(s);
  cudaFree(xstar);
  cudaFree(x0);
  cudaFree(e);
  return ret;
}

extern "C" hp_status hp_torso_copy_solution(HpTorso* h, double* x_rows, void* stream) {
  HP_REQUIRE(h && x_rows, "hp_torso_copy_solution: null argument");
  cudaStream_t s = (cudaStream_t)stream;
  double* tmp = nullptr;
  HP_CUDA_TRY(cudaMalloc((void**)&tmp, h->n_rows * 8));
  gather_rows<<<(unsigned)((h->n_rows + 255) / 256), 256, 0, s>>>(h->a.x, h->grid_of_row,
                                                                  h->n_rows, tmp);
  HP_CUDA_TRY(cudaMemcpyAsync(x_rows, tmp, h->n_rows * 8, cudaMemcpyDeviceToHost, s));
  HP_CUDA_TRY(cudaStreamSynchronize(s));
  HP_CUDA_TRY(cudaFree(tmp));
  return HP_OK;
}

extern "C" hp_status hp_torso_copy_rhs(HpTorso* h, float* b_rows, void* stream) {
  HP_REQUIRE(h && b_rows, "hp_torso_copy_rhs: null argument");
  cudaStream_t s = (cudaStream_t)stream;
  float* tmp = nullptr;
  HP_CUDA_TRY(cudaMalloc((void**)&tmp, h->n_rows * 4));
  gather_rows_f<<<(unsigned)((h->n_rows + 255) / 256), 256, 0, s>>>(h->a.b, h->grid_of_row,
                                                                    h->n_rows, tmp);
  HP_CUDA_TRY(cudaMemcpyAsync(b_rows, tmp, h->n_rows * 4, cudaMemcpyDeviceToHost, s));
  HP_CUDA_TRY(cudaStreamSynchronize(s));
  HP_CUDA_TRY(cudaFree(tmp));
  return HP_OK;
}

extern "C" hp_status hp_torso_reset(HpTorso* h) {
  HP_REQUIRE(h, "hp_torso_reset: null handle");
  // in the default stream, which a caller's non-blocking stream does not wait for
  HP_CUDA_TRY(cudaMemsetAsync(h->a.x, 0, h->a.ng * 8, cudaStreamLegacy));
  HP_CUDA_TRY(cudaStreamSynchronize(cudaStreamLegacy));
  h->have_x = false;
  return HP_OK;
}

extern "C" hp_status hp_torso_destroy(HpTorso* h) {
  if (!h) return HP_OK;
  for (int q = 0; q < 4; ++q)
    if (h->fcg_graph[q]) cudaGraphExecDestroy(h->fcg_graph[q]);
  for (void* p : h->allocs) cudaFree(p);
  if (h->h_scal) cudaFreeHost(h->h_scal);
  delete h;
  return HP_OK;
}
