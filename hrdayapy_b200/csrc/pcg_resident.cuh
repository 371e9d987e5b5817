// Jacobi-PCG iterations of the torso solve in one cooperative launch.
//
// A launch per pass (p update, A p, r update) bounded small and mid-size
// torsos by launch latency, host polls of the done flag and, on odd rows, a
// one-cell stencil, and had the full torso carry r through memory in two of
// the passes and decode labels per cell in all of them.  Here a warp owns
// whole tissue lines for the solve: r (and, while they fit, A p, x and the
// tables) stay in its block's shared memory, only p goes through L2, with one
// grid barrier after the p update and one all-reduce after each of A p and
// the r update.  All blocks hold the same scalars and take the same decisions.
//
// Cells are handled in pairs on a private copy of p of even row pitch.  A pair
// whose cells and neighbours all carry one material needs that material's
// conductance and Jacobi inverse only; every other pair (material boundaries,
// line ends, the pin, the smoothed boundary) has its six face conductances
// and inverses per cell precomputed, zero on air and at the pin.
//
// A solve that is warm-started from the last frame amplifies the last digit of
// its dot products: r = b - A x is rounded to FP32, so a step of 1e-16 in x
// flips the last bit of many residual entries, and hundreds of iterations
// later the stopped iterate has moved by up to 1e-4.  The order of the sums is
// therefore part of the method: 32 warps a multiprocessor take lines in turn,
// a lane adds its cells along the line (p.Ap pair by pair where the padded row
// is even, else cell by cell; the r update cell by cell), then the lanes of a
// warp, eight warps, and the eight-warp groups are added in a fixed tree.
// Per cell the FP32 arithmetic is the face-flux sum t (p_g - p_n) in face
// order +i -i +j -j +k -k, z = D^-1 r, p = z + beta p; x is FP64.
#pragma once
#include "grid_sync.cuh"

namespace hp {

// One tissue line: its first pair in p, pairs, first pair in the compact
// arrays and in its block's shared memory; the first cell's place in its pair
// and the cells.
struct PcgLine {
  uint32_t p2;
  int32_t n2, c2, s2, first, len;
};

struct PcgArgs {
  int32_t n_lines, n_pairs, n_mixed;
  int32_t room;           // pairs a block has room for in shared memory (a multiple of 4)
  const PcgLine* line;
  const uint32_t* meta;   // pair: material or PQ_MIXED | mixed index
  const float2* mixed;    // 7 x n_mixed: six face conductances, Jacobi inverse
  float tu[HP_MAX_MATERIALS], inv[HP_MAX_MATERIALS];  // of uniform pairs
  uint32_t sj, si;        // pair strides of a row and a plane of p
  float2* p;              // private pitch, zero off the rows
  float2* Ap;             // n_pairs (unless in shared memory)
  double2* x;             // n_pairs (unless in shared memory)
  float2* r;              // n_pairs (unless in shared memory)
  double* part;           // 2 x PCG_GROUPS x 4
  GridSync sync;
};
constexpr uint32_t PQ_MIXED = 0x80000000u;
constexpr int PCG_WARPS = 32;               // a block
constexpr int PCG_MAX_BLOCKS = 160;
constexpr int PCG_GROUPS = PCG_MAX_BLOCKS * (PCG_WARPS / 8);  // eight-warp groups
// where a block keeps its vectors: all in shared memory (36 bytes a pair), r
// alone (8 bytes a pair), none; PCG_MEM: nor its lines' records, for more of
// them than shared memory holds (24 bytes each, about 1.3 M on 148
// multiprocessors; nothing else would fit beside them there)
constexpr int PCG_ALL = 0, PCG_R = 1, PCG_NONE = 2, PCG_MEM = 3;
__host__ __device__ constexpr int pcg_pair_bytes(int mode) {
  return mode == PCG_ALL ? 36 : (mode == PCG_R ? 8 : 0);
}

// NV values over all threads of the launch: sums, or the maximum where bit k
// of MAXM is set, in the fixed order above (a lane's value, shuffles by 16, 8,
// .. 1, eight warps in turn, then the groups t, t + 256, .. of thread t and a
// tree over 256 threads).
template <int NV, uint32_t MAXM>
__device__ __forceinline__ bool grid_all(const PcgArgs& c, unsigned long long& epoch,
                                         double (&v)[NV]) {
  __shared__ double sh[PCG_WARPS][NV];
  __shared__ double tot[NV];
  __shared__ int s_ok;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int n_groups = gridDim.x * (PCG_WARPS / 8);
  double* part = c.part + (++epoch & 1) * (int64_t)PCG_GROUPS * 4;
  auto op = [](int k, double a, double b) { return (MAXM >> k) & 1u ? fmax(a, b) : a + b; };
  auto ident = [](int k) { return (MAXM >> k) & 1u ? -INFINITY : 0.0; };
  auto over_warp = [&]() {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      double w[NV];
#pragma unroll
      for (int k = 0; k < NV; ++k) w[k] = __shfl_down_sync(0xffffffffu, v[k], o);
#pragma unroll
      for (int k = 0; k < NV; ++k) v[k] = op(k, v[k], w[k]);
    }
  };
  over_warp();
  if (lane == 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k) sh[wid][k] = v[k];
  }
  __syncthreads();
  if (wid == 0) {
    if (lane < PCG_WARPS / 8) {
#pragma unroll
      for (int k = 0; k < NV; ++k) {
        double s = sh[8 * lane][k];
#pragma unroll
        for (int w = 1; w < 8; ++w) s = op(k, s, sh[8 * lane + w][k]);
        part[(blockIdx.x * (PCG_WARPS / 8) + lane) * 4 + k] = s;
      }
    }
    __syncwarp();
    if (lane == 0) s_ok = grid_arrive_wait(c.sync, epoch);
  }
  __syncthreads();
  // thread t < 256: groups t, t + 256, ..; then t and t + 128, t and t + 64, ..
  if (tid < 256) {
    double w[(PCG_GROUPS + 255) / 256][NV];
#pragma unroll
    for (int u = 0; u < (PCG_GROUPS + 255) / 256; ++u)
#pragma unroll
      for (int k = 0; k < NV; ++k)
        w[u][k] = tid + 256 * u < n_groups ? __ldcg(part + (tid + 256 * u) * 4 + k) : ident(k);
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      v[k] = ident(k);
#pragma unroll
      for (int u = 0; u < (PCG_GROUPS + 255) / 256; ++u) v[k] = op(k, v[k], w[u][k]);
    }
  }
  // the tree's steps by 128, 64 and 32 cross warps: every lane's column over
  // the eight warps, then the steps by 16 to 1 in one warp
  __shared__ double col[8][NV][32];
  if (tid < 256) {
#pragma unroll
    for (int k = 0; k < NV; ++k) col[wid][k][lane] = v[k];
  }
  __syncthreads();
  if (wid == 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      double t[8];
#pragma unroll
      for (int w = 0; w < 8; ++w) t[w] = col[w][k][lane];
#pragma unroll
      for (int w = 0; w < 4; ++w) t[w] = op(k, t[w], t[w + 4]);
      t[0] = op(k, t[0], t[2]);
      t[1] = op(k, t[1], t[3]);
      v[k] = op(k, t[0], t[1]);
    }
    over_warp();
    if (lane == 0) {
#pragma unroll
      for (int k = 0; k < NV; ++k) tot[k] = v[k];
    }
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < NV; ++k) v[k] = tot[k];
  return s_ok;
}

// The iterations from the residual and recursion that true_residual left
// (or an earlier launch: beta, r.z, p) until a stopping rule, the iteration
// limit or a breakdown.  At the end x holds the last iterate (nothing is
// pending) and r the recursive residual.
// P99 (the reference's 'p99' metric, compute_bspm.py:195-219): stop when the
// 0.99 quantile of |z| over the rows, linearly interpolated between order
// statistics as torch.quantile does, is below tol.  With N rows, position
// pos = 0.99 (N - 1), lo = floor(pos), and c rows at or above tol (their
// order statistics start at N - c), the quantile is below tol when lo + 1 <
// N - c, not below when lo >= N - c, and otherwise (lo = N - c - 1) equals
// m_lt + (pos - lo) (m_ge - m_lt) with m_lt the largest |z| below tol and
// m_ge the smallest at or above it: three reductions decide it exactly.
// The reported statistic is that value in the last case and otherwise
// m_lt (an upper bound of the quantile, below tol) or m_ge (a lower bound,
// not below tol).
template <int MODE, bool PAIRS, bool P99>
__global__ void __launch_bounds__(32 * PCG_WARPS, 1) pcg_resident(TorsoArgs a, PcgArgs c) {
  extern __shared__ __align__(16) unsigned char pcg_smem[];
  if (a.iscal[IS_DONE]) return;
  unsigned long long epoch = *(volatile unsigned long long*)c.sync.epoch;
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = blockIdx.x * PCG_WARPS + (tid >> 5), n_warps = gridDim.x * PCG_WARPS;
  __shared__ float s_t[HP_MAX_MATERIALS], s_inv[HP_MAX_MATERIALS];
  if (tid < HP_MAX_MATERIALS) {
    s_t[tid] = c.tu[tid];
    s_inv[tid] = c.inv[tid];
  }
  // shared memory: the vectors of `room` pairs, then this block's lines (the
  // warp's j-th line is line warp + j n_warps)
  const size_t room = c.room;
  PcgLine* sl = (PcgLine*)(pcg_smem + room * pcg_pair_bytes(MODE)) + (tid >> 5);
  const int nl = warp < c.n_lines ? (c.n_lines - 1 - warp) / n_warps + 1 : 0;
  if (MODE != PCG_MEM && lane == 0)
    for (int j = 0; j < nl; ++j) sl[j * PCG_WARPS] = c.line[warp + j * n_warps];
  __syncwarp();
  auto line = [&](int j) {
    return MODE == PCG_MEM ? c.line[warp + j * n_warps] : sl[j * PCG_WARPS];
  };
  // a line's vectors: [pair] of x, r, A p and meta
  auto xs = [&](const PcgLine& L) {
    return MODE == PCG_ALL ? (double2*)pcg_smem + L.s2 : c.x + L.c2;
  };
  auto rs = [&](const PcgLine& L) {
    return MODE == PCG_ALL ? (float2*)(pcg_smem + 16 * room) + L.s2
           : MODE == PCG_R ? (float2*)pcg_smem + L.s2
                           : c.r + L.c2;
  };
  auto As = [&](const PcgLine& L) {
    return MODE == PCG_ALL ? (float2*)(pcg_smem + 24 * room) + L.s2 : c.Ap + L.c2;
  };
  auto ms = [&](const PcgLine& L) {
    return MODE == PCG_ALL ? (const uint32_t*)(pcg_smem + 32 * room) + L.s2
                           : c.meta + L.c2;
  };
  auto inverse = [&](uint32_t m) {
    if (m & PQ_MIXED) return c.mixed[6 * (int64_t)c.n_mixed + (m & ~PQ_MIXED)];
    return make_float2(s_inv[m], s_inv[m]);
  };
  // the padded-grid cell of a line's first pair
  auto grid_cell = [&](const PcgLine& L) {
    return (int64_t)(L.p2 / c.sj) * a.pk + 2 * (L.p2 % c.sj);
  };
  for (int j = 0; j < nl; ++j) {
    const PcgLine L = line(j);
    const int64_t g = grid_cell(L);
    double* x = (double*)xs(L);
    float* r = (float*)rs(L);
    for (int k = lane; k < 2 * L.n2; k += 32) {
      const bool in = k >= L.first && k < L.first + L.len;
      r[k] = in ? a.r[g + k] : 0.0f;
      x[k] = in ? a.x[g + k] : 0.0;
    }
    if (MODE == PCG_ALL)
      for (int q = lane; q < L.n2; q += 32) ((uint32_t*)ms(L))[q] = c.meta[L.c2 + q];
  }
  __syncthreads();

  const int rule = a.iscal[IS_RULE], maxit = a.iscal[IS_MAXIT];
  const double tol = a.scal[SC_TOL], bb = a.scal[SC_BB];
  const float tolf = (float)tol;
  double rz = a.scal[SC_RZ], beta = a.scal[SC_BETA], alpha_prev = 0.0, pAp = 0.0, alpha = 0.0;
  double stat = a.scal[SC_STAT], zz = 0.0, rr = 0.0, zmax = 0.0;
  int it = a.iscal[IS_ITER], breakdown = 0, nonfinite = 0;
  for (bool done = false; !done;) {
    // x += alpha p (the last iteration's step), p = D^-1 r + beta p.  A
    // recursion starts with beta = 0 and forgets p, which may hold what a
    // non-finite solve left (0 * NaN is NaN).
    const float betaf = (float)beta;
    const bool start = betaf == 0.0f;
    for (int j = 0; j < nl; ++j) {
      const PcgLine L = line(j);
      double2* x = xs(L);
      const float2* r = rs(L);
      const uint32_t* m = ms(L);
      float2* p = c.p + L.p2;
#pragma unroll 2
      for (int q = lane; q < L.n2; q += 32) {
        const float2 rq = r[q], inv = inverse(m[q]);
        float2 pq = p[q];
        if (alpha_prev != 0.0) {
          double2 u = x[q];
          u.x += alpha_prev * (double)pq.x;
          u.y += alpha_prev * (double)pq.y;
          x[q] = u;
        }
        if (start) pq = make_float2(0.0f, 0.0f);
        pq.x = __fmaf_rn(betaf, pq.x, __fmul_rn(inv.x, rq.x));
        pq.y = __fmaf_rn(betaf, pq.y, __fmul_rn(inv.y, rq.y));
        p[q] = pq;
      }
    }
    alpha_prev = 0.0;
    if (!grid_sync(c.sync, epoch)) return;
    // A p and p.Ap
    double s1[1] = {0.0};
    for (int j = 0; j < nl; ++j) {
      const PcgLine L = line(j);
      float2* Ap = As(L);
      const uint32_t* m = ms(L);
      const float2* p = c.p + L.p2;
      if constexpr (PAIRS) {
        for (int q = lane; q < L.n2; q += 32) {
          const float2 pc = p[q], ip = p[q + (int64_t)c.si], im = p[q - (int64_t)c.si];
          const float2 jp = p[q + (int64_t)c.sj], jm = p[q - (int64_t)c.sj];
          const float km = ((const float*)p)[2 * q - 1], kp = ((const float*)p)[2 * q + 2];
          const uint32_t mq = m[q];
          const float pv[2] = {pc.x, pc.y};
          const float nb[6][2] = {{ip.x, ip.y}, {im.x, im.y}, {jp.x, jp.y},
                                  {jm.x, jm.y}, {pc.y, kp},   {km, pc.x}};
          float ap[2] = {0.0f, 0.0f};
          if (mq & PQ_MIXED) {
            const float2* W = c.mixed + (mq & ~PQ_MIXED);
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
          s1[0] += (double)pv[0] * (double)ap[0];
          s1[0] += (double)pv[1] * (double)ap[1];
        }
      } else {
        const float* p1 = (const float*)p;
        const int64_t sj = 2 * (int64_t)c.sj, si = 2 * (int64_t)c.si;
        for (int k = L.first + lane; k < L.first + L.len; k += 32) {
          const float pc = p1[k];
          const float nb[6] = {p1[k + si], p1[k - si], p1[k + sj], p1[k - sj], p1[k + 1], p1[k - 1]};
          const uint32_t mq = m[k >> 1];
          float ap = 0.0f;
          if (mq & PQ_MIXED) {
            const float* W = (const float*)(c.mixed + (mq & ~PQ_MIXED)) + (k & 1);
#pragma unroll
            for (int f = 0; f < 6; ++f)
              ap = __fmaf_rn(W[2 * f * (int64_t)c.n_mixed], __fsub_rn(pc, nb[f]), ap);
          } else {
            const float w = s_t[mq];
#pragma unroll
            for (int f = 0; f < 6; ++f) ap = __fmaf_rn(w, __fsub_rn(pc, nb[f]), ap);
          }
          ((float*)Ap)[k] = ap;
          s1[0] += (double)pc * (double)ap;
        }
      }
    }
    if (!grid_all<1, 0u>(c, epoch, s1)) return;
    pAp = s1[0];
    if (!(fabs(pAp) >= 1e-30) || !isfinite(pAp)) {  // breakdown, as the reference's |pAp| < 1e-30
      breakdown = isfinite(pAp) ? 1 : 0;
      nonfinite = isfinite(pAp) ? 0 : 1;
      alpha = 0.0;
      break;
    }
    alpha = rz / pAp;
    // r -= alpha A p; r.z, z.z, r.r and max |z|; P99: r.z, count |z| >= tol,
    // max of |z| below tol, max of -|z| at or above tol
    const float alphaf = (float)alpha;
    double v[4] = {0.0, 0.0, P99 ? -INFINITY : 0.0, -INFINITY};
    float m2 = -INFINITY, m3 = -INFINITY;
    for (int j = 0; j < nl; ++j) {
      const PcgLine L = line(j);
      float* r = (float*)rs(L);
      const float* Ap = (const float*)As(L);
      const uint32_t* m = ms(L);
#pragma unroll 2
      for (int k = L.first + lane; k < L.first + L.len; k += 32) {
        const uint32_t mq = m[k >> 1];
        const float inv = (mq & PQ_MIXED)
                              ? ((const float*)(c.mixed + 6 * (int64_t)c.n_mixed + (mq & ~PQ_MIXED)))[k & 1]
                              : s_inv[mq];
        const float re = __fmaf_rn(-alphaf, Ap[k], r[k]);
        r[k] = re;
        const float z = __fmul_rn(inv, re);
        v[0] += (double)re * (double)z;
        if constexpr (P99) {
          const float az = fabsf(z);
          if (az >= tolf) {
            v[1] += 1.0;
            m3 = fmaxf(m3, -az);
          } else {
            m2 = fmaxf(m2, az);
          }
        } else {
          v[1] += (double)z * (double)z;
          v[2] += (double)re * (double)re;
          m3 = fmaxf(m3, fabsf(z));
        }
      }
    }
    if (P99) v[2] = m2;
    v[3] = m3;
    if (!grid_all<4, P99 ? 12u : 8u>(c, epoch, v)) return;
    beta = v[0] / rz;
    rz = v[0];
    alpha_prev = alpha;
    ++it;
    bool below;
    if constexpr (P99) {
      const double N = (double)a.n_rows, m_lt = v[2], m_ge = -v[3];
      const double pos = 0.99 * (N - 1.0), lo = floor(pos);
      const double first_ge = N - v[1];
      if (lo + 1.0 < first_ge) {
        stat = m_lt;
        below = true;
      } else if (lo >= first_ge) {
        stat = m_ge;
        below = false;
      } else {
        stat = m_lt + (pos - lo) * (m_ge - m_lt);
        below = stat < tol;
      }
    } else {
      zz = v[1];
      rr = v[2];
      zmax = v[3];
      if (rule == HP_STOP_RMS) stat = sqrt(zz / (double)a.n_rows);
      else if (rule == HP_STOP_LINF) stat = zmax;
      else stat = sqrt(rr / fmax(bb, 1e-300));  // recursive estimate
      // REL: stop the recursion a little below tol; the true residual decides
      below = stat < (rule == HP_STOP_REL ? 0.5 * tol : tol);
    }
    if (!isfinite(rz)) {
      nonfinite = 1;
      done = true;
    } else if (below || it >= maxit) {
      done = true;
    }
  }
  // the last step's x, and the vectors back to the padded grid
  for (int j = 0; j < nl; ++j) {
    const PcgLine L = line(j);
    const int64_t g = grid_cell(L);
    const double* x = (const double*)xs(L);
    const float* r = (const float*)rs(L);
    const float* p = (const float*)(c.p + L.p2);
    for (int k = L.first + lane; k < L.first + L.len; k += 32) {
      a.r[g + k] = r[k];
      a.x[g + k] = alpha_prev != 0.0 ? x[k] + alpha_prev * (double)p[k] : x[k];
    }
  }
  if (grid_last_out(c.sync, epoch)) {
    a.scal[SC_RZ] = rz;
    a.scal[SC_PAP] = pAp;
    a.scal[SC_ALPHA] = alpha;
    a.scal[SC_BETA] = beta;
    a.scal[SC_STAT] = stat;
    if (!P99) {
      a.scal[SC_ZZ] = zz;
      a.scal[SC_RR] = rr;
      a.scal[SC_ZMAX] = zmax;
    }
    a.iscal[IS_ITER] = it;
    a.iscal[IS_BREAKDOWN] = breakdown;
    a.iscal[IS_NONFINITE] = nonfinite;
    a.iscal[IS_DONE] = 1;
  }
}

}  // namespace hp
