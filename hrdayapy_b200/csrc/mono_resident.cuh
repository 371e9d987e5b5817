// Resident monodomain steps: many time steps per launch, for hearts whose
// cells all fit on the chip at one thread per cell.
//
// The split step costs two launches per time step and the theta-scheme four
// more per CG iteration; on a heart of a few ten thousand cells these are
// bound by launch and ramp latency, not by work.  Here one cooperative launch
// (every block resident) advances n steps.  A thread owns one tissue cell of
// the compact list, or one Purkinje node, for the whole launch: its 18 TTP06
// states, its potential and its CG entries stay in registers, its operator
// row (neighbour slots and coefficients) in shared memory.  Only what
// neighbours read -- W, and in the theta-scheme r, q and p -- goes through
// L2, with a grid barrier between writing and reading it: one per explicit
// step, one per CG iteration.
//
// The arithmetic per cell is the split step's in the same order, so the
// explicit step is bit-identical to it.  What bounds it: an explicit step of a
// small heart is one chain of L2 round trips (neighbours 0.5 us, barrier
// 0.9 us) and the TTP06 update's own latency, about 3 us; from about 40,000
// cells on it is the update's issue and special-function rate.  A CG iteration
// (4.6 us) is the neighbour loads, a block sum, the barrier and the partials'
// round trip in turn; at 12,473 cells and 35 iterations a step the whole step
// went from 730 to 160 us.
#pragma once
#include "grid_sync.cuh"

namespace hp {

struct ResArgs {
  const int32_t* idx;       // NQ x n_active: neighbour slot, -1 no term, -2 a term that reads 0
  const float* coef;        // NQ x n_active (19-point operator): the term's coefficient
  GridSync sync;
  double* part;               // 2 x RES_MAX_BLOCKS rows of 8 partial sums
  float4* cg;               // theta: {r, q, p, D^-1} by iteration parity, 2 x cg_n
  int64_t cg_n;             // ([slots | Purkinje])
};
constexpr int RES_MAX_BLOCKS = 160;
constexpr int RES_BATCH = 20;  // partials in flight a thread: all of them from 64 threads on
// threads a block: register budgets (res_kernel) and the most there may be
constexpr int RES_SMALL_THREADS = 256;
constexpr int RES_MID_THREADS = 448;
constexpr int RES_MAX_THREADS = 640;
// shorter explicit runs take the split kernels: a launch reads 144 bytes of
// operator row per cell before its first step
constexpr int RES_MIN_STEPS = 4;

template <bool ANISO>
struct ResGeom {
  static constexpr int NQ = ANISO ? 18 : 6;
};

// Operator rows of the compact tissue cells (once per handle): the face
// terms, then the edge terms, in stencil_sum's order and rounding.  A term
// whose neighbour brick is absent reads 0, as the staged tiles do.
__global__ void resident_rows_kernel(MonoArgs a, int bi, int bj, int bk, int nq,
                                     int32_t* __restrict__ idx, float* __restrict__ coef) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.n_active) return;
  const int off[18][3] = {{1, 0, 0},  {-1, 0, 0},  {0, 1, 0},  {0, -1, 0}, {0, 0, 1},  {0, 0, -1},
                          {1, 1, 0},  {-1, -1, 0}, {1, -1, 0}, {-1, 1, 0}, {1, 0, 1},  {-1, 0, -1},
                          {1, 0, -1}, {-1, 0, 1},  {0, 1, 1},  {0, -1, -1}, {0, 1, -1}, {0, -1, 1}};
  const int slot = a.active_slot[i], bv = bi * bj * bk;
  const int b = slot / bv, loc = slot % bv;
  const int l[3] = {loc / (bj * bk), (loc / bk) % bj, loc % bk}, d[3] = {bi, bj, bk};
  const uint32_t tag = a.tag[slot];
  for (int q = 0; q < nq; ++q) {
    int32_t s = -1;
    float c = 0.0f;
    if (tag & (1u << (q < 6 ? HP_TAG_FACE_SHIFT + q : HP_TAG_DIAG_SHIFT + q - 6))) {
      int dir = 0, pos = 0;
      for (int x = 0; x < 3; ++x) {
        int v = l[x] + off[q][x];
        const int step = v < 0 ? -1 : (v >= d[x] ? 1 : 0);
        v -= step * d[x];
        dir = 3 * dir + step + 1;
        pos = pos * d[x] + v;
      }
      const int nb = a.nbr[(int64_t)b * 27 + dir];
      s = nb < 0 ? -2 : nb * bv + pos;
      if (nq > 6 && q < 6) {
        const int64_t at = (q & 1) ? s : slot;  // weights live on the lower voxel of a face
        c = at < 0 ? 0.0f : a.wface[(q >> 1) * a.n_slots + at];
      } else if (nq > 6) {
        const float* D = a.doff + ((q - 6) >> 2) * a.n_slots;
        c = __fmul_rn(((q - 6) & 2) ? -0.25f : 0.25f,
                      __fadd_rn(D[slot], s < 0 ? 0.0f : D[s]));
      }
    }
    idx[(int64_t)q * a.n_active + i] = s;
    if (coef) coef[(int64_t)q * a.n_active + i] = c;
  }
}

// FP64 sums over all threads of the launch, in a barrier; every block adds
// the blocks' sums in the same order, so all hold the same totals.  The
// partials alternate between two sets: a block writes set e + 2 only after
// every block has arrived at e + 1, i.e. has read e.  About 2 us.
//
// Sums run over eight values at a time: a warp halves the values a lane holds
// at each of three exchanges (9 exchanges for 8 values instead of 40), after
// which lane 4 k holds value k; the blocks' partials lie as rows of eight, so
// that all threads of a block read them side by side.
__device__ __forceinline__ double warp_sum8(double (&v)[8]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int h = 4, o = 16; h >= 1; h >>= 1, o >>= 1) {
    const bool up = lane & o;
    double give[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (k < h) give[k] = up ? v[k] : v[k + h];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (k < h) give[k] = __shfl_xor_sync(0xffffffffu, give[k], o);
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (k < h) v[k] = (up ? v[k + h] : v[k]) + give[k];
  }
  double t = v[0];
  t += __shfl_xor_sync(0xffffffffu, t, 2);
  t += __shfl_xor_sync(0xffffffffu, t, 1);
  return t;
}

// v (any number of values up to eight, the rest zero) becomes the totals.
__device__ __forceinline__ bool grid_sum8(const ResArgs& r, unsigned long long& epoch,
                                        double (&v)[8]) {
  __shared__ double sh[32][8];
  __shared__ double tot[8];
  __shared__ int s_ok;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nw = blockDim.x >> 5;
  const int G = gridDim.x;
  double* part = r.part + (++epoch & 1) * (int64_t)RES_MAX_BLOCKS * 8;
  const double t = warp_sum8(v);
  if ((lane & 3) == 0) sh[wid][lane >> 2] = t;
  __syncthreads();
  if (tid < 32) {
    // lane: value lane / 4, every fourth warp; then the four quarters
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < 32; w += 4)
      if (w + (lane & 3) < nw) s += sh[w + (lane & 3)][lane >> 2];
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    if ((lane & 3) == 0) part[blockIdx.x * 8 + (lane >> 2)] = s;
    __syncwarp();
    if (lane == 0) s_ok = grid_arrive_wait(r.sync, epoch);
  }
  __syncthreads();
  // the totals, in the same order in every block: thread t adds value t % 8
  // of every (threads / 8)-th block, then the threads' sums are added
  double s = 0.0;
  const int rows = blockDim.x >> 3;
  for (int b = tid >> 3; b < G; b += RES_BATCH * rows) {
    double w[RES_BATCH];
#pragma unroll
    for (int u = 0; u < RES_BATCH; ++u)
      w[u] = b + u * rows < G ? __ldcg(part + (b + u * rows) * 8 + (tid & 7)) : 0.0;
#pragma unroll
    for (int u = 0; u < RES_BATCH; ++u) s += w[u];
  }
  s += __shfl_xor_sync(0xffffffffu, s, 16);
  s += __shfl_xor_sync(0xffffffffu, s, 8);
  if (lane < 8) sh[wid][lane] = s;
  __syncthreads();
  if (tid < 32) {
    double q = 0.0;
#pragma unroll
    for (int w = 0; w < 32; w += 4)
      if (w + (lane & 3) < nw) q += sh[w + (lane & 3)][lane >> 2];
    q += __shfl_xor_sync(0xffffffffu, q, 2);
    q += __shfl_xor_sync(0xffffffffu, q, 1);
    if ((lane & 3) == 0) tot[lane >> 2] = q;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 8; ++k) v[k] = tot[k];
  return s_ok;
}

// The terms of one operator row: a field's values at its NQ neighbours,
// loaded unconditionally (a missing term holds the cell's own slot) so that
// all loads are in flight at once.
template <int NQ>
__device__ __forceinline__ void row_load(const float* f, const int32_t* sidx, int ld,
                                         float (&v)[NQ]) {
#pragma unroll
  for (int q = 0; q < NQ; ++q) v[q] = __ldcg(f + sidx[q * ld]);
}

// Operator row on the values v, own value Vc, in stencil_sum's order and
// rounding.  have: the row's terms; zero: those that read 0.
template <bool ANISO, int NQ>
__device__ __forceinline__ float row_sum(const MonoArgs& a, const float* scoef, int ld,
                                         uint32_t have, uint32_t zero, float Vc,
                                         const float (&v)[NQ]) {
  float acc = 0.0f;
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    const float d = __fsub_rn((zero & (1u << q)) ? 0.0f : v[q], Vc);
    const float c = ANISO ? scoef[q * ld] : 0.0f;
    if (have & (1u << q)) acc = ANISO ? __fmaf_rn(c, d, acc) : __fadd_rn(acc, d);
  }
  return ANISO ? acc : __fmul_rn(a.iso_coef, acc);
}

// Row sum of a Purkinje node whose first NQ entries sit in shared memory:
// purkinje_row's order and rounding, the loads of a batch issued together.
template <int NQ, class VAL>
__device__ __forceinline__ float resident_pk_row(const MonoArgs& a, const int32_t* sidx,
                                                 const float* scoef, int ld, int q0, int q1,
                                                 float Vc, VAL&& val) {
  const int n = q1 - q0;
  float acc = 0.0f;
  constexpr int B = NQ < 6 ? NQ : 6;
#pragma unroll
  for (int b = 0; b < NQ; b += B) {
    if (b >= n) break;
    float v[B];
#pragma unroll
    for (int u = 0; u < B; ++u) v[u] = b + u < n ? val(sidx[(b + u) * ld]) : 0.0f;
#pragma unroll
    for (int u = 0; u < B; ++u)
      if (b + u < n) acc += scoef[(b + u) * ld] * (v[u] - Vc);
  }
  for (int q = q0 + NQ; q < q1; ++q) acc += a.pk_coef[q] * (val(a.pk_idx[q]) - Vc);
  return acc;
}

// n steps from the state the split step leaves (W_step in its buffer, Vpost,
// compact states) to the same state n steps later.
template <bool ANISO, bool THETA, int MAXT>
__global__ void __launch_bounds__(MAXT, 1)
mono_resident_kernel(MonoArgs a, CnArgs cn, ResArgs rs, int n) {
  constexpr int NQ = ResGeom<ANISO>::NQ;
  extern __shared__ __align__(16) float smem[];
  const int ld = blockDim.x;
  int32_t* sidx = (int32_t*)smem + threadIdx.x;  // NQ x ld
  float* scoef = smem + NQ * ld + threadIdx.x;   // NQ x ld
  float* sstate = scoef + NQ * ld;               // theta: N_STATE x ld
  const int64_t step0 = *a.d_step;
  unsigned long long epoch = *(volatile unsigned long long*)rs.sync.epoch;

  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool tissue = i < a.n_active;
  const int p = i - a.n_active_pad;
  const bool pk = p >= 0 && p < a.n_pk;
  int slot = 0, var = 0;
  uint32_t tag = 0, have = 0, zero = 0;  // have, zero: see row_sum
  CellState cs;
#pragma unroll
  for (int v = 0; v < N_STATE; ++v) cs.v[v] = 0.0f;
  float V = 0.0f, W = 0.0f;
  float dinv = 0.0f;
  // the cell's range of junction entries (tissue; its first entry is kept) or
  // its whole row (Purkinje; the first NQ entries are kept in shared memory)
  int q0 = 0, q1 = 0, j0 = 0;
  float c0 = 0.0f;
  if (tissue) {
    slot = a.active_slot[i];
    tag = a.tag[slot];
    var = a.brick_variant ? a.brick_variant[slot >> a.bv_shift] : 0;
#pragma unroll
    for (int v = 0; v < N_STATE; ++v) cs.v[v] = a.state[(int64_t)v * a.n_active + i];
    V = a.Vpost[slot];
    W = ((step0 & 1) ? a.Vs1 : a.Vs0)[slot];
    if constexpr (THETA) dinv = cn.dinv[slot];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int32_t s = rs.idx[(int64_t)q * a.n_active + i];
      sidx[q * ld] = s >= 0 ? s : slot;
      have |= s != -1 ? 1u << q : 0u;
      zero |= s == -2 ? 1u << q : 0u;
      if constexpr (ANISO) scoef[q * ld] = rs.coef[(int64_t)q * a.n_active + i];
    }
    if (tag & HP_TAG_PMJ) {
      const int r = a.pmj_row[slot];
      q0 = a.pmj_ptr[r];
      q1 = a.pmj_ptr[r + 1];
      if (q0 < q1) {
        j0 = a.pmj_pk[q0];
        c0 = a.pmj_coef[q0];
      }
    }
  } else if (pk) {
    var = a.pk_variant ? a.pk_variant[p] : 0;
    tag = 1u | ((uint32_t)a.pk_stim[p] << HP_TAG_STIM_SHIFT);  // Purkinje cells are endocardial
#pragma unroll
    for (int v = 0; v < N_STATE; ++v) cs.v[v] = a.pk_state[(int64_t)v * a.n_pk + p];
    V = a.pk_Vpost[p];
    W = ((step0 & 1) ? a.pk_Vs1 : a.pk_Vs0)[p];
    if constexpr (THETA) dinv = cn.dinv[a.n_slots + p];
    q0 = a.pk_ptr[p];
    q1 = a.pk_ptr[p + 1];
    for (int q = 0; q < NQ && q0 + q < q1; ++q) {
      sidx[q * ld] = a.pk_idx[q0 + q];
      scoef[q * ld] = a.pk_coef[q0 + q];
    }
  }
  const CellParams cp = pheno_params(tag & HP_TAG_PHENO_MASK, a.var_gks[var], a.var_gkr[var]);
  const uint8_t* on_tab = a.site_on + var * a.site_stride;
  // steps to the next snapshot / animation frame and its index
  int64_t vm_frame = 0, anim_frame = 0, vm_left = -1, anim_left = -1;
  if (a.vm_every > 0) {
    vm_frame = (step0 + a.vm_every - 1) / a.vm_every;
    vm_left = vm_frame * a.vm_every - step0;
  }
  if (a.frame_every > 0) {
    anim_frame = (step0 + a.frame_every - 1) / a.frame_every;
    anim_left = anim_frame * a.frame_every - step0;
  }
  int total = 0, unconv = 0, breaks = 0;
  // junction currents of a tissue cell, the first entry's value given
  auto junctions = [&](float acc, float Vc, float first, auto&& get) {
    if (q0 < q1) acc = __fmaf_rn(c0, __fsub_rn(first, Vc), acc);
    for (int q = q0 + 1; q < q1; ++q)
      acc = __fmaf_rn(a.pmj_coef[q], __fsub_rn(get(a.pmj_pk[q]), Vc), acc);
    return acc;
  };

  for (int it = 0; it < n; ++it) {
    const int64_t step = step0 + it;
    const bool odd = step & 1;
    const float* Win = odd ? a.Vs1 : a.Vs0;
    const float* Wpk = odd ? a.pk_Vs1 : a.pk_Vs0;
    float* Wout = odd ? a.Vs0 : a.Vs1;
    float* Wpk_out = odd ? a.pk_Vs0 : a.pk_Vs1;
    const uint32_t on = on_tab[step + 1];
    // the operator on W_step
    float acc = 0.0f;
    if (tissue) {
      const float first = q0 < q1 ? __ldcg(Wpk + j0) : 0.0f;
      float v[NQ];
      row_load<NQ>(Win, sidx, ld, v);
      acc = row_sum<ANISO, NQ>(a, scoef, ld, have, zero, W, v);
      acc = junctions(acc, W, first, [&](int j) { return __ldcg(Wpk + j); });
    } else if (pk) {
      acc = resident_pk_row<NQ>(a, sidx, scoef, ld, q0, q1, W, [&](int j) {
        return j >= 0 ? __ldcg(Wpk + j) : __ldcg(Win + (-j - 1));
      });
    }
    float Vn;
    if constexpr (!THETA) {
      Vn = fminf(fmaxf(__fadd_rn(W, acc), -150.0f), 80.0f);
    } else {
      // Jacobi-CG from x = W, r = Lh W (see diffuse_pass), one barrier per
      // iteration: <p, q>_w, ||r||^2 and <r, z>_w are summed together with
      // <r, q>, <q, q>, <r, D^-1 q>_w and <q, D^-1 q>_w, which predict the
      // norms of the next residual r - alpha q, hence beta and the stopping
      // test.  The sums are taken afresh from the residual in every iteration,
      // since a carried prediction would keep the first iterations' rounding.
      // A neighbour's
      // next direction is formed from its published r, q and p as its owner
      // forms it: r - alpha q, then D^-1 r + beta p.
      const int64_t e = tissue ? slot : a.n_slots + p;
      const float wgt = pk ? cn.pk_weight : 1.0f;
      float x = W, r = acc, pd = 0.0f, qd = 0.0f;
      // the 18 states wait in shared memory: the row's loads need the registers
#pragma unroll
      for (int v = 0; v < N_STATE; ++v) sstate[v * ld] = cs.v[v];
      double sm[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
      if (tissue || pk) {
        const float b = W + cn.omt * acc;
        rs.cg[rs.cg_n + e] = make_float4(r, 0.0f, 0.0f, dinv);  // the parity "before iteration 0"
        sm[0] = (double)b * b;
        sm[1] = (double)acc * acc;
      }
      if (!grid_sum8(rs, epoch, sm)) return;
      const double bb = sm[0];
      float alpha = 0.0f, beta = 0.0f;
      bool done = sm[1] <= cn.tol2 * bb || bb == 0.0;
      for (int k = 0; !done; ++k) {
        const float4* old = rs.cg + ((k & 1) ? 0 : rs.cg_n);  // of iteration k - 1
        float4* mine = rs.cg + ((k & 1) ? rs.cg_n : 0);
        auto dir = [&](int64_t j) {
          const float4 t = __ldcg(old + j);
          return __fmaf_rn(beta, t.z, __fmul_rn(t.w, __fmaf_rn(-alpha, t.y, t.x)));
        };
#pragma unroll
        for (int u = 0; u < 8; ++u) sm[u] = 0.0;
        if (tissue || pk) {
          pd = __fmaf_rn(beta, pd, __fmul_rn(dinv, r));
          float ac;
          if (tissue) {
            const float first = q0 < q1 ? dir(a.n_slots + j0) : 0.0f;
            float4 t[NQ];
#pragma unroll
            for (int q = 0; q < NQ; ++q) t[q] = __ldcg(old + sidx[q * ld]);
            float v[NQ];
#pragma unroll
            for (int q = 0; q < NQ; ++q)
              v[q] = __fmaf_rn(beta, t[q].z, __fmul_rn(t[q].w, __fmaf_rn(-alpha, t[q].y, t[q].x)));
            ac = row_sum<ANISO, NQ>(a, scoef, ld, have, zero, pd, v);
            ac = junctions(ac, pd, first, [&](int j) { return dir(a.n_slots + j); });
          } else {
            ac = resident_pk_row<NQ>(a, sidx, scoef, ld, q0, q1, pd, [&](int j) {
              return dir(j >= 0 ? a.n_slots + j : (int64_t)(-j - 1));
            });
          }
          qd = pd - cn.theta * ac;
          mine[e] = make_float4(r, qd, pd, dinv);
          const double wd = (double)wgt * dinv;
          sm[0] = (double)wgt * pd * qd;
          sm[1] = (double)r * r;
          sm[2] = (double)r * qd;
          sm[3] = (double)qd * qd;
          sm[4] = wd * sm[1];
          sm[5] = wd * sm[2];
          sm[6] = wd * sm[3];
        }
        if (!grid_sum8(rs, epoch, sm)) return;
        const double pq = sm[0], rz = sm[4];
        if (!(pq > 0.0) || !isfinite(pq)) {  // breakdown: keep the current x
          ++breaks;
          break;
        }
        alpha = (float)(rz / pq);
        x = x + alpha * pd;
        r = __fmaf_rn(-alpha, qd, r);
        const double al = alpha;
        const double rz_new = rz + al * (al * sm[6] - 2.0 * sm[5]);
        const double rr = sm[1] + al * (al * sm[3] - 2.0 * sm[2]);
        ++total;
        beta = (float)(rz > 0.0 ? rz_new / rz : 0.0);
        if (rr <= cn.tol2 * bb) {
          done = true;
        } else if (k + 1 >= cn.max_iter || !isfinite(rr)) {
          ++unconv;
          done = true;
        }
      }
#pragma unroll
      for (int v = 0; v < N_STATE; ++v) cs.v[v] = sstate[v * ld];
      Vn = fminf(fmaxf(x, -150.0f), 80.0f);
    }
    const int64_t vf = vm_left == 0 ? vm_frame : -1, af = anim_left == 0 ? anim_frame : -1;
    if (tissue) {
      voxel_outputs(a, slot, tag, Vn, V, step, vf, af);
    } else if (pk) {
      a.pk_Vpost[p] = Vn;
      if (af >= 0) a.pk_frames[af * (int64_t)a.n_pk + p] = Vn;
    }
    if (a.vm_every > 0) {
      if (vm_left == 0) { ++vm_frame; vm_left = a.vm_every; }
      --vm_left;
    }
    if (a.frame_every > 0) {
      if (anim_left == 0) { ++anim_frame; anim_left = a.frame_every; }
      --anim_left;
    }
    V = Vn;
    if (tissue || pk) {
      const float Iion = ttp06_step(Vn, cs, a.dt, cp);
      const float Is = site_current(a, (tag >> HP_TAG_STIM_SHIFT) & on, var);
      W = Vn + a.dt_over_Cm * (-(Iion * a.Cm) + Is);
      if (tissue) Wout[slot] = W;
      else Wpk_out[p] = W;
    }
    if (it + 1 < n && !grid_sync(rs.sync, epoch)) return;
  }
  if (tissue) {
#pragma unroll
    for (int v = 0; v < N_STATE; ++v) a.state[(int64_t)v * a.n_active + i] = cs.v[v];
  } else if (pk) {
#pragma unroll
    for (int v = 0; v < N_STATE; ++v) a.pk_state[(int64_t)v * a.n_pk + p] = cs.v[v];
  }
  if (THETA && blockIdx.x == 0 && threadIdx.x == 0) {
    cn.iscal[CI_TOTAL] += total;
    cn.iscal[CI_SOLVES] += n;
    cn.iscal[CI_UNCONV] += unconv;
    cn.iscal[CI_BREAK] += breaks;
  }
  if (grid_last_out(rs.sync, epoch)) *(int64_t*)a.d_step = step0 + n;
}

}  // namespace hp
