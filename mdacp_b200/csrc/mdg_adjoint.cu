// Differentiable LJ trajectories: the gradient of a trajectory loss with
// respect to the potential's epsilon and sigma and to the initial positions,
// by a hand-written adjoint (reverse) sweep over the drift-kick-drift steps.
//
// Model (FP64 throughout):
//   U(r) = epsilon * phi(r / sigma), phi(s) = 4 (s^-12 - s^-6 + C2 s^2 + C0)
//   for s <= s_c, 0 beyond: the reference's smoothed potential
//   (Variables::Variables, src/variables.cc:16-33) with the cut-off s_c in
//   units of sigma, so U and U' vanish at the cut-off.
//   Step (MDManager::Calculate, NVE, src/mdmanager.cc:153-186):
//     q_h = q + v dt/2;  v' = v + F(q_h) dt;  q' = q_h + v' dt/2.
//   Loss: L = 1/(T N) sum_{t=1..T} [ PE(q_t) + S(q_t) ], PE the pair energy
//   and S = sum over pairs of g((r - a)/w) g((b - r)/w), a smoothed count of
//   the pairs in the shell a < r < b (g the logistic function).
//
// Reverse sweep, per step, from the adjoints (lq, lv) of (q', v'):
//   lq += dL/dq'          (the loss term of this step)
//   lv' = lv + lq dt/2
//   u = lv' dt;  lq_h = lq - H(q_h) u;  dL/dtheta += u . dF/dtheta
//   lv = lv';  lq = lq_h;  lv += lq_h dt/2
// H(q_h) u is the Hessian-vector product of the pair energy, assembled pair
// by pair: (H u)_i = sum_j K_ij (u_i - u_j), K = U'' d d^T + U'/r (I - d d^T)
// with d the unit separation.  Positions and velocities are checkpointed every
// k steps in the forward pass; each k-step segment is recomputed forward
// (keeping q_h and v') before its reverse sweep.
//
// Pairs come from a Verlet list of search length r_c + skin (r_c = s_c
// sigma; skin 0.3 sigma, less where the box is narrow).  The kernel that makes
// the positions of an evaluation also checks them against the list's build
// positions, and the evaluation's kernel rebuilds the list first when an atom
// has moved more than skin/2, which keeps every pair within r_c in the rows.
// A row is ordered by (hash of the partner, partner): eight buckets of the
// hash, which the lanes that share an atom divide among them, so that a lane's
// pairs within r_c and their order are a function of the positions alone,
// whichever build the row comes from.  This component has no counterpart in
// the reference, which has no gradients.
//
// A gradient of 32,000 atoms x 200 steps takes 31 ms, of 500 atoms x 50 steps
// 2.1 ms; with one kernel per operation (12 launches a step forward, 19 in
// reverse), a one-block cell grid (170 us a rebuild, 180 more for the rows; 133
// us in all here), roots and two divisions a pair and ballots to share out a
// row they took 86 and 8.9 ms.  Per pass at 32,000 atoms, four lanes an atom:
// force 15 us (37), loss with gradient 34 (51), Hessian 35 (47); of the 29 ms
// of kernels in that run 19.5 are 780 passes and 9.5 are 71 rebuilds.
//
// One launch per evaluation: a step is a force pass (kick and both drifts in
// its end), a loss pass (forward: the sums; reverse: the loss gradient and the
// first half of the reverse step) and, in reverse, a Hessian pass (and the
// second half).  The passes are cooperative launches because a rebuild inside
// one has grid barriers; without a rebuild no block waits for another.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <tuple>
#include <vector>

#include "mdacp_b200.h"
#include "mdg_device.cuh"

namespace {

constexpr int kAB = 128;        // threads per block
// Blocks an SM that the passes are held to: 72 registers, which the force and
// loss sums keep to; the loss with its gradient and the Hessian spill some 110
// and 150 bytes a thread.  Other caps have not been measured.
constexpr int kABlocks = 7;
constexpr int kBuckets = 8;     // hash buckets of a row
constexpr int kReduceSlots = 32;  // steps whose block partials are kept before they are summed

struct Pot {
  double rc2;                   // cut-off^2 (absolute)
  double c0, c2;                // smoothed-LJ constants in units of sigma
  double sigma2, inv_sigma, inv_sigma2, inv_eps;
  double e4;                    // 4 eps
  double k4;                    // 4 eps / sigma^2
  double a, b, inv_w;           // shell of the smoothed pair count
  double mid, h;                // (a + b) / 2, exp((a - b) / (2 w))
  int one_exp;                  // the shell's exponents stay in range for every r < r_c: one exp per pair
};

// n points: (x, y) pairs, then z.  24 bytes a gathered partner, spread over
// all bank columns of the L1 (a 32-byte point leaves half of them unused).
struct Vec {
  double *p;
  size_t ns;  // n rounded up to an even number
  __device__ __forceinline__ double3 at(int i) const {
    const double2 a = reinterpret_cast<const double2 *>(p)[i];
    return make_double3(a.x, a.y, p[2 * ns + i]);
  }
  __device__ __forceinline__ void set(int i, const double3 &x) const {
    reinterpret_cast<double2 *>(p)[i] = make_double2(x.x, x.y);
    p[2 * ns + i] = x.z;
  }
};

// A grid barrier's arrivals and generation (meet).
struct Meeting {
  unsigned count, gen;
};

// The cell grid and the Verlet list.  Row of atom i: nbr[i * maxnb + k], the
// end of bucket b at ends[i * kBuckets + b].
struct List {
  int ms[3], ncell, maxnb, n;
  double L[3], inv_L[3], inv_cs[3];
  // search length^2: enlarged by the rounding of box coordinates for an FP32
  // search; negative for an FP64 one (boxes too long for FP32)
  float Lf[3], inv_Lf[3], reach2;
  double half_skin2;
  int *count, *start, *cell, *rank, *cursor;  // cells: atoms, first place; atoms: cell, place in it
  float4 *sorted;                             // box coordinates and index in cell order
  int *nbr;
  unsigned short *ends;
  Vec qb;                                     // positions at the last build
  int *overflow, *timeout;
  Meeting *bar;
};

__device__ __forceinline__ double3 axpy(double h, const double3 &v, const double3 &q) {
  return make_double3(fma(v.x, h, q.x), fma(v.y, h, q.y), fma(v.z, h, q.z));
}
__device__ __forceinline__ double dist2(const double3 &a, const double3 &b) {
  const double x = a.x - b.x, y = a.y - b.y, z = a.z - b.z;
  return x * x + y * y + z * z;
}

// d - L rint(d / L): the rounding by adding and taking away 1.5 2^52, which
// leaves the nearest whole number for any |d / L| a trajectory reaches.
__device__ __forceinline__ double min_image(double d, double L, double inv_L) {
  const double big = 6755399441055744.0;
  const double k = fma(d, inv_L, big) - big;
  return fma(-L, k, d);
}

__device__ __forceinline__ int cell_axis(double x, double L, double inv_cs, int ms, float *boxed) {
  x -= L * floor(x / L);
  *boxed = (float)x;
  int c = (int)(x * inv_cs);
  return c < 0 ? 0 : (c >= ms ? ms - 1 : c);
}

__device__ __forceinline__ int bucket_of(int j) { return (int)(((unsigned)j * 0x9E3779B1u) >> 29); }

// ---------------------------------------------------------- Verlet list
// Every block of the (resident) grid arrives; false when the wait ran out.
__device__ __forceinline__ bool meet(const List &l) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    ok = 1;
    const unsigned gen = mdg::ld_acquire_gpu(&l.bar->gen);
    __threadfence();
    if (atomicAdd(&l.bar->count, 1u) + 1u == gridDim.x) {
      l.bar->count = 0u;
      __threadfence();
      atomicAdd(&l.bar->gen, 1u);
    } else {
      long long polls = 0;
      while (mdg::ld_acquire_gpu(&l.bar->gen) == gen) {
        if (++polls > mdg::kBarrierPolls) {
          atomicOr(l.timeout, 1);
          ok = 0;
          break;
        }
        __nanosleep(20);
      }
    }
  }
  __syncthreads();
  return ok != 0;
}

// Ascending sort of a warp's 128 values, v[e] = element e * 32 + lane (bitonic
// network).
__device__ __forceinline__ void warp_sort(unsigned (&v)[4], int lane) {
#pragma unroll
  for (int k = 2; k <= 128; k <<= 1) {
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
      if (j >= 32) {  // partner in the same lane
#pragma unroll
        for (int e = 0; e < 4; e++) {
          const int f = e ^ (j / 32);
          if (f > e) {
            const bool up = ((e * 32) & k) == 0;
            const unsigned x = v[e], y = v[f];
            v[e] = up ? min(x, y) : max(x, y);
            v[f] = up ? max(x, y) : min(x, y);
          }
        }
      } else {  // partner in lane ^ j
#pragma unroll
        for (int e = 0; e < 4; e++) {
          const unsigned o = __shfl_xor_sync(0xffffffffu, v[e], j);
          const bool up = ((e * 32 + lane) & k) == 0, lower = (lane & j) == 0;
          v[e] = lower == up ? min(v[e], o) : max(v[e], o);
        }
      }
    }
  }
}

// Row of atom i by one warp: the atoms of the 27 cells around it within the
// search length (FP32 minimum image on box coordinates; the reach is enlarged
// by more than its rounding, and rows may hold more than they must; FP64 where
// that would be more than a hundredth of the search length), put in
// (bucket, index) order.  The cells of an x-row are consecutive in `sorted`:
// the 27 cells are 9 runs, and 9 more of one cell each where x wraps; the next
// 32 atoms' load is in flight while 32 are tested.  keys: maxnb words of shared
// memory.
template <bool EXACT>
__device__ __forceinline__ void build_row(const List &l, const Vec &x, int i, unsigned *keys) {
  const int lane = threadIdx.x & 31;
  const double3 q = x.at(i);
  float bx, by, bz;
  const int cx = cell_axis(q.x, l.L[0], l.inv_cs[0], l.ms[0], &bx);
  const int cy = cell_axis(q.y, l.L[1], l.inv_cs[1], l.ms[1], &by);
  const int cz = cell_axis(q.z, l.L[2], l.inv_cs[2], l.ms[2], &bz);
  if (lane == 0) l.qb.set(i, q);
  const bool wraps = cx == 0 || cx == l.ms[0] - 1;
  const int runs = wraps ? 18 : 9;
  int first = 0, len = 0;  // lane < runs: one of the runs
  if (lane < runs) {
    const int r = lane % 9;
    const int z = (cz + r / 3 - 1 + l.ms[2]) % l.ms[2], y = (cy + r % 3 - 1 + l.ms[1]) % l.ms[1];
    const int row = (z * l.ms[1] + y) * l.ms[0];
    int c0 = max(cx - 1, 0), c1 = min(cx + 1, l.ms[0] - 1);
    if (lane >= 9) c0 = c1 = cx == 0 ? l.ms[0] - 1 : 0;
    first = __ldcg(&l.start[row + c0]);
    len = __ldcg(&l.start[row + c1]) + __ldcg(&l.count[row + c1]) - first;
  }
  int run = -1, f = 0, left = 0;  // the atoms loaded next: left ones from f on
  auto next = [&]() {
    f += 32;
    left -= 32;
    while (left <= 0 && ++run < runs) {
      f = __shfl_sync(0xffffffffu, first, run);
      left = __shfl_sync(0xffffffffu, len, run);
    }
  };
  next();
  float4 pn = make_float4(0.f, 0.f, 0.f, 0.f);
  if (lane < left) pn = __ldcg(&l.sorted[f + lane]);
  int m = 0;
  while (run < runs) {
    const float4 p = pn;
    const bool in = lane < left;
    next();
    if (lane < left) pn = __ldcg(&l.sorted[f + lane]);
    const int j = __float_as_int(p.w);
    float dx = p.x - bx, dy = p.y - by, dz = p.z - bz;
    dx = fmaf(-l.Lf[0], rintf(dx * l.inv_Lf[0]), dx);
    dy = fmaf(-l.Lf[1], rintf(dy * l.inv_Lf[1]), dy);
    dz = fmaf(-l.Lf[2], rintf(dz * l.inv_Lf[2]), dz);
    bool keep = in && j != i && fmaf(dx, dx, fmaf(dy, dy, dz * dz)) <= l.reach2;
    if (EXACT) {
      const double3 o = x.at(j);
      const double ex = min_image(q.x - o.x, l.L[0], l.inv_L[0]), ey = min_image(q.y - o.y, l.L[1], l.inv_L[1]),
                   ez = min_image(q.z - o.z, l.L[2], l.inv_L[2]);
      keep = in && j != i && ex * ex + ey * ey + ez * ez <= -(double)l.reach2;
    }
    const unsigned bal = __ballot_sync(0xffffffffu, keep);
    const int at = m + __popc(bal & ((1u << lane) - 1u));
    if (keep && at < l.maxnb) keys[at] = ((unsigned)bucket_of(j) << 29) | (unsigned)j;
    m += __popc(bal);
  }
  if (m > l.maxnb && lane == 0) atomicOr(l.overflow, 1);
  m = min(m, l.maxnb);
  __syncwarp();
  int *row = l.nbr + (size_t)i * l.maxnb;
  // in parts of 128, sorted in registers; an entry of a longer row comes after
  // the smaller ones of every part (a binary search each)
  for (int part = 0; part < m; part += 128) {
    unsigned v[4];
#pragma unroll
    for (int e = 0; e < 4; e++) v[e] = part + e * 32 + lane < m ? keys[part + e * 32 + lane] : 0xffffffffu;
    warp_sort(v, lane);
#pragma unroll
    for (int e = 0; e < 4; e++)
      if (part + e * 32 + lane < m) {
        if (m <= 128) row[e * 32 + lane] = (int)(v[e] & 0x1fffffffu);
        else keys[part + e * 32 + lane] = v[e];
      }
  }
  if (m > 128) {
    __syncwarp();
    for (int e = lane; e < m; e += 32) {
      const unsigned key = keys[e];
      int r = e & 127;
      for (int part = 0; part < m; part += 128) {
        if (part == (e & ~127)) continue;
        int lo = part, hi = min(part + 128, m);  // the first key of the part above this one
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if (keys[mid] < key) lo = mid + 1;
          else hi = mid;
        }
        r += lo - part;
      }
      row[r] = (int)(key & 0x1fffffffu);
    }
  }
  // ends of the buckets: entries of each, and their running sum
  int mine = 0;
  for (int e = 0; e < m; e += 32) {
    const int bk = e + lane < m ? (int)(keys[e + lane] >> 29) : -1;
#pragma unroll
    for (int c = 0; c < kBuckets; c++) {
      const int k = __popc(__ballot_sync(0xffffffffu, bk == c));
      mine += lane >= c ? k : 0;
    }
  }
  if (lane < kBuckets) l.ends[(size_t)i * kBuckets + lane] = (unsigned short)mine;
  __syncwarp();
}

// The list at x, by the whole grid; false when a barrier's wait ran out.
// x-rows of cells get their places in the order in which they ask for them:
// the list does not depend on it.
__device__ __noinline__ bool rebuild(const List &l, const Vec &x, unsigned *smem) {
  if (*(volatile const int *)l.timeout) return false;  // an earlier launch gave up: the run has failed
  const int t = blockIdx.x * kAB + threadIdx.x, nt = gridDim.x * kAB;
  for (int c = t; c < l.ncell; c += nt) l.count[c] = 0;
  if (t == 0) *l.cursor = 0;
  if (!meet(l)) return false;
  for (int i = t; i < l.n; i += nt) {
    const double3 q = x.at(i);
    float f;
    const int cx = cell_axis(q.x, l.L[0], l.inv_cs[0], l.ms[0], &f);
    const int cy = cell_axis(q.y, l.L[1], l.inv_cs[1], l.ms[1], &f);
    const int cz = cell_axis(q.z, l.L[2], l.inv_cs[2], l.ms[2], &f);
    const int c = (cz * l.ms[1] + cy) * l.ms[0] + cx;
    l.cell[i] = c;
    l.rank[i] = atomicAdd(&l.count[c], 1);
  }
  if (!meet(l)) return false;
  {  // a warp per x-row of cells: its place, and the running sum of its cells
    const int lane = threadIdx.x & 31, ms0 = l.ms[0], rows = l.ms[1] * l.ms[2];
    for (int r = t >> 5; r < rows; r += nt >> 5) {
      int total = 0;
      for (int c = lane; c < ms0; c += 32) total += __ldcg(&l.count[r * ms0 + c]);
      total = __reduce_add_sync(0xffffffffu, total);
      int at = 0;
      if (lane == 0) at = atomicAdd(l.cursor, total);
      at = __shfl_sync(0xffffffffu, at, 0);
      for (int c = 0; c < ms0; c += 32) {
        const int k = c + lane < ms0 ? __ldcg(&l.count[r * ms0 + c + lane]) : 0;
        int sum = k;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int v = __shfl_up_sync(0xffffffffu, sum, o);
          if (lane >= o) sum += v;
        }
        if (c + lane < ms0) l.start[r * ms0 + c + lane] = at + sum - k;
        at += __shfl_sync(0xffffffffu, sum, 31);
      }
    }
  }
  if (!meet(l)) return false;
  for (int i = t; i < l.n; i += nt) {  // the thread's own cell[i] and rank[i]
    const double3 q = x.at(i);
    float4 f;
    cell_axis(q.x, l.L[0], l.inv_cs[0], l.ms[0], &f.x);
    cell_axis(q.y, l.L[1], l.inv_cs[1], l.ms[1], &f.y);
    cell_axis(q.z, l.L[2], l.inv_cs[2], l.ms[2], &f.z);
    f.w = __int_as_float(i);
    l.sorted[__ldcg(&l.start[l.cell[i]]) + l.rank[i]] = f;
  }
  if (!meet(l)) return false;
  unsigned *keys = smem + (threadIdx.x >> 5) * l.maxnb;
  if (l.reach2 < 0.f)
    for (int i = t >> 5; i < l.n; i += nt >> 5) build_row<true>(l, x, i, keys);
  else
    for (int i = t >> 5; i < l.n; i += nt >> 5) build_row<false>(l, x, i, keys);
  return meet(l);
}

// ------------------------------------------------------------ evaluations
enum Kind { kForce, kLoss, kHess };

// One evaluation.  Kind kForce: F at x, then v' = v + F dt (into v_out), q' = x
// + v' dt/2 and the next step's x' = q' + v' dt/2; kLoss: block sums of PE, S
// and dPE/dsigma at x, with grad the loss gradient into lq and the first half
// of the reverse step (lv' = lv + lq dt/2, u = lv' dt); kHess: H(x) u, block
// sums of u . dF/d(eps, sigma), the second half (lq -= w, lv += lq dt/2), and
// the positions of the step before.
struct Eval {
  Vec x;
  const int *want;      // rebuild the list at x first
  int *move, *jump;     // flags of the next evaluation and of the one after it
  double dt;
  // kForce
  Vec v, v_out, q_out, x_out;  // q_out, x_out: p = null where not needed
  // kLoss, kHess
  Vec lq, lv, u;
  double scale;                // dL/d(sums); 0: sums only
  double *part;                // block sums of this step
  // kHess: the step before (x_prev.p = null: none); q_out gets its q'
  Vec x_prev, v_prev;
};

// Terms of the partners at d[0], d[1] (x_i - x_j, minimum image) into s.
template <Kind K, bool GRAD>
struct Terms {
  static constexpr int N = K == kForce ? 3 : (K == kLoss ? (GRAD ? 6 : 3) : 5);
};

template <Kind K, bool GRAD>
__device__ __forceinline__ void pair_terms(const Pot &p, const double3 (&d)[2], const bool (&on)[2],
                                           const double3 &ui, const double3 (&uj)[2],
                                           double (&s)[Terms<K, GRAD>::N]) {
  constexpr int N = Terms<K, GRAD>::N;
  double t[2][N];
  bool in[2];
#pragma unroll
  for (int e = 0; e < 2; e++) {
    const double3 &v = d[e];
    // products that sums follow are written out (fma or rounded), so that the
    // loss's sums do not depend on what else a pass computes
    double r2 = fma(v.x, v.x, fma(v.y, v.y, v.z * v.z));
    in[e] = on[e] && r2 < p.rc2;
    r2 = in[e] ? r2 : p.sigma2;
    // powers of sigma / r; U'/r and U'' need no root
    const double ir2 = mdg::quotient(1.0, r2);
    const double is2 = p.sigma2 * ir2, is6 = __dmul_rn(is2 * is2, is2);
    const double is8 = is6 * is2;
    const double A = p.k4 * fma(is8, fma(-12.0, is6, 6.0), 2.0 * p.c2);  // U'/r
    if (K == kForce) {
      t[e][0] = -A * v.x;
      t[e][1] = -A * v.y;
      t[e][2] = -A * v.z;
    } else if (K == kLoss) {
      const double s2 = r2 * p.inv_sigma2;
      const double u = p.e4 * fma(is6, is6 - 1.0, fma(p.c2, s2, p.c0));
      const double ir = rsqrt(r2), r = __dmul_rn(r2, ir);
      // the smoothed count g1 g2 and its derivative g1 g2 (g2 - g1) / w
      double g1, g2, g;
      if (p.one_exp) {
        const double E = exp(__dmul_rn(r - p.mid, p.inv_w));
        const double P = E + p.h, Q = fma(p.h, E, 1.0);
        const double inv = mdg::quotient(1.0, P * Q);
        g1 = E * Q * inv;
        g2 = P * inv;
        g = E * inv;
      } else {
        g1 = 1.0 / (1.0 + exp(-__dmul_rn(r - p.a, p.inv_w)));
        g2 = 1.0 / (1.0 + exp(-__dmul_rn(p.b - r, p.inv_w)));
        g = g1 * g2;
      }
      t[e][0] = 0.5 * u;
      t[e][1] = 0.5 * g;
      t[e][2] = -0.5 * (A * r2) * p.inv_sigma;  // dU/dsigma at fixed r
      if (GRAD) {
        const double c = A + g * (g2 - g1) * p.inv_w * ir;
        t[e][N - 3] = c * v.x;
        t[e][N - 2] = c * v.y;
        t[e][N - 1] = c * v.z;
      }
    } else {
      const double u2 = p.k4 * fma(is8, fma(156.0, is6, -42.0), 2.0 * p.c2);  // U''
      const double3 du = make_double3(ui.x - uj[e].x, ui.y - uj[e].y, ui.z - uj[e].z);
      const double B = (u2 - A) * ir2 * (v.x * du.x + v.y * du.y + v.z * du.z);
      // K du = U'' e (e.du) + U'/r (du - e (e.du))
      t[e][0] = fma(B, v.x, A * du.x);
      t[e][1] = fma(B, v.y, A * du.y);
      t[e][2] = fma(B, v.z, A * du.z);
      // F_i = sum_j -U'(r) e: dF_i/deps = -(U'/eps) e, dF_i/dsigma = (U' + r U'')/sigma e
      const double eu = v.x * ui.x + v.y * ui.y + v.z * ui.z;
      t[e][N - 2] = -(A * p.inv_eps) * eu;
      t[e][N - 1] = (A + u2) * p.inv_sigma * eu;
    }
  }
#pragma unroll
  for (int e = 0; e < 2; e++)
#pragma unroll
    for (int k = 0; k < N; k++) s[k] = __dadd_rn(s[k], in[e] ? t[e][k] : 0.0);
}

// Sum over the TPA lanes of one atom (fixed butterfly order); every lane of
// the group gets the total.
template <int TPA>
__device__ __forceinline__ double group_sum(double x) {
#pragma unroll
  for (int o = 1; o < TPA; o <<= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// Fixed-order block sum of NS values into part[blockIdx.x * NS + k].
template <int NS>
__device__ __forceinline__ void block_sums(double (&v)[NS], double *part) {
  __shared__ double sm[NS][kAB / 32];
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < NS; k++) {
    double x = v[k];
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (l == 0) sm[k][w] = x;
  }
  __syncthreads();
  if (threadIdx.x < NS) {
    double x = 0.0;
    for (int q = 0; q < kAB / 32; q++) x += sm[threadIdx.x][q];
    part[(size_t)blockIdx.x * NS + threadIdx.x] = x;
  }
}

// Flags for the evaluations at q (the next) and x (the one after): `move` when
// the list does not serve both, `jump` when a list made at q would not serve x.
__device__ __forceinline__ void flag_moves(const List &l, const Eval &e, int i, const double3 &q, const double3 &x) {
  const double3 b = l.qb.at(i);
  if (dist2(q, b) > l.half_skin2 || dist2(x, b) > l.half_skin2) atomicOr(e.move, 1);
  if (dist2(q, x) > l.half_skin2) atomicOr(e.jump, 1);
}

template <Kind K, bool GRAD, int TPA>
__global__ void __launch_bounds__(kAB, kABlocks)
    a_eval(const __grid_constant__ List l, const __grid_constant__ Pot p, const __grid_constant__ Eval e) {
  extern __shared__ unsigned smem[];
  if (*(volatile const int *)e.want && !rebuild(l, e.x, smem)) return;
  constexpr int N = Terms<K, GRAD>::N, NP = kBuckets / TPA;
  const long long threads = (long long)l.n * TPA, step = (long long)gridDim.x * kAB;
  double sums[3] = {0.0, 0.0, 0.0};
  const double3 zero = make_double3(0.0, 0.0, 0.0);
  // warps walk whole warps of threads, so the lane shuffles stay converged
  for (long long base = (long long)blockIdx.x * kAB + (threadIdx.x & ~31); base < threads; base += step) {
    const long long t = base + (threadIdx.x & 31);
    const bool on = t < threads;
    const int i = on ? (int)(t / TPA) : 0, sub = (int)(t % TPA);
    const double3 xi = e.x.at(i), ui = K == kHess ? e.u.at(i) : zero;
    // the lane's buckets, one run of the row
    int k = 0, end = 0;
    if (on) {
      const unsigned short *ends = l.ends + (size_t)i * kBuckets + sub * NP;
      k = sub ? ends[-1] : 0;
      end = ends[NP - 1];
    }
    const int *row = l.nbr + (size_t)i * l.maxnb;
    double s[N];
#pragma unroll
    for (int c = 0; c < N; c++) s[c] = 0.0;
    // two partners at once; the next two's positions and the list entries of
    // the two after them are in flight
    int j[2], jn[2];
    double3 x[2], u[2] = {zero, zero};
#pragma unroll
    for (int c = 0; c < 2; c++) {
      j[c] = k + c < end ? row[k + c] : i;
      jn[c] = k + 2 + c < end ? row[k + 2 + c] : i;
      x[c] = e.x.at(j[c]);
      if (K == kHess) u[c] = e.u.at(j[c]);
    }
#pragma unroll 1
    for (; k < end; k += 2) {
      double3 d[2], uc[2];
      const bool in[2] = {true, k + 1 < end};
#pragma unroll
      for (int c = 0; c < 2; c++) {
        d[c] = make_double3(min_image(xi.x - x[c].x, l.L[0], l.inv_L[0]), min_image(xi.y - x[c].y, l.L[1], l.inv_L[1]),
                            min_image(xi.z - x[c].z, l.L[2], l.inv_L[2]));
        uc[c] = u[c];
        x[c] = e.x.at(jn[c]);
        if (K == kHess) u[c] = e.u.at(jn[c]);
        jn[c] = k + 4 + c < end ? row[k + 4 + c] : i;
      }
      pair_terms<K, GRAD>(p, d, in, ui, uc, s);
    }
    // the atom's end, on its first lane
    if (K == kForce || K == kHess || GRAD) {
      constexpr int F = K == kLoss ? N - 3 : 0;
      const double3 w =
          make_double3(group_sum<TPA>(s[F]), group_sum<TPA>(s[F + 1]), group_sum<TPA>(s[F + 2]));
      if (on && sub == 0) {
        const double half = 0.5 * e.dt;
        if (K == kForce) {
          const double3 v = axpy(e.dt, w, e.v.at(i));
          e.v_out.set(i, v);
          const double3 q = axpy(half, v, xi), xn = axpy(half, v, q);
          if (e.q_out.p) e.q_out.set(i, q);
          if (e.x_out.p) e.x_out.set(i, xn);
          // the next evaluations: q' and x', or x' alone, or (no x') q' and x
          flag_moves(l, e, i, e.q_out.p ? q : xn, e.x_out.p ? xn : xi);
        } else if (K == kLoss) {
          const double3 a = axpy(e.scale, w, e.lq.at(i));
          const double3 b = axpy(half, a, e.lv.at(i));
          e.lq.set(i, a);
          e.lv.set(i, b);
          e.u.set(i, make_double3(b.x * e.dt, b.y * e.dt, b.z * e.dt));
        } else {
          const double3 a = axpy(-1.0, w, e.lq.at(i));
          e.lq.set(i, a);
          e.lv.set(i, axpy(half, a, e.lv.at(i)));
          if (e.x_prev.p) {
            const double3 xp = e.x_prev.at(i), q = axpy(half, e.v_prev.at(i), xp);
            e.q_out.set(i, q);
            flag_moves(l, e, i, q, xp);
          }
        }
      }
    }
    if (K == kLoss) {
#pragma unroll
      for (int c = 0; c < 3; c++) sums[c] += s[c];
    }
    if (K == kHess) {
      sums[0] += s[N - 2];
      sums[1] += s[N - 1];
    }
  }
  if (K == kLoss) block_sums<3>(sums, e.part);
  if (K == kHess) {
    double two[2] = {sums[0], sums[1]};
    block_sums<2>(two, e.part);
  }
}

// x = q + v h, and the flag of the evaluation at x.
__global__ void __launch_bounds__(kAB) a_half(List l, Vec q, Vec v, Vec x, double h, int *move) {
  const int i = blockIdx.x * kAB + threadIdx.x;
  if (i >= l.n) return;
  const double3 a = axpy(h, v.at(i), q.at(i));
  x.set(i, a);
  if (dist2(a, l.qb.at(i)) > l.half_skin2) atomicOr(move, 1);
}

// n x 3 arrays of the caller to points and back.
__global__ void __launch_bounds__(kAB) a_unpack(const double *in, Vec out, int n) {
  const int i = blockIdx.x * kAB + threadIdx.x;
  if (i < n) out.set(i, make_double3(in[3 * (size_t)i], in[3 * (size_t)i + 1], in[3 * (size_t)i + 2]));
}
__global__ void __launch_bounds__(kAB) a_pack(Vec in, double *out, int n) {
  const int i = blockIdx.x * kAB + threadIdx.x;
  if (i >= n) return;
  const double3 a = in.at(i);
  out[3 * (size_t)i] = a.x;
  out[3 * (size_t)i + 1] = a.y;
  out[3 * (size_t)i + 2] = a.z;
}

// Fixed-order sums of nb blocks' ns (<= 3) partials, one block per step:
// step blockIdx.x's partials at part + blockIdx.x * stride, its sums to out +
// blockIdx.x * ns (out_step < 0: to earlier places, as the reverse sweep goes).
constexpr int kRB = 256;
__global__ void __launch_bounds__(kRB) a_reduce(const double *part, size_t stride, int nb, int ns, double *out,
                                                int out_step) {
  __shared__ double sm[3][kRB];
  const int t = threadIdx.x;
  part += blockIdx.x * stride;
  out += (long long)blockIdx.x * out_step;
  for (int k = 0; k < ns; k++) {
    double x = 0.0;
    for (int b = t; b < nb; b += kRB) x += part[(size_t)b * ns + k];
    sm[k][t] = x;
  }
  __syncthreads();
  for (int o = kRB / 2; o > 0; o >>= 1) {
    if (t < o)
      for (int k = 0; k < ns; k++) sm[k][t] += sm[k][t + o];
    __syncthreads();
  }
  if (t < ns) out[t] = sm[t][0];
}

int nblk(int n) { return n > 0 ? (n + kAB - 1) / kAB : 1; }

// Device buffers, stream and pinned flag copy of the adjoint, kept per
// device between calls: a call takes its buffers in a fixed order and reuses
// every kept buffer that is large enough, replacing the others, so repeated
// calls of one shape allocate nothing.  One run at a time per process
// (g_ws_mutex); mdg_adjoint_release frees everything.
struct Workspace {
  std::vector<void *> buf;
  std::vector<size_t> bytes;
  cudaStream_t s = nullptr;
  int *hflag = nullptr;
};
std::mutex g_ws_mutex;
std::map<int, Workspace> g_ws;

void free_workspace(Workspace &w) {
  for (void *x : w.buf)
    if (x) cudaFree(x);
  if (w.hflag) cudaFreeHost(w.hflag);
  if (w.s) cudaStreamDestroy(w.s);
  w = Workspace();
}

struct Run {
  Workspace *ws = nullptr;
  size_t slot = 0;  // next workspace buffer
  int n = 0, tpa = 1, device = 0;
  cudaStream_t s = nullptr;
  List l{};
  Pot p{};
  double dt = 0.0;
  size_t ns = 0;                                // n rounded up to an even number
  Vec q{}, v{}, x[2]{}, lq{}, lv{}, u{};        // q': step end states; x: half-step positions, taking turns
  double *raw = nullptr;                        // n x 3 transfers
  double *ck_q = nullptr, *ck_v = nullptr;      // checkpoints
  double *seg_x = nullptr, *seg_v = nullptr;    // one segment's half-step positions and v'
  double *part = nullptr;                       // block partials of kReduceSlots steps
  double *loss_sums = nullptr;                  // per step: PE, S, dPE/dsigma
  double *adj_sums = nullptr;                   // per reverse step: u . dF/d(eps, sigma)
  int *flags = nullptr;                         // rebuild flags, one per evaluation
  int *state = nullptr;                         // row overflow, barrier timeout
  int next_flag = 0;
  int sms = 0, max_blocks = 0;
  cudaError_t err = cudaSuccess;

  template <typename T>
  cudaError_t alloc(T **ptr, size_t count_) {
    const size_t b = sizeof(T) * (count_ ? count_ : 1);
    if (slot == ws->buf.size()) {
      ws->buf.push_back(nullptr);
      ws->bytes.push_back(0);
    }
    if (ws->bytes[slot] < b) {
      if (ws->buf[slot]) cudaFree(ws->buf[slot]);
      ws->buf[slot] = nullptr;
      ws->bytes[slot] = 0;
      void *p_ = nullptr;
      const cudaError_t e = cudaMalloc(&p_, b);
      if (e != cudaSuccess) return e;
      ws->buf[slot] = p_;
      ws->bytes[slot] = b;
    }
    *ptr = static_cast<T *>(ws->buf[slot++]);
    return cudaSuccess;
  }
  cudaError_t alloc(Vec *out) {
    out->ns = ns;
    return alloc(&out->p, 3 * ns);
  }
  Vec at(double *base, size_t k) const { return Vec{base + k * 3 * ns, ns}; }
  int *flag() { return flags + next_flag++; }
  void note(cudaError_t e) {
    if (err == cudaSuccess) err = e;
  }
  size_t row_smem() const { return sizeof(unsigned) * (size_t)l.maxnb * (kAB / 32); }

  // Blocks of an evaluation: enough for its lanes and for a warp per row of a
  // rebuild, at most what is resident at once (a rebuild's barriers need every
  // block).  Fixed for a lane count, and the same for both loss passes, so that
  // the block sums are.
  template <Kind K, bool GRAD, int TPA>
  int grid() {
    int per_sm = 0;
    note(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, a_eval<K, GRAD, TPA>, kAB, row_smem()));
    if (K == kLoss) {
      int other = 0;
      note(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&other, a_eval<kLoss, !GRAD, TPA>, kAB, row_smem()));
      per_sm = std::min(per_sm, other);
    }
    const long long need = ((long long)n * std::max(TPA, 32) + kAB - 1) / kAB;
    return (int)std::max<long long>(1, std::min<long long>(need, (long long)std::max(per_sm, 1) * sms));
  }
  int grids[4][8] = {};  // by kind (a loss with gradients: 3) and lanes, 0: not computed yet
  template <Kind K, bool GRAD, int TPA>
  int eval_tpa(Eval &e) {
    int &g = grids[K == kLoss && GRAD ? 3 : K][TPA - 1];
    if (g == 0) g = grid<K, GRAD, TPA>();
    void *args[] = {&l, &p, &e};
    note(cudaLaunchCooperativeKernel((const void *)a_eval<K, GRAD, TPA>, dim3(g), dim3(kAB), args, row_smem(), s));
    return g;
  }
  // Launches one evaluation; returns its blocks.
  template <Kind K, bool GRAD>
  int eval(Eval &e) {
    switch (tpa) {
      case 1: return eval_tpa<K, GRAD, 1>(e);
      case 2: return eval_tpa<K, GRAD, 2>(e);
      case 4: return eval_tpa<K, GRAD, 4>(e);
      default: return eval_tpa<K, GRAD, 8>(e);
    }
  }
  size_t part_stride() const { return (size_t)max_blocks * 3; }
  void half(const Vec &a, const Vec &b, const Vec &out, int *move) {
    a_half<<<nblk(n), kAB, 0, s>>>(l, a, b, out, 0.5 * dt, move);
  }
  void copy(double *to, const double *from) {
    note(cudaMemcpyAsync(to, from, sizeof(double) * 3 * ns, cudaMemcpyDeviceToDevice, s));
  }
  // Row overflow (the sums are then incomplete) or a barrier that timed out.
  mdg_status list_status() {
    if (cudaMemcpyAsync(ws->hflag, state, 2 * sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess)
      return MDG_ERR_CUDA;
    if (cudaStreamSynchronize(s) != cudaSuccess) return MDG_ERR_CUDA;
    if (ws->hflag[1]) return MDG_ERR_TIMEOUT;
    return ws->hflag[0] ? MDG_ERR_CAPACITY : MDG_OK;
  }
};

// Lanes per atom of the passes, chosen once per device and problem shape by
// timing the loss pass with 1, 2, 4 and 8 lanes (the fastest is kept for the
// process, so repeated runs of one shape use the same lanes and give the same
// sums).  `want`: the list's first build.
std::mutex g_tune_mutex;
std::map<std::tuple<int, int, int>, int> g_tune;

int autotune_tpa(Run &R, int device, int *want) {
  const auto key = std::make_tuple(device, R.n, R.l.ncell);
  {
    std::lock_guard<std::mutex> lock(g_tune_mutex);
    auto it = g_tune.find(key);
    if (it != g_tune.end()) return it->second;
  }
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  int best = 1;
  float best_ms = 1e30f;
  Eval e{};
  e.x = R.x[0];
  e.dt = R.dt;
  e.part = R.part;
  e.want = want;
  int *never = R.flag();
  // the best of three rounds, the first of which warms up (and its first
  // launch builds the list)
  for (int round = 0; round < 3; round++)
    for (int t : {1, 2, 4, 8}) {
      R.tpa = t;
      cudaEventRecord(e0, R.s);
      for (int r = 0; r < 3; r++) {
        R.eval<kLoss, false>(e);
        e.want = never;
      }
      cudaEventRecord(e1, R.s);
      cudaEventSynchronize(e1);
      float ms = 0.f;
      cudaEventElapsedTime(&ms, e0, e1);
      if (round > 0 && ms < best_ms) {
        best_ms = ms;
        best = t;
      }
    }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  std::lock_guard<std::mutex> lock(g_tune_mutex);
  g_tune[key] = best;
  return best;
}

}  // namespace

extern "C" {

void mdg_adjoint_release(void) {
  std::lock_guard<std::mutex> lock(g_ws_mutex);
  int cur = 0;
  const bool have = cudaGetDevice(&cur) == cudaSuccess;
  for (auto &kv : g_ws) {
    if (cudaSetDevice(kv.first) == cudaSuccess) free_workspace(kv.second);
  }
  g_ws.clear();
  if (have) cudaSetDevice(cur);
}

void mdg_adjoint_default_params(mdg_adjoint_params *p) {
  if (!p) return;
  memset(p, 0, sizeof(*p));
  p->L[0] = p->L[1] = p->L[2] = 10.0;
  p->cutoff = 2.5;
  p->time_step = 0.005;
  p->epsilon = 1.0;
  p->sigma = 1.0;
  p->shell_lo = 1.0;
  p->shell_hi = 1.5;
  p->shell_width = 0.05;
  p->steps = 200;
  p->checkpoint_every = 20;
  p->threads_per_atom = 0;
  p->device = 0;
}

mdg_status mdg_adjoint_run(const mdg_adjoint_params *prm, const double *q0, const double *v0, int n, double *loss,
                           double *dloss_deps, double *dloss_dsigma, double *dloss_dq0) {
  if (!prm || !q0 || !v0 || !loss || n < 1 || prm->steps < 1 || prm->checkpoint_every < 1 ||
      !(prm->time_step > 0.0) || !(prm->epsilon > 0.0) || !(prm->sigma > 0.0) || !(prm->cutoff > 0.0) ||
      !(prm->shell_width > 0.0) ||
      (prm->threads_per_atom != 0 && prm->threads_per_atom != 1 && prm->threads_per_atom != 2 &&
       prm->threads_per_atom != 4 && prm->threads_per_atom != 8))
    return MDG_ERR_INVALID_ARGUMENT;
  const bool grad = dloss_deps || dloss_dsigma || dloss_dq0;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return MDG_ERR_NO_DEVICE;
  if (prm->device < 0 || prm->device >= ndev) return MDG_ERR_INVALID_ARGUMENT;
  if (cudaSetDevice(prm->device) != cudaSuccess) return MDG_ERR_CUDA;

  if (n >= 1 << 29) return MDG_ERR_CAPACITY;  // a row key holds 29 bits of index
  Run R;
  R.n = n;
  R.ns = ((size_t)n + 1) / 2 * 2;
  R.device = prm->device;
  R.dt = prm->time_step;
  List &l = R.l;
  l.n = n;
  const double rc = prm->cutoff * prm->sigma;
  // list skin: 0.3 sigma, less where a box axis holds fewer than three
  // cells of r_c + skin (no skin at all: the list is rebuilt whenever an
  // atom moved)
  double skin = 0.3 * prm->sigma;
  double longest = 0.0;
  for (int d = 0; d < 3; d++) {
    const double L = prm->L[d];
    if (!(L > 0.0) || !std::isfinite(L)) return MDG_ERR_INVALID_ARGUMENT;
    if ((int)(L / rc) < 3) return MDG_ERR_BOX_TOO_SMALL;
    skin = std::min(skin, L / 3.0 * (1.0 - 1e-9) - rc);  // cells of L/ms >= r_c + skin, ms >= 3
    longest = std::max(longest, L);
  }
  skin = std::max(skin, 0.0);
  const double sl = rc + skin;
  for (int d = 0; d < 3; d++) {
    const double L = prm->L[d];
    l.ms[d] = std::max(3, (int)(L / sl));
    l.L[d] = L;
    l.inv_cs[d] = l.ms[d] / L;
    l.inv_L[d] = 1.0 / L;
    l.Lf[d] = (float)L;
    l.inv_Lf[d] = (float)(1.0 / L);
  }
  // rows keep pairs up to sl and, for the FP32 rounding of box coordinates
  // (each difference is off by less than 4 u L, u = 2^-24; eight times that
  // here), a little more; where that is much, FP64 decides
  const double margin = 32.0 / 16777216.0 * longest;
  const double wide = sl * (1.0 + 1e-5) + margin;
  const bool exact = margin > 0.01 * sl;
  l.reach2 = (float)(exact ? -sl * sl * (1.0 + 1e-6) : wide * wide);
  l.half_skin2 = 0.25 * skin * skin;
  {
    const double reach = exact ? sl : wide;
    const double vol = prm->L[0] * prm->L[1] * prm->L[2];
    const double sphere = 4.0 / 3.0 * M_PI * reach * reach * reach;
    const double est = sphere * (double)n / vol;
    // twice the mean density's count plus 64, and at least the count at
    // density 1.3 (above a close-packed LJ solid) plus 32, so that a dense
    // region of a dilute box fits; at most 1024 within sl, which is 1056 within
    // a reach a hundredth longer.  A longer row is MDG_ERR_CAPACITY.
    const double dense = sphere * 1.3 / (prm->sigma * prm->sigma * prm->sigma);
    const double want = std::max(std::ceil(2.0 * est + 64.0), std::ceil(dense + 32.0));
    l.maxnb = (int)std::min<double>(std::min(std::max(n - 1, 1), 1056), want);
  }
  l.ncell = l.ms[0] * l.ms[1] * l.ms[2];
  const double sc = prm->cutoff;
  Pot &p = R.p;
  p.rc2 = rc * rc;
  p.c2 = 6.0 * pow(sc, -14.0) - 3.0 * pow(sc, -8.0);
  p.c0 = -pow(sc, -12.0) + pow(sc, -6.0) - p.c2 * sc * sc;
  p.sigma2 = prm->sigma * prm->sigma;
  p.inv_sigma = 1.0 / prm->sigma;
  p.inv_sigma2 = 1.0 / p.sigma2;
  p.inv_eps = 1.0 / prm->epsilon;
  p.e4 = 4.0 * prm->epsilon;
  p.k4 = p.e4 / p.sigma2;
  p.a = prm->shell_lo;
  p.b = prm->shell_hi;
  p.inv_w = 1.0 / prm->shell_width;
  p.mid = 0.5 * (p.a + p.b);
  p.h = exp(0.5 * (p.a - p.b) * p.inv_w);
  {
    // E = exp((r - mid)/w) and h as factors of a product of four stay finite
    // and normal
    const double most = 150.0 * prm->shell_width;
    p.one_exp = fabs(p.mid) < most && fabs(rc - p.mid) < most && fabs(0.5 * (p.a - p.b)) < most;
  }
  const int T = prm->steps, k = prm->checkpoint_every;
  const int nck = (T + k - 1) / k + 1;
  const int seg = std::min(k, T);

  std::lock_guard<std::mutex> ws_lock(g_ws_mutex);
  Workspace &ws = g_ws[prm->device];
  if (!ws.buf.empty()) {
    // buffers of an earlier call: still this context's device memory? (a
    // device reset in between drops them)
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, ws.buf[0]) != cudaSuccess || at.type != cudaMemoryTypeDevice) {
      cudaGetLastError();
      ws = Workspace();
    }
  }
  R.ws = &ws;
  cudaError_t e = cudaDeviceGetAttribute(&R.sms, cudaDevAttrMultiProcessorCount, prm->device);
  R.max_blocks = (int)std::min<long long>(((long long)n * 32 + kAB - 1) / kAB, (long long)R.sms * 16);
  if (e == cudaSuccess && !ws.s) e = cudaStreamCreateWithFlags(&ws.s, cudaStreamNonBlocking);
  if (e == cudaSuccess && !ws.hflag) e = cudaMallocHost((void **)&ws.hflag, 2 * sizeof(int));
  R.s = ws.s;
  const size_t nflags = 6 * (size_t)T + 2 * (size_t)nck + 16;
  if (e == cudaSuccess) e = R.alloc(&R.q);
  if (e == cudaSuccess) e = R.alloc(&R.v);
  if (e == cudaSuccess) e = R.alloc(&R.x[0]);
  if (e == cudaSuccess) e = R.alloc(&R.x[1]);
  if (e == cudaSuccess) e = R.alloc(&l.qb);
  if (e == cudaSuccess) e = R.alloc(&R.raw, 3 * (size_t)n);
  if (e == cudaSuccess) e = R.alloc(&l.cell, n);
  if (e == cudaSuccess) e = R.alloc(&l.rank, n);
  if (e == cudaSuccess) e = R.alloc(&l.count, l.ncell);
  if (e == cudaSuccess) e = R.alloc(&l.start, l.ncell);
  if (e == cudaSuccess) e = R.alloc(&l.sorted, n);
  if (e == cudaSuccess) e = R.alloc(&l.nbr, (size_t)l.maxnb * n);
  if (e == cudaSuccess) e = R.alloc(&l.ends, (size_t)kBuckets * n);
  if (e == cudaSuccess) e = R.alloc(&R.part, R.part_stride() * kReduceSlots * (grad ? 2 : 1));
  if (e == cudaSuccess) e = R.alloc(&R.loss_sums, (size_t)T * 3);
  if (e == cudaSuccess) e = R.alloc(&R.flags, nflags);
  if (e == cudaSuccess) e = R.alloc(&R.state, 8);
  if (grad) {
    if (e == cudaSuccess) e = R.alloc(&R.lq);
    if (e == cudaSuccess) e = R.alloc(&R.lv);
    if (e == cudaSuccess) e = R.alloc(&R.u);
    if (e == cudaSuccess) e = R.alloc(&R.adj_sums, (size_t)T * 2);
    if (e == cudaSuccess) e = R.alloc(&R.ck_q, (size_t)nck * 3 * R.ns);
    if (e == cudaSuccess) e = R.alloc(&R.ck_v, (size_t)nck * 3 * R.ns);
    if (e == cudaSuccess) e = R.alloc(&R.seg_x, (size_t)seg * 3 * R.ns);
    if (e == cudaSuccess) e = R.alloc(&R.seg_v, (size_t)seg * 3 * R.ns);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();  // reported here, not by the next call
    return e == cudaErrorMemoryAllocation ? MDG_ERR_CAPACITY : MDG_ERR_CUDA;
  }
  l.overflow = R.state;
  l.timeout = R.state + 1;
  l.cursor = R.state + 2;
  l.bar = reinterpret_cast<Meeting *>(R.state + 4);
  R.note(cudaMemsetAsync(R.flags, 0, sizeof(int) * nflags, R.s));
  R.note(cudaMemsetAsync(R.state, 0, sizeof(int) * 8, R.s));
  R.note(cudaMemsetAsync(l.qb.p, 0, sizeof(double) * 3 * R.ns, R.s));

  R.note(cudaMemcpyAsync(R.raw, q0, sizeof(double) * 3 * n, cudaMemcpyHostToDevice, R.s));
  a_unpack<<<nblk(n), kAB, 0, R.s>>>(R.raw, R.q, n);
  R.note(cudaMemcpyAsync(R.raw, v0, sizeof(double) * 3 * n, cudaMemcpyHostToDevice, R.s));
  a_unpack<<<nblk(n), kAB, 0, R.s>>>(R.raw, R.v, n);

  // the first evaluation builds the list
  int *move = R.flag();
  R.note(cudaMemsetAsync(move, 1, 1, R.s));
  R.half(R.q, R.v, R.x[0], move);
  bool built = false;
  if (prm->threads_per_atom) {
    R.tpa = prm->threads_per_atom;
  } else {
    const int before = R.next_flag;
    R.tpa = autotune_tpa(R, prm->device, move);
    built = R.next_flag != before;
    if (built) move = R.flag();  // timed: the list is there
  }

  // forward pass.  Without gradients: loss terms per step.  With them:
  // checkpoints every k steps; the reverse sweep passes every step's end
  // state again, and its loss passes give the loss terms too.
  int slots = 0, nb = 0;
  for (int t = 0; t < T; t++) {
    if (grad && t % k == 0) {
      R.copy(R.ck_q + (size_t)(t / k) * 3 * R.ns, R.q.p);
      R.copy(R.ck_v + (size_t)(t / k) * 3 * R.ns, R.v.p);
    }
    if (grad && t / k == (T - 1) / k) break;  // the sweep runs the last segment itself
    Eval f{};
    f.x = R.x[t & 1];
    f.want = move;
    f.dt = R.dt;
    f.v = f.v_out = R.v;
    if (!grad || (t + 1) % k == 0) f.q_out = R.q;
    f.x_out = R.x[(t + 1) & 1];
    int *at_q = f.move = R.flag();
    f.jump = R.flag();
    move = grad ? f.move : f.jump;
    R.eval<kForce, false>(f);
    built = true;
    if (grad) continue;
    Eval o{};
    o.x = R.q;
    o.want = at_q;
    o.dt = R.dt;
    o.part = R.part + R.part_stride() * slots;
    nb = R.eval<kLoss, false>(o);
    if (++slots == kReduceSlots || t == T - 1) {
      a_reduce<<<slots, kRB, 0, R.s>>>(R.part, R.part_stride(), nb, 3, R.loss_sums + (size_t)3 * (t + 1 - slots), 3);
      slots = 0;
    }
  }
  std::vector<double> sums((size_t)T * 3);
  const double norm = 1.0 / ((double)T * n);
  double sum = 0.0, dl_deps = 0.0, dl_dsig = 0.0;
  auto read_loss = [&]() {
    R.note(cudaMemcpyAsync(sums.data(), R.loss_sums, sizeof(double) * sums.size(), cudaMemcpyDeviceToHost, R.s));
    R.note(cudaStreamSynchronize(R.s));
    for (int t = 0; t < T; t++) {
      sum += sums[3 * t] + sums[3 * t + 1];
      dl_deps += sums[3 * t] / prm->epsilon;  // PE is linear in epsilon
      dl_dsig += sums[3 * t + 2];
    }
    *loss = sum * norm;
  };
  if (!grad) {
    read_loss();
    if (R.err != cudaSuccess || cudaGetLastError() != cudaSuccess) return MDG_ERR_CUDA;
    return R.list_status();
  }

  // reverse sweep, one checkpointed segment at a time
  R.note(cudaMemsetAsync(R.lq.p, 0, sizeof(double) * 3 * R.ns, R.s));
  R.note(cudaMemsetAsync(R.lv.p, 0, sizeof(double) * 3 * R.ns, R.s));
  double *hess_part = R.part + R.part_stride() * kReduceSlots;
  int nb_loss = 0;
  for (int sg = (T - 1) / k; sg >= 0; sg--) {
    const int t0 = sg * k, t1 = std::min(T, t0 + k);
    // forward again from the checkpoint; the last step leaves q' for the sweep
    move = R.flag();
    if (!built) R.note(cudaMemsetAsync(move, 1, 1, R.s));  // no evaluation yet (one segment)
    built = true;
    R.half(R.at(R.ck_q, sg), R.at(R.ck_v, sg), R.at(R.seg_x, 0), move);
    int *jump = nullptr;
    for (int t = t0; t < t1; t++) {
      Eval f{};
      f.x = R.at(R.seg_x, t - t0);
      f.want = move;
      f.dt = R.dt;
      f.v = t == t0 ? R.at(R.ck_v, sg) : R.at(R.seg_v, t - 1 - t0);
      f.v_out = R.at(R.seg_v, t - t0);
      if (t == t1 - 1) f.q_out = R.q;
      else f.x_out = R.at(R.seg_x, t + 1 - t0);
      move = f.move = R.flag();
      jump = f.jump = R.flag();
      R.eval<kForce, false>(f);
    }
    for (int t = t1 - 1; t >= t0; t--) {
      Eval g{};
      g.x = R.q;
      g.want = move;
      g.dt = R.dt;
      g.lq = R.lq;
      g.lv = R.lv;
      g.u = R.u;
      g.scale = norm;
      g.part = R.part + R.part_stride() * slots;
      nb_loss = R.eval<kLoss, true>(g);
      Eval h{};
      h.x = R.at(R.seg_x, t - t0);
      h.want = jump;
      h.dt = R.dt;
      h.lq = R.lq;
      h.lv = R.lv;
      h.u = R.u;
      h.part = hess_part + R.part_stride() * slots;
      if (t > t0) {
        h.x_prev = R.at(R.seg_x, t - 1 - t0);
        h.v_prev = R.at(R.seg_v, t - 1 - t0);
        h.q_out = R.q;
      }
      move = h.move = R.flag();
      jump = h.jump = R.flag();
      nb = R.eval<kHess, false>(h);
      if (++slots == kReduceSlots || t == 0) {
        // slot s holds step t + slots - 1 - s
        a_reduce<<<slots, kRB, 0, R.s>>>(R.part, R.part_stride(), nb_loss, 3,
                                         R.loss_sums + (size_t)3 * (t + slots - 1), -3);
        a_reduce<<<slots, kRB, 0, R.s>>>(hess_part, R.part_stride(), nb, 2, R.adj_sums + (size_t)2 * (t + slots - 1),
                                         -2);
        slots = 0;
      }
    }
  }
  std::vector<double> adj((size_t)T * 2);
  R.note(cudaMemcpyAsync(adj.data(), R.adj_sums, sizeof(double) * adj.size(), cudaMemcpyDeviceToHost, R.s));
  if (dloss_dq0) {
    a_pack<<<nblk(n), kAB, 0, R.s>>>(R.lq, R.raw, n);
    R.note(cudaMemcpyAsync(dloss_dq0, R.raw, sizeof(double) * 3 * n, cudaMemcpyDeviceToHost, R.s));
  }
  read_loss();
  if (R.err != cudaSuccess || cudaGetLastError() != cudaSuccess) return MDG_ERR_CUDA;
  dl_deps *= norm;
  dl_dsig *= norm;
  // dynamics terms summed in reverse-sweep order, as the sweep produced them
  for (int t = T - 1; t >= 0; t--) {
    dl_deps += adj[(size_t)2 * t];
    dl_dsig += adj[(size_t)2 * t + 1];
  }
  if (dloss_deps) *dloss_deps = dl_deps;
  if (dloss_dsigma) *dloss_dsigma = dl_dsig;
  return R.list_status();
}

}  // extern "C"
