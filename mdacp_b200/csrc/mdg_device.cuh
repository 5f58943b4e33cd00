// Device code of the B200 LJ timestep: cell sort, Verlet list build, force
// kick (FP64 drop-in and FP32-mixed), drift, skin bookkeeping, thermostats
// and FP64 observables.  Host orchestration lives in mdg_api.cu.
//
// Data layout in HBM (n atoms, slots renumbered in cell order at every
// rebuild):
//   q, v      double4[cap]   position (unwrapped between rebuilds), velocity
//   qfix      int4[cap]      fixed-point copy of q for the FP32-mixed force:
//                            x_fix = round(frac(x/L) * 2^32) as uint32, so the
//                            int32 difference of two atoms is the minimum-image
//                            displacement in units of L/2^32 (no shift tables)
//   nbr       int32[maxnb][stride]  full Verlet list, column-major: entry k
//                            of atom i at nbr[k*stride + i] (coalesced per warp)
//   nnbr      int32[cap]     row lengths; rows are padded with the atom's own
//                            index up to a multiple of 4 (the FP32 force loop
//                            walks 4 partners at a time; a self entry has r = 0
//                            and is masked)
//   qloc      float4[cap]    FP32 coordinates at the last build for the list
//                            prefilter: x in box coordinates, y and z
//                            relative to the atom's cell
//   cxyz      int32[cap]     the slot's cell coordinates at the last build,
//                            packed x | y << 11 | z << 22
//   xsub      int32[rows*(8*ms_x+1)]  list-build trim table, one block per
//                            x-row of cells: atoms inside a cell are in x
//                            order, entry 8*cx + k of a row's block is the first
//                            slot of its cell cx at or beyond x0 + k cs_x / 8,
//                            and entry 8*ms_x is the end of the row
//   nbr16     uint2[maxnb/4][stride]  FP32-mixed only: the same rows as 16-bit
//                            indices into the block's staged partner positions
//                            (four per 8-byte load); see k_stage_plan
//   stage_rng int4[blocks][kStageRanges]  per 128-atom block: the cell ranges
//                            whose atoms the force pass stages in shared memory
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

namespace mdg {

constexpr int kErrCapacity = 1;
constexpr int kErrTooFast = 2;
constexpr int kErrInvalidPosition = 4;
constexpr int kErrNonFinite = 8;
constexpr int kErrTimeout = 16;
constexpr int kErrStage = 32;  // a staged row index outside its block's stage (an inconsistent plan)

// Geometry and force constants, passed by value to every kernel.
struct Box {
  double L[3];
  double hL[3];        // L/2, minimum-image threshold
  double inv_cs[3];    // 1 / cell size
  int ms[3];           // cells per axis (MeshList::ChangeScale: int(L/SL))
  int ncell;
  double sl;           // SearchLength
  double sl2;          // SearchLength^2
  double rc2;          // CUTOFF_LENGTH^2
  double rc;           // CUTOFF_LENGTH
  double c0, c2;       // smoothed-LJ constants (Variables::C0, C2)
  double dt;           // TimeStep
  double buffer_length;
  float fix_scale[3];  // L / 2^32
  float rc2f;
  float c2x8f;
  int check_list_length;
  double cs[3];        // cell size L / ms
  float sl2_lo, sl2_hi;  // FP32 prefilter band around SearchLength^2
  // z-slab of a decomposed system (slab = 1): the owned cell layers are the
  // global layers z0 .. z0 + nzl - 1, and cell indices, packed cell
  // coordinates and trim-table rows use the local layer z - z0; the trim
  // table has two more blocks of rows, the ghost layers below (block nzl)
  // and above (block nzl + 1).  A single domain has slab = 0, z0 = 0 and
  // nzl = ms[2].
  int slab, z0, nzl;
  long long stage_wait;  // staged FP32 pass: cycles of the first wait for the stage copy
};

// Mutable device-side state of one handle.
struct Status {
  int error;                        // kErr* flags; any set flag halts the step kernels
  int list_stale;                   // 1: next step rebuilds unconditionally
  unsigned long long vmax2_bits;    // max |v|^2 of the last velocity update (double bits)
  double budget;                    // PairList::buffer_length
  unsigned long long dr2max_bits;   // displacement check: max |dq|^2
  int cand_weighted;                // candidate copies (real atoms and ghost images)
  int cand_n;                       // candidate copies stored
  int max_row;                      // longest neighbour row of the last build
  int want_build;                   // this step rebuilds the list
  long long list_entries;
  long long total_images;           // real atoms + ghost images (PairList Nl bound)
  long long rebuilds;
  long long steps;
  long long disp_checks;
  double zeta;                      // Nose-Hoover friction (Variables::Zeta)
  double sim_time;
  double too_fast_v;                // speed that tripped kErrTooFast
  double ext_position;              // external executor: current piston position
  double ext_impulse;               // external executor: impulse of the last pass
  // 1 while Arrays::v_lag holds the velocities of the last second half
  // drift: an executor changed v after the step, and the reconstruction of
  // the reference's half-step-old ghost copies (q - v dt/2) must use the
  // velocities the drift used.  Cleared once the next step's skin check is
  // decided, and by a rebuild (fresh copies).
  int vlag_set;
  // persistent pipeline (mdg_calculate with the persistent pass): the step
  // count the queued launches stop at, the fixed-point buffer the next
  // fused step reads (0: qfix, 1: qfix2), and the steps the persistent
  // pass took
  long long target_steps;
  int fix_parity;
  long long persistent_steps;
  unsigned long long vmax2_ring[3];  // the persistent pass's |v| maxima, step k in slot k % 3
};

// An executor the reference's projects run after every Calculate() (on the
// real atoms' momenta = velocities), applied on the device after each step.
struct External {
  int kind;          // 0 none, 1 gravity, 2 piston, 3 shell wall
  int axis;          // gravity: axis of the acceleration
  double strength;   // gravity: acceleration
  double dt;         // the time step the executor multiplies by
  double velocity;   // piston: displacement per pass (towards -z)
  double center[3];  // shell: centre
  double radius;     // shell: radius of the wall surface
};

struct Arrays {
  double4 *q, *v, *q_old;
  int4 *qfix;
  int4 *qfix2;        // second fixed-point buffer: the fused NVE step reads one and writes the other
  double *pz, *pz2;   // FP64 handles: z of the packed positions whose (x, y) are qfix, qfix2 as double2; null otherwise
  float4 *qloc;       // FP32 coordinates at the last build (list prefilter): x global, y z cell-local
  int *cxyz;          // packed cell coordinates of each slot at the last build
  int *xsub;          // x sub-bin starts of every cell and row ends (list-build trim table)
  int *ids, *type;
  int *cell;          // cell of each slot at the last build
  int *nbr, *nnbr;
  int *cell_count, *cell_start;
  int *slot;          // rank inside the cell from the atomic scatter
  int *perm, *perm2;  // new slot -> old slot
  double4 *q_tmp, *v_tmp;
  double4 *v_lag;     // velocities of the last second half drift (Status::vlag_set); null in slabs
  int *ids_tmp, *type_tmp, *cell_tmp;
  unsigned char *mult; // ghost-border membership at the last build (bits, see border_bits)
  int2 *cand;         // displacement-check candidates: (slot, image code)
  double *disp2;      // per atom: the largest squared copy displacement of the last skin check (k_disp_max); null: not kept
  double *partials;   // per-block partial sums for reductions
  Status *st;
  int stride;         // column stride of nbr (>= cap, multiple of 32)
  int maxnb;          // neighbour-row capacity
  // staged FP32 force (null / 0 when off)
  int4 *stage_rng;    // per block: (first cell, end cell, first atom, offset in the block's stage)
  int *stage_n;       // per block: ranges, -1 = partners gathered from global memory
  uint2 *nbr16;       // rows as stage indices, four 16-bit entries per element
  int stage_cap;      // atoms one block stages at most
};

// The FP32 prefilter band of the list build: candidates whose FP32 r^2 lies
// in [lo, hi] around SearchLength^2 are decided by the exact FP64 test.  The
// prefilter's x coordinate is the box coordinate (error up to one rounding
// of L_x) and y, z are cell-local, so with u = 2^-24 the FP32 r^2 of a
// candidate near the search length is within u (6 L_x / SL + 37) SL^2 of
// the exact value; the band is four times that, and at least 1e-4 SL^2.
inline void prefilter_band(double sl2, double sl, double lx, float *lo, float *hi) {
  const double u = 1.0 / 16777216.0;
  const double rel = fmax(1e-4, 4.0 * u * (6.0 * lx / sl + 37.0));
  *lo = (float)(sl2 * (1.0 - rel));
  *hi = (float)(sl2 * (1.0 + rel));
}

// ------------------------------------------------------------------ helpers
__device__ __forceinline__ double dadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double dsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double dmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double ddiv(double a, double b) { return __ddiv_rn(a, b); }

// a / b for normal b: one Newton step on the hardware's approximate
// reciprocal, then the quotient corrected by its residual with fused
// multiply-adds (P. W. Markstein, "Computation of elementary functions on the
// IBM RISC System/6000 processor", 1990).  The reciprocal is good to about
// 2^-40, so the quotient before its last rounding is to about 2^-80: the
// correctly rounded one but for some 10^-8 of the operands, where it is its
// neighbour (tests/test_gpu_quotient.py: none differs from the IEEE quotient in
// 10^5 pairs of the force and observer terms from 1e-12 to the cut-off).  Unlike
// the operator it has no branch for unusual operands, so the quotients of several
// pairs overlap; one that overflows, or whose denominator is zero or subnormal
// (pairs nearer than 1e-22), is NaN where the operator gives an infinity.
__device__ __forceinline__ double quotient(double a, double b) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
  y = fma(y, fma(-b, y, 1.0), y);
  const double q = a * y;
  return fma(fma(-b, q, a), y, q);
}

// The skin budget's cost of one step, 2 vmax dt, each operation separately
// rounded as in PairList::IsPairListExpired (src/pairlist.cc:25-65), so
// every kernel that spends the budget spends the same amount.
__device__ __forceinline__ double skin_cost(double vmax, double dt) { return dmul(dmul(vmax, 2.0), dt); }

__device__ __forceinline__ void atomic_max_double_bits(unsigned long long *addr, double v) {
  // non-negative doubles order like their bit patterns
  atomicMax(addr, (unsigned long long)__double_as_longlong(v));
}

template <typename T>
__device__ __forceinline__ T warp_max(T v) {
  for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Block-wide max of a non-negative double, one atomic per block.
template <int BLOCK>
__device__ __forceinline__ void block_max_to(unsigned long long *addr, double v) {
  __shared__ double sm[BLOCK / 32];
  v = warp_max(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) sm[w] = v;
  __syncthreads();
  if (w == 0) {
    v = (l < BLOCK / 32) ? sm[l] : 0.0;
    v = warp_max(v);
    if (l == 0) atomic_max_double_bits(addr, v);
  }
}

// Warp maximum folded into a global maximum without a block barrier, so a
// warp that finishes its rows early leaves at once; the atomic is skipped
// when the global value is already at least as large (non-negative v).
__device__ __forceinline__ void warp_max_to(unsigned long long *addr, double v) {
  v = warp_max(v);
  if ((threadIdx.x & 31) == 0 && v > 0.0) {
    const unsigned long long cur = *(volatile unsigned long long *)addr;
    const unsigned long long mine = (unsigned long long)__double_as_longlong(v);
    if (mine > cur) atomicMax(addr, mine);
  }
}

// The error flag as one lane of the warp read it: the lanes of an atom must
// agree on whether they take its row (they exchange values), and the flag
// can be raised by another block at any time.  All lanes must call.
__device__ __forceinline__ int warp_error(const Status *st) {
  return __shfl_sync(0xffffffffu, *(volatile const int *)&st->error, 0);
}

// Fixed order block sum written to partials[blockIdx.x * nsum + k].
template <int BLOCK, int NSUM>
__device__ __forceinline__ void block_sum_to(double (&v)[NSUM], double *partials) {
  __shared__ double sm[NSUM][BLOCK / 32];
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < NSUM; k++) {
    double x = warp_sum(v[k]);
    if (l == 0) sm[k][w] = x;
  }
  __syncthreads();
  if (w == 0) {
#pragma unroll
    for (int k = 0; k < NSUM; k++) {
      double x = (l < BLOCK / 32) ? sm[k][l] : 0.0;
      x = warp_sum(x);
      if (l == 0) partials[(size_t)blockIdx.x * NSUM + k] = x;
    }
  }
}

__device__ __forceinline__ int cell_coord(double x, double inv_cs, int ms) {
  int c = (int)(x * inv_cs);
  return c < 0 ? 0 : (c >= ms ? ms - 1 : c);
}

// Fixed-point image of one coordinate: frac(x / L) * 2^32 rounded, mod 2^32.
__device__ __forceinline__ int fixed_coord(double x, double L) {
  double u = x / L;
  u -= floor(u);
  const long long k = __double2ll_rn(u * 4294967296.0);
  return (int)(unsigned int)(unsigned long long)k;
}

// Position (x, y, z) of atom i into a packed copy: fixed-point, or with a z
// array (FP64 handles) as (x, y) and z apart.  The FP64 pair kernels gather 24
// bytes a partner from the split copy: in a double4 array the 16-byte halves
// of consecutive atoms fall on every other 16-byte column of the L1's data
// banks and z on every fourth, which made the gathers' bank conflicts the
// bound of the pass.
__device__ __forceinline__ void pack_position(int4 *out, double *out_z, int i, double x, double y, double z,
                                              const double L[3]) {
  if (out_z) {
    reinterpret_cast<double2 *>(out)[i] = make_double2(x, y);
    out_z[i] = z;
  } else {
    out[i] = make_int4(fixed_coord(x, L[0]), fixed_coord(y, L[1]), fixed_coord(z, L[2]), 0);
  }
}

// Minimum-image ghost coordinate as the reference forms it: the copy of
// atom j that lies next to atom i is q_j + diff with diff in {-L, 0, +L}
// (MDUnit::MakeBufferForBorderParticles, src/mdunit.cc:152-192).
__device__ __forceinline__ double image_of(double xj, double xi, double L, double hL) {
  const double t = xj - xi;
  if (t > hL) return dsub(xj, L);
  if (t < -hL) return dadd(xj, L);
  return xj;
}

// ---------------------------------------------------------------- kernels
// Upload indices of a fresh state: slot i holds atom i.
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) k_upload_ids(Arrays a, int n) {
  const int i = blockIdx.x * BLOCK + threadIdx.x;
  if (i < n) a.ids[i] = i;
}

// Initial |v|^2 maximum (used before the first step after an upload) and a
// finiteness check of the uploaded state.
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) k_vmax(Arrays a, int n) {
  const int i = blockIdx.x * BLOCK + threadIdx.x;
  double v2 = 0.0;
  if (i < n) {
    const double4 v = a.v[i];
    const double4 q = a.q[i];
    v2 = dadd(dadd(dmul(v.x, v.x), dmul(v.y, v.y)), dmul(v.z, v.z));
    if (!isfinite(v2) || !isfinite(q.x) || !isfinite(q.y) || !isfinite(q.z)) {
      atomicOr(&a.st->error, kErrNonFinite);
      v2 = 0.0;
    }
  }
  block_max_to<BLOCK>(&a.st->vmax2_bits, v2);
}

// PairList::IsPairListExpired (src/pairlist.cc:25-65): budget -= 2 vmax dt
// while the budget is positive (a too-fast atom is an error), then arm the
// displacement check once the budget is spent.  One thread: *disp_out = run
// the displacement check this step; returns whether the step rebuilds
// unconditionally (a stale list).
__device__ __forceinline__ int expiry_decide(Status *st, const Box &b, int *disp_out) {
  int disp = 0, build = 0;
  if (st->error == 0) {
    if (st->list_stale) {
      build = 1;
    } else {
      if (st->budget > 0.0) {
        const double vmax = sqrt(__longlong_as_double((long long)st->vmax2_bits));
        if (skin_cost(vmax, b.dt) > b.buffer_length) {
          st->too_fast_v = vmax;
          atomicOr(&st->error, kErrTooFast);
        } else {
          st->budget = dsub(st->budget, skin_cost(vmax, b.dt));
        }
      }
      if (st->error == 0 && st->budget < 0.0) {
        disp = 1;
        st->dr2max_bits = 0ull;
        st->cand_weighted = 0;
        st->cand_n = 0;
        st->disp_checks++;
      }
    }
  }
  st->want_build = build;
  st->vmax2_bits = 0ull;
  if (!disp) st->vlag_set = 0;  // no displacement check reads the ghost copies this step
  *disp_out = disp;
  return build;
}

// expiry_decide in a graph: the step's conditional branch (skin check, then
// rebuild) runs if either may be due.  One thread.  A conditional node costs
// 6.5 us where its branch is not taken (a rate every step pays), so a step has
// one, and the rebuild's is inside its branch.
__device__ __forceinline__ void expiry_in_graph(Status *st, const Box &b, cudaGraphConditionalHandle h_any) {
  int disp = 0;
  const int build = expiry_decide(st, b, &disp);
  cudaGraphSetConditional(h_any, disp || (st->error == 0 && build));
}

// expiry_decide as a kernel: for a graph, or setting device flags in eager
// mode (there the check and the rebuild are launched apart).
static __global__ void k_expiry(Arrays a, Box b, cudaGraphConditionalHandle h_any, int in_graph, int *eager_flags) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  Status *st = a.st;
  if (in_graph) {
    expiry_in_graph(st, b, h_any);
    return;
  }
  int disp = 0;
  const int build = expiry_decide(st, b, &disp);
  // the rebuild decision when no displacement check runs; otherwise k_decide,
  // after the check, sets it again
  eager_flags[0] = disp;
  eager_flags[1] = st->error == 0 && build;
}

// Sets the rebuild condition of this step from the expiry and displacement
// decisions.
static __global__ void k_decide(Arrays a, cudaGraphConditionalHandle h_build, int in_graph, int *eager_flags) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  const int build = (a.st->error == 0) && a.st->want_build;
  a.st->vlag_set = 0;  // the displacement check has read the ghost copies
  if (in_graph) cudaGraphSetConditional(h_build, build);
  else eager_flags[1] = build;
}

// ---- ghost copies of the reference, for the skin check -----------------
// The reference checks displacements over real atoms AND their ghost
// copies (src/pairlist.cc:67-121 loops over GetTotalParticleNumber()).  A
// ghost is q + diff with diff = +L for atoms in a low-face strip and -L for a
// high-face strip, per axis, for every combination of the strips the atom was
// in at the last build (the six sequential border passes,
// src/mdmanager.cc:395-401).  Its old position is the build-time copy; its
// current one dates from the last SendBorderParticles, i.e. half a step back
// after a full NVE / Nose-Hoover step (lag = dt/2; 0 otherwise).  An image
// code holds 2 bits per axis: 0 no shift, 1 +L, 2 -L; code 0 is the atom.
__device__ __forceinline__ double image_coord(double x, int c, double L) {
  return c == 1 ? dadd(x, L) : (c == 2 ? dadd(x, -L) : x);
}

// The axis options of an atom's copies: mask bits 2d (low strip) and 2d+1
// (high strip) for axis d.
__device__ __forceinline__ int axis_options(int mask, int d, int opt[2]) {
  int k = 0;
  if (mask & (1 << (2 * d))) opt[k++] = 1;
  if (mask & (1 << (2 * d + 1))) opt[k++] = 2;
  return k;
}

// The state arrays the copy helpers read.
struct CopyView {
  const double4 *q_old, *q, *v;
  const unsigned char *mask;
};

// Old and current position of copy `code` of atom i in a box of lengths L.
__device__ __forceinline__ void copy_positions(const CopyView &cv, const double L[3], int i, int code, double lag,
                                               double old_p[3], double new_p[3]) {
  const double4 o = cv.q_old[i], q = cv.q[i];
  const double oo[3] = {o.x, o.y, o.z};
  double qq[3] = {q.x, q.y, q.z};
  if (code != 0 && lag > 0.0) {
    const double4 v = cv.v[i];
    qq[0] = dsub(q.x, dmul(v.x, lag));
    qq[1] = dsub(q.y, dmul(v.y, lag));
    qq[2] = dsub(q.z, dmul(v.z, lag));
  }
  for (int d = 0; d < 3; d++) {
    const int c = (code >> (2 * d)) & 3;
    old_p[d] = image_coord(oo[d], c, L[d]);
    new_p[d] = image_coord(qq[d], c, L[d]);
  }
}

__device__ __forceinline__ double dist2(const double a[3], const double c[3]) {
  const double dx = dsub(a[0], c[0]), dy = dsub(a[1], c[1]), dz = dsub(a[2], c[2]);
  return dadd(dadd(dmul(dx, dx), dmul(dy, dy)), dmul(dz, dz));
}

// Calls f(code, d2) for every copy of atom i (the atom first), d2 the
// squared displacement since the last build as the reference forms it
// (qb_old - q, src/pairlist.cc:75-79).
template <typename F>
__device__ __forceinline__ void for_each_copy(const CopyView &cv, const double L[3], int i, double lag, F f) {
  const int mask = cv.mask[i];
  int ox[3] = {0, 0, 0}, oy[3] = {0, 0, 0}, oz[3] = {0, 0, 0};
  int tx[2], ty[2], tz[2];
  const int nx = axis_options(mask, 0, tx), ny = axis_options(mask, 1, ty), nz = axis_options(mask, 2, tz);
  for (int k = 0; k < nx; k++) ox[k + 1] = tx[k];
  for (int k = 0; k < ny; k++) oy[k + 1] = ty[k];
  for (int k = 0; k < nz; k++) oz[k + 1] = tz[k];
  for (int z = 0; z <= nz; z++)
    for (int y = 0; y <= ny; y++)
      for (int x = 0; x <= nx; x++) {
        const int code = ox[x] | (oy[y] << 2) | (oz[z] << 4);
        double op[3], np[3];
        copy_positions(cv, L, i, code, lag, op, np);
        f(code, dist2(op, np));
      }
}

// Velocities that date the ghost copies: v_lag after an executor changed v.
__device__ __forceinline__ const double4 *lag_velocities(const Arrays &a) {
  return (a.v_lag && a.st->vlag_set) ? a.v_lag : a.v;
}

__device__ __forceinline__ CopyView copy_view(const Arrays &a) {
  return CopyView{a.q_old, a.q, lag_velocities(a), a.mult};
}

// PairList::CheckByDisplacement, first pass: max |qb_old - q|^2 over all
// copies (src/pairlist.cc:67-84).
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) k_disp_max(Arrays a, Box b, int n, double lag) {
  const int i = blockIdx.x * BLOCK + threadIdx.x;
  double d2 = 0.0;
  if (a.st->list_stale) return;  // a graph's branch that only rebuilds
  if (i < n) for_each_copy(copy_view(a), b.L, i, lag, [&](int, double x) { d2 = fmax(d2, x); });
  if (a.disp2 && i < n) a.disp2[i] = d2;
  block_max_to<BLOCK>(&a.st->dr2max_bits, d2);
}

// Files atom i's copies that moved further than sqrt(c_d2) as candidates
// (slot, image code): counted first, so that an atom waits for one atomic
// instead of one per copy (24 replicas' collection 8.9 -> 5.3 us, 256
// replicas' 23 -> 18).  weighted counts them all, stored those with a
// place offered.
__device__ __forceinline__ void collect_copies(const CopyView &cv, const double L[3], int i, double lag, double c_d2,
                                               int *weighted, int *stored, int2 *cand, int cand_cap) {
  unsigned long long codes = 0ull;  // 6 bits a copy, at most 8 copies
  int k = 0;
  for_each_copy(cv, L, i, lag, [&](int code, double d2) {
    if (d2 > c_d2) codes |= (unsigned long long)code << (6 * k++);
  });
  if (k == 0) return;
  atomicAdd(weighted, k);
  const int at = atomicAdd(stored, k);
  for (int u = 0; u < k && at + u < cand_cap; u++, codes >>= 6) cand[at + u] = make_int2(i, (int)(codes & 63ull));
}

// Second pass: copies that moved more than BufferLength - sqrt(dr2_max)
// (src/pairlist.cc:86-97); each is stored as (slot, image code).
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) k_disp_collect(Arrays a, Box b, int n, int cand_cap, double lag) {
  const int i = blockIdx.x * BLOCK + threadIdx.x;
  if (i >= n || a.st->list_stale) return;
  const double c = b.buffer_length - sqrt(__longlong_as_double((long long)a.st->dr2max_bits));
  const double c_d2 = c * c;
  // no copy of this atom moved more than c (k_disp_max's per-atom maximum
  // of the same displacements): nothing to collect
  if (a.disp2 && !(a.disp2[i] > c_d2)) return;
  // a full list: the number of copies has decided (k_disp_pairs; over several
  // slabs too), and thousands of atomics to one address would follow
  if (*(volatile const int *)&a.st->cand_weighted >= cand_cap) return;
  collect_copies(copy_view(a), b.L, i, lag, c_d2, &a.st->cand_weighted, &a.st->cand_n, a.cand, cand_cap);
}

// Candidate copies staged in shared memory for the pair test: old and
// current position of each, one array per axis so that consecutive lanes
// read consecutive doubles.  960 copies (45 KB) covers the reference's
// CheckListLength of 500 with room; longer lists are read from global memory.
constexpr int kPairStage = 960;

struct PairStage {
  double o[3][kPairStage], n[3][kPairStage];
};

// candidate_pair_test reading the copies' positions from global memory (any l,
// no barrier).
template <int BLOCK>
__device__ __forceinline__ void candidate_pair_test_global(const CopyView &cv, const double L[3], const int2 *cand,
                                                           int l, double lag, double sl2, double rc2, int part,
                                                           int parts, volatile int *found) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int a = part * (BLOCK / 32) + w; a < l - 1 && !*found; a += parts * (BLOCK / 32)) {
    double o1[3], n1[3];
    copy_positions(cv, L, cand[a].x, cand[a].y, lag, o1, n1);
    for (int c = a + 1 + lane; c < l; c += 32) {
      double o2[3], n2[3];
      copy_positions(cv, L, cand[c].x, cand[c].y, lag, o2, n2);
      if (dist2(o1, o2) < sl2) continue;
      if (dist2(n1, n2) < rc2) *found = 1;
    }
  }
}

// The pair test of PairList::CheckByDisplacement (src/pairlist.cc:99-121)
// over the candidate list's rows, a warp each, dealt over `parts` blocks: sets *found
// if a pair of candidate copies (a < b) that was at least SearchLength apart
// at the last build is now inside the cut-off.  Copies carry their shifts,
// so the distances are the reference's direct differences.  The result is
// an "any" over the pairs, so splitting the rows over blocks and the columns
// over threads changes only the time.  l must be the same for every thread
// of the block (the staging pass ends in a barrier).
template <int BLOCK>
__device__ __forceinline__ void candidate_pair_test(const CopyView &cv, const double L[3], const int2 *cand, int l,
                                                    double lag, double sl2, double rc2, int part, int parts,
                                                    PairStage &sm, volatile int *found) {
  if (l <= kPairStage) {
    for (int k = threadIdx.x; k < l; k += BLOCK) {
      const int2 c = cand[k];
      double o[3], p[3];
      copy_positions(cv, L, c.x, c.y, lag, o, p);
      for (int d = 0; d < 3; d++) {
        sm.o[d][k] = o[d];
        sm.n[d][k] = p[d];
      }
    }
    __syncthreads();
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int a = part * (BLOCK / 32) + w; a < l - 1 && !*found; a += parts * (BLOCK / 32)) {
      const double o1[3] = {sm.o[0][a], sm.o[1][a], sm.o[2][a]};
      const double n1[3] = {sm.n[0][a], sm.n[1][a], sm.n[2][a]};
      for (int c = a + 1 + lane; c < l; c += 32) {
        const double o2[3] = {sm.o[0][c], sm.o[1][c], sm.o[2][c]};
        if (dist2(o1, o2) < sl2) continue;
        const double n2[3] = {sm.n[0][c], sm.n[1][c], sm.n[2][c]};
        if (dist2(n1, n2) < rc2) *found = 1;
      }
    }
  } else {
    candidate_pair_test_global<BLOCK>(cv, L, cand, l, lag, sl2, rc2, part, parts, found);
  }
}

// Third pass, kPairParts blocks sharing the rows: expired if the copies
// found reach min(total copies, CheckListLength), or if the pair test finds
// a pair (src/pairlist.cc:86-121).
constexpr int kPairParts = 16;

template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) k_disp_pairs(Arrays a, Box b, double lag) {
  __shared__ PairStage sm;
  __shared__ volatile int found;
  if (threadIdx.x == 0) found = 0;
  __syncthreads();
  Status *st = a.st;
  if (st->list_stale) return;
  const long long tn = st->total_images;
  const int nl = (int)((tn > b.check_list_length) ? b.check_list_length : tn);
  if (st->cand_weighted >= nl) {
    if (threadIdx.x == 0) found = 1;
  } else {
    const int l = min(st->cand_n, b.check_list_length);
    candidate_pair_test<BLOCK>(copy_view(a), b.L, a.cand, l, lag, b.sl2, b.rc2, blockIdx.x, gridDim.x, sm, &found);
  }
  __syncthreads();
  if (threadIdx.x == 0 && found) st->want_build = 1;
}

// ------------------------------------------------------ staged partners
// The FP32-mixed force pass stages, per block of kStageBlock consecutive
// atoms, the fixed-point positions of every atom in the union of the
// block's 27-cell stencils in shared memory, and reads partners from there.
// Atoms are in cell order, so that union is a few runs of consecutive cells
// (the stencil rows of the block's home cells), i.e. a few runs of
// consecutive atoms, which the pass copies with bulk asynchronous copies.
// Rows hold, besides the global partner index, its index in the stage
// (16 bits, four per 8-byte element).  The pair terms and their order are
// the global-gather pass's; only where the positions are read from changes.
constexpr int kStageBlock = 128;
constexpr int kStageRanges = 32;
constexpr int kStageRaw = 96;  // stencil-row cell runs per block before merging

// Offset from a global atom index to its stage index, for an atom of cell nc:
// the plan range that holds nc (ranges are sorted by first cell).
__device__ __forceinline__ int stage_shift(const int4 *plan, int npl, int nc) {
  int lo = 0, hi = npl - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (plan[mid].x <= nc) lo = mid;
    else hi = mid - 1;
  }
  return plan[lo].w - plan[lo].z;
}

// Entry k of atom i's staged row: four 16-bit entries per uint2, written
// when the fourth arrives (rows are padded to a multiple of 4).
__device__ __forceinline__ void stage_entry(uint2 *nbr16, int stride, int i, int k, int v, unsigned &g0,
                                            unsigned &g1) {
  const unsigned val = (unsigned)v & 0xffffu;
  switch (k & 3) {
    case 0: g0 = val; g1 = 0u; break;
    case 1: g0 |= val << 16; break;
    case 2: g1 = val; break;
    default:
      g1 |= val << 16;
      nbr16[(size_t)(k >> 2) * stride + i] = make_uint2(g0, g1);
  }
}

// Rebuild, after the permutation and the cell scan: the stage plan of every
// block of kStageBlock atoms, one thread per block.  The block's home cells
// lie in [cell of its first atom, cell of its last atom]; each run of them
// along x contributes, per (dz, dy), the cells x-1 .. x+1 of that row (one
// or two runs with the periodic wrap).  The runs are sorted and merged; a
// block that needs more than kStageRanges runs or more than stage_cap atoms
// is marked -1 and gathers its partners from global memory.
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) k_stage_plan(Arrays a, Box b, int n) {
  const int blk = blockIdx.x * BLOCK + threadIdx.x;
  const int nblk = (n + kStageBlock - 1) / kStageBlock;
  if (blk >= nblk || a.st->error) return;
  const int i0 = blk * kStageBlock, i1 = min(n, i0 + kStageBlock) - 1;
  const int c_first = a.cell_tmp[i0], c_last = a.cell_tmp[i1];
  const int ms0 = b.ms[0], ms1 = b.ms[1], ms2 = b.ms[2];
  int2 run[kStageRaw];
  int nrun = 0;
  bool over = false;
  for (int c = c_first; c <= c_last && !over;) {
    const int xa = c % ms0, y = (c / ms0) % ms1, z = c / (ms0 * ms1);
    const int xb = min(ms0 - 1, xa + (c_last - c));
    c += xb - xa + 1;
    if (nrun + 18 > kStageRaw) {
      over = true;
      break;
    }
    const int lo = xa - 1, hi = xb + 1;  // inclusive, before the wrap
    int s0, e0, s1 = 0, e1 = 0;
    if (hi - lo + 1 >= ms0) {
      s0 = 0; e0 = ms0;
    } else if (lo < 0) {
      s0 = 0; e0 = hi + 1; s1 = lo + ms0; e1 = ms0;
    } else if (hi >= ms0) {
      s0 = 0; e0 = hi - ms0 + 1; s1 = lo; e1 = ms0;
    } else {
      s0 = lo; e0 = hi + 1;
    }
    for (int dz = -1; dz <= 1; dz++) {
      const int zz = (z + dz + ms2) % ms2;
      for (int dy = -1; dy <= 1; dy++) {
        const int base = (zz * ms1 + (y + dy + ms1) % ms1) * ms0;
        run[nrun++] = make_int2(base + s0, base + e0);
        if (e1 > s1) run[nrun++] = make_int2(base + s1, base + e1);
      }
    }
  }
  int m = 0;
  if (!over) {
    for (int k = 1; k < nrun; k++) {  // insertion sort by first cell
      const int2 x = run[k];
      int j = k - 1;
      while (j >= 0 && run[j].x > x.x) {
        run[j + 1] = run[j];
        j--;
      }
      run[j + 1] = x;
    }
    for (int k = 0; k < nrun; k++) {  // merge overlapping and touching runs
      if (m > 0 && run[k].x <= run[m - 1].y) run[m - 1].y = max(run[m - 1].y, run[k].y);
      else run[m++] = run[k];
    }
    over = m > kStageRanges;
  }
  int total = 0;
  if (!over) {
    for (int r = 0; r < m; r++) {
      const int first = a.cell_start[run[r].x];
      a.stage_rng[blk * kStageRanges + r] = make_int4(run[r].x, run[r].y, first, total);
      total += a.cell_start[run[r].y] - first;
    }
    over = total > a.stage_cap;
  }
  a.stage_n[blk] = over ? -1 : m;
}

// ------------------------------------------------------------- list build
// x sub-bins per cell of the list build's trim table (see xsub above).
constexpr int kXSub = 8;

// Cell coordinates packed into one int (x and y below 2048, z below 1024).
__device__ __forceinline__ int pack_cell(int cx, int cy, int cz) { return cx | (cy << 11) | (cz << 22); }

// Trim-table entries of a cell: the block of its x-row, at its x position.
__device__ __forceinline__ int *trim_entries(int *tab, int ms0, int row, int cx) {
  return tab + (size_t)row * (ms0 * kXSub + 1) + cx * kXSub;
}

// One warp orders the cnt slots perm[beg, beg + cnt) of a cell by (x, upload
// id) into perm2 and writes the cell's entries of the trim table: ent[k] =
// beg + (atoms with x < x0 + k bin), k < kXSub, and for the last cell of a
// row (last) the row's end ent[kXSub] = beg + cnt.  Ties in x (a lattice) go
// by id, so the order is a function of the state alone.
__device__ __forceinline__ void sort_cell_x(const double4 *q, const int *ids, const int *perm, int *perm2, int beg,
                                            int cnt, double x0, double bin, int *ent, bool last, int lane) {
  int below[kXSub];
#pragma unroll
  for (int k = 0; k < kXSub; k++) below[k] = 0;
  for (int base = 0; base < cnt; base += 32) {
    const int me = base + lane;
    int my_slot = -1, my_id = 0x7fffffff;
    double my_x = 0.0;
    if (me < cnt) {
      my_slot = perm[beg + me];
      my_x = q[my_slot].x;
      my_id = ids[my_slot];
    }
    int rank = 0;
    for (int ob = 0; ob < cnt; ob += 32) {
      const int other = ob + lane;
      double ox = 0.0;
      int oid = 0x7fffffff;
      if (other < cnt) {
        const int os = perm[beg + other];
        ox = q[os].x;
        oid = ids[os];
      }
      const int lim = min(32, cnt - ob);
      for (int k = 0; k < lim; k++) {
        const double kx = __shfl_sync(0xffffffffu, ox, k);
        const int kid = __shfl_sync(0xffffffffu, oid, k);
        rank += (kx < my_x || (kx == my_x && kid < my_id)) ? 1 : 0;
      }
    }
    if (me < cnt) perm2[beg + rank] = my_slot;
#pragma unroll
    for (int k = 1; k < kXSub; k++)
      below[k] += __popc(__ballot_sync(0xffffffffu, me < cnt && my_x < x0 + k * bin));
  }
  int v = 0;
#pragma unroll
  for (int k = 1; k < kXSub; k++)
    if (lane == k) v = below[k];
  if (lane < kXSub) ent[lane] = beg + v;
  if (last && lane == 0) ent[kXSub] = beg + cnt;
}

// Rebuild 1/6: wrap into [0,L] (Variables::AdjustPeriodicBoundary,
// src/variables.cc:63-84), validity check, cell index and rank inside the cell.
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) k_cell_assign(Arrays a, Box b, int n) {
  const int i = blockIdx.x * BLOCK + threadIdx.x;
  if (i >= n || a.st->error) return;
  double4 q = a.q[i];
  double x[3] = {q.x, q.y, q.z};
  int cc[3];
  bool bad = false;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    if (!isfinite(x[d])) {
      atomicOr(&a.st->error, kErrNonFinite);
      return;
    }
    if (x[d] < 0.0) x[d] = dadd(x[d], b.L[d]);
    else if (x[d] > b.L[d]) x[d] = dsub(x[d], b.L[d]);
    bad |= (x[d] < 0.0 || x[d] > b.L[d]);
    cc[d] = cell_coord(x[d], b.inv_cs[d], b.ms[d]);
  }
  if (bad) {
    atomicOr(&a.st->error, kErrInvalidPosition);
    return;
  }
  q.x = x[0]; q.y = x[1]; q.z = x[2];
  a.q[i] = q;
  if (b.slab) {  // the slab's own layers only (migration moved every other atom away)
    cc[2] -= b.z0;
    if (cc[2] < 0 || cc[2] >= b.nzl) {
      atomicOr(&a.st->error, kErrInvalidPosition);
      return;
    }
  }
  const int c = (cc[2] * b.ms[1] + cc[1]) * b.ms[0] + cc[0];
  a.cell[i] = c;
  a.slot[i] = atomicAdd(&a.cell_count[c], 1);
}

template <int BLOCK>
__device__ __forceinline__ int block_exclusive_scan(int x, int *total) {
  __shared__ int warp_tot[BLOCK / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int inc = x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += y;
  }
  if (lane == 31) warp_tot[w] = inc;
  __syncthreads();
  if (w == 0) {
    int t = lane < BLOCK / 32 ? warp_tot[lane] : 0;
    int ti = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, ti, o);
      if (lane >= o) ti += y;
    }
    if (lane < BLOCK / 32) warp_tot[lane] = ti - t;
    if (lane == BLOCK / 32 - 1) *total = ti;
  }
  __syncthreads();
  const int r = warp_tot[w] + inc - x;
  __syncthreads();
  return r;
}

// Rebuild 2/6: exclusive scan of the cell counts in three passes -- tiles of
// BLOCK cells scanned in parallel, the tile totals scanned by one block,
// the tile offsets added back.
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) k_scan_tiles(Arrays a, int ncell, int *tile_sum) {
  __shared__ int total;
  if (a.st->error) return;
  const int c = blockIdx.x * BLOCK + threadIdx.x;
  const int x = c < ncell ? a.cell_count[c] : 0;
  const int ex = block_exclusive_scan<BLOCK>(x, &total);
  if (c < ncell) a.cell_start[c] = ex;
  if (threadIdx.x == 0) tile_sum[blockIdx.x] = total;
}

template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) k_scan_tile_sums(Arrays a, int ncell, int *tile_sum, int ntiles) {
  __shared__ int total;
  if (a.st->error) return;
  int carry = 0;
  for (int base = 0; base < ntiles; base += BLOCK) {
    const int k = base + threadIdx.x;
    const int x = k < ntiles ? tile_sum[k] : 0;
    const int ex = block_exclusive_scan<BLOCK>(x, &total);
    if (k < ntiles) tile_sum[k] = carry + ex;
    carry += total;
    __syncthreads();
  }
  if (threadIdx.x == 0) a.cell_start[ncell] = carry;
}

template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) k_scan_add(Arrays a, int ncell, const int *tile_sum) {
  if (a.st->error) return;
  const int c = blockIdx.x * BLOCK + threadIdx.x;
  if (c < ncell && blockIdx.x > 0) a.cell_start[c] += tile_sum[blockIdx.x];
}

// The same in one block, for grids of few cells: the carry runs over
// chunks of BLOCK cells (one launch instead of three).
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) k_scan_single(Arrays a, int ncell) {
  __shared__ int total;
  if (a.st->error) return;
  int carry = 0;
  for (int base = 0; base < ncell; base += BLOCK) {
    const int c = base + threadIdx.x;
    const int x = c < ncell ? a.cell_count[c] : 0;
    const int ex = block_exclusive_scan<BLOCK>(x, &total);
    if (c < ncell) a.cell_start[c] = carry + ex;
    carry += total;
    __syncthreads();
  }
  if (threadIdx.x == 0) a.cell_start[ncell] = carry;
}

// Rebuild 3/6: scatter old slots to their cell ranges.
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) k_scatter(Arrays a, int n) {
  const int i = blockIdx.x * BLOCK + threadIdx.x;
  if (i >= n || a.st->error) return;
  a.perm[a.cell_start[a.cell[i]] + a.slot[i]] = i;
}

// Rebuild 4/6: order every cell by (x, upload id), one warp per cell, which
// makes the slot order a function of the state alone (independent of
// atomics) and puts each cell's atoms in x order for the list build's trim
// table; the cell's row of that table is written too (sort_cell_x).
static __global__ void k_sort_cells(Arrays a, Box b, int ncell) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= ncell || a.st->error) return;
  const int beg = a.cell_start[warp], cnt = a.cell_start[warp + 1] - beg;
  const int cx = warp % b.ms[0];
  sort_cell_x(a.q, a.ids, a.perm, a.perm2, beg, cnt, cx * b.cs[0], b.cs[0] / kXSub,
              trim_entries(a.xsub, b.ms[0], warp / b.ms[0], cx), cx == b.ms[0] - 1, lane);
}

// Ghost-strip membership of a wrapped position at a build: bit 2d for
// 0 < x_d < SL, bit 2d+1 for L_d - SL < x_d < L_d (MDRect::IsInsideEdge,
// src/mdrect.cc:23-47); the copies are every combination of the strips, so
// their count including the atom is the product over axes of (1 + bits).
__device__ __forceinline__ int border_bits(const double x[3], const Box &b, int *copies) {
  int mask = 0, m = 1;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const int lo = (x[d] < b.sl && x[d] > 0.0) ? 1 : 0;
    const int hi = (x[d] > b.L[d] - b.sl && x[d] < b.L[d]) ? 1 : 0;
    mask |= (lo << (2 * d)) | (hi << (2 * d + 1));
    m *= 1 + lo + hi;
  }
  *copies = m;
  return mask;
}

// Rebuild 5/6: gather into cell order (temporary arrays), snapshot q_old
// (PairList::Init), ghost-strip membership and the total copy count.
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) k_permute(Arrays a, Box b, int n, int4 *pack, double *pack_z) {
  const int s = blockIdx.x * BLOCK + threadIdx.x;
  int m = 0;
  if (s < n && !a.st->error) {
    const int o = a.perm2[s];
    const double4 q = a.q[o];
    a.q_tmp[s] = q;
    a.v_tmp[s] = a.v[o];
    a.ids_tmp[s] = a.ids[o];
    a.type_tmp[s] = a.type[o];
    a.cell_tmp[s] = a.cell[o];
    a.q_old[s] = q;
    const double x[3] = {q.x, q.y, q.z};
    const int strips = border_bits(x, b, &m);
    a.mult[s] = (unsigned char)strips;
    // FP32 coordinates for the list prefilter (x in box coordinates, y and z
    // relative to the cell), with the strip bits, and the packed cell coordinates
    const int c = a.cell_tmp[s];
    const int cx = c % b.ms[0], cy = (c / b.ms[0]) % b.ms[1], cz = c / (b.ms[0] * b.ms[1]);
    const int gz = cz + b.z0;  // global layer (the local one in a slab)
    a.qloc[s] = make_float4((float)q.x, (float)(q.y - cy * b.cs[1]), (float)(q.z - gz * b.cs[2]), __int_as_float(strips));
    a.cxyz[s] = pack_cell(cx, cy, cz);
    if (pack) {
      // the coming step's first-drift positions for the fused NVE pass
      const double4 v = a.v[o];
      const double dt2 = b.dt * 0.5;
      pack_position(pack, pack_z, s, dadd(q.x, dmul(v.x, dt2)), dadd(q.y, dmul(v.y, dt2)), dadd(q.z, dmul(v.z, dt2)),
                    b.L);
    }
  }
  const int tot = __reduce_add_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0 && tot) atomicAdd((unsigned long long *)&a.st->total_images, (unsigned long long)tot);
}

// Strip bits a partner needs for its ghost copy with shift (sx, sy, sz) to
// exist: +L images come from the low-face strip, -L images from the high-face
// strip (MDUnit::MakeBufferForBorderParticles, src/mdunit.cc:156-192).  A
// partner outside the strip -- e.g. exactly on a face, which the strict
// MDRect::IsInsideEdge test leaves out (src/mdrect.cc:27-43) -- has no copy
// there, and the reference's search does not see that pair from this side.
__device__ __forceinline__ int needed_strips(double sx, double sy, double sz) {
  return (sx > 0.0 ? 1 : 0) | (sx < 0.0 ? 2 : 0) | (sy > 0.0 ? 4 : 0) | (sy < 0.0 ? 8 : 0) |
         (sz > 0.0 ? 16 : 0) | (sz < 0.0 ? 32 : 0);
}

// Exact test of one candidate, the reference's arithmetic
// (MeshList::SearchMesh, src/meshlist.cc:276-289): ghost image q_j + diff
// first, then dx = x_i - image, then ((dx*dx + dy*dy) + dz*dz), each
// operation separately rounded; kept when r^2 <= SearchLength^2.
__device__ __forceinline__ bool within_search_exact(const double4 &qi, const double4 &qj, double sx, double sy,
                                                    double sz, double sl2) {
  const double gx = dadd(qj.x, sx), gy = dadd(qj.y, sy), gz = dadd(qj.z, sz);
  const double ex = dsub(qi.x, gx), ey = dsub(qi.y, gy), ez = dsub(qi.z, gz);
  const double r2 = dadd(dadd(dmul(ex, ex), dmul(ey, ey)), dmul(ez, ez));
  return !(r2 > sl2);
}

// Image shift of a stencil piece, 2 bits per axis (0: none, 1: -L, 2: +L).
__device__ __forceinline__ double shift_of(int code, int d, const double L[3]) {
  const int c = (code >> (2 * d)) & 3;
  return c == 1 ? -L[d] : (c == 2 ? L[d] : 0.0);
}

// The exact test of candidate j of atom i through image shift `shift`
// (within_search_exact).  Reached only for candidates in the FP32 band, so
// the FP64 positions and shifts are read here rather than held in registers
// across the candidate loop.
__device__ __forceinline__ bool band_test(const double4 *__restrict__ q, int i, int j, int shift, const Box &b) {
  return within_search_exact(q[i], q[j], shift_of(shift, 0, b.L), shift_of(shift, 1, b.L), shift_of(shift, 2, b.L),
                             b.sl2);
}

// Candidates [beg, end) of one stencil row of atom i, in slot order: FP32
// prefilter r^2 <= hi on the prefilter coordinates moved by the row's base
// (bx, by, bz); the ghost-existence rule for image shifts (NEED); the exact
// FP64 test for candidates in the band [lo, hi] (band_test, image shift
// `shift`); emit(j, k) files partner j as entry k of the row.  SELF: the
// range holds atom i itself.  Four loads are issued before the first test.
//
// With BTPA lanes per atom (the lanes of one atom are consecutive and all
// walk the same ranges), lane s tests candidates beg + s, beg + BTPA + s, ...
// and the lanes file the ones they keep in slot order through a ballot over
// the atom's lanes, so the row is the same for every lane count; cnt stays
// equal on all of them.
template <bool NEED, bool SELF, int BTPA, typename Emit>
__device__ __forceinline__ void build_range(const float4 *__restrict__ qloc, const double4 *__restrict__ q,
                                            const unsigned char *__restrict__ mult, int beg, int end, float bx,
                                            float by, float bz, int need, int shift, const Box &b, int i, int &cnt,
                                            Emit &emit) {
  auto keep_of = [&](int j, const float4 &l) {
    const float ex = l.x + bx, ey = l.y + by, ez = l.z + bz;
    const float r2 = fmaf(ex, ex, fmaf(ey, ey, ez * ez));
    bool keep = r2 <= b.sl2_hi;
    if (SELF) keep = keep && j != i;
    if (NEED) keep = keep && (mult[j] & need) == need;
    if (keep && r2 >= b.sl2_lo) keep = band_test(q, i, j, shift, b);
    return keep;
  };
  if (BTPA == 1) {
    // four candidates at a time: the four prefilter tests are independent
    // (one pass over them), the rare band candidates are decided in one
    // branch, then the kept ones are filed in slot order; the loads run one
    // batch ahead
    auto prefilter = [&](int j, const float4 &l, float &r2) {
      const float ex = l.x + bx, ey = l.y + by, ez = l.z + bz;
      r2 = fmaf(ex, ex, fmaf(ey, ey, ez * ez));
      bool keep = r2 <= b.sl2_hi;
      if (SELF) keep = keep && j != i;
      return keep;
    };
    int j = beg;
    float4 n0, n1, n2, n3;
    if (j + 4 <= end) {
      n0 = __ldg(qloc + j);
      n1 = __ldg(qloc + j + 1);
      n2 = __ldg(qloc + j + 2);
      n3 = __ldg(qloc + j + 3);
    }
    for (; j + 4 <= end; j += 4) {
      const float4 l0 = n0, l1 = n1, l2 = n2, l3 = n3;
      if (j + 8 <= end) {
        n0 = __ldg(qloc + j + 4);
        n1 = __ldg(qloc + j + 5);
        n2 = __ldg(qloc + j + 6);
        n3 = __ldg(qloc + j + 7);
      }
      float r0, r1, r2, r3;
      bool k0 = prefilter(j, l0, r0), k1 = prefilter(j + 1, l1, r1), k2 = prefilter(j + 2, l2, r2),
           k3 = prefilter(j + 3, l3, r3);
      if (NEED) {
        k0 = k0 && (mult[j] & need) == need;
        k1 = k1 && (mult[j + 1] & need) == need;
        k2 = k2 && (mult[j + 2] & need) == need;
        k3 = k3 && (mult[j + 3] & need) == need;
      }
      const float lo = b.sl2_lo;
      if ((k0 && r0 >= lo) || (k1 && r1 >= lo) || (k2 && r2 >= lo) || (k3 && r3 >= lo)) {
        if (k0 && r0 >= lo) k0 = band_test(q, i, j, shift, b);
        if (k1 && r1 >= lo) k1 = band_test(q, i, j + 1, shift, b);
        if (k2 && r2 >= lo) k2 = band_test(q, i, j + 2, shift, b);
        if (k3 && r3 >= lo) k3 = band_test(q, i, j + 3, shift, b);
      }
      if (k0) emit(j, cnt);
      cnt += k0;
      if (k1) emit(j + 1, cnt);
      cnt += k1;
      if (k2) emit(j + 2, cnt);
      cnt += k2;
      if (k3) emit(j + 3, cnt);
      cnt += k3;
    }
    for (; j < end; j++) {
      if (keep_of(j, __ldg(qloc + j))) {
        emit(j, cnt);
        cnt++;
      }
    }
  } else {
    const int lane = threadIdx.x & 31, sub = lane & (BTPA - 1), first = lane & ~(BTPA - 1);
    const unsigned gmask = (BTPA == 32) ? 0xffffffffu : (((1u << BTPA) - 1u) << first);
    const unsigned below = (1u << sub) - 1u;
    auto file = [&](int j, bool keep) {
      const unsigned m = __ballot_sync(gmask, keep) >> first;
      if (keep) emit(j, cnt + __popc(m & below));
      cnt += __popc(m);
    };
    for (int base = beg; base < end; base += 2 * BTPA) {
      const int j0 = base + sub, j1 = base + BTPA + sub;
      float4 l0 = make_float4(0.f, 0.f, 0.f, 0.f), l1 = l0;
      if (j0 < end) l0 = __ldg(qloc + j0);
      if (j1 < end) l1 = __ldg(qloc + j1);
      const bool k0 = j0 < end && keep_of(j0, l0);
      const bool k1 = j1 < end && keep_of(j1, l1);
      file(j0, k0);
      file(j1, k1);
    }
  }
}

// The full Verlet row of atom i (MeshList::SearchMesh's pair set, src/
// meshlist.cc:242-292, seen from i): the 27 cells around i's own cell
// (periodic, >= 3 cells per axis so they are distinct) are walked as 9 rows
// along x.  Cells of a row are consecutive in slot order and atoms inside a
// cell are in x order, so one row is one contiguous slot range (two or
// three where the periodic wrap splits it), trimmed at both ends through the
// trim table to the sub-bins that reach within SearchLength of x_i; rows
// whose y-z gap to i already exceeds SearchLength are skipped.  Row order:
// rows in (dz, dy) order, then x order across the row's cells -- the cells
// in dx order, as a 27-cell walk visits them.  Returns the partners found
// (entries beyond the capacity are counted, not filed).
template <int BTPA, typename Emit>
__device__ __forceinline__ int build_rows(const Box &b, const float4 *__restrict__ qloc,
                                          const double4 *__restrict__ q, const unsigned char *__restrict__ mult,
                                          const int *__restrict__ tab, int pc, int i, Emit &emit) {
  const float4 li = qloc[i];
  const int cx = pc & 2047, cy = (pc >> 11) & 2047, cz = (int)((unsigned)pc >> 22);  // layers from 512 on use the sign bit
  const int ms0 = b.ms[0], ms1 = b.ms[1], ms2 = b.ms[2];
  const float hi = b.sl2_hi;
  const int mx = ms0 * kXSub;
  // x_i in sub-bins from the start of the virtual row of cells cx-1 .. cx+1
  // (unwrapped x; bins of width cs/kXSub from each cell's lower face, as the
  // trim table counts them), and the x bases of the three pieces (image
  // shifts -L, 0, +L; prefilter x is global)
  const int vbase = (cx - 1) * kXSub;
  float ubin, per_binf, bxm, bx0, bxp;
  {
    const double qx = q[i].x;
    const double cs0 = b.cs[0], per_bin = kXSub / cs0;
    ubin = (float)((qx - (cx - 1) * cs0) * per_bin);
    per_binf = (float)per_bin;
    bxm = (float)(-b.L[0] - qx);
    bx0 = (float)(-qx);
    bxp = (float)(b.L[0] - qx);
  }
  const float csy = (float)b.cs[1], csz = (float)b.cs[2];
  int cnt = 0;
  for (int dz = -1; dz <= 1; dz++) {
    int z = cz + dz, zc = 0;  // zc: the row's image shift along z (shift_of's code)
    if (z < 0) { z += ms2; zc = 1; } else if (z >= ms2) { z -= ms2; zc = 2; }
    const double sz = zc == 1 ? -b.L[2] : (zc == 2 ? b.L[2] : 0.0);
    const float bz = (float)((z - cz) * b.cs[2] + sz) - li.z;
    const float gz = dz == 0 ? 0.f : (dz < 0 ? li.z : csz - li.z);
    for (int dy = -1; dy <= 1; dy++) {
      const float gy = dy == 0 ? 0.f : (dy < 0 ? li.y : csy - li.y);
      const float g2 = fmaf(gy, gy, gz * gz);
      if (g2 > hi) continue;  // the whole row is out of reach
      // sub-bins [vlo, vhi) of the row that can hold a partner: every bin
      // that reaches x_i -/+ sqrt(hi - g2), the x reach left by the row's
      // y-z gap g (hi is above SearchLength^2 by more than the FP32 error of
      // g2; the bin edges get 1e-3 of a bin more)
      const float reach = sqrtf(hi - g2) * per_binf;
      int vlo = vbase + (int)floorf(ubin - reach - 1e-3f);
      int vhi = vbase + (int)floorf(ubin + reach + 1e-3f) + 1;
      vlo = max(vlo, vbase);
      vhi = min(vhi, vbase + 3 * kXSub);
      int y = cy + dy, yc = 0;
      if (y < 0) { y += ms1; yc = 1; } else if (y >= ms1) { y -= ms1; yc = 2; }
      const double sy = yc == 1 ? -b.L[1] : (yc == 2 ? b.L[1] : 0.0);
      const float by = (float)((y - cy) * b.cs[1] + sy) - li.y;
      const int *xr = tab + (size_t)(z * ms1 + y) * (mx + 1);
      const int yz = (yc << 2) | (zc << 4);
      if (vlo < 0)  // through the -x face: the row's last cells, image shift -L
        build_range<true, false, BTPA>(qloc, q, mult, xr[vlo + mx], xr[mx], bxm, by, bz,
                                       needed_strips(-b.L[0], sy, sz), 1 | yz, b, i, cnt, emit);
      {
        const int a0 = max(vlo, 0), a1 = min(vhi, mx);
        const int beg = xr[a0], end = xr[a1];
        const int need = needed_strips(0.0, sy, sz);
        if (dz == 0 && dy == 0)
          build_range<false, true, BTPA>(qloc, q, mult, beg, end, bx0, by, bz, 0, yz, b, i, cnt, emit);
        else if (need)
          build_range<true, false, BTPA>(qloc, q, mult, beg, end, bx0, by, bz, need, yz, b, i, cnt, emit);
        else
          build_range<false, false, BTPA>(qloc, q, mult, beg, end, bx0, by, bz, 0, yz, b, i, cnt, emit);
      }
      if (vhi > mx)  // through the +x face: the row's first cells, image shift +L
        build_range<true, false, BTPA>(qloc, q, mult, xr[0], xr[vhi - mx], bxp, by, bz,
                                       needed_strips(b.L[0], sy, sz), 2 | yz, b, i, cnt, emit);
    }
  }
  return cnt;
}

// ---- rows of a warp's atoms, one lane per atom
// What a lane's row walk needs of its box (the replica's own in an ensemble).
struct RowGeom {
  double L[3], cs0, inv_cs0, sl2;
  float csy, csz, lo, hi;  // cell edges along y and z; the FP32 prefilter band
  int ms[3], z0, nzl;
};

__device__ __forceinline__ RowGeom row_geom(const Box &b) {
  return RowGeom{{b.L[0], b.L[1], b.L[2]}, b.cs[0],   b.inv_cs[0], b.sl2, (float)b.cs[1], (float)b.cs[2], b.sl2_lo,
                 b.sl2_hi,  {b.ms[0], b.ms[1], b.ms[2]}, b.z0, b.nzl};
}

// Strip bits an image shift needs (needed_strips), from its code (shift_of):
// code 1 (-L) needs the high strip, code 2 (+L) the low one.
__device__ __forceinline__ int strips_of(int code) { return ((code & 0x15) << 1) | ((code & 0x2a) >> 1); }

__device__ __forceinline__ float sqrt_approx(float x) {
  float y;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Candidates of one run that a warp stages at a time, and words of found
// partners that a lane keeps before they go to the list.
constexpr int kRunStage = 128;

// Shared memory of one warp's row walk.
template <int WORDS>
struct WarpRows {
  float4 xy[kRunStage / 2];  // staged candidates in pairs: x0, x1, y0, y1
  float2 zz[kRunStage / 2];  //                             z0, z1
  // column l: lane l's words, 32 candidates each: partners as bits (the first
  // candidate at bit 31) and the first candidate's slot
  uint2 word[WORDS][32];
};

// The exact test of candidate j of atom i (within_search_exact) through the
// y and z images of the row (code yz, see shift_of) and the minimum image in
// x.  A candidate near SearchLength is less than half the box away in x, so
// that image is the one it was staged for; it must also lie in cells cx - 1
// .. cx + 1 as the reference's search sees them, which a walk past the lane's
// own window does not promise.
static __device__ __noinline__ bool band_test_row(const RowGeom &g, const double4 *__restrict__ q, int i, int j, int cx,
                                           int yz) {
  const double4 qi = q[i], qj = q[j];
  const double t = qj.x - qi.x;
  const int xc = t > 0.5 * g.L[0] ? 1 : (t < -0.5 * g.L[0] ? 2 : 0);
  const int cj = cell_coord(qj.x, g.inv_cs0, g.ms[0]) + (xc == 1 ? -g.ms[0] : (xc == 2 ? g.ms[0] : 0));
  if (cj < cx - 1 || cj > cx + 1) return false;
  return within_search_exact(qi, qj, shift_of(xc, 0, g.L), shift_of(yz, 1, g.L), shift_of(yz, 2, g.L), g.sl2);
}

// Entries of atom i's row from runs [first, last) of the nine, walked by one lane
// (rows as build_rows', entry for entry); filed from entry cnt on, or only
// counted (nbr null).  Returns the next entry.  For atoms that lie thin: see
// build_rows_warp.
template <bool SLAB>
__device__ __forceinline__ int walk_own_runs(const RowGeom &g, const float4 *__restrict__ qloc,
                                          const double4 *__restrict__ q, const int *__restrict__ tab, int pc, int i,
                                          int first, int last, int cnt, int *__restrict__ nbr, int stride, int maxnb) {
  const float4 li = qloc[i];
  const int cx = pc & 2047, cy = (pc >> 11) & 2047, lz = (int)((unsigned)pc >> 22);
  const int cz = SLAB ? g.z0 + lz : lz;
  const int mx = g.ms[0] * kXSub, vbase = (cx - 1) * kXSub;
  const double qx = q[i].x;
  const double per_bin = kXSub / g.cs0;
  const float ubin = (float)((qx - (cx - 1) * g.cs0) * per_bin), per_binf = (float)per_bin;
#pragma unroll 1
  for (int r = first; r < last; r++) {
    const int dz = r / 3 - 1, dy = r % 3 - 1;
    const float gz = dz == 0 ? 0.f : (dz < 0 ? li.z : g.csz - li.z);
    const float gy = dy == 0 ? 0.f : (dy < 0 ? li.y : g.csy - li.y);
    const float g2 = fmaf(gy, gy, gz * gz);
    if (g2 > g.hi) continue;
    const float reach = sqrt_approx(g.hi - g2) * per_binf;
    const int lo = vbase + max((int)floorf(ubin - reach - 1e-3f), 0);
    const int hi = vbase + min((int)floorf(ubin + reach + 1e-3f) + 1, 3 * kXSub);
    int z = cz + dz, y = cy + dy, yz = 0;
    if (z < 0) { z += g.ms[2]; yz = 1 << 4; } else if (z >= g.ms[2]) { z -= g.ms[2]; yz = 2 << 4; }
    if (y < 0) { y += g.ms[1]; yz |= 1 << 2; } else if (y >= g.ms[1]) { y -= g.ms[1]; yz |= 2 << 2; }
    int blk = z;
    if (SLAB) {
      const int nl = lz + dz;
      blk = nl < 0 ? g.nzl : (nl >= g.nzl ? g.nzl + 1 : nl);
    }
    const int *xr = tab + (size_t)(blk * g.ms[1] + y) * (mx + 1);
    const float byf = (float)dy * g.csy - li.y, bzf = (float)dz * g.csz - li.z;
    // the run's pieces: through the -x face, inside the row, through the +x face
#pragma unroll 1
    for (int xc = lo < 0 ? 1 : 0; xc <= 2; xc = xc == 1 ? 0 : (xc == 0 && hi > mx ? 2 : 3)) {
      const int b0 = xc == 1 ? lo + mx : (xc == 2 ? 0 : max(lo, 0));
      const int b1 = xc == 1 ? mx : (xc == 2 ? hi - mx : min(hi, mx));
      const int code = yz | xc, need = strips_of(code);
      const float bx = (float)(shift_of(xc, 0, g.L) - qx);
      const int end = xr[b1];
      for (int j = xr[b0]; j < end; j++) {
        const float4 l = __ldg(qloc + j);
        const float ex = l.x + bx, ey = l.y + byf, ez = l.z + bzf;
        const float r2 = fmaf(ex, ex, fmaf(ey, ey, ez * ez));
        if (r2 > g.hi || (__float_as_int(l.w) & need) != need || (j == i && code == 0)) continue;
        if (r2 >= g.lo && !within_search_exact(q[i], q[j], shift_of(code, 0, g.L), shift_of(code, 1, g.L),
                                               shift_of(code, 2, g.L), g.sl2))
          continue;
        if (nbr && cnt < maxnb) nbr[(size_t)cnt * stride + i] = j;
        cnt++;
      }
    }
  }
  return cnt;
}

// Whether a warp's atoms lie thin: many x-rows of cells among them and few atoms
// a cell that has any (the rule's figures: build_rows_warp); shared: the lanes
// would walk their runs twice.  All lanes call.
__device__ __forceinline__ bool rows_lie_thin(int owner, int pc, bool active, bool all_pairs, bool shared) {
  constexpr unsigned kAll = 0xffffffffu;
  const int key = active ? pc : -1;  // no packed cell is -1
  const int before_key = __shfl_up_sync(kAll, key, 1), before_owner = __shfl_up_sync(kAll, owner, 1);
  const bool first = (threadIdx.x & 31) == 0 || owner != before_owner;
  const int atoms = __popc(__ballot_sync(kAll, active));
  const int cells = __popc(__ballot_sync(kAll, active && (first || key != before_key)));
  const int turns = __popc(__ballot_sync(kAll, active && (first || (unsigned)key >> 11 != (unsigned)before_key >> 11)));
  const bool others = __any_sync(kAll, (int)all_pairs);
  return !others && turns * (5 * cells + atoms) * 25 > (15 * cells + 27 * atoms) * (shared ? 8 : 5);
}

// build_rows_warp for atoms that lie thin.
template <bool SLAB, int SPLIT>
static __device__ __noinline__ int rows_alone(const RowGeom &g, const float4 *__restrict__ qloc,
                                              const double4 *__restrict__ q, const int *__restrict__ tab, int pc, int i,
                                              bool active, int (*counts)[32], int part, int *__restrict__ nbr, int stride,
                                              int maxnb) {
  const int lane = threadIdx.x & 31, first = part * (9 / SPLIT), last = first + 9 / SPLIT;
  int cnt = 0;
  for (int pass = SPLIT == 1 ? 1 : 0; pass < 2; pass++) {
    // pass 0 counts, so that the entries of the parts have their places
    const int at = cnt;
    if (active) cnt = walk_own_runs<SLAB>(g, qloc, q, tab, pc, i, first, last, cnt, pass ? nbr : nullptr, stride, maxnb);
    if (SPLIT > 1) {
      if (pass == 0) {
        counts[part][lane] = cnt - at;
        __syncthreads();
      }
      cnt = 0;
      for (int w = 0; w < (pass ? SPLIT : part); w++) cnt += counts[w][lane];
    }
  }
  const bool mine = part == 0 && active;
  if (mine)
    for (int k = cnt; (k & 3) && k < maxnb; k++) nbr[(size_t)k * stride + i] = i;
  return mine ? cnt : 0;
}

// Words a lane has room for: nine warps' rows fit a block's 48 KB.
__host__ __device__ constexpr int row_words(int split) { return split == 9 ? 14 : 16; }

// A lane's atom of a system narrower than three cells an axis (ensembles),
// whose partners are its system's other atoms [beg, end) in slot order, each
// through its minimum image (unique: L > 2 SearchLength).
struct SmallRow {
  bool on;
  int beg, end;
};

// The full Verlet rows of a warp's 32 atoms, one lane each: build_rows' rows
// entry for entry (the same 9 runs of slots in the same order, the same FP32
// prefilter, ghost-existence rule and exact test of the band).  All 32 lanes
// call; lanes without an atom pass active = false and any valid slot i.
// owner tells lanes of different systems apart.  With SMALL, lanes whose
// small.on is set take that row instead (active = false).
//
// SPLIT warps of a block (1, 3 or 9; the block has SPLIT warps when more than
// 1) share the same 32 atoms: warp `part` walks 9 / SPLIT of the runs, or that
// share of a small row, and the lanes' entries follow those of the parts
// before (counts: SPLIT x 32 shared words; all threads of the block call).  A
// single warp's walk is a chain of nine look-ups, loads and walks; with too few
// atoms to fill the chip that chain is the build's time.  Before its place is
// known (pass 0) a part keeps its words; one whose words do not fit walks again.  Returns the
// row length on the first part's lanes, 0 on the others.
//
// build_rows is bound by the L1 data path, its latency and its branches: every
// lane loads its own candidates (32 addresses a load, two thirds of the lanes
// busy), about 38 instructions a candidate, and files each partner with a
// scattered 4-byte store.  Here the lanes of one x-row of cells walk together
// (slots are in cell order, so a warp's atoms are of one x-row, or of a few,
// which take turns):
// - the run of slots that their windows cover is staged in shared memory by
//   coalesced loads, already moved through the x face where the run wraps,
//   with the images that the reference never builds put out of reach, so the
//   walk tests neither;
// - every lane walks as many candidates as the longest window, from its own
//   window's start: candidates outside the window lie out of reach in x and
//   fail the test, so the walk has no bound to test; four consecutive lanes of
//   one cell walk the union of their windows and read one address;
// - packed FP32 instructions take two candidates, and a candidate's verdict
//   is the sign of r^2 - hi shifted into a word: 8 instructions a candidate
//   and no branch.  Words with a candidate in the band (the sign of
//   (r^2 - hi)(r^2 - lo)) take the exact test for all their partners;
// - the words are turned into entries at the end, all lanes at the same
//   entry, so that 32 stores fill a 128-byte line of the list.
// On the 256,000-atom liquid the kernel takes 152 us against 235 us (300
// warp instructions an atom against 470, issue 65% against 57%); a rebuild of
// the 2.05M-atom liquid 1.13 ms against 2.05 ms.  64 registers (32 warps an
// SM, a few spills outside the walk) against 80: 1.13 and 1.17 ms; partners
// filed one by one in a shared-memory ring instead of words: 1.6 ms.
//
// Turns cost about the same however little there is to walk, so where atoms lie
// thin (many x-rows among 32, few candidates a run) every lane walks alone
// (rows_alone).  With T turns a warp and p atoms in a cell that has any, turns
// pay up to T (5 + p) = 3 + 5.4 p, and up to 1.6 times that T where the lanes
// alone would walk twice (count, then file) because warps share their atoms.  In
// turns, alone, and by build_rows with one lane an atom, us: 400,000 atoms, p =
// 1, T = 4.4: 226, 115, 101; p = 1.4, T = 1.5: 111, 102, 110; p = 2.6, T = 1.9:
// 133, 153, 153; T = 3: 199, 166, 173; p = 4.7, T = 2: 158, 218, 212; T = 3.2:
// 238, 233, 231; 30,000 atoms, nine warps, p = 1, T = 9: 44, 18, 16; p = 1.4, T =
// 3.9: 27, 23, 25; p = 2.6, T = 5.4: 36, 31, 37; T = 2.9: 25, 29, 35.
template <bool SLAB, int SPLIT, bool SMALL>
__device__ __forceinline__ int build_rows_warp(const RowGeom &g, const float4 *__restrict__ qloc,
                                               const double4 *__restrict__ q, const int *__restrict__ tab, int owner,
                                               int pc, int i, bool active, const SmallRow &small,
                                               WarpRows<row_words(SPLIT)> &sm,
                                               int (*counts)[32], int part, int *__restrict__ nbr, int stride,
                                               int maxnb) {
  static_assert(SPLIT == 1 || SPLIT == 3 || SPLIT == 9, "whole runs per warp");
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int kNoSlot = 1 << 30;  // above every slot; differences with slots stay in range
  const int lane = threadIdx.x & 31;
  if (rows_lie_thin(owner, pc, active, SMALL && small.on, SPLIT > 1))
    return rows_alone<SLAB, SPLIT>(g, qloc, q, tab, pc, i, active, counts, part, nbr, stride, maxnb);
  const float4 li = qloc[i];
  const int cx = pc & 2047;
  const int mx = g.ms[0] * kXSub, vbase = (cx - 1) * kXSub;
  // x_i in sub-bins from the lower face of cell cx - 1
  const double qx = q[i].x;
  const double per_bin = kXSub / g.cs0;
  const float ubin = (float)((qx - (cx - 1) * g.cs0) * per_bin), per_binf = (float)per_bin;
  const float2 bx = make_float2((float)(-qx), (float)(-qx));
  // lanes 4k .. 4k + 3 of one cell of one system
  const int key = active ? pc : -1;  // no packed cell is -1
  const int k1 = __shfl_xor_sync(kAll, key, 1), k2 = __shfl_xor_sync(kAll, key, 2);
  const int o1 = __shfl_xor_sync(kAll, owner, 1), o2 = __shfl_xor_sync(kAll, owner, 2);
  const int s1 = active && key == k1 && owner == o1, s2 = active && key == k2 && owner == o2;
  const int s12 = __shfl_xor_sync(kAll, s1, 2);  // the other pair's
  const bool quad = s1 && s2 && s12;
  int cnt = 0;             // the lane's next entry in the list
  int nw = 0, fresh = 0;   // the lane's words, and the partners in them
  bool filing = SPLIT == 1;  // the place of the lane's entries is known: full words may go to the list
  bool lost = false;         // words did not fit before that (warp-uniform)

  // the words' partners into the list
  auto flush = [&]() {
    const int mine = min(fresh, maxnb - cnt), n = __reduce_max_sync(kAll, mine);
    int *dst = nbr + (size_t)cnt * stride + i;
    const uint2 *w = &sm.word[0][lane];
    uint2 m = make_uint2(0u, 0u);
    for (int t = 0; t < n; t++, dst += stride) {
      if (t < mine) {
        if (m.x == 0u) {  // the next word (none is empty)
          m = *w;
          w += 32;
        }
        const int b = __clz(m.x);
        *dst = (int)m.y + b;
        m.x ^= 0x80000000u >> b;
      }
    }
    cnt += fresh;
    nw = fresh = 0;
  };
  // room for three more words a lane
  auto make_room = [&]() {
    if (__any_sync(kAll, nw > row_words(SPLIT) - 3)) {
      if (filing) {
        flush();
      } else {
        lost = true;
        nw = 0;
      }
    }
  };

  for (int pass = SPLIT == 1 ? 1 : 0; pass < 2; pass++) {
    if (SMALL && __any_sync(kAll, small.on)) {
      // an FP32 minimum image on the prefilter coordinates (box coordinates
      // here, the system being one cell) drops the far atoms: its band is 1e-4
      // SL^2 plus the rounding of coordinates up to the box lengths (each
      // difference is off by less than 4 u L, u = 2^-24, and 2 SL of that
      // reaches r^2)
      const float lx = (float)g.L[0], ly = (float)g.L[1], lz = (float)g.L[2];
      const float ix = 1.f / lx, iy = 1.f / ly, iz = 1.f / lz;
      const float wide = (float)(16.0 / 16777216.0 * (g.L[0] + g.L[1] + g.L[2]) * sqrt(g.sl2));
      const float hi = (float)(g.sl2 * 1.0001) + wide, lo = (float)(g.sl2 * 0.9999) - wide;
      const float round_big = 12582912.f;  // + and - it: the nearest whole number
      auto whole = [&](float x) { return __fsub_rn(__fadd_rn(x, round_big), round_big); };
      const int n = small.on ? small.end - small.beg : 0;
      const int share = ((n + SPLIT - 1) / SPLIT + 31) & ~31;  // whole words
      const int beg = small.beg + min(n, part * share), end = small.beg + min(n, (part + 1) * share);
      const int trip = __reduce_max_sync(kAll, small.on ? end - beg : 0);
      for (int k = 0; k < trip; k += 32) {
        const int first = beg + k;
        unsigned m = 0u;
#pragma unroll 1
        for (int u = 0; u < 32; u += 4) {
          float4 l[4];
#pragma unroll
          for (int c = 0; c < 4; c++) l[c] = __ldg(qloc + (small.on ? min(first + u + c, small.end - 1) : i));
#pragma unroll
          for (int c = 0; c < 4; c++) {
            float dx = l[c].x - li.x, dy = l[c].y - li.y, dz = l[c].z - li.z;
            dx = fmaf(-lx, whole(__fmul_rn(dx, ix)), dx);
            dy = fmaf(-ly, whole(__fmul_rn(dy, iy)), dy);
            dz = fmaf(-lz, whole(__fmul_rn(dz, iz)), dz);
            m = __funnelshift_l(__float_as_uint(fmaf(dx, dx, fmaf(dy, dy, dz * dz)) - hi), m, 1);
          }
        }
        const int have = small.on ? min(max(end - first, 0), 32) : 0, self = i - first;
        m = have == 0 ? 0u : m & (0xffffffffu << (32 - have));
        if (self >= 0 && self < 32) m &= ~(0x80000000u >> self);
        for (unsigned rest = m; rest;) {
          const int b = __clz(rest);
          rest ^= 0x80000000u >> b;
          const float4 l = __ldg(qloc + first + b);
          float dx = l.x - li.x, dy = l.y - li.y, dz = l.z - li.z;
          const float kx = whole(__fmul_rn(dx, ix)), ky = whole(__fmul_rn(dy, iy)), kz = whole(__fmul_rn(dz, iz));
          dx = fmaf(-lx, kx, dx);
          dy = fmaf(-ly, ky, dy);
          dz = fmaf(-lz, kz, dz);
          // image shift of the partner (shift_of's code) and the strips it
          // needs; atoms half a box apart, where FP32 may take the wrong image,
          // are further than SearchLength and so in the band
          int code = (kx > 0.f ? 1 : (kx < 0.f ? 2 : 0)) | (ky > 0.f ? 4 : (ky < 0.f ? 8 : 0)) |
                     (kz > 0.f ? 16 : (kz < 0.f ? 32 : 0));
          const bool band = fmaf(dx, dx, fmaf(dy, dy, dz * dz)) >= lo;
          if (band) {
            const double4 qi = q[i], qj = q[first + b];
            const double tx = qj.x - qi.x, ty = qj.y - qi.y, tz = qj.z - qi.z;
            code = (tx > 0.5 * g.L[0] ? 1 : (tx < -0.5 * g.L[0] ? 2 : 0)) |
                   (ty > 0.5 * g.L[1] ? 4 : (ty < -0.5 * g.L[1] ? 8 : 0)) |
                   (tz > 0.5 * g.L[2] ? 16 : (tz < -0.5 * g.L[2] ? 32 : 0));
          }
          const int need = strips_of(code);
          bool keep = (__float_as_int(l.w) & need) == need;
          if (keep && band)
            keep = within_search_exact(q[i], q[first + b], shift_of(code, 0, g.L), shift_of(code, 1, g.L),
                                       shift_of(code, 2, g.L), g.sl2);
          if (!keep) m ^= 0x80000000u >> b;
        }
        if (m) sm.word[nw++][lane] = make_uint2(m, (unsigned)first);
        fresh += __popc(m);
        make_room();
      }
    }
    // one turn per x-row of cells among the lanes' atoms
    for (unsigned left = __ballot_sync(kAll, active); left;) {
      const int lead = __ffs(left) - 1;
      const unsigned row = (unsigned)__shfl_sync(kAll, pc, lead) >> 11;
      const int row_owner = __shfl_sync(kAll, owner, lead);
      const bool on = active && ((unsigned)pc >> 11) == row && owner == row_owner;
      left &= ~__ballot_sync(kAll, on);
      // a candidate is kept when r^2 - hi < 0: never on the other lanes
      const float2 nhi = on ? make_float2(-g.hi, -g.hi) : make_float2(1.f, 1.f);
      const float2 nlo = on ? make_float2(-g.lo, -g.lo) : make_float2(1.f, 1.f);
      const int cy = (int)(row & 2047u), lz = (int)(row >> 11);
      // the row's geometry, from the turn's own lanes
      const int ms1 = __shfl_sync(kAll, g.ms[1], lead), ms2 = __shfl_sync(kAll, g.ms[2], lead);
      const int rmx = __shfl_sync(kAll, mx, lead);
      const float Lx = __shfl_sync(kAll, (float)g.L[0], lead);
      const int *rtab = (const int *)__shfl_sync(kAll, (unsigned long long)tab, lead);
      const int cz = SLAB ? g.z0 + lz : lz;  // global layer

#pragma unroll 1
      for (int r = part * (9 / SPLIT); r < (part + 1) * (9 / SPLIT); r++) {
        const int dz = r / 3 - 1, dy = r % 3 - 1;
        int z = cz + dz, y = cy + dy, yz = 0;  // yz: the run's image shift along y and z (shift_of's code)
        if (z < 0) { z += ms2; yz = 1 << 4; } else if (z >= ms2) { z -= ms2; yz = 2 << 4; }
        if (y < 0) { y += ms1; yz |= 1 << 2; } else if (y >= ms1) { y -= ms1; yz |= 2 << 2; }
        int blk = z;
        if (SLAB) {
          const int nl = lz + dz;
          blk = nl < 0 ? g.nzl : (nl >= g.nzl ? g.nzl + 1 : nl);
        }
        // the lane's window [wl, wh) in sub-bins of the 3 kXSub bins of cells
        // cx - 1 .. cx + 1 (build_rows' windows; empty when out of reach)
        const float gz = dz == 0 ? 0.f : (dz < 0 ? li.z : g.csz - li.z);
        const float gy = dy == 0 ? 0.f : (dy < 0 ? li.y : g.csy - li.y);
        const float g2 = fmaf(gy, gy, gz * gz);
        const float reach = sqrt_approx(fmaxf(g.hi - g2, 0.f)) * per_binf;
        const bool out = !on || g2 > g.hi;
        int wl = out ? 3 * kXSub : max((int)floorf(ubin - reach - 1e-3f), 0);
        int wh = out ? 0 : min((int)floorf(ubin + reach + 1e-3f) + 1, 3 * kXSub);
#pragma unroll
        for (int o = 1; o <= 2; o <<= 1) {
          const int lo2 = __shfl_xor_sync(kAll, wl, o), hi2 = __shfl_xor_sync(kAll, wh, o);
          if (quad) {
            wl = min(wl, lo2);
            wh = max(wh, hi2);
          }
        }
        // as slots [e0, e1) of the row continued through its x faces: slots
        // below x0 are those of the row's end (image shift -L), slots from x1
        // on those of its start (+L)
        const int *xr = rtab + (size_t)(blk * ms1 + y) * (rmx + 1);
        const int x0 = xr[0], x1 = xr[rmx], nrow = x1 - x0;
        int e0 = kNoSlot, e1 = -kNoSlot;
        if (wl < wh) {
          const int b0 = vbase + wl, b1 = vbase + wh;
          e0 = b0 < 0 ? xr[b0 + rmx] - nrow : xr[b0];
          e1 = b1 > rmx ? xr[b1 - rmx] + nrow : xr[b1];
          if (e0 >= e1) {
            e0 = kNoSlot;
            e1 = -kNoSlot;
          }
        }
        const int c0 = __reduce_min_sync(kAll, e0), c1 = __reduce_max_sync(kAll, e1);
        const bool wraps = c0 < x0 || c1 > x1, plain = !wraps && yz == 0;
        const float byf = (float)dy * g.csy - li.y, bzf = (float)dz * g.csz - li.z;
        const float2 by = make_float2(byf, byf), bz = make_float2(bzf, bzf);
        for (int c = c0; c < c1; c += kRunStage) {
          const int total = min(c1 - c, kRunStage);
          __syncwarp();  // the last walk has read the stage
          if (plain) {
            for (int t = 2 * lane; t < ((total + 3) & ~3); t += 64) {
              const float4 *p = qloc + c + t;
              float4 l0 = make_float4(1e18f, 0.f, 0.f, 0.f), l1 = l0;
              if (t < total) l0 = __ldg(p);
              if (t + 1 < total) l1 = __ldg(p + 1);
              sm.xy[t >> 1] = make_float4(l0.x, l1.x, l0.y, l1.y);
              sm.zz[t >> 1] = make_float2(l0.z, l1.z);
            }
          } else {
            for (int t = 2 * lane; t < ((total + 3) & ~3); t += 64) {
              float4 p[2];
#pragma unroll
              for (int u = 0; u < 2; u++) {
                p[u] = make_float4(1e18f, 0.f, 0.f, 0.f);
                if (t + u < total) {
                  int s = c + t + u, code = yz;
                  float sx = 0.f;
                  if (s < x0) {
                    s += nrow;
                    sx = -Lx;
                    code |= 1;
                  } else if (s >= x1) {
                    s -= nrow;
                    sx = Lx;
                    code |= 2;
                  }
                  const int need = strips_of(code);
                  p[u] = __ldg(qloc + s);
                  p[u].x = (__float_as_int(p[u].w) & need) == need ? p[u].x + sx : 1e18f;
                }
              }
              sm.xy[t >> 1] = make_float4(p[0].x, p[1].x, p[0].y, p[1].y);
              sm.zz[t >> 1] = make_float2(p[0].z, p[1].z);
            }
          }
          __syncwarp();
          // the lane's part of the stage, from an even candidate; the longest
          // one sets the warp's walk, and starts move down to end in the stage
          const int f0 = max(e0, c), f1 = min(e1, c + total);
          int st = f0 < f1 ? (f0 - c) & ~1 : 0;
          const int trip = (__reduce_max_sync(kAll, f0 < f1 ? f1 - c - st : 0) + 3) & ~3;
          st = min(st, ((total + 3) & ~3) - trip);
          const float4 *pxy = sm.xy + (st >> 1);
          const float2 *pzz = sm.zz + (st >> 1);
          for (int k = 0; k < trip; k += 32, st += 32) {
            unsigned m = 0u, band = 0u;
            const int kn = min(trip - k, 32);
#pragma unroll 2
            for (int u = 0; u < kn; u += 4, pxy += 2, pzz += 2) {
              const float4 a0 = pxy[0], a1 = pxy[1];
              const float2 z0 = pzz[0], z1 = pzz[1];
              const float2 ex0 = __fadd2_rn(make_float2(a0.x, a0.y), bx), ey0 = __fadd2_rn(make_float2(a0.z, a0.w), by);
              const float2 ex1 = __fadd2_rn(make_float2(a1.x, a1.y), bx), ey1 = __fadd2_rn(make_float2(a1.z, a1.w), by);
              const float2 ez0 = __fadd2_rn(z0, bz), ez1 = __fadd2_rn(z1, bz);
              const float2 r0 = __ffma2_rn(ex0, ex0, __ffma2_rn(ey0, ey0, __fmul2_rn(ez0, ez0)));
              const float2 r1 = __ffma2_rn(ex1, ex1, __ffma2_rn(ey1, ey1, __fmul2_rn(ez1, ez1)));
              const float2 h0 = __fadd2_rn(r0, nhi), h1 = __fadd2_rn(r1, nhi);
              const float2 b0 = __fmul2_rn(h0, __fadd2_rn(r0, nlo)), b1 = __fmul2_rn(h1, __fadd2_rn(r1, nlo));
              m = __funnelshift_l(__float_as_uint(h0.x), m, 1);
              m = __funnelshift_l(__float_as_uint(h0.y), m, 1);
              m = __funnelshift_l(__float_as_uint(h1.x), m, 1);
              m = __funnelshift_l(__float_as_uint(h1.y), m, 1);
              band |= __float_as_uint(b0.x) | __float_as_uint(b0.y);
              band |= __float_as_uint(b1.x) | __float_as_uint(b1.y);
            }
            m <<= 32 - kn;
            const int first = c + st;  // virtual slot of bit 31
            const int self = i - first;
            if (r == 4 && self >= 0 && self < 32) m &= ~(0x80000000u >> self);
            if (__any_sync(kAll, (int)(band & 0x80000000u))) {
              // some candidate of some lane in the band: exact test of that
              // lane's partners
              if (band >> 31)
                for (unsigned left2 = m; left2;) {
                  const int b = __clz(left2);
                  left2 &= ~(0x80000000u >> b);
                  int s = first + b;
                  s += s < x0 ? nrow : (s >= x1 ? -nrow : 0);
                  if (!band_test_row(g, q, i, s, cx, yz)) m &= ~(0x80000000u >> b);
                }
            }
            if (!wraps) {
              if (m) sm.word[nw++][lane] = make_uint2(m, (unsigned)first);
            } else {
              // the run wraps: the slots before, in and after the row in words
              // of their own
              const int h0 = x0 - first, h1 = x1 - first;
              const unsigned lt0 = h0 <= 0 ? 0u : (h0 >= 32 ? 0xffffffffu : ~(0xffffffffu >> h0));
              const unsigned lt1 = h1 <= 0 ? 0u : (h1 >= 32 ? 0xffffffffu : ~(0xffffffffu >> h1));
              if (m & lt0) sm.word[nw++][lane] = make_uint2(m & lt0, (unsigned)(first + nrow));
              if (m & lt1 & ~lt0) sm.word[nw++][lane] = make_uint2(m & lt1 & ~lt0, (unsigned)first);
              if (m & ~lt1) sm.word[nw++][lane] = make_uint2(m & ~lt1, (unsigned)(first - nrow));
            }
            fresh += __popc(m);
            make_room();
          }
        }
      }
    }
    if (SPLIT > 1 && pass == 0) {
      // the entries' places: after those of the parts before
      counts[part][lane] = fresh;
      __syncthreads();
      int before = 0, all = 0;
#pragma unroll
      for (int w = 0; w < SPLIT; w++) {
        if (w == part) before = all;
        all += counts[w][lane];
      }
      cnt = before;
      filing = true;
      if (!lost) {
        flush();
        cnt = all;
        break;
      }
      nw = fresh = 0;  // once more, filing as it goes
    } else {
      flush();
      if (SPLIT > 1) {
        cnt = 0;
#pragma unroll
        for (int w = 0; w < SPLIT; w++) cnt += counts[w][lane];
      }
    }
  }
  // padded with the atom itself to a multiple of 4
  const bool mine = part == 0 && (active || (SMALL && small.on));
  if (mine)
    for (int k = cnt; (k & 3) && k < maxnb; k++) nbr[(size_t)k * stride + i] = i;
  return mine ? cnt : 0;
}

// Stage offset of global slot j: the plan range whose atoms hold j (ranges
// are sorted by first cell, so by first atom).
__device__ __forceinline__ int stage_shift_atom(const int4 *plan, int npl, int j) {
  int lo = 0, hi = npl - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (plan[mid].z <= j) lo = mid;
    else hi = mid - 1;
  }
  return plan[lo].w - plan[lo].z;
}

// Longest row and list entries of a warp's atoms (cnt: a lane's row, 0 for
// none).  All lanes must call.
__device__ __forceinline__ void count_rows(Status *st, int cnt) {
  const int wmax = __reduce_max_sync(0xffffffffu, cnt);
  const int wsum = __reduce_add_sync(0xffffffffu, cnt);
  if ((threadIdx.x & 31) == 0 && wsum) {
    atomicMax(&st->max_row, wmax);
    atomicAdd((unsigned long long *)&st->list_entries, (unsigned long long)wsum);
  }
}

// Rebuild 6/6: full Verlet list, one thread per atom (build_rows_warp, which
// walks thin atoms' rows alone) or BTPA of them (build_rows; also the rows that carry stage indices).  Each
// candidate is first tested in FP32; only candidates whose FP32 r^2 falls in
// a band around SearchLength^2 -- wider than the FP32 error bound, which
// mdg_create derives from the box -- are decided by the exact FP64 test, so
// the pair set is the reference's bit for bit.  Rows are padded with the
// atom's own index to a multiple of 4.
template <int BLOCK, bool STAGE, bool SLAB = false, int BTPA = 1>
__global__ void __launch_bounds__(BLOCK, !STAGE && BTPA == 1 ? 1024 / BLOCK : 0) k_build(Arrays a, Box b, int n) {
  static_assert(!SLAB || (!STAGE && BTPA == 1), "slabs: one lane per atom, rows not staged");
  static_assert(!STAGE || BTPA == 1, "staged rows are built one lane per atom");
  const int t = blockIdx.x * BLOCK + threadIdx.x;
  const int i = t / BTPA, sub = t % BTPA;
  int cnt = 0;
  if (!STAGE && BTPA == 1) {
    __shared__ WarpRows<row_words(1)> rows[STAGE || BTPA > 1 ? 1 : BLOCK / 32];
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    // the lanes of a warp walk together: they agree on the error flag
    if (t - l < n && !warp_error(a.st)) {
      const bool active = i < n;
      const int ii = active ? i : n - 1;
      cnt = build_rows_warp<SLAB, 1, false>(row_geom(b), a.qloc, a.q, a.xsub, 0, a.cxyz[ii], ii, active, SmallRow{},
                                            rows[w], nullptr, 0, a.nbr, a.stride, a.maxnb);
      if (active) {
        a.nnbr[i] = min(cnt, a.maxnb);
        if (cnt > a.maxnb) atomicOr(&a.st->error, kErrCapacity);
      }
    }
    count_rows(a.st, cnt);
    return;
  }
  // STAGE: also the rows as stage indices (FP32-mixed staged force), from
  // the block's stage plan, see k_stage_plan
  __shared__ int4 plan[STAGE ? kStageRanges : 1];
  __shared__ int nplan;
  __shared__ int nstaged;
  int npl = -1, staged_atoms = 0;
  if (STAGE) {
    static_assert(!STAGE || BLOCK == kStageBlock, "stage plans are per kStageBlock atoms");
    if (threadIdx.x == 0) {
      const int m = a.nbr16 ? a.stage_n[blockIdx.x] : -1;
      nplan = (m > 0 && m <= kStageRanges) ? m : -1;
    }
    __syncthreads();
    npl = nplan;
    if ((int)threadIdx.x < npl) plan[threadIdx.x] = a.stage_rng[blockIdx.x * kStageRanges + threadIdx.x];
    __syncthreads();
    if (threadIdx.x == 0 && npl > 0) {
      const int4 last = plan[npl - 1];
      nstaged = last.w + a.cell_start[last.y] - last.z;
    }
    __syncthreads();
    // a stage index outside the stage would be a plan that misses a stencil
    // cell: flagged, and the entry points at the atom's own slot 0 instead
    staged_atoms = npl > 0 ? nstaged : 0;
  }
  unsigned g0 = 0u, g1 = 0u;  // the row's current group of four stage indices
  // one decision per atom: the lanes of an atom must walk its rows together
  // (their ballots name each other), so they all see its first lane's read
  // of the error flag
  int err = a.st->error;
  if (BTPA > 1) err = __shfl_sync(0xffffffffu, err, (threadIdx.x & 31) & ~(BTPA - 1));
  if (i < n && !err) {
    const int maxnb = a.maxnb, stride = a.stride;
    int *__restrict__ nbr = a.nbr;
    auto emit = [&](int j, int k) {
      if (k >= maxnb) return;
      nbr[(size_t)k * stride + i] = j;
      if (STAGE && npl > 0) {
        int v = j + stage_shift_atom(plan, npl, j);
        if (v < 0 || v >= staged_atoms) {
          atomicOr(&a.st->error, kErrStage);
          v = 0;
        }
        stage_entry(a.nbr16, stride, i, k, v, g0, g1);
      }
    };
    cnt = build_rows<BTPA>(b, a.qloc, a.q, a.mult, a.xsub, a.cxyz[i], i, emit);
    if (sub == 0) a.nnbr[i] = min(cnt, maxnb);
    if (cnt > maxnb) {
      if (sub == 0) atomicOr(&a.st->error, kErrCapacity);
    } else if (sub == 0) {
      int self = (STAGE && npl > 0) ? i + stage_shift(plan, npl, a.cell_tmp[i]) : 0;
      if (STAGE && npl > 0 && (self < 0 || self >= staged_atoms)) {
        atomicOr(&a.st->error, kErrStage);
        self = 0;
      }
      for (int k = cnt; k < ((cnt + 3) & ~3); k++) {
        nbr[(size_t)k * stride + i] = i;
        if (STAGE && npl > 0) stage_entry(a.nbr16, stride, i, k, self, g0, g1);
      }
    }
  }
  if (sub != 0) cnt = 0;  // the atom's row is counted once
  count_rows(a.st, cnt);
}

// The same for few atoms: SPLIT warps share every 32 of them.
template <int SPLIT>
__global__ void __launch_bounds__(SPLIT * 32, 27 / SPLIT) k_build_split(Arrays a, Box b, int n) {
  __shared__ WarpRows<row_words(SPLIT)> rows[SPLIT];
  __shared__ int counts[SPLIT][32];
  __shared__ int err;
  const int w = threadIdx.x >> 5, i = blockIdx.x * 32 + (threadIdx.x & 31);
  if (threadIdx.x == 0) err = *(volatile const int *)&a.st->error;
  __syncthreads();
  if (err) return;
  const bool active = i < n;
  const int ii = active ? i : n - 1;
  const int cnt = build_rows_warp<false, SPLIT, false>(row_geom(b), a.qloc, a.q, a.xsub, 0, a.cxyz[ii], ii, active,
                                                       SmallRow{}, rows[w], counts, w, a.nbr, a.stride, a.maxnb);
  if (active && w == 0) {
    a.nnbr[i] = min(cnt, a.maxnb);
    if (cnt > a.maxnb) atomicOr(&a.st->error, kErrCapacity);
  }
  count_rows(a.st, cnt);
}

// Warps that share 32 atoms' rows, so that few atoms fill the chip too: nine
// while that makes up to 64 warps a multiprocessor, then three up to 128 (its
// 32 warps at a time finish unevenly; more parts even them out).  A rebuild of
// the liquid with one / three / nine warps, us: 6,912 atoms - / 97 / 94 (109
// with eight lanes an atom), 32,000 - / 121 / 119 (144), 55,296 152 / 134 /
// 135, 108,000 175 / 167 / -, 157,216 205 / 196 / -, 340,736 298 / 302 / -.
// Three warps that would all walk alone (a system whose atoms lie thin on
// average) are one: 100,000 atoms, T = 20: 41 us with three, 35 with one.
inline int build_split(long long atoms, int sms, double per_cell, double per_row) {
  const long long warps = atoms / 32;
  if (warps * 9 <= 64LL * sms) return 9;
  const double p = fmax(per_cell / -expm1(-per_cell), 1.0);  // atoms in a cell that has any, scattered at random
  const double turns = 1.0 + 31.0 / fmax(per_row, 1.0);
  return warps * 3 <= 128LL * sms && turns * (5.0 + p) <= 3.0 + 5.4 * p ? 3 : 1;
}

// Before a build: clear the build counters.
static __global__ void k_build_begin(Arrays a) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  a.st->max_row = 0;
  a.st->list_entries = 0;
  a.st->total_images = 0;
}

// k_build_begin and the clear of the cell counts in one launch.
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) k_build_begin_clear(Arrays a, int ncell) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    a.st->max_row = 0;
    a.st->list_entries = 0;
    a.st->total_images = 0;
  }
  for (int c = blockIdx.x * BLOCK + threadIdx.x; c < ncell; c += gridDim.x * BLOCK) a.cell_count[c] = 0;
}

// The permuted state back into place (q, v, ids, types), one launch.
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) k_copy_back(Arrays a, int n) {
  const int i = blockIdx.x * BLOCK + threadIdx.x;
  if (i >= n || a.st->error) return;  // nothing was permuted: the atoms stay
  a.q[i] = a.q_tmp[i];
  a.v[i] = a.v_tmp[i];
  a.ids[i] = a.ids_tmp[i];
  a.type[i] = a.type_tmp[i];
}

// After a build: fresh skin budget (PairList::Init, src/pairlist.cc:10-23),
// counters, |v|^2 max for the next expiry test is untouched.
static __global__ void k_build_done(Arrays a, Box b) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  Status *st = a.st;
  if (st->error) return;
  st->budget = b.buffer_length;
  st->list_stale = 0;
  st->vlag_set = 0;  // fresh ghost copies, and v_lag is in the old slot order
  st->rebuilds++;
}

// Nose-Hoover: T = KE/N/1.5 from the blocks' partial sums, zeta += (T -
// T0)/tau^2 * dt/2 (ForceCalculator::HeatbathZeta, src/fcalculator.cc:979-985).
// All threads of one block; the sum has the same order for every block size.
template <int BLOCK>
__device__ __forceinline__ void add_zeta(const Arrays &a, const Box &b, int nblocks, int n, double aimed_t,
                                         double tau) {
  constexpr int kTerms = 1024;
  __shared__ double sm[kTerms];
  for (int t = threadIdx.x; t < kTerms; t += BLOCK) {
    double s = 0.0;
    for (int k = t; k < nblocks; k += kTerms) s += __ldcg(a.partials + k);  // other blocks' stores
    sm[t] = s;
  }
  for (int off = kTerms / 2; off >= 32; off >>= 1) {
    __syncthreads();
    for (int t = threadIdx.x; t < off; t += BLOCK) sm[t] += sm[t + off];
  }
  __syncthreads();
  if (threadIdx.x >= 32) return;
  double s = sm[threadIdx.x];
  for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
  if (threadIdx.x == 0 && !a.st->error) {
    const double t = s / (double)n / 1.5;
    const double t1 = (t - aimed_t) / (tau * tau);
    a.st->zeta += t1 * (b.dt * 0.5);
  }
}

// First zeta update of a Nose-Hoover step, made by k_drift's last block (of
// the kinetic energy that the drift leaves alone): ticket counts the blocks.
struct DriftZeta {
  int *ticket;
  double aimed_t, tau;
};

// q += v dt/2 (ForceCalculator::UpdatePositionHalf, src/fcalculator.cc:17-30);
// FIX also writes the packed copy that the force pass reads.  ZETA: with the
// kinetic energy partials (KineticEnergyObserver, src/observer.cc:4-15) and the
// zeta update in the pass; as kernels of their own they took 2.0 + 2.9 us of a
// 118,661-atom step besides the drift's 3.0.
template <int BLOCK, bool FIX, bool ZETA = false>
__global__ void __launch_bounds__(BLOCK) k_drift(Arrays a, Box b, int n, int track_vmax, DriftZeta zeta = DriftZeta{}) {
  const int i = blockIdx.x * BLOCK + threadIdx.x;
  double v2 = 0.0, ke[1] = {0.0};
  if (i < n && !a.st->error) {
    const double dt2 = b.dt * 0.5;
    double4 q = a.q[i];
    const double4 v = a.v[i];
    q.x = dadd(q.x, dmul(v.x, dt2));
    q.y = dadd(q.y, dmul(v.y, dt2));
    q.z = dadd(q.z, dmul(v.z, dt2));
    a.q[i] = q;
    if (FIX) pack_position(a.qfix, a.pz, i, q.x, q.y, q.z, b.L);
    if (track_vmax) {
      v2 = dadd(dadd(dmul(v.x, v.x), dmul(v.y, v.y)), dmul(v.z, v.z));
      if (!isfinite(v2) || !isfinite(q.x + q.y + q.z)) atomicOr(&a.st->error, kErrNonFinite);
    }
    if (ZETA)
      ke[0] = dadd(dadd(dmul(dmul(0.5, v.x), v.x), dmul(dmul(0.5, v.y), v.y)), dmul(dmul(0.5, v.z), v.z));
  }
  if (track_vmax) block_max_to<BLOCK>(&a.st->vmax2_bits, v2);
  if constexpr (ZETA) {
    __shared__ bool last;
    block_sum_to<BLOCK, 1>(ke, a.partials);
    if (threadIdx.x == 0) {
      __threadfence();  // the partial before the ticket
      last = atomicAdd(zeta.ticket, 1) == (int)gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    add_zeta<BLOCK>(a, b, gridDim.x, n, zeta.aimed_t, zeta.tau);
    if (threadIdx.x == 0) *zeta.ticket = 0;
  }
}

// ------------------------------------------------------------ executors
// The wall term of the reference's executors: the pair-force expression at
// distance d, each operation separately rounded (src/rankine.cc:78-82,
// src/burst.cc:91-93).
__device__ __forceinline__ double wall_df(double d, double c2, double dt) {
  const double r2 = dmul(d, d);
  const double r6 = dmul(dmul(r2, r2), r2);
  return dmul(dadd(ddiv(dsub(dmul(24.0, r6), 48.0), dmul(dmul(r6, r6), r2)), dmul(c2, 8.0)), dt);
}

// Before an executor pass: the pass re-takes the |v| maximum the next skin
// check reads (PairList::IsPairListExpired reads the momenta after it).
static __global__ void k_external_begin(Arrays a) {
  if (threadIdx.x == 0 && blockIdx.x == 0 && !a.st->error) {
    a.st->vmax2_bits = 0ull;
    if (a.v_lag) a.st->vlag_set = 1;  // k_external keeps the pre-pass velocities
  }
}

// One executor pass over all atoms: GravityImposer (src/phaseflow.cc:58-73),
// MyPiston (src/rankine.cc:55-97), ShellForce (src/burst.cc:67-99); block
// partial sums of the piston impulse into a.partials.
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) k_external(Arrays a, Box b, External x, int n) {
  const int i = blockIdx.x * BLOCK + threadIdx.x;
  double v2 = 0.0, imp = 0.0;
  if (i < n && !a.st->error) {
    const double4 q = a.q[i];
    double4 v = a.v[i];
    if (a.v_lag) a.v_lag[i] = v;  // the velocities the step's second drift used
    const double CL = b.rc;
    if (x.kind == 1) {
      const double g = dmul(x.strength, x.dt);
      if (x.axis == 0) v.x = dadd(v.x, g);
      else if (x.axis == 1) v.y = dadd(v.y, g);
      else v.z = dadd(v.z, g);
    } else if (x.kind == 2) {
      if (q.z < CL) {
        const double df = wall_df(q.z, b.c2, x.dt);
        v.z = dsub(v.z, dmul(df, q.z));
      }
      const double pos = a.st->ext_position;
      if (q.z > pos) {
        const double dz = dadd(dsub(pos, q.z), CL);
        const double df = wall_df(dz, b.c2, x.dt);
        v.z = dadd(v.z, dmul(df, dz));
        imp = -dmul(df, dz);
      }
    } else if (x.kind == 3) {
      const double dx = dsub(q.x, x.center[0]), dy = dsub(q.y, x.center[1]), dz = dsub(q.z, x.center[2]);
      const double r = dsub(x.radius, sqrt(dadd(dadd(dmul(dx, dx), dmul(dy, dy)), dmul(dz, dz))));
      if (!(dmul(r, r) > b.rc2)) {
        const double df = wall_df(r, b.c2, x.dt);
        v.x = dadd(v.x, dmul(df, dx));
        v.y = dadd(v.y, dmul(df, dy));
        v.z = dadd(v.z, dmul(df, dz));
      }
    }
    a.v[i] = v;
    v2 = dadd(dadd(dmul(v.x, v.x), dmul(v.y, v.y)), dmul(v.z, v.z));
  }
  block_max_to<BLOCK>(&a.st->vmax2_bits, v2);
  double s1[1] = {imp};
  block_sum_to<BLOCK, 1>(s1, a.partials);
}

// After a pass: impulse (fixed-order sum of the block partials) and the
// piston's move, as Rankine::Run moves it after each pass
// (src/rankine.cc:117-121).
static __global__ void k_external_done(Arrays a, External x, int nblocks) {
  if (threadIdx.x != 0 || blockIdx.x != 0 || a.st->error) return;
  double s = 0.0;
  for (int k = 0; k < nblocks; k++) s += a.partials[k];
  a.st->ext_impulse = s;
  if (x.kind == 2) a.st->ext_position = dsub(a.st->ext_position, x.velocity);
}

// Variables::ChangeScale (src/variables.cc:141-148): q *= alpha.
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) k_scale_positions(Arrays a, int n, double alpha) {
  const int i = blockIdx.x * BLOCK + threadIdx.x;
  if (i >= n) return;
  double4 q = a.q[i];
  q.x = dmul(q.x, alpha);
  q.y = dmul(q.y, alpha);
  q.z = dmul(q.z, alpha);
  a.q[i] = q;
}

// Atoms per cell of a regular grid (BubbleHist::AnalyseSub,
// src/cavitation.cc:117-146): index int((x - 0) / grid_size) per axis on the
// wrapped position, x fastest; counts kept in int, cast to unsigned char by
// the caller as the reference's counters wrap.
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) k_density(Arrays a, Box b, int n, double gsinv, int gx, int gy, int gz,
                                                   int *count) {
  const int i = blockIdx.x * BLOCK + threadIdx.x;
  if (i >= n) return;
  const double4 q = a.q[i];
  double x[3] = {q.x, q.y, q.z};
  int g[3] = {gx, gy, gz}, c[3];
  for (int d = 0; d < 3; d++) {
    x[d] -= b.L[d] * floor(x[d] / b.L[d]);
    const int k = (int)(x[d] * gsinv);
    c[d] = k < 0 ? 0 : (k >= g[d] ? g[d] - 1 : k);
  }
  atomicAdd(&count[c[0] + c[1] * gx + c[2] * gx * gy], 1);
}

// Packs q + v dt/2 (the coming step's first half drift) into out without
// moving atoms: the copy the fused NVE force pass reads.
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) k_pack_half(Arrays a, Box b, int n, int4 *out, double *out_z) {
  const int i = blockIdx.x * BLOCK + threadIdx.x;
  if (i >= n || a.st->error) return;
  const double4 q = a.q[i];
  const double4 v = a.v[i];
  const double dt2 = b.dt * 0.5;
  pack_position(out, out_z, i, dadd(q.x, dmul(v.x, dt2)), dadd(q.y, dmul(v.y, dt2)), dadd(q.z, dmul(v.z, dt2)), b.L);
}

// Writes the packed copy of q without moving atoms.
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) k_pack_fix(Arrays a, Box b, int n) {
  const int i = blockIdx.x * BLOCK + threadIdx.x;
  if (i >= n) return;
  const double4 q = a.q[i];
  pack_position(a.qfix, a.pz, i, q.x, q.y, q.z, b.L);
}

enum ForceMode { kKick = 0, kForceOut = 1, kKickNoseHoover = 2, kKickLangevin = 3 };

__device__ __forceinline__ void philox4x32_10(uint32_t c[4], uint32_t k0, uint32_t k1) {
#pragma unroll
  for (int r = 0; r < 10; r++) {
    const uint32_t lo0 = 0xD2511F53u * c[0], hi0 = __umulhi(0xD2511F53u, c[0]);
    const uint32_t lo1 = 0xCD9E8D57u * c[2], hi1 = __umulhi(0xCD9E8D57u, c[2]);
    const uint32_t n0 = hi1 ^ c[1] ^ k0, n2 = hi0 ^ c[3] ^ k1;
    c[0] = n0; c[1] = lo1; c[2] = n2; c[3] = lo0;
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
}

// Three standard normals for (atom id, step) from one Philox4x32-10 block and
// two Box-Muller pairs; the same stream as the oracle's ljo_langevin_normals.
__device__ __forceinline__ void langevin_normals(unsigned long long seed, uint32_t id,
                                                 unsigned long long step, double z[3]) {
  uint32_t c[4] = {id, (uint32_t)step, (uint32_t)(step >> 32), 0x4C414E47u};
  philox4x32_10(c, (uint32_t)seed, (uint32_t)(seed >> 32));
  const double scale = 2.3283064365386963e-10;
  const double u0 = ((double)c[0] + 0.5) * scale, u1 = ((double)c[1] + 0.5) * scale;
  const double u2 = ((double)c[2] + 0.5) * scale, u3 = ((double)c[3] + 0.5) * scale;
  const double twopi = 6.283185307179586;
  const double r0 = sqrt(-2.0 * log(u0)), r1 = sqrt(-2.0 * log(u2));
  z[0] = r0 * cos(twopi * u1);
  z[1] = r0 * sin(twopi * u1);
  z[2] = r1 * cos(twopi * u3);
}

struct Thermo {
  double gamma, noise_sd;      // Langevin friction and noise amplitude sqrt(2 gamma T / dt)
  unsigned long long seed;     // Langevin key; the counter is the device step count
};

// Per-atom epilogue shared by both precisions: apply the kick in the mode's
// form and emit the quantities the next kernels need.
template <int MODE>
__device__ __forceinline__ void finish_atom(Arrays &a, const Box &b, const Thermo &th, int i,
                                            double fx, double fy, double fz, double &v2,
                                            double &ke) {
  if (MODE == kForceOut) {
    a.v_tmp[i] = make_double4(fx, fy, fz, 0.0);
    return;
  }
  double4 v = a.v[i];
  double exp1 = 1.0;
  if (MODE == kKickNoseHoover) {
    exp1 = exp(-(b.dt * 0.5) * a.st->zeta);
    v.x = dmul(v.x, exp1); v.y = dmul(v.y, exp1); v.z = dmul(v.z, exp1);
  }
  v.x = dadd(v.x, fx); v.y = dadd(v.y, fy); v.z = dadd(v.z, fz);
  if (MODE == kKickNoseHoover) {
    v.x = dmul(v.x, exp1); v.y = dmul(v.y, exp1); v.z = dmul(v.z, exp1);
    ke = dadd(dadd(dmul(dmul(0.5, v.x), v.x), dmul(dmul(0.5, v.y), v.y)), dmul(dmul(0.5, v.z), v.z));
  }
  if (MODE == kKickLangevin) {
    // ForceCalculator::Langevin, src/fcalculator.cc:1001-1017
    double z[3];
    langevin_normals(th.seed, (uint32_t)a.ids[i], (unsigned long long)a.st->steps, z);
    const double dt = b.dt;
    v.x = dadd(v.x, dmul(dadd(dmul(-th.gamma, v.x), dmul(th.noise_sd, z[0])), dt));
    v.y = dadd(v.y, dmul(dadd(dmul(-th.gamma, v.y), dmul(th.noise_sd, z[1])), dt));
    v.z = dadd(v.z, dmul(dadd(dmul(-th.gamma, v.z), dmul(th.noise_sd, z[2])), dt));
    v2 = dadd(dadd(dmul(v.x, v.x), dmul(v.y, v.y)), dmul(v.z, v.z));
  }
  a.v[i] = v;
}

// The per-atom end of a force pass: the FP64 kick (fx, fy, fz) and, with
// DRIFT, the second half drift (DRIFT == 2 also this step's first half drift
// of the atom itself and the pack of the next step's first-drift position).
template <int MODE, int DRIFT>
__device__ __forceinline__ void kick_and_drift(Arrays &a, const Box &b, const Thermo &th, int i, double fx, double fy,
                                               double fz, int4 *next, double *next_z, double &v2, double &ke) {
  const double dt2 = b.dt * 0.5;
  double4 q;
  if (DRIFT) q = a.q[i];
  if (DRIFT == 2) {
    // this step's first half drift (the partners' copies already have it)
    const double4 v0 = a.v[i];
    q.x = dadd(q.x, dmul(v0.x, dt2));
    q.y = dadd(q.y, dmul(v0.y, dt2));
    q.z = dadd(q.z, dmul(v0.z, dt2));
  }
  finish_atom<MODE>(a, b, th, i, fx, fy, fz, v2, ke);
  if (DRIFT) {
    const double4 v = a.v[i];
    q.x = dadd(q.x, dmul(v.x, dt2));
    q.y = dadd(q.y, dmul(v.y, dt2));
    q.z = dadd(q.z, dmul(v.z, dt2));
    a.q[i] = q;
    v2 = dadd(dadd(dmul(v.x, v.x), dmul(v.y, v.y)), dmul(v.z, v.z));
    if (!isfinite(v2) || !isfinite(q.x + q.y + q.z)) atomicOr(&a.st->error, kErrNonFinite);
    // the next step's first half drift, packed for its force pass
    if (DRIFT == 2)
      pack_position(next, next_z, i, dadd(q.x, dmul(v.x, dt2)), dadd(q.y, dmul(v.y, dt2)), dadd(q.z, dmul(v.z, dt2)),
                    b.L);
  }
}

// ------------------------------------------------ FP64 rows, 1, 4 or 8 lanes per atom
// Whether some partner of an atom of (local) cell pc sat beyond a periodic face
// when the list was built: only atoms of the outermost cells have such
// partners, since a row reaches one cell out.  Says where to look for images
// first (pair_displacements), not that the others need none.
__device__ __forceinline__ bool row_wraps(const int ms[3], int z0, int pc) {
  const int cx = pc & 2047, cy = (pc >> 11) & 2047, cz = z0 + (int)((unsigned)pc >> 22);
  return cx == 0 || cx == ms[0] - 1 || cy == 0 || cy == ms[1] - 1 || cz == 0 || cz == ms[2] - 1;
}

// FP64 positions as the pair kernels gather them: the state's array, or a
// packed copy (pack_position).
struct PosState {
  const double4 *q;
  __device__ __forceinline__ double3 at(int j) const {
    const double4 p = q[j];
    return make_double3(p.x, p.y, p.z);
  }
};
struct PosSplit {
  const double2 *xy;
  const double *z;
  __device__ __forceinline__ double3 at(int j) const {
    const double2 p = xy[j];
    return make_double3(p.x, p.y, z[j]);
  }
};

// Blocks of 128 threads an SM that the FP64 pair kernels are held to (72
// registers, 28 warps).  The fused pass of the 2.05M-atom liquid: 0.464 ms with
// 7, 0.524 with 6, 0.476 with 8, 0.540 with 9; the serial branching loop over
// double4 positions that it replaced 0.600 ms and 0.054 ms of drift kernels.
constexpr int kFp64Blocks = 7;

// Lanes per atom of the FP64 pair kernels (every count gives the same sums,
// fp64_row).  Few atoms leave the chip to the latency of one row, many are
// bound by the pair arithmetic and the gathers.  Fused pass with 8, 4 and 1
// lanes: 4,000 atoms 7.5, 9.0, 24.6 us; 8,788 atoms 9.0, 9.6, 24.3; 16,384
// atoms 12.8, 11.2, 24.8; 55,296 atoms 33, 24, 28; 118,661 atoms (Nose-Hoover)
// 63, 45, 40.
inline int fp64_lanes(int n) { return n <= 10000 ? 8 : (n <= 65536 ? 4 : 1); }

// Sums over an atom's row in FP64, NS of them, in one fixed order whatever
// the number of lanes that share the row: the row falls into chunks of four
// entries (the last one shorter), each is summed in row order from 0, and the
// row's sum is ((0 + c0) + c1) + ...  With TPA lanes per atom (consecutive
// lanes; all lanes of the warp call together), lane `sub` sums chunks sub, sub
// + TPA, ..., and after each round every lane adds the round's chunk sums in
// chunk order, so every lane holds the sums.  pair(p, j, on, s) adds the terms
// of two partners j at p to s, in order; entries past the row's end arrive as
// the atom itself with on = false.  Two pairs are formed at once and without
// branches, so that their latencies overlap, and the next two partners'
// positions and the next chunk's entries are in flight meanwhile.
template <int TPA, int NS, typename Pos, typename Pair>
__device__ __forceinline__ void fp64_row(const Pos &q, const int *__restrict__ nbr, int stride, int nn, int i, int sub,
                                         double (&out)[NS], Pair pair) {
  const int chunks = (nn + 3) >> 2;
  const int rounds = TPA > 1 ? __reduce_max_sync(0xffffffffu, (chunks + TPA - 1) / TPA) : chunks;
  const int first = (threadIdx.x & 31) & ~(TPA - 1);
  const size_t hop = (size_t)(4 * TPA) * stride;
  const int *row = nbr + (size_t)(4 * sub) * stride + i;  // the chunk whose entries are loaded next
  int c = sub;                                            // its number
  // entries of a chunk (the row is padded to whole chunks)
  auto load = [&](int (&j)[4]) {
    const bool in = c < chunks;
#pragma unroll
    for (int u = 0; u < 4; u++) j[u] = in ? row[(size_t)u * stride] : i;
    row += hop;
    c += TPA;
  };
#pragma unroll
  for (int k = 0; k < NS; k++) out[k] = 0.0;
  int jc[4], jn[4];
  load(jc);
  double3 p[2] = {q.at(jc[0]), q.at(jc[1])};
  int k = 4 * sub;  // the chunk's first entry
#pragma unroll 1
  for (int r = 0; r < rounds; r++, k += 4 * TPA) {
    double s[NS];
#pragma unroll
    for (int m = 0; m < NS; m++) s[m] = 0.0;
    load(jn);
    const double3 p2[2] = {q.at(jc[2]), q.at(jc[3])};
    {
      const int j[2] = {jc[0], jc[1]};
      const bool on[2] = {k < nn, k + 1 < nn};
      pair(p, j, on, s);
    }
    p[0] = q.at(jn[0]);
    p[1] = q.at(jn[1]);
    {
      const int j[2] = {jc[2], jc[3]};
      const bool on[2] = {k + 2 < nn, k + 3 < nn};
      pair(p2, j, on, s);
    }
#pragma unroll
    for (int u = 0; u < 4; u++) jc[u] = jn[u];
#pragma unroll
    for (int l = 0; l < TPA; l++)
#pragma unroll
      for (int m = 0; m < NS; m++) out[m] += TPA > 1 ? __shfl_sync(0xffffffffu, s[m], first + l) : s[m];
  }
}

// Box edges as the FP64 pair terms need them; near_hi is the upper word of the
// shortest half edge.
struct Edges {
  const double *L, *hL;
  int near_hi;
};

__device__ __forceinline__ Edges edges_of(const double *L, const double *hL) {
  return Edges{L, hL, __double2hiint(fmin(fmin(hL[0], hL[1]), hL[2]))};
}

// Displacements from qi to the images of p[0] and p[1] that image_of takes.
// With WRAP (a warp with an atom of an outermost cell) the image is looked for
// at once.  Elsewhere partners are their own images, being nearer than half
// the shortest edge along every axis, unless an atom went far since the list
// was built -- the reference's skin check lets it while no other atom moves
// much -- or is not finite: the upper words of the differences tell, with
// integer instructions, and the image search is a branch.  A pass of the
// 2.05M-atom liquid takes 0.464 ms with the test and without it, 0.468 with no
// WRAP path; a 118,661-atom Nose-Hoover pass 40.2, 39.5 and 42.0 us.
template <bool WRAP>
__device__ __forceinline__ void pair_displacements(const Edges &e, const double3 &qi, const double3 (&p)[2],
                                                   double (&d)[2][3]) {
  if (!WRAP) {
    int far = 0;
#pragma unroll
    for (int u = 0; u < 2; u++) {
      d[u][0] = dsub(p[u].x, qi.x);
      d[u][1] = dsub(p[u].y, qi.y);
      d[u][2] = dsub(p[u].z, qi.z);
#pragma unroll
      for (int c = 0; c < 3; c++) far = max(far, __double2hiint(d[u][c]) & 0x7fffffff);
    }
    if (far < e.near_hi) return;
  }
#pragma unroll
  for (int u = 0; u < 2; u++) {
    d[u][0] = dsub(image_of(p[u].x, qi.x, e.L[0], e.hL[0]), qi.x);
    d[u][1] = dsub(image_of(p[u].y, qi.y, e.L[1], e.hL[1]), qi.y);
    d[u][2] = dsub(image_of(p[u].z, qi.z, e.L[2], e.hL[2]), qi.z);
  }
}

// FP64 force kick, TPA lanes per atom (BLOCK / TPA atoms per block).  Every
// pair term is the reference's (ForceCalculator::CalculateForceNext,
// src/fcalculator.cc:228-290): dx = image(q_j) - q_i, r2 = (dx*dx + dy*dy) +
// dz*dz, 0 if r2 > rc^2, r6 = (r2*r2)*r2, df = ((24 r6 - 48) /
// ((r6*r6)*r2) + 8 C2) * dt, term = df * dx, all separately rounded but for the
// division's last bit in some 10^-8 of pairs (quotient); and the summation order
// differs (fp64_row).
struct Fp64Pair {
  Edges e;
  double rc2, c2x8, dt;
  double3 qi;
};

template <bool WRAP>
__device__ __forceinline__ void lj_pairs_fp64(const Fp64Pair &f, const double3 (&p)[2], const bool (&on)[2],
                                              double (&s)[3]) {
  double d[2][3], df[2];
  pair_displacements<WRAP>(f.e, f.qi, p, d);
#pragma unroll
  for (int u = 0; u < 2; u++) {
    double r2 = dadd(dadd(dmul(d[u][0], d[u][0]), dmul(d[u][1], d[u][1])), dmul(d[u][2], d[u][2]));
    const bool in = on[u] && !(r2 > f.rc2);
    r2 = in ? r2 : 1.0;  // an ordinary operand for the division
    const double r6 = dmul(dmul(r2, r2), r2);
    df[u] = dmul(dadd(quotient(dsub(dmul(24.0, r6), 48.0), dmul(dmul(r6, r6), r2)), f.c2x8), f.dt);
    df[u] = in ? df[u] : 0.0;
  }
#pragma unroll
  for (int u = 0; u < 2; u++) {
    s[0] = dadd(s[0], dmul(df[u], d[u][0]));
    s[1] = dadd(s[1], dmul(df[u], d[u][1]));
    s[2] = dadd(s[2], dmul(df[u], d[u][2]));
  }
}

template <int TPA, typename Pos>
__device__ __forceinline__ void fp64_force_row(const Pos &q, const int *nbr, int stride, int nn, int i, int sub,
                                               const Fp64Pair &f, bool wraps, double (&s)[3]) {
  // one path for the whole warp
  if (__any_sync(0xffffffffu, (int)wraps))
    fp64_row<TPA>(q, nbr, stride, nn, i, sub, s,
                  [&](const double3 (&p)[2], const int (&)[2], const bool (&on)[2], double (&t)[3]) {
                    lj_pairs_fp64<true>(f, p, on, t);
                  });
  else
    fp64_row<TPA>(q, nbr, stride, nn, i, sub, s,
                  [&](const double3 (&p)[2], const int (&)[2], const bool (&on)[2], double (&t)[3]) {
                    lj_pairs_fp64<false>(f, p, on, t);
                  });
}

// DRIFT as in k_force_fp32 (the positions come from the packed copy `pos`,
// so moving q races with no other thread): 1 also makes the second half
// drift, 2 the whole NVE step, with the next step's first-drift positions
// packed into next, next_z.
template <int BLOCK, int MODE, int DRIFT, int TPA, typename Pos>
__global__ void __launch_bounds__(BLOCK, kFp64Blocks) k_force_fp64(Arrays a, Box b, int n, Thermo th, Pos pos, int4 *next,
                                                      double *next_z) {
  const int t = blockIdx.x * BLOCK + threadIdx.x;
  const int i = t / TPA, sub = t % TPA;
  double v2 = 0.0, ke = 0.0;
  if (DRIFT == 2 && t == 0 && !a.st->error) {
    // the step counter (k_step_done's work): nothing in this pass reads it
    a.st->steps++;
    a.st->sim_time += b.dt;
  }
  // the lanes of a warp walk together: they agree on the error flag
  const int err = warp_error(a.st);
  const bool on = i < n && !err;
  const int ii = i < n ? i : 0;
  const Fp64Pair f{edges_of(b.L, b.hL), b.rc2, b.c2 * 8.0, MODE == kForceOut ? 1.0 : b.dt, pos.at(ii)};
  double s[3];
  fp64_force_row<TPA>(pos, a.nbr, a.stride, on ? a.nnbr[ii] : 0, ii, sub, f,
                      on && row_wraps(b.ms, b.z0, a.cxyz[ii]), s);
  if (on && sub == 0) kick_and_drift<MODE, DRIFT>(a, b, th, i, s[0], s[1], s[2], next, next_z, v2, ke);
  if (MODE == kKickLangevin || DRIFT) warp_max_to(&a.st->vmax2_bits, v2);
  if (MODE == kKickNoseHoover) {
    double sum[1] = {ke};  // 0 on lanes other than the atom's first
    block_sum_to<BLOCK, 1>(sum, a.partials);
  }
}

// FP32 reciprocal on the special-function unit (rcp.approx.ftz.f32, PTX ISA):
// relative error at most one unit in the last place, well inside the FP32
// force error budget.
__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// One FP32 pair term from fixed-point positions: the wrapped int32
// difference is the minimum-image displacement in units of L/2^32.  r^2 = 0
// (the padding entries, the atom itself) contributes nothing: the unsigned
// compare of the float bits keeps 0 < r^2 <= rc^2 in one test.
__device__ __forceinline__ void lj_pair_fp32(const int4 &pi, const int4 &pj, float sx, float sy, float sz,
                                             unsigned rc2_bits, float c2x8, float &fx, float &fy, float &fz) {
  const float dx = (float)(pj.x - pi.x) * sx;
  const float dy = (float)(pj.y - pi.y) * sy;
  const float dz = (float)(pj.z - pi.z) * sz;
  const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
  const float ir2 = rcp_approx(r2);
  const float ir6 = ir2 * ir2 * ir2;
  float df = fmaf(ir2 * ir6, fmaf(-48.f, ir6, 24.f), c2x8);
  df = (__float_as_uint(r2) - 1u < rc2_bits) ? df : 0.f;
  fx = fmaf(df, dx, fx);
  fy = fmaf(df, dy, fy);
  fz = fmaf(df, dz, fz);
}

template <int MODE, int DRIFT>
__device__ __forceinline__ void fp32_finish(Arrays &a, const Box &b, const Thermo &th, int i, double Fx, double Fy,
                                            double Fz, int4 *qf_next, double &v2, double &ke) {
  const double dt = (MODE == kForceOut) ? 1.0 : b.dt;
  kick_and_drift<MODE, DRIFT>(a, b, th, i, Fx * dt, Fy * dt, Fz * dt, qf_next, nullptr, v2, ke);
}

// ------------------------------------------------ FP32 row sums, 1-4 lanes per atom
// The row sum of an atom in one fixed order whatever the number of lanes
// that share the row, so that 1, 2 or 4 lanes per atom give bit-identical
// forces.  The row's G groups of four entries (rows are padded to a
// multiple of 4 with masked self entries) form chunks of two groups (the
// last chunk may hold one): chunk c is groups 2c and 2c + 1, its eight pair
// terms summed in FP32 in entry order from 0; the row sum is the FP64 sum
// of the chunk sums in chunk order, S = ((0 + s_0) + s_1) + ...  With TPA
// lanes per atom, lane s sums chunks s, s + TPA, s + 2 TPA, ...; after each
// round of TPA chunks every lane of the atom reads the round's chunk sums
// from its neighbours (shuffles of FP32 values) and adds them in chunk
// order, so every lane holds S at the end.  Chunks past the row's end add
// +0.0, which leaves S unchanged (S starts at +0.0 and is never -0.0).

// A packed position.  LIVE: the copy changes while the kernel runs (the
// persistent pass), so the load is an ordinary one: the read-only path promises
// nothing for such data, and the compiler may move its loads across a barrier.
template <bool LIVE>
__device__ __forceinline__ int4 packed_at(const int4 *qf, int i) {
  return LIVE ? qf[i] : __ldg(qf + i);
}

// Partner positions of a lane's groups from the global fixed-point copy.
// The list entries of the group after the next are in flight while a group
// is summed (the list is the pass's one stream from HBM); with AHEAD the
// next group's positions are too (software pipeline: the gathers are the
// pass's long-latency loads; four more int4 registers).  Group -1 is none:
// its entries are the atom itself.
template <bool AHEAD = true, bool LIVE = false>
struct GlobalGroups {
  const int *row;  // nbr + atom
  int st;          // list stride
  const int4 *qf;
  int self;
  int n0, n1, n2, n3;      // entries of the current group (without AHEAD)
  int m0, m1, m2, m3;      // entries of the next group
  int4 c0, c1, c2, c3;     // positions of the current group (with AHEAD)
  __device__ __forceinline__ void load(int g, int &x0, int &x1, int &x2, int &x3) const {
    if (g < 0) {
      x0 = x1 = x2 = x3 = self;
      return;
    }
    const int *r = row + (size_t)(4 * g) * st;
    x0 = __ldg(r);
    x1 = __ldg(r + st);
    x2 = __ldg(r + 2 * st);
    x3 = __ldg(r + 3 * st);
  }
  // the lane's first two groups
  __device__ __forceinline__ void start(int ga, int gb) {
    load(ga, n0, n1, n2, n3);
    if (AHEAD) {
      c0 = packed_at<LIVE>(qf, n0);
      c1 = packed_at<LIVE>(qf, n1);
      c2 = packed_at<LIVE>(qf, n2);
      c3 = packed_at<LIVE>(qf, n3);
    }
    load(gb, m0, m1, m2, m3);
  }
  // positions of the lane's current group; the entries of the group after
  // the next (gnext) start loading, with AHEAD also the next group's positions
  __device__ __forceinline__ void take(int gnext, int4 &p0, int4 &p1, int4 &p2, int4 &p3) {
    if (AHEAD) {
      p0 = c0;
      p1 = c1;
      p2 = c2;
      p3 = c3;
      c0 = packed_at<LIVE>(qf, m0);
      c1 = packed_at<LIVE>(qf, m1);
      c2 = packed_at<LIVE>(qf, m2);
      c3 = packed_at<LIVE>(qf, m3);
    } else {
      p0 = packed_at<LIVE>(qf, n0);
      p1 = packed_at<LIVE>(qf, n1);
      p2 = packed_at<LIVE>(qf, n2);
      p3 = packed_at<LIVE>(qf, n3);
      n0 = m0;
      n1 = m1;
      n2 = m2;
      n3 = m3;
    }
    load(gnext, m0, m1, m2, m3);
  }
};

// The same from the block's stage in shared memory: one 8-byte load brings
// four 16-bit stage indices; indices outside the stage are flagged and read
// as entry 0.  One lane per atom.
__device__ __forceinline__ unsigned stage_index(unsigned v, unsigned nstage, bool &bad) {
  const bool out = v >= nstage;
  bad |= out;
  return out ? 0u : v;
}

struct StagedGroups {
  const uint2 *row;  // nbr16 + atom
  int st;
  const int4 *pos;   // the stage
  unsigned nstage;
  bool bad;
  uint2 g0, g1;
  __device__ __forceinline__ uint2 load(int g) const {
    return g < 0 ? make_uint2(0u, 0u) : __ldg(row + (size_t)g * st);
  }
  __device__ __forceinline__ void start(int ga, int gb) {
    bad = false;
    g0 = load(ga);
    g1 = load(gb);
  }
  __device__ __forceinline__ void take(int gnext, int4 &p0, int4 &p1, int4 &p2, int4 &p3) {
    p0 = pos[stage_index(g0.x & 0xffffu, nstage, bad)];
    p1 = pos[stage_index(g0.x >> 16, nstage, bad)];
    p2 = pos[stage_index(g0.y & 0xffffu, nstage, bad)];
    p3 = pos[stage_index(g0.y >> 16, nstage, bad)];
    g0 = g1;
    g1 = load(gnext);
  }
};

// Fixed-point scales and force constants of the FP32 pair term.
struct PairConst {
  float sx, sy, sz;
  unsigned rc2_bits;
  float c2x8;
};

__device__ __forceinline__ PairConst pair_const(const float fix_scale[3], float rc2f, float c2x8f) {
  return PairConst{fix_scale[0], fix_scale[1], fix_scale[2], __float_as_uint(rc2f), c2x8f};
}

__device__ __forceinline__ void lj_group_fp32(const int4 &pi, const int4 &p0, const int4 &p1, const int4 &p2,
                                              const int4 &p3, const PairConst &k, float &fx, float &fy, float &fz) {
  lj_pair_fp32(pi, p0, k.sx, k.sy, k.sz, k.rc2_bits, k.c2x8, fx, fy, fz);
  lj_pair_fp32(pi, p1, k.sx, k.sy, k.sz, k.rc2_bits, k.c2x8, fx, fy, fz);
  lj_pair_fp32(pi, p2, k.sx, k.sy, k.sz, k.rc2_bits, k.c2x8, fx, fy, fz);
  lj_pair_fp32(pi, p3, k.sx, k.sy, k.sz, k.rc2_bits, k.c2x8, fx, fy, fz);
}

// Row sum of an atom with G groups (see above), lane `sub` of TPA.  All TPA
// lanes of the atom must call together (they exchange chunk sums); every
// lane returns the row sum.
template <int TPA, typename Groups>
__device__ __forceinline__ void fp32_row(Groups &f, int G, int sub, const int4 &pi, const PairConst &k, double &Fx,
                                         double &Fy, double &Fz) {
  static_assert(TPA == 1 || TPA == 2 || TPA == 4, "1, 2 or 4 lanes per atom");
  double Sx = 0.0, Sy = 0.0, Sz = 0.0;
  float fx = 0.f, fy = 0.f, fz = 0.f;
  if (TPA == 1) {
    f.start(G > 0 ? 0 : -1, G > 1 ? 1 : -1);
    for (int g = 0; g < G; g++) {
      int4 p0, p1, p2, p3;
      f.take(g + 2 < G ? g + 2 : -1, p0, p1, p2, p3);
      lj_group_fp32(pi, p0, p1, p2, p3, k, fx, fy, fz);
      if (g & 1) {
        Sx += (double)fx;
        Sy += (double)fy;
        Sz += (double)fz;
        fx = fy = fz = 0.f;
      }
    }
    Sx += (double)fx;  // the last chunk when it holds one group (else +0)
    Sy += (double)fy;
    Sz += (double)fz;
  } else {
    const int lane = threadIdx.x & 31;
    const unsigned amask = ((1u << TPA) - 1u) << (lane & ~(TPA - 1));
    const int C = (G + 1) >> 1, R = (C + TPA - 1) / TPA;
    // the lane's m-th group: group 2c + (m & 1) of chunk c = sub + (m >> 1) TPA
    auto grp = [&](int m) {
      const int g = 2 * (sub + (m >> 1) * TPA) + (m & 1);
      return g < G ? g : -1;
    };
    f.start(grp(0), grp(1));
    for (int r = 0; r < R; r++) {
      const int ga = grp(2 * r), gb = grp(2 * r + 1);
      int4 p0, p1, p2, p3;
      fx = fy = fz = 0.f;
      f.take(grp(2 * r + 2), p0, p1, p2, p3);
      if (ga >= 0) lj_group_fp32(pi, p0, p1, p2, p3, k, fx, fy, fz);
      f.take(grp(2 * r + 3), p0, p1, p2, p3);
      if (gb >= 0) lj_group_fp32(pi, p0, p1, p2, p3, k, fx, fy, fz);
#pragma unroll
      for (int j = 0; j < TPA; j++) {
        Sx += (double)__shfl_sync(amask, fx, j, TPA);
        Sy += (double)__shfl_sync(amask, fy, j, TPA);
        Sz += (double)__shfl_sync(amask, fz, j, TPA);
      }
    }
  }
  Fx = Sx;
  Fy = Sy;
  Fz = Sz;
}

// fp32_row<1> over the global fixed-point copy in one plain loop (the same
// sums in the same order): rows are padded to a multiple of 4 with the atom
// itself, so the row is walked four partners at a time without masks, with
// the list entries of the next two groups always in flight.  Measured at
// 0.282 ms per fused pass on the 2.05M-atom liquid against 0.304 ms for
// fp32_row<1> over GlobalGroups (whose per-group selects the compiler
// schedules worse).
__device__ __forceinline__ void fp32_row_global(const int *nbr, int st, const int4 *qf, int i, const int4 &pi, int nn4,
                                                const PairConst &c, double &Fx, double &Fy, double &Fz) {
  const float sx = c.sx, sy = c.sy, sz = c.sz;
  const unsigned rc2_bits = c.rc2_bits;
  const float c2x8 = c.c2x8;
  const int *row = nbr + i;
  float fx = 0.f, fy = 0.f, fz = 0.f;
  int n0 = i, n1 = i, n2 = i, n3 = i;
  int m0 = i, m1 = i, m2 = i, m3 = i;
  if (nn4 > 0) {
    n0 = __ldg(row);
    n1 = __ldg(row + st);
    n2 = __ldg(row + 2 * st);
    n3 = __ldg(row + 3 * st);
  }
  if (nn4 > 4) {
    m0 = __ldg(row + 4 * st);
    m1 = __ldg(row + 5 * st);
    m2 = __ldg(row + 6 * st);
    m3 = __ldg(row + 7 * st);
  }
  Fx = Fy = Fz = 0.0;
  for (int k = 0; k < nn4; k += 4) {
    const int4 p0 = __ldg(qf + n0);
    const int4 p1 = __ldg(qf + n1);
    const int4 p2 = __ldg(qf + n2);
    const int4 p3 = __ldg(qf + n3);
    n0 = m0;
    n1 = m1;
    n2 = m2;
    n3 = m3;
    if (k + 8 < nn4) {
      const int *r = row + (size_t)(k + 8) * st;
      m0 = __ldg(r);
      m1 = __ldg(r + st);
      m2 = __ldg(r + 2 * st);
      m3 = __ldg(r + 3 * st);
    }
    lj_pair_fp32(pi, p0, sx, sy, sz, rc2_bits, c2x8, fx, fy, fz);
    lj_pair_fp32(pi, p1, sx, sy, sz, rc2_bits, c2x8, fx, fy, fz);
    lj_pair_fp32(pi, p2, sx, sy, sz, rc2_bits, c2x8, fx, fy, fz);
    lj_pair_fp32(pi, p3, sx, sy, sz, rc2_bits, c2x8, fx, fy, fz);
    if (k & 4) {  // the second group of a chunk
      Fx += (double)fx;
      Fy += (double)fy;
      Fz += (double)fz;
      fx = fy = fz = 0.f;
    }
  }
  Fx += (double)fx;  // the last chunk when it holds one group (else +0)
  Fy += (double)fy;
  Fz += (double)fz;
}

// Sum of one value per atom over a block's BLOCK / TPA atoms (consecutive
// atoms, TPA lanes each, the value on the atom's first lane), written to
// partials[blockIdx.x].  The tree is block_sum_to<BLOCK / TPA, 1>'s over
// one lane per atom whatever TPA is, so the sum does not depend on the lane
// count.  All threads of the block must call.
template <int BLOCK, int TPA>
__device__ __forceinline__ void atom_block_sum(double x, double *partials) {
  constexpr int ATOMS = BLOCK / TPA;
  static_assert(ATOMS % 32 == 0, "whole warps of atoms");
  __shared__ double per_atom[TPA > 1 ? ATOMS : 1];
  __shared__ double per_warp[ATOMS / 32];
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (TPA > 1) {
    if (threadIdx.x % TPA == 0) per_atom[threadIdx.x / TPA] = x;
    __syncthreads();
    x = threadIdx.x < ATOMS ? per_atom[threadIdx.x] : 0.0;
  }
  if (w < ATOMS / 32) {
    const double s = warp_sum(x);
    if (l == 0) per_warp[w] = s;
  }
  __syncthreads();
  if (w == 0) {
    double y = l < ATOMS / 32 ? per_warp[l] : 0.0;
    y = warp_sum(y);
    if (l == 0) partials[blockIdx.x] = y;
  }
}

// FP32-mixed force kick, TPA lanes per atom (BLOCK / TPA atoms per block).
// Displacements come from the fixed-point copy (no ghost atoms, no shift
// codes); the row sum is fp32_row's fixed-order sum and the kick is FP64
// (the atom's first lane).  With DRIFT the second half drift q += v dt/2 and the |v| maximum
// of the step are done in the same pass: this kernel reads only the
// fixed-point copy, so moving q here races with no other thread.  DRIFT == 2
// is the whole NVE step in one pass: qf holds every atom's position after
// this step's first half drift (packed by the previous step's pass, or by
// k_pack_half after a rebuild); the kernel applies that drift to its own
// atom, kicks, drifts again and packs the next step's first-drift position
// into qf_next (the other buffer, so no thread overwrites a copy that
// another still reads).  The arithmetic is the separate drift kernels',
// operation for operation.
template <int BLOCK, int MODE, int DRIFT, int TPA>
__global__ void __launch_bounds__(BLOCK) k_force_fp32(Arrays a, Box b, int n, Thermo th, const int4 *qf,
                                                      int4 *qf_next) {
  const int t = blockIdx.x * BLOCK + threadIdx.x;
  const int i = t / TPA, sub = t % TPA;
  double v2 = 0.0, ke = 0.0;
  if (DRIFT == 2 && MODE == kKick && t == 0 && !a.st->error) {
    // the step counter (k_step_done's work): nothing in this pass reads it
    a.st->steps++;
    a.st->sim_time += b.dt;
  }
  const int err = TPA > 1 ? warp_error(a.st) : a.st->error;
  if (i < n && !err) {
    const int4 pi = qf[i];
    double Fx, Fy, Fz;
    const PairConst k = pair_const(b.fix_scale, b.rc2f, b.c2x8f);
    if (TPA == 1) {
      fp32_row_global(a.nbr, a.stride, qf, i, pi, (a.nnbr[i] + 3) & ~3, k, Fx, Fy, Fz);
    } else {
      GlobalGroups<> f{a.nbr + i, a.stride, qf, i};
      fp32_row<TPA>(f, (a.nnbr[i] + 3) >> 2, sub, pi, k, Fx, Fy, Fz);
    }
    if (sub == 0) fp32_finish<MODE, DRIFT>(a, b, th, i, Fx, Fy, Fz, qf_next, v2, ke);
  }
  if (MODE == kKickLangevin || DRIFT) warp_max_to(&a.st->vmax2_bits, v2);
  if (MODE == kKickNoseHoover) atom_block_sum<BLOCK, TPA>(ke, a.partials);
}

// ---------------------------------------------- mbarrier and bulk copies
// (PTX ISA: mbarrier, cp.async.bulk; sm_90 and later)
__device__ __forceinline__ uint32_t smem_addr(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
               : "memory");
}

// Bulk copy of `bytes` (a multiple of 16, both addresses 16-byte aligned)
// from global to shared memory, completing on the mbarrier's transaction
// count.  A plain load: no multicast.
__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_addr(dst)),
      "l"(src), "r"(bytes), "r"(smem_addr(bar))
      : "memory");
}

// Waits for the mbarrier's phase `parity` to complete, for at most `limit`
// clock cycles; false if it gave up.  The test is the non-blocking
// mbarrier.test_wait (PTX ISA), polled with a short sleep, so that a short
// limit is kept to within a poll.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, long long limit) {
  const long long t0 = clock64();
  while (true) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(done)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    if (done) return true;
    if (clock64() - t0 > limit) return false;
    __nanosleep(20);
  }
}

// About one second at the B200's clocks: a stage copy takes microseconds.
constexpr long long kStageWaitCycles = 2000000000ll;

// The staged FP32-mixed pass: k_force_fp32 with the partners' positions read
// from the block's stage (k_stage_plan) in dynamic shared memory, which one
// thread fills with one bulk copy per plan range while the others wait on an
// mbarrier.  Blocks without a plan (-1) gather from global memory.  If the
// wait gives up (Box::stage_wait cycles, mdg_params.stage_wait_cycles), the
// block sets kErrTimeout, waits once more (up to kStageWaitCycles) for its
// copies in flight, and kicks no atom.
template <int BLOCK, int MODE, int DRIFT>
__global__ void __launch_bounds__(BLOCK) k_force_fp32_staged(Arrays a, Box b, int n, Thermo th, const int4 *qf,
                                                             int4 *qf_next) {
  extern __shared__ __align__(16) int4 pos[];
  __shared__ __align__(8) uint64_t bar;
  static_assert(BLOCK == kStageBlock, "stage plans are per kStageBlock atoms");
  const int i = blockIdx.x * BLOCK + threadIdx.x;
  double v2 = 0.0, ke = 0.0;
  if (DRIFT == 2 && MODE == kKick && i == 0 && !a.st->error) {
    a.st->steps++;
    a.st->sim_time += b.dt;
  }
  // thread 0 checks the plan against the stage and the atom count (a plan
  // left from an earlier layout is never copied) and fills the stage
  __shared__ int staged;
  __shared__ unsigned nstage;
  uint32_t total = 0;
  if (threadIdx.x == 0) {
    const int npl = a.stage_n[blockIdx.x];
    int use = npl > 0 && npl <= kStageRanges && !a.st->error;
    const int4 *plan = a.stage_rng + (size_t)blockIdx.x * kStageRanges;
    for (int r = 0; use && r < npl; r++) {
      const int4 pr = plan[r];
      if (pr.x < 0 || pr.y > b.ncell || pr.x >= pr.y) {
        use = 0;
        break;
      }
      const int cnt = a.cell_start[pr.y] - pr.z;
      if (cnt < 0 || pr.z < 0 || pr.z + cnt > n || pr.w != (int)total || pr.w + cnt > a.stage_cap) use = 0;
      // bulk copies start on 16-byte boundaries at both ends
      if (cnt > 0 && (((smem_addr(pos + pr.w) | (uint32_t)(uintptr_t)(qf + pr.z)) & 15u) != 0u)) use = 0;
      total += (uint32_t)cnt;
    }
    if (!use && npl > 0 && npl <= kStageRanges && !a.st->error) atomicOr(&a.st->error, kErrStage);
    if (use) mbar_init(&bar, 1);
    staged = use;
    nstage = use ? total : 0u;
  }
  __syncthreads();
  const bool use_stage = staged != 0;
  bool ok = true;
  if (use_stage) {
    if (threadIdx.x == 0) {
      const int npl = a.stage_n[blockIdx.x];
      const int4 *plan = a.stage_rng + (size_t)blockIdx.x * kStageRanges;
      mbar_arrive_expect_tx(&bar, total * (uint32_t)sizeof(int4));
      for (int r = 0; r < npl; r++) {
        const int4 pr = plan[r];
        const int cnt = a.cell_start[pr.y] - pr.z;
        if (cnt > 0) bulk_load(pos + pr.w, qf + pr.z, (uint32_t)cnt * (uint32_t)sizeof(int4), &bar);
      }
    }
    ok = mbar_wait(&bar, 0, b.stage_wait);
    if (!ok) {
      atomicOr(&a.st->error, kErrTimeout);
      mbar_wait(&bar, 0, kStageWaitCycles);
    }
  }
  if (ok && i < n && !a.st->error) {
    const int4 pi = qf[i];
    const int G = (a.nnbr[i] + 3) >> 2;
    const PairConst k = pair_const(b.fix_scale, b.rc2f, b.c2x8f);
    double Fx = 0.0, Fy = 0.0, Fz = 0.0;
    if (use_stage) {
      StagedGroups f{a.nbr16 + i, a.stride, pos, nstage};
      fp32_row<1>(f, G, 0, pi, k, Fx, Fy, Fz);
      if (f.bad) atomicOr(&a.st->error, kErrStage);
    } else {
      GlobalGroups<> f{a.nbr + i, a.stride, qf, i};
      fp32_row<1>(f, G, 0, pi, k, Fx, Fy, Fz);
    }
    fp32_finish<MODE, DRIFT>(a, b, th, i, Fx, Fy, Fz, qf_next, v2, ke);
  }
  if (MODE == kKickLangevin || DRIFT) warp_max_to(&a.st->vmax2_bits, v2);
  if (MODE == kKickNoseHoover) {
    double s[1] = {ke};
    block_sum_to<BLOCK, 1>(s, a.partials);
  }
}

// ------------------------------------------- persistent multi-step NVE pass
// Grid barrier for a cooperative launch (every block resident): a count of
// arrivals that only grows (cleared before the launch); each barrier waits for
// gridDim.x more.  (With arrivals by groups of 16 blocks, on lines of their
// own, a step took a microsecond longer.)  A block waits at most `limit` polls;
// one that gives up sets kErrTimeout and returns false, and the caller leaves
// its loop (so does every other block at its next barrier).  dr2: the largest
// squared displacement of a check, alternating between two slots.
struct GridBarrier {
  unsigned count;
  unsigned long long dr2[2];
};

__device__ __forceinline__ unsigned ld_acquire_gpu(const unsigned *p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Every block of the (cooperative, fully resident) grid arrives; false if
// this block gave up waiting after `limit` polls (kErrTimeout is set).  The
// block's writes before the barrier are visible to every block after it:
// a gpu-scope fence before the arrival, acquire loads while waiting.  goal:
// the arrivals so far, 0 at the launch.  max_to: where the maximum of the
// block's `warps` values goes with the arrival.
__device__ __forceinline__ bool grid_barrier(GridBarrier *g, Status *st, long long limit, unsigned &goal,
                                             unsigned long long *max_to = nullptr, const double *values = nullptr,
                                             int warps = 0) {
  __shared__ int ok;
  goal += gridDim.x;
  __syncthreads();
  if (threadIdx.x == 0) {
    ok = 1;
    if (max_to) {
      double m = values[0];
      for (int w = 1; w < warps; w++) m = fmax(m, values[w]);
      atomic_max_double_bits(max_to, m);
    }
    __threadfence();
    atomicAdd(&g->count, 1u);
    long long polls = 0;
    while ((int)(ld_acquire_gpu(&g->count) - goal) < 0) {
      if (++polls > limit) {
        atomicOr(&st->error, kErrTimeout);
        ok = 0;
        break;
      }
      __nanosleep(20);
    }
  }
  __syncthreads();
  return ok != 0;
}

// About a second of polling (a poll and a 20 ns sleep take some 60 ns): a
// step takes microseconds.
constexpr long long kBarrierPolls = 16000000ll;

// The expiry test of PairList::IsPairListExpired (k_expiry's arithmetic)
// for a step the persistent pass may take on its own: the list is current,
// the skin budget is positive and stays non-negative after this step's
// 2 vmax dt.  Only then is the budget spent and the |v| maximum cleared;
// otherwise nothing changes and the caller's ordinary step (k_expiry, the
// displacement check, the rebuild) takes this step.
__device__ __forceinline__ bool take_step_alone(Status *st, const Box &b) {
  if (st->error || st->list_stale || !(st->budget > 0.0)) return false;
  const double vmax = sqrt(__longlong_as_double((long long)st->vmax2_bits));
  if (skin_cost(vmax, b.dt) > b.buffer_length) return false;  // k_expiry reports the too-fast atom
  const double budget = dsub(st->budget, skin_cost(vmax, b.dt));
  if (budget < 0.0) return false;
  st->budget = budget;
  st->vmax2_bits = 0ull;
  st->vlag_set = 0;
  return true;
}

// The first two chunks (of eight entries) of a lane's share of its row, and
// the row's groups; entries past the end are the atom itself.
struct RowHead {
  int first[8], second[8];
  int groups;
};

template <int TPA>
__device__ __forceinline__ void row_chunk(const Arrays &a, int i, int groups, int c, int (&e)[8]) {
  const int *row = a.nbr + (size_t)(8 * c) * a.stride + i;
#pragma unroll
  for (int u = 0; u < 8; u++) e[u] = 2 * c + u / 4 < groups ? __ldg(row + (size_t)u * a.stride) : i;
}

template <int TPA>
__device__ __forceinline__ RowHead row_head(const Arrays &a, int i, int sub) {
  RowHead h;
  h.groups = (a.nnbr[i] + 3) >> 2;
  row_chunk<TPA>(a, i, h.groups, sub, h.first);
  row_chunk<TPA>(a, i, h.groups, sub + TPA, h.second);
  return h;
}

// fp32_row's sum (the same terms in the same order) with the next chunk's
// eight positions and the entries of the one after it in flight, and the row's
// head in registers.
template <int TPA>
__device__ __forceinline__ void fp32_row_deep(const Arrays &a, const int4 *qf, int i, int sub, const RowHead &h,
                                              const int4 &pi, const PairConst &k, double &Fx, double &Fy, double &Fz) {
  const int chunks = (h.groups + 1) >> 1, rounds = (chunks + TPA - 1) / TPA;
  const unsigned lane = threadIdx.x & 31, amask = ((1u << TPA) - 1u) << (lane & ~(TPA - 1));
  int4 p[8];
  int e[8];
#pragma unroll
  for (int u = 0; u < 8; u++) {
    p[u] = packed_at<true>(qf, h.first[u]);
    e[u] = h.second[u];
  }
  Fx = Fy = Fz = 0.0;
#pragma unroll 2
  for (int r = 0; r < rounds; r++) {
    int4 pn[8];
#pragma unroll
    for (int u = 0; u < 8; u++) pn[u] = packed_at<true>(qf, e[u]);
    row_chunk<TPA>(a, i, h.groups, sub + (r + 2) * TPA, e);
    float fx = 0.f, fy = 0.f, fz = 0.f;
#pragma unroll
    for (int u = 0; u < 8; u++) lj_pair_fp32(pi, p[u], k.sx, k.sy, k.sz, k.rc2_bits, k.c2x8, fx, fy, fz);
#pragma unroll
    for (int j = 0; j < TPA; j++) {
      Fx += (double)(TPA > 1 ? __shfl_sync(amask, fx, j, TPA) : fx);
      Fy += (double)(TPA > 1 ? __shfl_sync(amask, fy, j, TPA) : fy);
      Fz += (double)(TPA > 1 ? __shfl_sync(amask, fz, j, TPA) : fz);
    }
#pragma unroll
    for (int u = 0; u < 8; u++) p[u] = pn[u];
  }
}

// kick_and_drift<kKick, 2> on an atom in registers; returns |v|^2, and the
// packed position of the next step's first half drift.
__device__ __forceinline__ double step_atom(const Box &b, double4 &q, double4 &v, double fx, double fy, double fz,
                                            int4 *packed) {
  const double dt2 = b.dt * 0.5;
  q.x = dadd(q.x, dmul(v.x, dt2));
  q.y = dadd(q.y, dmul(v.y, dt2));
  q.z = dadd(q.z, dmul(v.z, dt2));
  v.x = dadd(v.x, fx);
  v.y = dadd(v.y, fy);
  v.z = dadd(v.z, fz);
  q.x = dadd(q.x, dmul(v.x, dt2));
  q.y = dadd(q.y, dmul(v.y, dt2));
  q.z = dadd(q.z, dmul(v.z, dt2));
  pack_position(packed, nullptr, 0, dadd(q.x, dmul(v.x, dt2)), dadd(q.y, dmul(v.y, dt2)), dadd(q.z, dmul(v.z, dt2)),
                b.L);
  return dadd(dadd(dmul(v.x, v.x), dmul(v.y, v.y)), dmul(v.z, v.z));
}

// FP32-mixed NVE steps in one cooperative launch, for systems small enough
// that per-step launch latency dominates: each step is the fused pass of
// k_force_fp32<.., kKick, 2, TPA> over all atoms (grid-stride) followed by
// one grid barrier.  Every decision of PairList::IsPairListExpired and
// CheckByDisplacement is a function of values every block holds or reads
// after a barrier, so every block takes it by itself:
// - the skin budget lives in a register (budget -= 2 vmax dt while
//   positive; a check once it is negative);
// - the step's |v| maximum comes from a ring of three slots (pass k fills
//   slot k % 3; block 0 clears slot k + 1 during step k, which no block
//   reads any more and none fills before the next barrier);
// - a displacement check runs as k_disp_max, k_disp_collect and
//   k_disp_pairs do it (copies dated `lag` back), three phases each ending
//   in a grid barrier, and every block reads the verdict (want_build) after
//   the last one; block 0 clears the check's counters after it (the next
//   check starts at least one barrier later) and want_build while the next
//   check's first phase runs.  The last two phases are left out when the
//   largest displacement makes no copy a candidate.
// The pass stops before the first step that needs a rebuild -- it marks the
// list stale, so the caller's ordinary step rebuilds without deciding again
// -- before a step whose atom is too fast (the caller's step reports it),
// or when the step count reaches Status::target_steps; block 0 then writes
// the budget, the |v| maximum, the counters and the buffer parity back.
// Errors raised inside the passes stop the work of later passes (they
// check the flag) and are reported by the caller; the decisions never read
// the flag, which a block may raise while another still decides.  The
// fixed-point buffer the next step reads comes from, and goes back to,
// Status::fix_parity (0: qf0, 1: qf1).  The arithmetic is k_force_fp32's
// and the decisions are the graph path's, so trajectories and counters
// equal the graph path's bit for bit.
//
// A step is a chain of latencies: the barrier, the row's gathers and the
// atom's update.  DEEP, for grids whose threads cover every atom's lanes, keeps
// each thread's atom and the head of its row in registers (128, four blocks an
// SM) between steps and walks the row with eight gathers in flight
// (fp32_row_deep).  Launches of 100 steps of the 32,000-atom gas-like liquid
// (rho 0.5) take 1.25 ms in all against 1.61 ms without, 5,324 atoms (rho 0.8)
// 0.99 against 1.35 ms.
template <int BLOCK, int TPA, bool DEEP>
__global__ void __launch_bounds__(BLOCK, DEEP ? 512 / BLOCK : 0) k_nve_persistent(Arrays a, Box b, int n, int4 *qf0, int4 *qf1, double lag,
                                                          GridBarrier *bar) {
  __shared__ volatile int found;
  __shared__ double values[BLOCK / 32];  // the warps' |v|^2 maxima (DEEP)
  const Thermo th{};
  const PairConst k = pair_const(b.fix_scale, b.rc2f, b.c2x8f);
  const long long nthreads = (long long)n * TPA;
  const long long stride = (long long)gridDim.x * BLOCK;
  const int gtid = blockIdx.x * BLOCK + threadIdx.x, gthreads = gridDim.x * BLOCK;
  Status *st = a.st;
  const bool lead = blockIdx.x == 0 && threadIdx.x == 0;
  // the values the decisions start from, read by every block before any is
  // written (the first barrier)
  int parity = *(volatile int *)&st->fix_parity;
  double budget = *(volatile double *)&st->budget;
  unsigned long long vmax2 = *(volatile unsigned long long *)&st->vmax2_bits;
  const long long steps0 = *(volatile long long *)&st->steps;
  const long long target = *(volatile long long *)&st->target_steps;
  const bool startable = !*(volatile int *)&st->error && !*(volatile int *)&st->list_stale;
  double sim_time = st->sim_time;  // block 0's copy
  unsigned goal = 0;
  // DEEP: this thread's lane of its atom
  const bool mine = DEEP && gtid < nthreads && startable;
  const int own = mine ? gtid / TPA : 0, lane = gtid % TPA;
  RowHead head{};
  double4 q0 = make_double4(0.0, 0.0, 0.0, 0.0), v0 = q0;
  int4 pown = make_int4(0, 0, 0, 0);
  if (mine) {
    q0 = a.q[own];
    v0 = a.v[own];
    pown = (parity ? qf1 : qf0)[own];
    head = row_head<TPA>(a, own, lane);
  }
  if (lead) {
    st->vmax2_ring[0] = st->vmax2_ring[1] = 0ull;
    st->dr2max_bits = 0ull;
    st->cand_weighted = 0;
    st->cand_n = 0;
  }
  if (!grid_barrier(bar, st, kBarrierPolls, goal)) return;
  bool stale = false, checked = false;
  long long taken = 0, checks = 0;
  for (;; taken++) {
    // 0: stop; 1: take the step; 2: check displacements first
    int g = 0;
    if (startable && steps0 + taken < target) {
      if (budget > 0.0) {
        const double cost = skin_cost(sqrt(__longlong_as_double((long long)vmax2)), b.dt);
        if (cost <= b.buffer_length) {  // else too fast: the caller's step reports it
          budget = dsub(budget, cost);
          g = budget < 0.0 ? 2 : 1;
        }
      } else {
        g = budget < 0.0 ? 2 : 1;
      }
    }
    checked = false;
    if (g == 2) {
      checks++;
      checked = true;
      if (lead) st->want_build = 0;
      double d2 = 0.0;
      for (int i = gtid; i < n; i += gthreads)
        for_each_copy(copy_view(a), b.L, i, lag, [&](int, double x) { d2 = fmax(d2, x); });
      unsigned long long *dr2 = &bar->dr2[checks & 1];
      block_max_to<BLOCK>(dr2, d2);
      if (!grid_barrier(bar, st, kBarrierPolls, goal)) break;
      const double dr2max = __longlong_as_double(*(volatile long long *)dr2);
      const double c = b.buffer_length - sqrt(dr2max);
      const double c_d2 = c * c;
      // every block has read the other slot (at the last check, before the
      // barrier above), and none fills it before the next barrier
      if (lead) bar->dr2[(checks + 1) & 1] = 0ull;
      if (dr2max > c_d2) {
        for (int i = gtid; i < n; i += gthreads)
          collect_copies(copy_view(a), b.L, i, lag, c_d2, &st->cand_weighted, &st->cand_n, a.cand,
                         b.check_list_length);
        if (!grid_barrier(bar, st, kBarrierPolls, goal)) break;
        if (threadIdx.x == 0) found = 0;
        __syncthreads();
        const long long tn = st->total_images;
        const int nl = (int)((tn > b.check_list_length) ? b.check_list_length : tn);
        if (*(volatile int *)&st->cand_weighted >= nl) {
          if (threadIdx.x == 0) found = 1;
        } else {
          const int l = min(*(volatile int *)&st->cand_n, b.check_list_length);
          candidate_pair_test_global<BLOCK>(copy_view(a), b.L, a.cand, l, lag, b.sl2, b.rc2, blockIdx.x, gridDim.x,
                                            &found);
        }
        __syncthreads();
        if (threadIdx.x == 0 && found) st->want_build = 1;
        if (!grid_barrier(bar, st, kBarrierPolls, goal)) break;
        stale = *(volatile int *)&st->want_build != 0;
      }  // else no copy is a candidate: the check has passed
      if (lead) {
        // the check is over: its counters are free for the next one
        st->cand_weighted = 0;
        st->cand_n = 0;
        st->vlag_set = 0;  // k_decide: the check has read the ghost copies
      }
      if (stale) break;  // a rebuild is left to the caller's ordinary step
    }
    if (g == 0) break;
    // the step: block 0 clears the ring slot step taken + 1 will fill
    if (lead) {
      st->vmax2_ring[(taken + 1) % 3] = 0ull;
      if (!checked) st->vlag_set = 0;  // expiry_decide's clear: no check reads the copies this step
      sim_time += b.dt;
    }
    const int4 *qf = parity ? qf1 : qf0;
    int4 *qf_next = parity ? qf0 : qf1;
    unsigned long long *ring = &st->vmax2_ring[taken % 3];
    if constexpr (DEEP) {
      const int err = *(volatile const int *)&st->error;  // read late: the gathers need not wait for it
      double v2 = 0.0;
      if (mine) {
        double Fx, Fy, Fz;
        fp32_row_deep<TPA>(a, qf, own, lane, head, pown, k, Fx, Fy, Fz);
        if (!err) {
          v2 = step_atom(b, q0, v0, Fx * b.dt, Fy * b.dt, Fz * b.dt, &pown);
          if (lane == 0) {
            a.q[own] = q0;
            a.v[own] = v0;
            qf_next[own] = pown;
            if (!isfinite(v2) || !isfinite(q0.x + q0.y + q0.z)) atomicOr(&st->error, kErrNonFinite);
          }
        }
      }
      v2 = warp_max(v2);
      if ((threadIdx.x & 31) == 0) values[threadIdx.x >> 5] = v2;
    } else {
      // warps walk whole warps of threads, so the lane shuffles stay converged
      for (long long base = (long long)blockIdx.x * BLOCK + (threadIdx.x & ~31); base < nthreads; base += stride) {
        const long long t = base + (threadIdx.x & 31);
        const int i = (int)(t / TPA), sub = (int)(t % TPA);
        const int err = warp_error(st);
        double v2 = 0.0, ke = 0.0;
        if (t < nthreads && !err) {
          const int4 pi = qf[i];
          double Fx, Fy, Fz;
          GlobalGroups<true, true> f{a.nbr + i, a.stride, qf, i};
          fp32_row<TPA>(f, (a.nnbr[i] + 3) >> 2, sub, pi, k, Fx, Fy, Fz);
          if (sub == 0) fp32_finish<kKick, 2>(a, b, th, i, Fx, Fy, Fz, qf_next, v2, ke);
        }
        warp_max_to(ring, v2);
      }
    }
    parity ^= 1;
    if (!grid_barrier(bar, st, kBarrierPolls, goal, DEEP ? ring : nullptr, values, BLOCK / 32)) {
      taken++;
      break;
    }
    vmax2 = *(volatile unsigned long long *)ring;
  }
  if (lead) {
    st->steps = steps0 + taken;
    st->sim_time = sim_time;
    st->budget = budget;
    // expiry_decide's clear at a step that stopped for a rebuild; else the
    // last pass's maximum, which the next decision reads
    st->vmax2_bits = checked && stale ? 0ull : vmax2;
    st->disp_checks += checks;
    if (stale) {
      st->list_stale = 1;
      st->want_build = 1;
    }
    st->fix_parity = parity;
    st->persistent_steps += taken;
  }
}

// The rebuild step of the persistent pipeline: queued after each persistent
// launch, it runs only when that launch stopped for a rebuild (a stale
// list, no error, steps left).  Then it takes expiry_decide's stale-list
// branch (want_build, the |v| maximum cleared) and the graph body rebuilds,
// packs buffer 0 and runs the fused step from it.
static __global__ void k_rebuild_guard(Arrays a, Box b, cudaGraphConditionalHandle h_run) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  Status *st = a.st;
  int run = !st->error && st->list_stale && st->steps < st->target_steps;
  if (run) {
    int disp = 0;
    run = expiry_decide(st, b, &disp) && !st->error;
  }
  cudaGraphSetConditional(h_run, run);
}

static __global__ void k_set_parity(Arrays a, int parity) {
  if (threadIdx.x == 0 && blockIdx.x == 0 && !a.st->error) a.st->fix_parity = parity;
}

// Start of a persistent pipeline run: the step count to stop at and the
// buffer the next fused step reads.
static __global__ void k_set_target(Arrays a, long long target, int parity) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  a.st->target_steps = target;
  a.st->fix_parity = parity;
}

// What a step's last kernel does besides its own work: counts the step and, in
// a graph, decides the next step's branch (expiry_in_graph).
struct StepEnd {
  int expiry;
  cudaGraphConditionalHandle h_any;
};

// One thread.
__device__ __forceinline__ void end_step(Status *st, const Box &b, const StepEnd &end) {
  if (!st->error) {
    st->steps++;
    st->sim_time += b.dt;
  }
  if (end.expiry) expiry_in_graph(st, b, end.h_any);
}

// The second zeta update of a Nose-Hoover step, and the step's end.
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) k_zeta(Arrays a, Box b, int nblocks, int n, double aimed_t, double tau,
                                                StepEnd end) {
  add_zeta<BLOCK>(a, b, nblocks, n, aimed_t, tau);
  if (threadIdx.x == 0) end_step(a.st, b, end);
}

// Observers: KE, PE, virial per atom over the full list, x 1/2 for pair sums
// (PotentialEnergyObserver / VirialObserver, src/observer.cc:17-79: each
// pair term formed as the reference forms it).  lag > 0 reproduces what the
// reference's observers see after a full NVE or Nose-Hoover step: a partner
// reached through the periodic boundary is a ghost copy refreshed after the
// first half drift (MDManager::SendBorderParticles, src/mdmanager.cc:165-167),
// i.e. the partner's position lag = dt/2 earlier, q_j - v_j dt/2.
// Energy and virial terms of the partners at p[0] and p[1] (t[0] and t[1],
// counted from both ends); WRAP as in lj_pairs_fp64.
template <bool WRAP>
__device__ __forceinline__ void observe_pairs(const Edges &box, double rc2, double c0, double c2, const double3 &qi,
                                              const double3 (&p)[2], const bool (&on)[2], double (&t)[2]) {
  double d[2][3], e[2], w[2];
  pair_displacements<WRAP>(box, qi, p, d);
#pragma unroll
  for (int u = 0; u < 2; u++) {
    double r2 = dadd(dadd(dmul(d[u][0], d[u][0]), dmul(d[u][1], d[u][1])), dmul(d[u][2], d[u][2]));
    const bool in = on[u] && !(r2 > rc2);
    r2 = in ? r2 : 1.0;
    const double r4 = dmul(r2, r2), r6 = dmul(r4, r2), r8 = dmul(r6, r2), r10 = dmul(r8, r2), r12 = dmul(r10, r2);
    e[u] = dmul(4.0, dadd(dadd(dsub(quotient(1.0, r12), quotient(1.0, r6)), dmul(c2, r2)), c0));
    w[u] = dmul(dadd(quotient(dsub(dmul(24.0, r6), 48.0), dmul(dmul(r6, r6), r2)), c2 * 8.0), r2);
    e[u] = in ? e[u] : 0.0;
    w[u] = in ? w[u] : 0.0;
  }
#pragma unroll
  for (int u = 0; u < 2; u++) {
    t[0] = dadd(t[0], e[u]);
    t[1] = dadd(t[1], w[u]);
  }
}

template <int BLOCK, int TPA>
__global__ void __launch_bounds__(BLOCK, kFp64Blocks) k_observe(Arrays a, Box b, int n, double lag) {
  const int tid = blockIdx.x * BLOCK + threadIdx.x;
  const int i = tid / TPA, sub = tid % TPA;
  const bool on = i < n;
  const int ii = on ? i : 0;
  const PosState pos{a.q};
  const double3 qi = pos.at(ii);
  const Edges box = edges_of(b.L, b.hL);
  const int nn = on ? a.nnbr[ii] : 0;
  double t[2];
  // a lagging copy is looked for like an image, and only a partner with one has it
  if (__any_sync(0xffffffffu, (int)(on && (lag > 0.0 || row_wraps(b.ms, b.z0, a.cxyz[ii]))))) {
    const double4 *vl = lag_velocities(a);
    fp64_row<TPA>(pos, a.nbr, a.stride, nn, ii, sub, t,
                  [&](const double3 (&p)[2], const int (&j)[2], const bool (&in)[2], double (&u)[2]) {
                    double3 qj[2] = {p[0], p[1]};
                    for (int k = 0; k < 2; k++) {
                      if (lag > 0.0 && (fabs(qj[k].x - qi.x) > b.hL[0] || fabs(qj[k].y - qi.y) > b.hL[1] ||
                                        fabs(qj[k].z - qi.z) > b.hL[2])) {
                        const double4 vj = vl[j[k]];
                        qj[k].x = dsub(qj[k].x, dmul(vj.x, lag));
                        qj[k].y = dsub(qj[k].y, dmul(vj.y, lag));
                        qj[k].z = dsub(qj[k].z, dmul(vj.z, lag));
                      }
                    }
                    observe_pairs<true>(box, b.rc2, b.c0, b.c2, qi, qj, in, u);
                  });
  } else {
    fp64_row<TPA>(pos, a.nbr, a.stride, nn, ii, sub, t,
                  [&](const double3 (&p)[2], const int (&)[2], const bool (&in)[2], double (&u)[2]) {
                    observe_pairs<false>(box, b.rc2, b.c0, b.c2, qi, p, in, u);
                  });
  }
  double s[3] = {0.0, 0.0, 0.0};
  if (on && sub == 0) {
    const double4 v = a.v[i];
    s[0] = dadd(dadd(dmul(dmul(0.5, v.x), v.x), dmul(dmul(0.5, v.y), v.y)), dmul(dmul(0.5, v.z), v.z));
    s[1] = 0.5 * t[0];
    s[2] = 0.5 * t[1];
  }
  block_sum_to<BLOCK, 3>(s, a.partials);
}

// Fixed-order final sum of NSUM-wide partials into out[0..NSUM).
template <int BLOCK, int NSUM>
__global__ void __launch_bounds__(BLOCK) k_final_sum(const double *partials, int nblocks, double *out) {
  __shared__ double sm[NSUM][BLOCK];
  for (int k = 0; k < NSUM; k++) {
    double s = 0.0;
    for (int b = threadIdx.x; b < nblocks; b += BLOCK) s += partials[(size_t)b * NSUM + k];
    sm[k][threadIdx.x] = s;
  }
  __syncthreads();
  for (int off = BLOCK / 2; off > 0; off >>= 1) {
    if (threadIdx.x < off)
      for (int k = 0; k < NSUM; k++) sm[k][threadIdx.x] += sm[k][threadIdx.x + off];
    __syncthreads();
  }
  if (threadIdx.x == 0)
    for (int k = 0; k < NSUM; k++) out[k] = sm[k][0];
}

// Directed list entries within the cut-off (the pairs whose force is
// evaluated), with the reference's r^2 test (src/fcalculator.cc:268), summed
// into counts[0]; counts[1] gets all list entries.
template <bool WRAP>
__device__ __forceinline__ void count_pairs(const Edges &box, double rc2, const double3 &qi, const double3 (&p)[2],
                                            const bool (&on)[2], double (&t)[1]) {
  double d[2][3];
  pair_displacements<WRAP>(box, qi, p, d);
#pragma unroll
  for (int u = 0; u < 2; u++) {
    const double r2 = dadd(dadd(dmul(d[u][0], d[u][0]), dmul(d[u][1], d[u][1])), dmul(d[u][2], d[u][2]));
    t[0] += on[u] && !(r2 > rc2) ? 1.0 : 0.0;
  }
}

template <int BLOCK, int TPA>
__global__ void __launch_bounds__(BLOCK, kFp64Blocks) k_count_pairs(Arrays a, Box b, int n,
                                                                    unsigned long long *counts) {
  const int tid = blockIdx.x * BLOCK + threadIdx.x;
  const int i = tid / TPA, sub = tid % TPA;
  const bool on = i < n;
  const int ii = on ? i : 0;
  const PosState pos{a.q};
  const double3 qi = pos.at(ii);
  const Edges box = edges_of(b.L, b.hL);
  const int nn = on ? a.nnbr[ii] : 0;
  double t[1];
  if (__any_sync(0xffffffffu, (int)(on && row_wraps(b.ms, b.z0, a.cxyz[ii]))))
    fp64_row<TPA>(pos, a.nbr, a.stride, nn, ii, sub, t,
                  [&](const double3 (&p)[2], const int (&)[2], const bool (&in)[2], double (&u)[1]) {
                    count_pairs<true>(box, b.rc2, qi, p, in, u);
                  });
  else
    fp64_row<TPA>(pos, a.nbr, a.stride, nn, ii, sub, t,
                  [&](const double3 (&p)[2], const int (&)[2], const bool (&in)[2], double (&u)[1]) {
                    count_pairs<false>(box, b.rc2, qi, p, in, u);
                  });
  const int ws = __reduce_add_sync(0xffffffffu, sub == 0 ? (int)t[0] : 0);
  const int ns = __reduce_add_sync(0xffffffffu, sub == 0 ? nn : 0);
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(&counts[0], (unsigned long long)ws);
    atomicAdd(&counts[1], (unsigned long long)ns);
  }
}

// End of step bookkeeping (MDManager::Calculate: s_time += TimeStep).
static __global__ void k_step_done(Arrays a, Box b, StepEnd end) {
  if (threadIdx.x == 0 && blockIdx.x == 0) end_step(a.st, b, end);
}

// Langevin alone (ForceCalculator::Langevin, src/fcalculator.cc:1001-1017),
// for callers that run the step piece by piece; the noise counter is the
// device step count, as in the fused kick.
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) k_langevin(Arrays a, Box b, int n, Thermo th) {
  const int i = blockIdx.x * BLOCK + threadIdx.x;
  if (i >= n || a.st->error) return;
  double4 v = a.v[i];
  double z[3];
  langevin_normals(th.seed, (uint32_t)a.ids[i], (unsigned long long)a.st->steps, z);
  const double dt = b.dt;
  v.x = dadd(v.x, dmul(dadd(dmul(-th.gamma, v.x), dmul(th.noise_sd, z[0])), dt));
  v.y = dadd(v.y, dmul(dadd(dmul(-th.gamma, v.y), dmul(th.noise_sd, z[1])), dt));
  v.z = dadd(v.z, dmul(dadd(dmul(-th.gamma, v.z), dmul(th.noise_sd, z[2])), dt));
  a.v[i] = v;
}

// HeatbathMomenta alone (src/fcalculator.cc:987-999).
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) k_scale_v(Arrays a, int n, double dt2) {
  const int i = blockIdx.x * BLOCK + threadIdx.x;
  if (i >= n) return;
  const double e = exp(-dt2 * a.st->zeta);
  double4 v = a.v[i];
  v.x = dmul(v.x, e); v.y = dmul(v.y, e); v.z = dmul(v.z, e);
  a.v[i] = v;
}

}  // namespace mdg
