// Kernels of the B200 force-and-integrate step.  Each kernel names the
// reference routine whose arithmetic it restates.  The file is compiled with
// --fmad=false, IEEE division and square root, so every REAL*4 expression is
// evaluated with the same roundings as gfortran -O2 on x86-64 (no FMA).
#pragma once
#include "ibg_common.cuh"

namespace ibg {

// ------------------------------------------------------------ precision policy
// FP32 path: REAL*4 geometry and table math, forces summed as 64-bit
// fixed-point integers (order independent, reproducible run to run).
// FP64 path: the same algorithm in double with double atomics.
template <typename R>
struct Prec;

template <>
struct Prec<float> {
  using pos_t = float4;
  using acc_t = unsigned long long;  // global accumulator element
  using reg_t = long long;           // per-thread partial sum
  static __device__ __forceinline__ reg_t q(float v, unsigned* err) {
    if (!(fabsf(v) < kFixMax)) {  // also catches NaN
      atomicOr(err, EB_FIXED);
      v = (v == v) ? copysignf(kFixMax, v) : 0.0f;
    }
    return __float2ll_rn(v * kFixScale);
  }
  static __device__ __forceinline__ void add(acc_t* p, reg_t v) { atomicAdd(p, (unsigned long long)v); }
  static __device__ __forceinline__ double get(acc_t v) { return (double)(long long)v * kFixInv; }
  static __device__ __forceinline__ reg_t from_double(double v, unsigned* err) {
    double s = v * 4294967296.0;
    if (!(fabs(s) < 9.2e18)) {
      atomicOr(err, EB_FIXED);
      s = (s == s) ? copysign(9.2e18, s) : 0.0;
    }
    return __double2ll_rn(s);
  }
  static __device__ __forceinline__ float tbits(int b) { return __int_as_float(b); }
  static __device__ __forceinline__ int bits(float w) { return __float_as_int(w); }
};

template <>
struct Prec<double> {
  using pos_t = double4;
  using acc_t = double;
  using reg_t = double;
  static __device__ __forceinline__ reg_t q(double v, unsigned*) { return v; }
  static __device__ __forceinline__ void add(acc_t* p, reg_t v) { atomicAdd(p, v); }
  static __device__ __forceinline__ double get(acc_t v) { return v; }
  static __device__ __forceinline__ reg_t from_double(double v, unsigned*) { return v; }
  static __device__ __forceinline__ double tbits(int b) { return __longlong_as_double((long long)b); }
  static __device__ __forceinline__ int bits(double w) { return (int)__double_as_longlong(w); }
};

__device__ __forceinline__ float r_round(float x) { return roundf(x); }
__device__ __forceinline__ double r_round(double x) { return round(x); }
__device__ __forceinline__ float r_sqrt(float x) { return sqrtf(x); }
__device__ __forceinline__ double r_sqrt(double x) { return sqrt(x); }
__device__ __forceinline__ float r_acos(float x) { return acosf(x); }
__device__ __forceinline__ double r_acos(double x) { return acos(x); }
__device__ __forceinline__ float r_abs(float x) { return fabsf(x); }
__device__ __forceinline__ double r_abs(double x) { return fabs(x); }

// Fortran INT: truncation; values outside the int range saturate.
template <typename R>
__device__ __forceinline__ int fint(R x) {
  if (!(x == x)) return INT_MIN;
  if (x >= (R)2147483647.0) return INT_MAX;
  if (x <= (R)-2147483647.0) return -INT_MAX;
  return (int)x;
}

template <typename R>
__device__ __forceinline__ void box_of(const Scalars* sc, R* b, R* bi, R* b2);
template <>
__device__ __forceinline__ void box_of<float>(const Scalars* sc, float* b, float* bi, float* b2) {
  for (int c = 0; c < 3; ++c) { b[c] = sc->boxf[c]; bi[c] = sc->boxinvf[c]; b2[c] = sc->box2f[c]; }
}
template <>
__device__ __forceinline__ void box_of<double>(const Scalars* sc, double* b, double* bi, double* b2) {
  for (int c = 0; c < 3; ++c) { b[c] = sc->box[c]; bi[c] = sc->boxinv[c]; b2[c] = sc->box2[c]; }
}

// ------------------------------------------------------------------ per step
// Fold into the primary box (SHIFT.f90:37-43): applied to all three
// components when any one lies outside [-L/2, L/2].
template <typename R>
__device__ __forceinline__ void fold3(R* r, const R* b2) {
  bool out = false;
#pragma unroll
  for (int c = 0; c < 3; ++c) out |= (r[c] > b2[c]) || (r[c] < -b2[c]);
  if (!out) return;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    R x = r[c] / b2[c];
    R sp = x - (R)2.0 * (R)fint(x / (R)2.0);
    r[c] = (sp - (R)2.0 * (R)fint(sp)) * b2[c];
  }
}

// A position as 32-bit fractions of the box per axis: round(x/L * 2^32)
// modulo 2^32, in FP64.  The wrapped difference of two of them, read as a
// signed integer, is the nearest-image displacement in units of L/2^32, exact
// to one unit (L/2^32: 3e-9 nm for a 12.6 nm box), whatever the particles'
// distance from the box centre.
__device__ __forceinline__ int4 box_fraction(const double* x, const double* boxinv, int w) {
  int q[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    double t = x[c] * boxinv[c];
    t -= floor(t + 0.5);
    q[c] = (int)(unsigned)(long long)llrint(t * 4294967296.0);
  }
  return make_int4(q[0], q[1], q[2], w);
}

struct PosArgs {
  Scalars* sc;
  int natoms, nvirta;
  int nupdate, nmts;
  const double* S;     // unwrapped positions (3,NITEMS), FP64 state
  double* Svs;         // VS rows of S (written for the FP64 path and output)
  const int* tbits;    // type | label<<16 per particle
  const int* gslot;    // slot*2 + list per particle
  void* pos4[2];       // per-list wrapped positions, slot order
  int4* posq[2];       // FP32 path: per-list positions as 32-bit fractions of the box, slot order
  const int* vcenter;  // VIRT_CENTER (0-based atom id or -1 for COM)
  const int* vnum;     // members per VS
  const int* vmem;     // members, [v*15 + k], 0-based
  const float* vmass;  // member masses per [v*15 + k]
  const float* vinv;   // VIRT_INVMASS per VS
  int com_carry;       // 1: the reference's centre-of-mass form (VIRTUAL_DEF.f90:31)
  // com_carry: per site the mass-weighted y and z member terms (R[32]: y at
  // 0..14, z at 16..30), then the x coordinates (R[nvirta]), then the member
  // counts (int[nvirta], -1 for a centre-atom site), for k_vsite_chain
  void* chain;
};

template <typename R>
struct ChainView {
  R* terms;
  R* xs;
  int* n;
  __device__ ChainView(const PosArgs& a)
      : terms((R*)a.chain), xs((R*)a.chain + 32 * (size_t)a.nvirta), n((int*)(xs + a.nvirta)) {}
};

// Bytes of the com_carry scratch for nvirta sites.
template <typename R>
constexpr size_t chain_bytes(long long nvirta) {
  return (size_t)nvirta * (33 * sizeof(R) + sizeof(int));
}

// A particle's wrapped position into its list's slot: the FP32/FP64 record
// with its type/label word, and on the FP32 path the 32-bit box fractions
// from the FP64 value sd.
template <typename R>
__device__ __forceinline__ void store_position(const PosArgs& a, const R* b2, const double* boxinv, int i, const R* s,
                                               const double* sd) {
  using PT = typename Prec<R>::pos_t;
  const int g = a.gslot[i];
  const int tb = a.tbits[i];
  R r[3] = {s[0], s[1], s[2]};
  fold3<R>(r, b2);
  PT p;
  p.x = r[0]; p.y = r[1]; p.z = r[2];
  p.w = Prec<R>::tbits(tb);
  ((PT*)a.pos4[g & 1])[g >> 1] = p;
  if (a.posq[g & 1]) a.posq[g & 1][g >> 1] = box_fraction(sd, boxinv, tb);
}

// SHIFT.f90:33-45 for atoms and VIRTUAL_DEF.f90:19-47 for virtual sites
// (centre-of-mass sums with all three components reset per site, or the
// reference's form, where only the x sum is reset: com_carry).
// begin: when set, block 0 first starts the step: it advances the step
// counter and sets this step's flags, or marks the step skipped when the run
// aborted.  A system that has run its last step (done) is left as it is, so
// its virtual-site rows keep the values of its last step.
template <typename R, bool B>
__global__ void k_positions(__grid_constant__ const PosArgs a0, const PosArgs* const* tab, const BlockMap bm,
                            int begin) {
  using PT = typename Prec<R>::pos_t;
  pdl_wait();
  pdl_trigger();
  const Blk bk = blk<B>(bm);
  const PosArgs& a = B ? *tab[bk.sys] : a0;
  Scalars* sc = a.sc;
  if (sc->done) {
    if (begin && bk.b == 0 && threadIdx.x == 0) sc->skip = 1;
    return;
  }
  if (begin && bk.b == 0 && threadIdx.x == 0) {
    if (sc->abort) {
      sc->skip = 1;
    } else {
      sc->skip = 0;
      for (int q = 0; q < 4; ++q) sc->work[q] = 0u;
      const int st = ++sc->step;
      sc->rebuild = (st % a.nupdate) == 0;
      sc->mts_m = a.nmts > 0 ? st % (3 + a.nmts) : -1;
      sc->miu = 1.0;
    }
  }
  R b[3], bi[3], b2[3];
  box_of<R>(sc, b, bi, b2);
  const double boxinv[3] = {sc->boxinv[0], sc->boxinv[1], sc->boxinv[2]};
  // sd: the position in FP64 for the fixed-point copy (FP32 path).  The slot
  // and label are loaded before the first store (the arrays may alias as far
  // as the compiler knows, and a load after a store would wait for it).
  auto store = [&](int i, const R* s, const double* sd) { store_position<R>(a, b2, boxinv, i, s, sd); };
  for (int i = bk.b * blockDim.x + threadIdx.x; i < a.natoms; i += bk.g * blockDim.x) {
    R s[3];
    double sd[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      sd[c] = a.S[3 * (size_t)i + c];
      s[c] = (R)sd[c];
    }
    store(i, s, sd);
  }
  const int hl = threadIdx.x & 15;
  // VIRTUAL_DEF.f90:30-39 with all three sums reset per site: 16 lanes per
  // site (half a warp), lane k holding member k's mass-weighted position; the
  // sum runs over the members in order (0 + p0 + p1 + ...), as the
  // reference's loop does.  The loop over sites is uniform within a warp, so
  // its shuffles see all 32 lanes.  In the reference's form (com_carry) only
  // the x sum is reset per site (:31): the x coordinate is formed here, and
  // the y and z member terms go to the chain scratch, whose sums
  // k_vsite_chain runs on from site to site.
  const ChainView<R> cv(a);
  const int w0 = (bk.b * blockDim.x + threadIdx.x) >> 5, nw = (bk.g * blockDim.x) >> 5;
  for (int w = w0; 2 * w < a.nvirta; w += nw) {
    const int v = 2 * w + ((threadIdx.x >> 4) & 1);
    const bool valid = v < a.nvirta;
    const int ctr = valid ? a.vcenter[v] : 0;
    const int nm = valid && ctr < 0 ? a.vnum[v] : 0;
    R pm[3] = {0, 0, 0};
    if (hl < nm) {
      const int m = a.vmem[v * 15 + hl];
      const R mm = (R)a.vmass[v * 15 + hl];
#pragma unroll
      for (int c = 0; c < 3; ++c) pm[c] = mm * (R)a.S[3 * (size_t)m + c];
    }
    if (a.com_carry && hl < nm) {
      cv.terms[32 * (size_t)v + hl] = pm[1];
      cv.terms[32 * (size_t)v + 16 + hl] = pm[2];
    }
    R acc[3] = {0, 0, 0};
#pragma unroll
    for (int q = 0; q < 15; ++q) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const R x = __shfl_sync(0xffffffffu, pm[c], q, 16);
        if (q < nm) acc[c] = acc[c] + x;
      }
    }
    if (!valid || hl != 0) continue;
    if (a.com_carry) {
      cv.n[v] = ctr >= 0 ? -1 : nm;  // -1: a centre-atom site, outside the sums
      if (ctr < 0) {  // finished by k_vsite_chain
        cv.xs[v] = acc[0] * (R)a.vinv[v];
        continue;
      }
    }
    R s[3];
    if (ctr >= 0) {
#pragma unroll
      for (int c = 0; c < 3; ++c) s[c] = (R)a.S[3 * (size_t)ctr + c];
    } else {
      const R inv = (R)a.vinv[v];
#pragma unroll
      for (int c = 0; c < 3; ++c) s[c] = acc[c] * inv;
    }
    double sd[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      sd[c] = (double)s[c];
      a.Svs[3 * (size_t)v + c] = sd[c];
    }
    store(a.natoms + v, s, sd);
  }
}

// VIRTUAL_DEF.f90:30-39 as the reference runs it (com_carry): SUMTOTXYZ(2)
// and (3) are not reset before a centre-of-mass site (only (1) is, :31), so
// the y and z sums run on from one such site to the next, from zero at the
// start of the pass.  k_positions has formed each site's x coordinate and its
// mass-weighted y and z member terms; one block per system adds the terms in
// the reference's order.  The sites go through shared memory in chunks, two
// buffers: thread 0 runs the sums over one chunk while warps 1..7 load the
// next and finish the one before (the sums times VIRT_INVMASS, the FP64 row
// and the list record).
// A row of 32 values from shared memory in 16-byte loads issued back to back
// (asm volatile keeps them together, ahead of the arithmetic that uses them).
__device__ __forceinline__ void lds_row(float* t, const float* row) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(row);
#pragma unroll
  for (int k = 0; k < 8; ++k)
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(t[4 * k]), "=f"(t[4 * k + 1]), "=f"(t[4 * k + 2]), "=f"(t[4 * k + 3])
                 : "r"(a + 16 * k));
}
__device__ __forceinline__ void lds_row(double* t, const double* row) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(row);
#pragma unroll
  for (int k = 0; k < 16; ++k)
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(t[2 * k]), "=d"(t[2 * k + 1]) : "r"(a + 16 * k));
}

template <typename R, bool B>
__global__ void __launch_bounds__(256) k_vsite_chain(__grid_constant__ const PosArgs a0, const PosArgs* const* tab,
                                                     const BlockMap bm) {
  constexpr int kC = sizeof(R) == 4 ? 128 : 64;  // sites per chunk
  __shared__ __align__(16) R s_t[2][kC][32];
  __shared__ int s_n[2][kC];
  __shared__ R s_c[2][kC][2];
  const Blk bk = blk<B>(bm);
  const PosArgs& a = B ? *tab[bk.sys] : a0;
  Scalars* sc = a.sc;
  if (!a.com_carry || bk.b != 0 || sc->done) return;
  const ChainView<R> cv(a);
  R b[3], bi[3], b2[3];
  box_of<R>(sc, b, bi, b2);
  const double boxinv[3] = {sc->boxinv[0], sc->boxinv[1], sc->boxinv[2]};
  const int nv = a.nvirta;
  // chunk c0 into buffer q, by the threads from t0 on
  auto load = [&](int c0, int q, int t0) {
    const int nc = min(kC, nv - c0);
    for (int k = (int)threadIdx.x - t0; k < nc * 32; k += (int)blockDim.x - t0)
      s_t[q][k >> 5][k & 31] = cv.terms[32 * (size_t)c0 + k];
    for (int k = (int)threadIdx.x - t0; k < nc; k += (int)blockDim.x - t0) s_n[q][k] = cv.n[c0 + k];
  };
  // the sites of chunk c0 from the sums in s_c[q], by the threads from t0 on:
  // the sums times VIRT_INVMASS, the FP64 row and the list record
  auto finish = [&](int c0, int q, int t0) {
    const int nc = min(kC, nv - c0);
    for (int u = (int)threadIdx.x - t0; u < nc; u += (int)blockDim.x - t0) {
      const int v = c0 + u;
      if (cv.n[v] < 0) continue;  // a centre-atom site: k_positions placed it
      const R inv = (R)a.vinv[v];
      R sv[3] = {cv.xs[v], s_c[q][u][0] * inv, s_c[q][u][1] * inv};
      double sd[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        sd[c] = (double)sv[c];
        a.Svs[3 * (size_t)v + c] = sd[c];
      }
      store_position<R>(a, b2, boxinv, a.natoms + v, sv, sd);
    }
  };
  if (nv > 0) load(0, 0, 0);
  __syncthreads();
  // step j: thread 0 sums chunk j (buffer j&1) while warps 1..7 load chunk
  // j+1 into the other buffer and finish chunk j-1 from its sums
  R cy = 0, cz = 0;  // the running sums, held by thread 0
  int last = -1;     // the chunk summed last, still to be finished
  for (int c0 = 0, q = 0; c0 < nv; c0 += kC, q ^= 1) {
    const int nc = min(kC, nv - c0);
    if (threadIdx.x == 0) {
      // two sites at a time: both sites' terms are loaded (whole rows, the
      // unused slots included) before the first addition, so the additions
      // wait on one another only
      for (int u = 0; u < nc; u += 2) {
        const int u1 = min(u + 1, nc - 1);
        R t0[32], t1[32];
        lds_row(t0, s_t[q][u]);
        lds_row(t1, s_t[q][u1]);
        const int n0 = s_n[q][u], n1 = s_n[q][u1];
#pragma unroll
        for (int k = 0; k < 15; ++k) {
          if (k < n0) {
            cy = cy + t0[k];
            cz = cz + t0[16 + k];
          }
        }
        s_c[q][u][0] = cy;
        s_c[q][u][1] = cz;
        if (u1 == u) break;
#pragma unroll
        for (int k = 0; k < 15; ++k) {
          if (k < n1) {
            cy = cy + t1[k];
            cz = cz + t1[16 + k];
          }
        }
        s_c[q][u1][0] = cy;
        s_c[q][u1][1] = cz;
      }
    } else if (threadIdx.x >= 32) {
      if (c0 + kC < nv) load(c0 + kC, q ^ 1, 32);
      if (last >= 0) finish(last, q ^ 1, 32);
    }
    __syncthreads();  // buffer q is summed, q^1 loaded and its sums used
    last = c0;
  }
  if (last >= 0) finish(last, ((last / kC) & 1), 0);
}

// ------------------------------------------------------------ cell lists
struct ListArgs {
  Scalars* sc;
  int n;             // particles in the list
  int which;         // 0 atoms, 1 beads
  int natoms;        // NATOMS (VS-VS exclusion)
  int hybrid;        // IBRDESCR == 0
  int maxnab;        // reference STOP threshold
  int cell_cap;      // capacity of the cell arrays
  int nslices;       // slices of the list storage
  float rlist, rlistsq;
  double rlistd, rlistsqd;
  // FP32 path: accepted pairs at r^2 >= rgroupsq (rc + skin/4, squared) are
  // stored after the others, each group in the reference's order, so that
  // list rows far beyond the cutoff are mostly skipped whole by the
  // nonbonded kernel's warps; 0 keeps the reference's order throughout
  float rgroupsq;
  const int* idx;    // INDEX_LIST, 0-based global ids
  int* cell_of;      // [n] cell of list entry A
  int* cell_count;   // [cell_cap]
  int* cell_start;   // [cell_cap + 1]
  int* place;        // [n] place of list entry A among its cell's entries
  int* cells;        // [n] the cells' entries, one cell after another
  int* sorted;       // [n] slot -> A
  int* slot_of;      // [n] A -> slot
  int* gslot;        // [NITEMS]
  void* pos4;        // [n]
  int4* posq;        // [n] FP32 path: fixed-point positions (box fractions), or null
  const double* S;   // FP64 state (3,NITEMS)
  const int* tbits;  // type | label<<16 per particle
  int* counts;       // [n] per slot
  int* slice_w;      // [nslices] rows of 32 entries used by each slice
  int* entries;      // list storage: slice g owns rows [g*w_cap, (g+1)*w_cap) of 32 entries
  int w_cap;         // rows of 32 entries per slice
  const int* excl_n; // CONNECTIONS, by global id
  const int* excl;   // CONNECTED_TO, [i*20 + c], 0-based
};

// List-rebuild kernels run when the step rebuilds its lists (or always, for
// the rebuild of ibg_set_state) and the step is not skipped.  The list builds
// themselves raise skip when a slot outgrows the storage, while blocks of the
// same launch may only be starting: there a block reads the flag together, so
// that no warp leaves whose work the others wait for.
__device__ __forceinline__ bool build_idle(const Scalars* sc, int always) {
  return __syncthreads_or(sc->skip || !(always || sc->rebuild));
}

// Five launches: cells and counts, their scan, the cells' entries, their order
// and new slots, the lists.  (They were eight; each costs ~4 us where the
// system is small.)
//
// UPDATE_NEIGHBOURLIST.F90:14-48 / ALLOCATEVAR2.f90:19-42: cells per
// dimension = INT(BOX/RLIST), and LINKS.f90:16-18.  A component equal to NCELL
// (coordinate at +L/2 after rounding) would address a cell outside the grid;
// it is clamped and counted.  The cell counters are zero at the start (when
// allocated, and again after k_cell_fill).  An entry's place among its cell's
// entries, in no particular order yet, is what its count returned.
template <typename R, bool B>
__global__ void k_cell_assign(__grid_constant__ const ListArgs L0, const ListArgs* const* tab, const BlockMap bm, int always) {
  pdl_wait();
  pdl_trigger();
  using PT = typename Prec<R>::pos_t;
  const Blk bk = blk<B>(bm);
  const ListArgs& L = B ? *tab[bk.sys] : L0;
  Scalars* sc = L.sc;
  if (sc->skip || !(always || sc->rebuild)) return;
  R b[3], bi[3], b2[3];
  box_of<R>(sc, b, bi, b2);
  int nc[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) nc[c] = fint(b[c] / (sizeof(R) == 4 ? (R)L.rlist : (R)L.rlistd));
  const bool bad = nc[0] < 3 || nc[1] < 3 || nc[2] < 3;
  const bool full = (long long)nc[0] * nc[1] * nc[2] > L.cell_cap;
  if (bad || full) nc[0] = nc[1] = nc[2] = 1;
  if (bk.b == 0 && threadIdx.x == 0) {
    if (bad) atomicOr(&sc->err, EB_CELL_GRID);
    if (full) atomicOr(&sc->err, EB_CAPACITY);
    for (int c = 0; c < 3; ++c) sc->ncell[L.which][c] = nc[c];
    sc->rows_max[L.which] = 0;
  }
  const PT* pos = (const PT*)L.pos4;
  for (int a = bk.b * blockDim.x + threadIdx.x; a < L.n; a += bk.g * blockDim.x) {
    PT p = pos[L.slot_of[a]];
    R x[3] = {p.x, p.y, p.z};
    int k[3];
    int clamps = 0;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      k[c] = fint((x[c] * bi[c] + (R)0.5) * (R)nc[c]);
      if (k[c] >= nc[c]) { k[c] = nc[c] - 1; ++clamps; }
      if (k[c] < 0) { k[c] = 0; ++clamps; }
    }
    if (clamps) atomicAdd(&sc->cell_clamps, (unsigned long long)clamps);
    const int cell = (k[0] * nc[1] + k[1]) * nc[2] + k[2];
    L.cell_of[a] = cell;
    L.place[a] = atomicAdd(&L.cell_count[cell], 1);
  }
}

// Exclusive scan of the cell counts by one block per system (cell_start has
// cell_cap + 1 entries).
template <bool B>
__global__ void k_scan_cells(__grid_constant__ const ListArgs L0, const ListArgs* const* tab, const BlockMap bm, int always) {
  pdl_wait();
  pdl_trigger();
  const Blk bk = blk<B>(bm);
  const ListArgs& L = B ? *tab[bk.sys] : L0;
  Scalars* sc = L.sc;
  if (sc->skip || !(always || sc->rebuild)) return;
  const int* in = L.cell_count;
  int* out = L.cell_start;
  const int m = L.cell_cap;
  __shared__ int wsum[32];
  const int t = threadIdx.x, T = blockDim.x, lane = t & 31, warp = t >> 5, nw = (T + 31) >> 5;
  // tiles of V*T consecutive cells, thread t holding cells V*t..V*t+V-1 of
  // the tile (read and written as int4 where the tile is whole), the tiles in
  // order with the running total carried from one to the next
  constexpr int V = 16;
  int carry = 0, most = 0;
  for (int base = 0; base < m; base += V * T) {
    const int i0 = base + V * t;
    const bool whole = i0 + V <= m;
    int x[V], s = 0;
    if (whole) {
#pragma unroll
      for (int j = 0; j < V / 4; ++j) {
        const int4 q = ((const int4*)(in + i0))[j];
        x[4 * j] = q.x; x[4 * j + 1] = q.y; x[4 * j + 2] = q.z; x[4 * j + 3] = q.w;
      }
    } else {
#pragma unroll
      for (int j = 0; j < V; ++j) x[j] = i0 + j < m ? in[i0 + j] : 0;
    }
#pragma unroll
    for (int j = 0; j < V; ++j) {
      s += x[j];
      most = max(most, x[j]);
    }
    int v = s;  // inclusive scan of the threads' sums: warps, then warp totals
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += y;
    }
    if (lane == 31) wsum[warp] = v;
    __syncthreads();
    if (warp == 0) {
      int w = lane < nw ? wsum[lane] : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += y;
      }
      wsum[lane] = w;
    }
    __syncthreads();
    int run = carry + v - s + (warp ? wsum[warp - 1] : 0);
#pragma unroll
    for (int j = 0; j < V; ++j) {
      const int e = run;
      run += x[j];
      x[j] = e;
    }
    if (whole) {
#pragma unroll
      for (int j = 0; j < V / 4; ++j)
        ((int4*)(out + i0))[j] = make_int4(x[4 * j], x[4 * j + 1], x[4 * j + 2], x[4 * j + 3]);
    } else {
#pragma unroll
      for (int j = 0; j < V; ++j)
        if (i0 + j < m) out[i0 + j] = x[j];
    }
    carry += wsum[nw - 1];
    __syncthreads();  // wsum is rewritten by the next tile
  }
  // the fullest cell (the list build's units)
  __shared__ int s_most;
  if (t == 0) s_most = 0;
  __syncthreads();
  most = __reduce_max_sync(0xffffffffu, most);
  if (lane == 0) atomicMax(&s_most, most);
  __syncthreads();
  if (t == 0) {
    out[m] = carry;
    sc->cell_max[L.which] = s_most;
  }
}

// The cells' entries side by side, and the cell counters (for the next
// rebuild) and slice lengths (for this one's lists) cleared.
template <bool B>
__global__ void k_cell_fill(__grid_constant__ const ListArgs L0, const ListArgs* const* tab, const BlockMap bm, int always) {
  pdl_wait();
  pdl_trigger();
  const Blk bk = blk<B>(bm);
  const ListArgs& L = B ? *tab[bk.sys] : L0;
  Scalars* sc = L.sc;
  if (sc->skip || !(always || sc->rebuild)) return;
  const int t0 = bk.b * blockDim.x + threadIdx.x, nt = bk.g * blockDim.x;
  for (int a = t0; a < L.n; a += nt) L.cells[L.cell_start[L.cell_of[a]] + L.place[a]] = a;
  for (int c = t0; c < L.cell_cap; c += nt) L.cell_count[c] = 0;
  for (int g = t0; g < L.nslices; g += nt) L.slice_w[g] = 0;
}

// Within a cell the reference's linked list visits entries by decreasing A
// (LINKS.f90:19-20); slots are kept in increasing A so the list build can
// walk them backwards.  Each entry finds its rank among its cell's entries,
// and with it its new slot; its position goes there from the FP64 state, as
// k_positions stored it in the old slot (a site's row holds the value in the
// step's precision).
template <typename R, bool B>
__global__ void k_cell_rank(__grid_constant__ const ListArgs L0, const ListArgs* const* tab, const BlockMap bm, int always) {
  pdl_wait();
  pdl_trigger();
  using PT = typename Prec<R>::pos_t;
  const Blk bk = blk<B>(bm);
  const ListArgs& L = B ? *tab[bk.sys] : L0;
  Scalars* sc = L.sc;
  if (sc->skip || !(always || sc->rebuild)) return;
  R b[3], bi[3], b2[3];
  box_of<R>(sc, b, bi, b2);
  const double boxinv[3] = {sc->boxinv[0], sc->boxinv[1], sc->boxinv[2]};
  for (int s = bk.b * blockDim.x + threadIdx.x; s < L.n; s += bk.g * blockDim.x) {
    const int a = L.cells[s];
    const int c = L.cell_of[a], i = L.idx[a];
    const int lo = L.cell_start[c], hi = L.cell_start[c + 1];
    const double sd[3] = {L.S[3 * (size_t)i], L.S[3 * (size_t)i + 1], L.S[3 * (size_t)i + 2]};
    const int tb = L.tbits[i];
    int slot = lo;
    for (int k = lo; k < hi; ++k) slot += L.cells[k] < a;
    R r[3] = {(R)sd[0], (R)sd[1], (R)sd[2]};
    fold3<R>(r, b2);
    PT p;
    p.x = r[0]; p.y = r[1]; p.z = r[2];
    p.w = Prec<R>::tbits(tb);
    ((PT*)L.pos4)[slot] = p;
    if (L.posq) L.posq[slot] = box_fraction(sd, boxinv, tb);
    L.sorted[slot] = a;
    L.slot_of[a] = slot;
    L.gslot[i] = slot * 2 + L.which;
  }
}

// The 13 neighbour cells of the half stencil in MAPS.f90:39-51 order.
#define IBG_HALF_STENCIL                                                                                    \
  {{1, 0, 0}, {1, 1, 0},  {0, 1, 0},  {-1, 1, 0}, {1, 0, -1}, {1, 1, -1}, {0, 1, -1},                        \
   {-1, 1, -1}, {1, 0, 1}, {1, 1, 1}, {0, 1, 1}, {-1, 1, 1}, {0, 0, 1}}
__constant__ int kStencil[13][3] = IBG_HALF_STENCIL;
static const int kStencilHost[13][3] = IBG_HALF_STENCIL;  // the same, for host code

// NEW_NEIGHBOUR_WITHLIST.f90:34-123.  A unit of work is up to 32 particles of
// one cell; a block takes units dynamically.  It stages the cell's candidates
// in shared memory, in the reference's order: the cell's own slots, then the
// slots of the 13 cells of the MAPS.f90:39-51 stencil, each run by decreasing
// A (with more candidates than the stage holds, a stage at a time).
//
// Distances: a lane holds a particle and a warp walks 32 candidates at a time,
// each one a broadcast from shared memory, leaving a bit per candidate and
// lane for "inside RLIST" and for "outer group" (ListArgs::rgroupsq).  A unit
// of 16 or 8 particles gives each two or four lanes, which take different
// words of candidates, so that no lane is idle in a small group.
//
// Lists: bits of excluded partners are cleared (an exclusion's slot lies in one
// of the runs, so its bit is known).  Every lane then writes the entries of its
// own words one after another; counts of the words before them give their
// places, so that they keep the candidates' order, the outer group's after the
// others.
//
// The reference pairs a particle with the own-cell candidates below it only
// (later in the staged order), and a virtual site with no other site.  The
// list is stored in the nonbonded kernel's layout: T lanes per slot, slices of
// P = 32/T slots, entry k of slot s (slice g) at (g*w_cap + k/T)*32 + (s%P)*T +
// k%T.  A slot that needs more than w_cap rows records its need and raises the
// abort flag (the host enlarges the storage and repeats the step).
//
// Minimum image: d - s with s the run's image shift (0 or +-L per axis).  For a
// pair inside RLIST <= L/3 that shift is the nearest image, so s = ANINT(d/L)*L
// exactly and d - s is the reference's d - ANINT(d/L)*L bit for bit; with any
// other shift the distance is above RLIST either way.  A cell none of whose
// runs wrapped has no shifts to subtract.
//
// Bound by its block barriers and by instruction issue (ncu, 40,000-bead melt:
// 40 % of the stalls at barriers, issue 57 %; 160,000-bead melt: ~310 warp
// instructions a particle for the distances, ~370 for writing the entries, the
// rest for staging, exclusions and counts).  A warp per particle that tests 32
// candidates at a time took ~1,400 (two ballots, prefix counts, exclusion
// compares and the shift for every 32 tests): launch 276 us, now ~220; the
// hybrid melt's two lists 405 us a rebuild with the cell sort, now 246.
// Entries written by a lane per candidate, word by word, took 450 a particle;
// by a lane per word, 1,150 (the words next to the particle are full).
//
// Candidates a block stages: 1,536 in FP32, 768 in FP64.
// Entries of the outer group a thread of the thread-per-particle build holds
// back to append after the others.
constexpr int kLateThread = 24;
template <typename R>
struct ListStage {
  static constexpr int words = sizeof(R) == 4 ? 48 : 24;  // of 32 candidates
  static constexpr int cap = 32 * words;
};

template <typename R, int T, bool B>
__global__ void __launch_bounds__(256, 4) k_list_build_warp(__grid_constant__ const ListArgs L0, const ListArgs* const* tab,
                                                       const BlockMap bm, int always) {
  pdl_wait();
  pdl_trigger();
  using PT = typename Prec<R>::pos_t;
  constexpr int kWords = ListStage<R>::words, kCap = ListStage<R>::cap;
  constexpr int P = 32 / T;
  const Blk bk = blk<B>(bm);
  __shared__ ListArgs s_args;
  if (B) stage_args(&s_args, tab[bk.sys]);
  const ListArgs& L = B ? s_args : L0;
  Scalars* sc = L.sc;
  if (build_idle(sc, always)) return;
  // candidates, 33 places per word: lanes that read different words at the
  // same time then hit different banks
  __shared__ PT s_pos[kWords * 33];
  __shared__ int s_slot[kCap];
  __shared__ unsigned s_in[kWords * 33], s_out[kWords * 33];  // [word][particle]: accepted, of them outer
  __shared__ unsigned s_vs[kWords];      // virtual sites among a word's candidates
  __shared__ int s_hi[14], s_pre[15];    // run u: slots s_hi[u] down, candidates from s_pre[u]
  __shared__ R s_sh[14][3];              // run u: periodic image shift
  __shared__ int s_ex[32][20], s_ne[32], s_cnt[32], s_i[32];
  __shared__ int s_n[256];               // [share of the words][particle]: entries, the outer group's << 16
  __shared__ int s_unit[2], s_wrap;
  const int nx = sc->ncell[L.which][0], ny = sc->ncell[L.which][1], nz = sc->ncell[L.which][2];
  // units per cell: one where there are cells enough for two per block (its
  // groups of particles then share one stage), else one per group
  const int ncells = nx * ny * nz;
  const int G = ncells >= 2 * bk.g ? 1 : max(1, (sc->cell_max[L.which] + 31) / 32);
  const int nunits = ncells * G;
  R b[3], bi[3], b2[3];
  box_of<R>(sc, b, bi, b2);
  const R rlsq = sizeof(R) == 4 ? (R)L.rlistsq : (R)L.rlistsqd;
  const R rg = L.rgroupsq > 0.f ? (R)L.rgroupsq : rlsq;
  const PT* pos = (const PT*)L.pos4;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int kWarps = 8;  // blockDim.x = 256
  const int cap = L.w_cap * T;  // entries a slot may hold
  int most = 0;  // most rows of any particle this lane closed
  if (threadIdx.x == 0) s_unit[0] = (int)atomicAdd(&sc->work[2 + L.which], 1u);
  for (int turn = 0;; turn ^= 1) {
    __syncthreads();  // the unit's number is there; the last one's stage is no longer read
    const int unit = s_unit[turn];
    if (unit >= nunits) break;
    if (threadIdx.x == 0) s_unit[turn ^ 1] = (int)atomicAdd(&sc->work[2 + L.which], 1u);  // the next one's, meanwhile
    const int c0 = G == 1 ? unit : unit / G;
    const int first = L.cell_start[c0], last = L.cell_start[c0 + 1];
    const int start = first + (unit - c0 * G) * 32;
    if (start >= last) continue;
    if (warp == 0) {
      // run 0: the own cell from its last slot down; runs 1..13: the stencil
      // cells, each from its last slot down; exclusive prefix of the lengths
      int hi = 0, len = 0;
      int w[3] = {0, 0, 0};  // the neighbour cell wraps past the box's +L/2 (1) or -L/2 (-1) face
      if (lane == 0) {
        hi = last - 1;
        len = last - first;
      } else if (lane < 14) {
        const int ic[3] = {c0 / (nz * ny), (c0 / nz) % ny, c0 % nz}, nc[3] = {nx, ny, nz};
        int jc[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          const int j = ic[q] + kStencil[lane - 1][q];
          w[q] = j >= nc[q] ? 1 : (j < 0 ? -1 : 0);
          jc[q] = j - w[q] * nc[q];
        }
        const int c = jc[0] * nz * ny + jc[1] * nz + jc[2];
        const int lo = L.cell_start[c];
        hi = L.cell_start[c + 1] - 1;
        len = hi - lo + 1;
      }
      int incl = len;
#pragma unroll
      for (int o = 1; o < 16; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      const unsigned wraps = __ballot_sync(0xffffffffu, (w[0] | w[1] | w[2]) != 0);
      if (lane < 14) {
        s_hi[lane] = hi;
        s_pre[lane] = incl - len;
#pragma unroll
        for (int q = 0; q < 3; ++q) s_sh[lane][q] = w[q] > 0 ? b[q] : (w[q] < 0 ? -b[q] : (R)0);
      }
      if (lane == 13) s_pre[14] = incl;
      if (lane == 0) s_wrap = wraps != 0;
    }
    bool staged = false;
    for (int s0 = start; s0 < last; s0 += 32 * G) {
      const int np = min(32, last - s0);
      if (s0 > start) __syncthreads();  // the group before is done
      if (warp == 1) {
        int i = 0, ne = 0;
        if (lane < np) {
          i = L.idx[L.sorted[s0 + lane]];
          ne = min(L.excl_n[i], 20);
        }
        s_i[lane] = i;
        s_ne[lane] = ne;
        s_cnt[lane] = 0;
      }
      __syncthreads();
      const int total = s_pre[14];
      const bool wrap = s_wrap != 0;
      // the particles' exclusions, as slots of this list
      for (int k = threadIdx.x; k < 32 * 20; k += blockDim.x) {
        const int p = k / 20, e = k - 20 * p;
        if (e >= s_ne[p]) continue;
        const int gs = L.gslot[L.excl[(size_t)s_i[p] * 20 + e]];
        s_ex[p][e] = (gs & 1) == L.which ? gs >> 1 : -1;
      }
      // this lane's particle in the distance pass, and its share of the words
      const int PL = np > 16 ? 32 : (np > 8 ? 16 : 8), SL = 32 / PL;
      const int p1 = lane & (PL - 1), sub = lane / PL;
      const int own = last - 1 - (s0 + p1);  // its place among the candidates: it pairs with later ones
      PT pi;
      if (p1 < np) pi = pos[s0 + p1];
      else { pi.x = pi.y = pi.z = 0; pi.w = Prec<R>::tbits(0); }
      const unsigned site = L.hybrid && p1 < np && s_i[p1] >= L.natoms ? 0xffffffffu : 0u;
      for (int base = 0; base < total; base += kCap) {
        const int nv = min(kCap, total - base), W = (nv + 31) / 32;
        if (base > 0) __syncthreads();  // the stage before is no longer read
        for (int w = staged ? W : warp; w < W; w += kWarps) {
          const int v = 32 * w + lane;
          PT q;
          bool vs = false;
          if (v < nv) {
            // the run of candidate base + v: the largest u with s_pre[u] <= it
            // (that run is not empty)
            int lo = 0;
  #pragma unroll
            for (int step = 8; step > 0; step >>= 1)
              if (lo + step < 14 && s_pre[lo + step] <= base + v) lo += step;
            const int t = s_hi[lo] - (base + v - s_pre[lo]);
            s_slot[v] = t;
            q = pos[t];
            vs = (Prec<R>::bits(q.w) >> 16) == 3;
            q.w = Prec<R>::tbits(lo);
          } else {  // beyond the candidates: farther than any RLIST
            q.x = q.y = q.z = (R)1e18;
            q.w = Prec<R>::tbits(0);
          }
          s_pos[33 * w + lane] = q;
          const unsigned m = __ballot_sync(0xffffffffu, vs);
          if (lane == 0) s_vs[w] = m;
        }
        staged = total <= kCap;
        __syncthreads();
        // the words from w1 on are this lane's, nw of them: consecutive ones, so
        // that its entries are consecutive in its particle's list
        const int nw = (W + kWarps * SL - 1) / (kWarps * SL), share = warp * SL + sub, w1 = share * nw;
        for (int q0 = 0; q0 < nw; ++q0) {
          const int w = w1 + q0;
          if (!__any_sync(0xffffffffu, w < W)) break;
          const PT* cand = s_pos + 33 * min(w, W - 1);
          unsigned m = 0, far = 0;
          auto test = [&](R d0, R d1, R d2, unsigned bit) {
            R r2 = d0 * d0;
            r2 = r2 + d1 * d1;
            r2 = r2 + d2 * d2;
            if (r2 < rlsq) m |= bit;
            if (r2 >= rg) far |= bit;
          };
          if (!wrap) {
  #pragma unroll 16
            for (int k = 0; k < 32; ++k) {
              const PT q = cand[k];
              test(pi.x - q.x, pi.y - q.y, pi.z - q.z, 1u << k);
            }
          } else {
  #pragma unroll 8
            for (int k = 0; k < 32; ++k) {
              const PT q = cand[k];
              const R* sh = s_sh[Prec<R>::bits(q.w)];
              R d0 = pi.x - q.x, d1 = pi.y - q.y, d2 = pi.z - q.z;
              d0 = d0 - sh[0];
              d1 = d1 - sh[1];
              d2 = d2 - sh[2];
              test(d0, d1, d2, 1u << k);
            }
          }
          if (w < W && p1 < np) {
            const int skip = own + 1 - (base + 32 * w);  // candidates of this word up to the particle itself
            if (skip > 0) m = skip >= 32 ? 0u : m & ~((1u << skip) - 1u);
            m &= ~(site & s_vs[w]);
            s_in[33 * w + p1] = m;
            s_out[33 * w + p1] = m & far;
          }
        }
        __syncthreads();
        // an excluded slot lies in one of the runs: clear its candidate's bit
        // (warp: which exclusion; lane: whose)
        const bool closing = base + kCap >= total;
        for (int e = warp; e < 20; e += kWarps) {
          const int t = e < s_ne[lane] ? s_ex[lane][e] : -1;
          if (!__any_sync(0xffffffffu, t >= 0)) continue;
          for (int u = 0; u < 14; ++u) {
            const int hi = s_hi[u], pre = s_pre[u], v = pre + hi - t - base;
            if (t < 0 || t > hi || hi - t >= s_pre[u + 1] - pre || v < 0 || v >= nv) continue;
            atomicAnd(&s_in[33 * (v >> 5) + lane], ~(1u << (v & 31)));
            atomicAnd(&s_out[33 * (v >> 5) + lane], ~(1u << (v & 31)));
          }
        }
        __syncthreads();
        // how many entries each lane's words hold, the outer group's in the upper
        // half, and how many come before them
        const int last_w = min(W, w1 + nw);
        int mine = 0;
        if (p1 < np)
          for (int w = w1; w < last_w; ++w) {
            const unsigned m = s_in[33 * w + p1], o = closing ? s_out[33 * w + p1] : 0u;
            mine += __popc(m & ~o) + (__popc(o) << 16);
          }
        s_n[share * PL + p1] = mine;
        __syncthreads();
        int before = 0, all = 0;
        for (int r = 0; r < kWarps * SL; ++r) {
          const int x = s_n[r * PL + p1];
          if (r < share) before += x;
          all += x;
        }
        if (p1 < np) {
          const int s = s0 + p1, g = s / P, cnt0 = s_cnt[p1];
          int* row = L.entries + (long long)g * L.w_cap * 32 + (s % P) * T;
          int ki = cnt0 + (before & 0xffff), ko = cnt0 + (all & 0xffff) + (before >> 16);
          // the lane's bits one after another, whatever word they are in (a list
          // that another stage of candidates follows is stored as found, which
          // only mixes the groups)
          int w = w1 - 1;
          unsigned m = 0, o = 0;
          for (int left = (mine & 0xffff) + (mine >> 16); left > 0;) {
            if (m == 0) {
              ++w;
              m = s_in[33 * w + p1];
              o = closing ? s_out[33 * w + p1] : 0u;
              continue;
            }
            const int bit = __ffs(m) - 1;
            m &= m - 1u;
            --left;
            const int k = (o >> bit) & 1u ? ko++ : ki++;
            if (k < cap) row[(k / T) * 32 + (k % T)] = s_slot[32 * w + bit];
          }
          if (share == 0 && closing) {
            const int cnt = cnt0 + (all & 0xffff) + (all >> 16);
            L.counts[s] = cnt;
            if (cnt >= L.maxnab) atomicOr(&sc->err, EB_LIST_OVERFLOW);
            const int rows = (cnt + T - 1) / T;
            most = max(most, rows);
            atomicMax(&L.slice_w[g], rows);
            if (rows > L.w_cap) {
              atomicMax(&sc->need_rows[L.which], rows);
              sc->abort = 1;
              sc->skip = 1;
            }
          }
        }
        if (!closing) {
          __syncthreads();  // every lane has read the counts
          if (share == 0 && p1 < np) s_cnt[p1] += (all & 0xffff) + (all >> 16);
        }
      }
    }
  }
  if (most > 0) atomicMax(&sc->rows_max[L.which], most);
}

// NEW_NEIGHBOUR_WITHLIST.f90:34-123 for large lists: a thread builds one
// particle's list (k_list_build_warp, above, gives a block to up to 32 particles
// of a cell and suits lists too short to fill the GPU with one thread per
// particle).
// A warp takes 32 consecutive slots at a time (dynamically), so its lanes
// mostly share a cell and walk the same candidates in step: a candidate's
// position is one load that the lanes share, and each lane appends what it
// accepts to its own list in the order it visits the candidates.  That order
// is the reference's: the particle's own cell below it by decreasing A (slots
// keep increasing A within a cell), then the 13 cells of the MAPS.f90:39-51
// stencil, each by decreasing A.  The distance test runs first and the
// exclusion test only for candidates inside RLIST (the accepted set is the
// same); exclusions are compared as slots of this list (the first four in
// registers, the rest in shared memory), and a virtual site is recognised by
// its label in the position's w, so no candidate's global id is loaded.
//
// The minimum image needs no per-candidate test: each stencil cell carries
// its periodic shift s (0 or +-L per axis, from whether it wrapped around the
// box), and a candidate's displacement is (x_i - x_j) - s.  For a pair inside
// RLIST <= L/3 that shift is the nearest image, so s = ANINT(d/L)*L exactly
// and d - s is the reference's d - ANINT(d*BOXINV)*BOX
// (NEW_NEIGHBOUR_WITHLIST.f90:65) bit for bit; with any other shift the
// distance is above RLIST either way.
//
// The list is stored in the nonbonded kernel's layout: T lanes per slot,
// slices of P = 32/T slots, entry k of slot s (slice g) at
// (g*w_cap + k/T)*32 + (s%P)*T + k%T.  A slot that needs more than w_cap rows
// records its need and raises the abort flag (the host enlarges the storage
// and repeats the step).
template <typename R, int T, bool B>
__global__ void __launch_bounds__(256) k_list_build_thread(__grid_constant__ const ListArgs L0, const ListArgs* const* tab,
                                                    const BlockMap bm, int always) {
  pdl_wait();
  pdl_trigger();
  using PT = typename Prec<R>::pos_t;
  const Blk bk = blk<B>(bm);
  __shared__ ListArgs s_args;
  if (B) stage_args(&s_args, tab[bk.sys]);
  const ListArgs& L = B ? s_args : L0;
  Scalars* sc = L.sc;
  if (build_idle(sc, always)) return;
  constexpr int P = 32 / T;
  __shared__ int s_ex[16][256];  // exclusions 5..20 of each thread's particle, as slots of this list
  __shared__ int s_late[kLateThread][256];  // each thread's entries of the outer group (rgroupsq), in order
  const int nx = sc->ncell[L.which][0], ny = sc->ncell[L.which][1], nz = sc->ncell[L.which][2];
  const int nc[3] = {nx, ny, nz};
  R b[3], bi[3], b2[3];
  box_of<R>(sc, b, bi, b2);
  const R rlsq = sizeof(R) == 4 ? (R)L.rlistsq : (R)L.rlistsqd;
  const R rg = L.rgroupsq > 0.f ? (R)L.rgroupsq : rlsq;
  const PT* pos = (const PT*)L.pos4;
  const int lane = threadIdx.x & 31;
  const int cap = L.w_cap * T;  // entries a slot may hold
  const int nchunks = (L.n + 31) / 32;
  int most = 0;  // most rows of any particle of this thread
  for (;;) {
    int ch = 0;
    if (lane == 0) ch = (int)atomicAdd(&sc->work[2 + L.which], 1u);
    ch = __shfl_sync(0xffffffffu, ch, 0);
    if (ch >= nchunks) break;
    const int s = ch * 32 + lane;
    if (s >= L.n) continue;
    const int a = L.sorted[s];
    const int i = L.idx[a];
    const int c0 = L.cell_of[a];
    const PT pi = pos[s];
    const int ne = min(L.excl_n[i], 20);
    int e0 = -1, e1 = -1, e2 = -1, e3 = -1;
    for (int e = 0; e < ne; ++e) {
      const int gs = L.gslot[L.excl[(size_t)i * 20 + e]];
      const int t = (gs & 1) == L.which ? gs >> 1 : -1;
      if (e == 0) e0 = t;
      else if (e == 1) e1 = t;
      else if (e == 2) e2 = t;
      else if (e == 3) e3 = t;
      else s_ex[e - 4][threadIdx.x] = t;
    }
    const bool i_vs = L.hybrid && i >= L.natoms;
    const int g = s / P;
    int* row = L.entries + (long long)g * L.w_cap * 32 + (s % P) * T;
    int cnt = 0, nlate = 0;
    // candidates slot hi down to lo, displaced by the run's image shift
    // a candidate inside RLIST: exclusions, the site-site rule, then stored
    auto accept = [&](int t, R r2, const PT& pj) {
      bool ok = !(i_vs && (Prec<R>::bits(pj.w) >> 16) == 3) && t != e0 && t != e1 && t != e2 && t != e3;
      if (ok && ne > 4)
        for (int e = 4; e < ne; ++e) ok &= s_ex[e - 4][threadIdx.x] != t;
      if (ok) {
        if (r2 >= rg && nlate < kLateThread) {
          s_late[nlate++][threadIdx.x] = t;  // the outer group, appended below
        } else {
          if (cnt < cap) row[(cnt / T) * 32 + cnt % T] = t;
          ++cnt;
        }
      }
    };
    auto scan = [&](int hi, int lo, R sh0, R sh1, R sh2) {
#pragma unroll 4
      for (int t = hi; t >= lo; --t) {
        const PT pj = pos[t];
        R d0 = pi.x - pj.x, d1 = pi.y - pj.y, d2 = pi.z - pj.z;
        d0 = d0 - sh0;
        d1 = d1 - sh1;
        d2 = d2 - sh2;
        R r2 = d0 * d0;
        r2 = r2 + d1 * d1;
        r2 = r2 + d2 * d2;
        if (r2 < rlsq) accept(t, r2, pj);
      }
    };
    scan(s - 1, L.cell_start[c0], (R)0, (R)0, (R)0);  // the own cell below this particle
    const int ic[3] = {c0 / (nz * ny), (c0 / nz) % ny, c0 % nz};
    for (int u = 0; u < 13; ++u) {
      int jc[3];
      R sh[3];
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const int j = ic[q] + kStencil[u][q];
        const int w = j >= nc[q] ? 1 : (j < 0 ? -1 : 0);
        jc[q] = j - w * nc[q];
        sh[q] = w > 0 ? b[q] : (w < 0 ? -b[q] : (R)0);
      }
      const int c = jc[0] * nz * ny + jc[1] * nz + jc[2];
      scan(L.cell_start[c + 1] - 1, L.cell_start[c], sh[0], sh[1], sh[2]);
    }
    for (int q = 0; q < nlate; ++q, ++cnt)
      if (cnt < cap) row[(cnt / T) * 32 + cnt % T] = s_late[q][threadIdx.x];
    L.counts[s] = cnt;
    if (cnt >= L.maxnab) atomicOr(&sc->err, EB_LIST_OVERFLOW);
    const int rows = (cnt + T - 1) / T;
    most = max(most, rows);
    atomicMax(&L.slice_w[g], rows);
    if (rows > L.w_cap) {
      atomicMax(&sc->need_rows[L.which], rows);
      sc->abort = 1;
      sc->skip = 1;
    }
  }
  most = __reduce_max_sync(0xffffffffu, most);
  if (lane == 0 && most > 0) atomicMax(&sc->rows_max[L.which], most);
}

// Slice lists (FP32 path, ListArgs/NBArgs form 1).  Slice g is the four
// slots 4g..4g+3.  Its list holds each neighbour once, as the entry
// slot | mask << 28, where bit k of the mask says that slot 4g+k pairs with
// it: the union of the four half lists, with no pair added or lost.  The
// four slots are consecutive in the cell order, so their lists share most of
// their neighbours (a stored entry stands for ~1.9 pairs on the melts), and
// the nonbonded kernel gathers each neighbour's position and adds its force
// once per slice instead of once per pair.  Entry e of slice g lives at
// g*w_cap*32 + e; the last row is filled up with empty entries (mask 0).
constexpr int kUSlots = 4;
constexpr unsigned kUSlotMask = (1u << 28) - 1u;
constexpr int kUBuf = 256;  // entries of a slice each warp sorts in shared memory

// NEW_NEIGHBOUR_WITHLIST.f90:34-123 in the slice form: a warp builds one
// slice's list.  For each cell that holds particles of the slice (one, or two
// when the slice straddles a cell boundary) it walks that cell's candidates,
// 32 at a time, one per lane: the own cell below the slice's last particle
// there, then the 13 stencil cells of MAPS.f90:39-51, each by decreasing slot.
// A lane tests its candidate against each particle of the slice in that cell
// with the reference's REAL*4 distance (the run's image shift gives the
// nearest image, as in k_list_build_thread), the own-cell rule (only slots
// below the particle), the virtual-site rule and the particle's exclusions.
// A candidate that two cells of a slice both reach is stored once per cell,
// with disjoint masks, so every pair is stored exactly once.
//
// The accepted entries are gathered in shared memory and stored sorted by
// the key (outer group, mask), stably: first the entries with a pair inside
// rgroupsq, by mask, then the rest, by mask.  So a row of 32 entries mostly
// shares one mask, and the nonbonded kernel's warp runs the pair arithmetic
// once per bit of that mask with all its lanes busy, instead of once per
// particle of the slice with the lanes whose masks hold it.  Entries beyond
// the first kUBuf of a slice are stored unsorted after them.  counts[s] is the
// number of pairs of slot s (its reference NNEBS).
template <bool B>
__global__ void __launch_bounds__(256) k_list_build_slices(__grid_constant__ const ListArgs L0,
                                                          const ListArgs* const* tab, const BlockMap bm, int always) {
  pdl_wait();
  pdl_trigger();
  const Blk bk = blk<B>(bm);
  __shared__ ListArgs s_args;
  if (B) stage_args(&s_args, tab[bk.sys]);
  const ListArgs& L = B ? s_args : L0;
  Scalars* sc = L.sc;
  if (build_idle(sc, always)) return;
  constexpr int kWarps = 8;
  __shared__ int s_ex[kWarps][kUSlots][20];  // each particle's exclusions as slots of this list
  __shared__ int s_buf[kWarps][kUBuf];       // the slice's entries, in the order accepted
  __shared__ unsigned char s_key[kWarps][kUBuf];  // their keys: mask | 16 for the outer group
  __shared__ int s_off[kWarps][32];          // per key: count, then next position
  __shared__ int2 s_run[kWarps][14];         // each candidate run: highest slot, first index
  __shared__ float s_sh[kWarps][14][3];      // each candidate run: image shift
  const int nx = sc->ncell[L.which][0], ny = sc->ncell[L.which][1], nz = sc->ncell[L.which][2];
  const int nc[3] = {nx, ny, nz};
  float b[3], bi[3], b2[3];
  box_of<float>(sc, b, bi, b2);
  const float rlsq = L.rlistsq;
  const float rg = L.rgroupsq > 0.f ? L.rgroupsq : rlsq;
  const float4* pos = (const float4*)L.pos4;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned below = (1u << lane) - 1u;
  int* buf = s_buf[warp];
  unsigned char* keys = s_key[warp];
  int* off = s_off[warp];
  const int cap = L.w_cap * 32;  // entries a slice may hold
  int most = 0;  // most rows of any slice of this warp
  for (;;) {
    int g = 0;
    if (lane == 0) g = (int)atomicAdd(&sc->work[2 + L.which], 1u);
    g = __shfl_sync(0xffffffffu, g, 0);
    if (g >= L.nslices) break;
    // the slice's particles: slot, cell, position, exclusions, site flag
    int my_cell = INT_MAX, my_ne = 0, my_vs = 0;
    float4 my_pos = make_float4(0.f, 0.f, 0.f, 0.f);
    int my_i = 0;
    if (lane < kUSlots && kUSlots * g + lane < L.n) {
      const int s = kUSlots * g + lane;
      const int a = L.sorted[s];
      my_i = L.idx[a];
      my_cell = L.cell_of[a];
      my_pos = pos[s];
      my_ne = min(L.excl_n[my_i], 20);
      my_vs = L.hybrid && my_i >= L.natoms;
    }
    float4 pi[kUSlots];
    int ci[kUSlots], ne[kUSlots];
    unsigned vsm = 0;
#pragma unroll
    for (int k = 0; k < kUSlots; ++k) {
      pi[k].x = __shfl_sync(0xffffffffu, my_pos.x, k);
      pi[k].y = __shfl_sync(0xffffffffu, my_pos.y, k);
      pi[k].z = __shfl_sync(0xffffffffu, my_pos.z, k);
      ci[k] = __shfl_sync(0xffffffffu, my_cell, k);
      ne[k] = __shfl_sync(0xffffffffu, my_ne, k);
      vsm |= (unsigned)__shfl_sync(0xffffffffu, my_vs, k) << k;
      const int ik = __shfl_sync(0xffffffffu, my_i, k);
      if (lane < ne[k]) {
        const int gs = L.gslot[L.excl[(size_t)ik * 20 + lane]];
        s_ex[warp][k][lane] = (gs & 1) == L.which ? gs >> 1 : -1;
      }
    }
    __syncwarp();
    const long long base = (long long)g * cap;
    int cnt = 0;
    int npair[kUSlots] = {0, 0, 0, 0};  // this lane's accepted pairs of each particle
    // each cell of the slice in turn (slots are in cell order, so the
    // particles of one cell are consecutive).  Its 14 runs (the own cell
    // below the group's last particle, then the 13 stencil cells) are walked
    // as one sequence of candidates, 32 at a time: lane u < 14 describes run
    // u (highest slot, image shift), a prefix sum gives each run's first index
    for (int k0 = 0; k0 < kUSlots && ci[k0] != INT_MAX;) {
      const int c0 = ci[k0];
      unsigned gm = 0;
      int k1 = k0;
      while (k1 < kUSlots && ci[k1] == c0) gm |= 1u << k1++;
      int hi = -1, len = 0;
      float sh[3] = {0.f, 0.f, 0.f};
      if (lane == 0) {
        hi = kUSlots * g + k1 - 2;
        len = max(0, hi - L.cell_start[c0] + 1);
      } else if (lane < 14) {
        const int ic[3] = {c0 / (nz * ny), (c0 / nz) % ny, c0 % nz};
        int jc[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          const int j = ic[q] + kStencil[lane - 1][q];
          const int w = j >= nc[q] ? 1 : (j < 0 ? -1 : 0);
          jc[q] = j - w * nc[q];
          sh[q] = w > 0 ? b[q] : (w < 0 ? -b[q] : 0.f);
        }
        const int c = jc[0] * nz * ny + jc[1] * nz + jc[2];
        hi = L.cell_start[c + 1] - 1;
        len = hi - L.cell_start[c] + 1;
      }
      int incl = len;
#pragma unroll
      for (int o = 1; o < 16; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      const int total = __shfl_sync(0xffffffffu, incl, 13);
      __syncwarp();  // the previous cell's run table is no longer read
      if (lane < 14) {
        s_run[warp][lane] = make_int2(hi, incl - len);
        s_sh[warp][lane][0] = sh[0];
        s_sh[warp][lane][1] = sh[1];
        s_sh[warp][lane][2] = sh[2];
      }
      __syncwarp();
      for (int v0 = 0; v0 < total; v0 += 32) {
        const int v = v0 + lane;
        unsigned m = 0;
        bool inner = false;
        int t = 0;
        if (v < total) {
          // the run of candidate v: the last run that starts at or before v
          // (empty runs start where the next one does, and are skipped)
          int u = 0;
#pragma unroll
          for (int step = 8; step > 0; step >>= 1)
            if (u + step < 14 && s_run[warp][u + step].y <= v) u += step;
          const int2 run = s_run[warp][u];
          t = run.x - (v - run.y);
          const float sh0 = s_sh[warp][u][0], sh1 = s_sh[warp][u][1], sh2 = s_sh[warp][u][2];
          const bool own = u == 0;
          const float4 pj = pos[t];
          const bool j_vs = (__float_as_int(pj.w) >> 16) == 3;
#pragma unroll
          for (int k = 0; k < kUSlots; ++k) {
            if (!((gm >> k) & 1u)) continue;
            // the reference's REAL*4 distance, scalar and uncontracted
            float d0 = pi[k].x - pj.x, d1 = pi[k].y - pj.y, d2 = pi[k].z - pj.z;
            d0 = d0 - sh0;
            d1 = d1 - sh1;
            d2 = d2 - sh2;
            float r2 = d0 * d0;
            r2 = r2 + d1 * d1;
            r2 = r2 + d2 * d2;
            if (!(r2 < rlsq)) continue;
            if (own && t >= kUSlots * g + k) continue;  // the own cell: only slots below the particle
            if (((vsm >> k) & 1u) && j_vs) continue;    // no site-site pair
            bool ok = true;
            for (int e = 0; e < ne[k]; ++e) ok &= s_ex[warp][k][e] != t;
            if (!ok) continue;
            m |= 1u << k;
            ++npair[k];
            inner |= r2 < rg;
          }
        }
        const unsigned ma = __ballot_sync(0xffffffffu, m != 0);
        if (m != 0) {
          const int k = cnt + __popc(ma & below);
          const int entry = t | (int)(m << 28);
          if (k < kUBuf) {
            buf[k] = entry;
            keys[k] = (unsigned char)(m | (inner ? 0u : 16u));
          } else if (k < cap) {
            L.entries[base + k] = entry;  // beyond the sort buffer: stored as found
          }
        }
        cnt += __popc(ma);
      }
      k0 = k1;
    }
#pragma unroll
    for (int k = 0; k < kUSlots; ++k)
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) npair[k] += __shfl_xor_sync(0xffffffffu, npair[k], o);
    // stable counting sort of the buffered entries by key
    __syncwarp();
    const int nb = min(cnt, kUBuf);
    off[lane] = 0;
    __syncwarp();
    for (int c = 0; c < nb; c += 32) {
      const int q = c + lane;
      const int key = q < nb ? keys[q] : 32 + lane;  // unique keys for the idle lanes
      const unsigned same = __match_any_sync(0xffffffffu, key);
      if (q < nb && (same & below) == 0) off[key] += __popc(same);
      __syncwarp();
    }
    {
      const int n_key = off[lane];
      int incl = n_key;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      __syncwarp();
      off[lane] = incl - n_key;  // first position of key `lane`
      __syncwarp();
    }
    for (int c = 0; c < nb; c += 32) {
      const int q = c + lane;
      const int key = q < nb ? keys[q] : 32 + lane;
      const unsigned same = __match_any_sync(0xffffffffu, key);
      int at = 0;
      if (q < nb) at = off[key] + __popc(same & below);
      __syncwarp();
      if (q < nb && (same & below) == 0) off[key] += __popc(same);
      if (q < nb && at < cap) L.entries[base + at] = buf[q];
      __syncwarp();
    }
    // empty entries up to the end of the last row
    const int rows = (cnt + 31) / 32;
    most = max(most, rows);
    if (cnt + lane < rows * 32 && cnt + lane < cap) L.entries[base + cnt + lane] = 0;
    if (lane < kUSlots && kUSlots * g + lane < L.n) {
      int np = npair[0];
#pragma unroll
      for (int k = 1; k < kUSlots; ++k) np = lane == k ? npair[k] : np;
      L.counts[kUSlots * g + lane] = np;
      if (np >= L.maxnab) atomicOr(&sc->err, EB_LIST_OVERFLOW);
    }
    if (lane == 0) {
      L.slice_w[g] = rows;
      if (rows > L.w_cap) {
        atomicMax(&sc->need_rows[L.which], rows);
        sc->abort = 1;
        sc->skip = 1;
      }
    }
    __syncwarp();  // s_ex, buf and keys are rewritten for the next slice
  }
  if (lane == 0 && most > 0) atomicMax(&sc->rows_max[L.which], most);
}

// ------------------------------------------------------------- nonbonded
// FP32 nonbonded energies and virials are summed in FP32 over this many list
// rows of a slice, then in fixed point.
constexpr int kEnergyRows = 8;

template <typename R>
struct NBArgs {
  Scalars* sc;
  int mts;                         // bead list of an MTS run: only steps m = 1..3 evaluate it
  int n, nslices, ntype;
  const void* pos4;
  const int4* posq;                // FP32 kernel: positions as box fractions
  const int* counts;
  const int* slice_w;
  const int* entries;
  int w_cap;                       // rows of 32 entries per slice
  int work;                        // index of this launch's work counter
  typename Prec<R>::acc_t* fsort;  // per slot, in blocks of 32 slots (fs_at)
  // tables of this list, per type pair: FP32 path {first row, NDAT, 1/bin bits,
  // 1 if a table}, FP64 path {first row or -1, NDAT, 1/bin low and high word}
  const int4* ptab;
  // FP32 kernel, UNI (all tables on one grid, 1/bin = uinv): the table numbers
  // per type, a byte per type of the neighbour, and the coefficient rows of
  // every table one after another, urows each, F scaled by -2^32; the last of
  // them is zero and holds r2_none
  const uint2* pbase;
  const float4* tuni;
  float uinv, r2_none;
  int urows;
  int chunk;         // 256ths of the units taken dynamically after the blocks' own ranges (0: all, per warp)
  int window;        // chunk > 0: 0 = each block one contiguous range of units; W > 0 = runs of W
                     // consecutive units dealt to the blocks in turn (block b takes runs b, b + G, b + 2G, ...)
  int rows;          // list rows per work unit, a multiple of kEnergyRows
  // FP32 kernel: pairs whose r^2 lies within a relative 1e-6 of the cutoff
  // are left to k_nb_near, which decides them as the FP64 path does from the
  // FP64 state (global ids from slot -> A -> global id)
  float rcut_lo, rcut_hi;
  int4* near;          // (i slot, j slot, i global id, j global id) of those pairs
  int near_cap;
  int near_in_collect;  // k_nb_collect takes those pairs along
  const int* sorted;
  const int* idx;
  const double* S;
  int natoms;
  const R* tfp;  // FP32 path: {F, P} per row, and X = RNBOND per row (k_nb_near)
  // FP32 kernel: per row {A, C, B, D}, -2^32 F = A + B u and P = C + D u with
  // u = r/bin - (row within the table); one 16-byte read per pair
  const float4* tcoef;
  const double4* tcoef64;  // FP64 kernel: the same unscaled, in FP64
  const R* tx;
  int ntab, nrows;
  R rcutsq;
};

// A nonbonded launch does nothing on a skipped step, and for the bead list
// of an MTS run on the steps MTS_APPROX extrapolates (MTS_LOOP.f90:100-110).
template <typename R>
__device__ __forceinline__ bool nb_idle(const NBArgs<R>& A) {
  const Scalars* sc = A.sc;
  if (sc->skip) return true;
  if (A.mts) {
    const int m = sc->mts_m;
    return !(m >= 1 && m <= 3);
  }
  return false;
}

// Work units of NBArgs::rows rows that cover the longest slice of a list.  (The
// storage holds a quarter more rows: units counted from it would be empty for
// every slice.)
template <typename R>
__device__ __forceinline__ int nb_units_per_slice(const NBArgs<R>& A) {
  return max(1, (min(A.sc->rows_max[A.work], A.w_cap) + A.rows - 1) / A.rows);
}

// The sequence of work units one warp of a nonbonded launch takes
// (NBArgs::chunk, NBArgs::window): first units of its block's share, taken
// through a shared counter -- a contiguous range of units (neighbouring
// slices), or with a window runs of W consecutive units dealt to the blocks in
// turn --, so that a block's warps gather from one region of space and share
// it in L1, with no barrier between them; then the last chunk/256 of all units (all of them with chunk 0),
// taken from a global counter by whichever warps get there first.  A warp
// knows its next unit while it still works on one, so that it can load ahead.
template <typename R>
struct NbUnits {
  const NBArgs<R>& A;
  const Blk& bk;
  int* own;  // the block's counter, in shared memory
  int U;     // units per slice
  int lo, hi;
  __device__ __forceinline__ NbUnits(const NBArgs<R>& A_, const Blk& bk_, int U_, int* own_)
      : A(A_), bk(bk_), own(own_), U(U_) {
    const int ns = nstat();
    lo = A.window > 0 ? 0 : (int)((long long)ns * bk.b / bk.g);
    hi = A.window > 0 ? ns : (int)((long long)ns * (bk.b + 1) / bk.g);
  }
  // units handed to the blocks; the rest are shared out
  __device__ __forceinline__ int nstat() const {
    const int n = A.nslices * U;
    return A.chunk > 0 ? n - (int)((long long)n * min(A.chunk, 256) / 256) : 0;
  }
  // the next unit, -1 when there is none left (every lane of the warp calls)
  __device__ __forceinline__ int next() {
    int u = 0;
    if (lo < hi) {
      if ((threadIdx.x & 31) == 0) u = atomicAdd(own, 1);
      u = __shfl_sync(0xffffffffu, u, 0);
      const int W = A.window;
      const long long v = W > 0 ? ((long long)(u / W) * bk.g + bk.b) * W + u % W : (long long)lo + u;
      if (v < hi) return (int)v;
      lo = hi;  // the block's share is taken
    }
    if ((threadIdx.x & 31) == 0) u = nstat() + (int)atomicAdd(&A.sc->work[A.work], 1u);
    u = __shfl_sync(0xffffffffu, u, 0);
    return u < A.nslices * U ? u : -1;
  }
};

// NONBONDED_FORCE.F90:45-104, FP64 path.  Persistent grid; a warp owns one
// slice of P = 32/T slots at a time and T lanes walk each slot's list; list
// reads are coalesced 128-byte rows, neighbour positions are 32-byte gathers
// from the cell-ordered array.  i-forces are summed in registers and reduced
// over the slot's lanes; j-forces are FP64 atomics.  Tables are staged in
// shared memory when SMEM.
//
// Bound by FP64 issue and by the latency of its gathers.  A pair cost two FP64
// divisions, three roundings to the nearest image and seven table reads; it
// now multiplies by 1/bin, picks the image by comparison, and reads a row of
// coefficients (A + B u, C + D u); two rows are evaluated in step and units are
// handed out as in k_nonbonded_f32.  16 warps per SM at 128 registers: at 24
// warps (80 registers, 108 bytes of spills) the launch took 189 us on the
// 160,000-bead melt, with 16 174 (before: 216), all without the block ranges.
// Between events, caches as the step leaves them: 174 us there, 50.5 on the
// 40,000-bead melt, with the tables staged or not.
template <bool SMEM, int T, bool B>
__global__ void __launch_bounds__(256, 2) k_nonbonded(__grid_constant__ const NBArgs<double> A0,
                                                      const NBArgs<double>* const* tab, const BlockMap bm) {
  using P = Prec<double>;
  pdl_wait();
  pdl_trigger();
  const Blk bk = blk<B>(bm);
  __shared__ NBArgs<double> s_args;
  if (B) stage_args(&s_args, tab[bk.sys]);
  const NBArgs<double>& A = B ? s_args : A0;
  Scalars* sc = A.sc;
  if (nb_idle(A)) return;
  constexpr int PS = 32 / T;
  extern __shared__ unsigned char smem_raw[];
  double* red = (double*)smem_raw;  // 9 * 9 doubles
  const int4* ptab = A.ptab;        // per type pair {first row or -1, NDAT, 1/bin}
  const double4* tco = A.tcoef64;
  if (SMEM) {
    double4* s_co = (double4*)(smem_raw + 96 * sizeof(double));
    int4* s_ptab = (int4*)(s_co + A.nrows);
    for (int k = threadIdx.x; k < A.nrows; k += blockDim.x) s_co[k] = A.tcoef64[k];
    for (int k = threadIdx.x; k < A.ntype * A.ntype; k += blockDim.x) s_ptab[k] = A.ptab[k];
    __syncthreads();
    ptab = s_ptab; tco = s_co;
  }
  double b[3], bi[3], b2[3];
  box_of<double>(sc, b, bi, b2);
  const double4* pos = (const double4*)A.pos4;
  const int lane = threadIdx.x & 31, grp = lane / T, q = lane % T;
  double acc[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) acc[k] = 0.0;
  unsigned err = 0;
  // a work unit is `rows` rows of 32 entries of one slice; the next one's
  // header is loaded while the warp works on this one
  const int rows = A.rows;
  const int U = nb_units_per_slice(A);
  struct Head {
    int u, w, cnt;
  };
  auto head = [&](int u) {
    const int g = U == 1 ? u : u / U;
    const int s = g * PS + grp;
    return Head{u, min(A.slice_w[g], A.w_cap), s < A.n ? A.counts[s] : 0};
  };
  __shared__ int s_next;
  if (threadIdx.x == 0) s_next = 0;
  __syncthreads();
  NbUnits<double> seq(A, bk, U, &s_next);
  struct Geo {
    double d0, d1, d2, r2;
  };
  auto unit = [&](const Head& h) {
    const int g = U == 1 ? h.u : h.u / U;
    const int r0 = (h.u - g * U) * rows, r1 = min(h.w, r0 + rows);
    if (r0 >= r1) return;
    const int s = g * PS + grp;
    // the lane's entries, T per row; a lane without one reads slot 0, which
    // then does not count
    int left = min(h.cnt, r1 * T) - r0 * T - q;
    const bool mine = left > 0;
    const int* e = A.entries + (size_t)g * ((unsigned)A.w_cap * 32u) + (unsigned)(r0 * 32 + lane);
    int t0 = left > 0 ? __ldcs(e) : 0, t1 = left > T ? __ldcs(e + 32) : 0;
    double4 pi;
    if (s < A.n) pi = pos[s];
    else { pi.x = pi.y = pi.z = 0; pi.w = P::tbits(0); }
    const int wi = P::bits(pi.w);
    const int ti = wi & 0xffff, li = wi >> 16;
    const int4* pti = ptab + ti * A.ntype;
    double fi0 = 0, fi1 = 0, fi2 = 0;
    // the nearest image: d - ANINT(d/L) L of two positions inside the box
    // (they could choose differently only at |d| = L/2, beyond the cutoff)
    auto image = [](double d, double L, double half) {
      return d > half ? d - L : (d < -half ? d + L : d);
    };
    auto geo = [&](const double4& pj) {
      Geo G;
      G.d0 = image(pi.x - pj.x, b[0], b2[0]);
      G.d1 = image(pi.y - pj.y, b[1], b2[1]);
      G.d2 = image(pi.z - pj.z, b[2], b2[2]);
      G.r2 = G.d0 * G.d0;
      G.r2 = G.r2 + G.d1 * G.d1;
      G.r2 = G.r2 + G.d2 * G.d2;
      return G;
    };
    // a pair's row and weight; clears `in` (and notes the error) where it has
    // no table or lies beyond it
    auto look = [&](const Geo& G, bool& in, int wj, double& u) {
      const int4 pt = pti[wj & 0xffff];
      const double r = r_sqrt(in ? G.r2 : 1.0);
      const double rb = r * __hiloint2double(pt.w, pt.z);
      const int ni = fint(rb);
      u = rb - (double)ni;
      if (in && pt.x < 0) { err |= EB_MISSING_TABLE; in = false; }
      if (in && (ni < 0 || ni > pt.y)) { err |= EB_TABLE_RANGE; in = false; }
      return in ? pt.x + ni : 0;
    };
    auto pair = [&](const Geo& G, int t, int wj, const double4& co, double u) {
      const double fij = co.x + co.z * u, vij = co.y + co.w * u;
      const int lj = wj >> 16;
      if (li == 1) acc[0] += vij;
      else if (li == 2) {
        if (lj == 2) acc[1] += vij;
        else if (lj == 3) acc[2] += vij;
      } else if (li == 3) acc[2] += vij;
      const double fx = fij * G.d0, fy = fij * G.d1, fz = fij * G.d2;
      fi0 += fx; fi1 += fy; fi2 += fz;
      double* fj = A.fsort + fs_at(t);
      P::add(fj, -fx);
      P::add(fj + 32, -fy);
      P::add(fj + 64, -fz);
      acc[3] += fx * G.d0;
      acc[4] += fy * G.d1;
      acc[5] += fz * G.d2;
      acc[6] += fy * G.d0;
      acc[7] += fz * G.d0;
      acc[8] += fz * G.d1;
    };
    for (int it = r0; it < r1; it += 2) {
      const double4 p0 = pos[(unsigned)t0];
      const double4 p1 = pos[(unsigned)t1];
      const bool v0 = left > 0, v1 = left > T;
      left -= 2 * T;
      e += 64;
      const int n0 = left > 0 ? __ldcs(e) : 0;
      const int n1 = left > T ? __ldcs(e + 32) : 0;
      const Geo g0 = geo(p0), g1 = geo(p1);
      bool in0 = v0 && g0.r2 < A.rcutsq, in1 = v1 && g1.r2 < A.rcutsq;
      if (in0 || in1) {
        const int w0 = P::bits(p0.w), w1 = P::bits(p1.w);
        double u0, u1;
        const int k0 = look(g0, in0, w0, u0), k1 = look(g1, in1, w1, u1);
        const double4 c0 = tco[k0], c1 = tco[k1];
        if (in0) pair(g0, t0, w0, c0, u0);
        if (in1) pair(g1, t1, w1, c1, u1);
      }
      t0 = n0;
      t1 = n1;
    }
#pragma unroll
    for (int o = T / 2; o > 0; o >>= 1) {
      fi0 += __shfl_down_sync(0xffffffffu, fi0, o, T);
      fi1 += __shfl_down_sync(0xffffffffu, fi1, o, T);
      fi2 += __shfl_down_sync(0xffffffffu, fi2, o, T);
    }
    if (q == 0 && mine) {
      double* fo = A.fsort + fs_at(s);
      P::add(fo, fi0);
      P::add(fo + 32, fi1);
      P::add(fo + 64, fi2);
    }
  };
  int u = seq.next();
  Head h{-1, 0, 0};
  if (u >= 0) h = head(u);
  while (h.u >= 0) {
    u = seq.next();
    Head hn{-1, 0, 0};
    if (u >= 0) hn = head(u);
    unit(h);
    h = hn;
  }
  if (err) atomicOr(&sc->err, err);
  __syncthreads();
  block_sums<9>(acc, red);
  if (threadIdx.x < 9) atomicAdd((double*)&sc->nbacc[A.work][threadIdx.x], red[threadIdx.x]);
}

// round(v * 2^S) to the nearest 64-bit integer: the scaling by a power of two
// is exact and the conversion rounds to nearest.  Values of magnitude
// 2^(63-S) and above (and Inf/NaN) raise EB_FIXED and count as 0.
// fabsf(fij) r below 0.99 kFixMax, tested on the force scaled by 2^32
constexpr float kFixLimScaled = 0.99f * kFixMax * kFixScale;
// The FP32 nonbonded kernels' energy and virial sums, at the start of their
// dynamic shared memory: 7 per lane of their blocks for a list of one label, 9
// for a list of several.  A lane adds to its own words, with no
// shuffle and no half-idle warp (per pair of lanes, they took 16 shuffles and
// nine half-warp updates for every eight list rows).
__host__ __device__ constexpr int nb_acc_bytes(bool mixed, int nt) { return (mixed ? 9 : 7) * nt * (int)sizeof(long long); }

template <int S>
__device__ __forceinline__ long long fixq(float v, unsigned& err) {
  const float s = v * (float)(1ull << S);
  if (!(fabsf(s) < 0x1p63f)) { err |= EB_FIXED; return 0; }
  return __float2ll_rn(s);
}

// 1/sqrt(x) of a normal x (squared distances are far above the denormals), as
// rsqrtf gives it there, without rsqrtf's scaling of denormals.
__device__ __forceinline__ float rsqrt_norm(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// The larger of two, NaN if either is.
__device__ __forceinline__ float max_nan(float a, float b) {
  float y;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(y) : "f"(a), "f"(b));
  return y;
}

// v * scale (a power of two) in 2^-24 fixed point, to nearest; saturates
// outside the 64-bit range (the caller checks the range).
__device__ __forceinline__ long long fix24(float v, float scale) { return __float2ll_rn(v * (scale * 0x1p24f)); }

// The block's energy and virial sums, [NE + 6][NT] per lane in lacc, into
// the list's accumulators: V_NB(1..3) and the six virial terms.  With one
// energy sum (NE = 1) it belongs to the label of the list's particles.
template <int NE, int NT>
__device__ __forceinline__ void nb_block_sums(const NBArgs<float>& A, long long* lacc) {
  constexpr int K = NE + 6;
  long long acc[K];
#pragma unroll
  for (int k = 0; k < K; ++k) acc[k] = lacc[k * NT + threadIdx.x];
  __syncthreads();
  block_sums<K>(acc, lacc);
  if (threadIdx.x < K && lacc[threadIdx.x] != 0) {
    int to = (int)threadIdx.x + (3 - NE);
    if (NE == 1 && threadIdx.x == 0) {
      const int li = A.posq[0].w >> 16;
      to = li == 1 ? 0 : (li == 2 ? 1 : 2);
    }
    atomicAdd(&A.sc->nbacc[A.work][to], (unsigned long long)lacc[threadIdx.x]);
  }
}

// NONBONDED_FORCE.F90:45-104, FP32 force path.  Same structure as
// k_nonbonded (slices of P = 32/T slots, T lanes per slot, dynamic units of
// `rows` list rows).  The arithmetic is REAL*4 as in the reference, with
// cheaper equivalents where only the force value (not a bit pattern) is
// compared: positions as 32-bit box fractions, whose wrapped difference is
// the nearest-image displacement at full precision anywhere in the box (a
// REAL*4 coordinate near the box edge carries only 24 bits), r from rsqrt,
// the table row and interpolation weight from a precomputed 1/bin,
// float-to-fixed by the hardware conversion of the exactly scaled value.  Energies and virials are
// summed in FP32 over kEnergyRows list rows, then as 64-bit fixed point
// (2^-24) per lane and per block, and added to the system's accumulators:
// integer sums depend neither on which warp took which unit nor on the rows
// per unit, so they are reproducible and the same alone or in a batch.
// MIXED: the list holds particles of more than one label, so each pair's
// energy term depends on j's label; otherwise every pair adds to the term of
// the list's one label.
// UNI: every type pair of the list has a table, all on one grid that reaches
// past the cutoff, and there are at most eight types (NBArgs::tuni): a pair's
// table number comes from a packed register, its row is that table's first
// row plus r/bin, and there is no descriptor to read and no range to check.
//
// What bounds it, on the 160,000-bead melt (ncu, one launch): L1 data-pipe
// wavefronts (70 %; position gathers ~40 %, table rows ~25 %, reductions ~16
// %) and issue (60 %).  Two rows are evaluated in step so that two positions
// and two table rows are in flight per lane; a pair that does not count reads
// a row of zeros instead of branching; lanes keep their own energy and virial
// sums; the next unit's header is loaded ahead.  58.2 M -> 47 M warp
// instructions.  A launch, between events, caches as the step leaves them:
// 40,000-bead melt 33 us, 160,000 beads 94, the hybrid melt's atoms and sites 52,
// 2,000,000 beads with k_nb_near 1,010 (ncu, cold caches, without it: 1,131
// before, 963 now).  Measured and dropped on 160,000 beads, each beside the kernel
// of its day: positions fetched a row pair ahead (107 us with spills at 64
// registers, 100 at 80 and 24 warps, against 101), units dealt to warps
// statically (94 against 88: uneven slices).  Tables staged in shared memory gain nothing
// (random 16-byte rows conflict on banks as they do on L1 tags: 40,000-bead
// melt 32.8 against 32.6, hybrid melt 61 to 69 against 52); they stay a choice
// of the caller's.
template <bool SMEM, bool MIXED, bool UNI, bool B, int NT>
__global__ void __launch_bounds__(NT, 1024 / NT) k_nonbonded_f32(__grid_constant__ const NBArgs<float> A0,
                                                          const NBArgs<float>* const* tab, const BlockMap bm) {
  constexpr int T = 8;  // lanes per particle (the lists are built for eight)
  constexpr int PS = 32 / T;
  constexpr int NE = MIXED ? 3 : 1;  // energy sums per lane
  pdl_wait();
  pdl_trigger();
  const Blk bk = blk<B>(bm);
  __shared__ NBArgs<float> s_args;
  if (B) stage_args(&s_args, tab[bk.sys]);
  const NBArgs<float>& A = B ? s_args : A0;
  Scalars* sc = A.sc;
  if (nb_idle(A)) return;
  extern __shared__ unsigned char smem_raw[];
  long long* lacc = (long long*)smem_raw;  // [NE + 6][NT] sums of each lane
  // per type pair {first row, last row index, 1/bin bits, has a table}
  const int4* ptab = A.ptab;
  const float4* tco = UNI ? A.tuni : A.tcoef;
  if (SMEM) {
    unsigned char* p = smem_raw + nb_acc_bytes(MIXED, NT);
    int4* s_ptab = (int4*)p;       p += sizeof(int4) * A.ntype * A.ntype;
    float4* s_co = (float4*)p;
    const int nr = UNI ? A.ntab * A.urows : A.nrows;
    for (int k = threadIdx.x; k < nr; k += NT) s_co[k] = tco[k];
    if (!UNI)
      for (int k = threadIdx.x; k < A.ntype * A.ntype; k += NT) s_ptab[k] = A.ptab[k];
    ptab = s_ptab; tco = s_co;
  }
#pragma unroll
  for (int k = 0; k < NE + 6; ++k) lacc[k * NT + threadIdx.x] = 0;
  __shared__ int s_next;
  if (threadIdx.x == 0) s_next = 0;
  __syncthreads();
  // displacement unit per axis: L / 2^32
  const float ux = (float)(sc->box[0] * 0x1p-32), uy = (float)(sc->box[1] * 0x1p-32), uz = (float)(sc->box[2] * 0x1p-32);
  const float2 uxy = make_float2(ux, uy);
  const float inv = A.uinv;
  const int urows = A.urows;
  const float r2_none = A.r2_none, rcut_lo = A.rcut_lo, rcut_hi = A.rcut_hi;
  const int4* pos = A.posq;
  const int lane = threadIdx.x & 31, grp = lane / T, q = lane % T;
  unsigned err = 0;
  float fmax = 0.f;  // largest |F| r, scaled by 2^32 (NaN stays)
  // a work unit is `rows` list rows of one slice (a multiple of kEnergyRows)
  const int rows = A.rows;
  const int U = nb_units_per_slice(A);
  long long* la = lacc + threadIdx.x;
  // a unit, the rows of its slice and the lane's particle's list length: what
  // the next unit's first entries wait for, loaded while the warp works on this one
  struct Head {
    int u, w, cnt;
  };
  auto head = [&](int u) {
    const int g = U == 1 ? u : u / U;
    const int s = g * PS + grp;
    return Head{u, min(A.slice_w[g], A.w_cap), s < A.n ? A.counts[s] : 0};
  };
  auto unit = [&](const Head& h) {
    const int g = U == 1 ? h.u : h.u / U;
    const int r0 = (h.u - g * U) * rows, r1 = min(h.w, r0 + rows);
    if (r0 >= r1) return;
    const int s = g * PS + grp;
    // the lane's entries, T per row, and how many are left from the current
    // row on (a lane without one reads slot 0, which then does not count)
    const int* e = A.entries + (size_t)g * ((unsigned)A.w_cap * 32u) + (unsigned)(r0 * 32 + lane);
    int left = min(h.cnt, r1 * T) - r0 * T - q;
    const bool mine = left > 0;
    int t0 = left > 0 ? __ldcs(e) : 0, t1 = left > T ? __ldcs(e + 32) : 0;
    const int4 pi = s < A.n ? pos[s] : make_int4(0, 0, 0, 0);
    const int ti = pi.w & 0xffff, li = pi.w >> 16;
    const int4* pti = ptab + ti * A.ntype;  // descriptors of (ti, tj) for every tj
    // UNI: table numbers of (ti, 0..7), a byte each
    const uint2 pk = UNI ? A.pbase[ti] : make_uint2(0u, 0u);
    // the energy term of a pair follows from j's label once i's is fixed:
    // V_NB(1) when i is an atom, V_NB(3) when i is a virtual site; when i is
    // a bead, V_NB(2) for a bead j and V_NB(3) for a site j
    const bool i_bead = li == 2;
    long long fi0 = 0, fi1 = 0, fi2 = 0;
    // energies and virials: FP32 over kEnergyRows rows (aligned to multiples of
    // kEnergyRows), then fixed point, so that their sums depend neither on the
    // rows per unit nor on which warp took which unit
    for (int b0 = r0; b0 < r1; b0 += kEnergyRows) {
      const int b1 = min(r1, b0 + kEnergyRows);
      // em: the term of i's label (and bead-bead); e3: bead i with site j.
      // The virials are summed scaled by -2^32 (exact: a power of two):
      // {xx, yy}, {zx, zy}, yx, zz
      float em = 0.f, e3 = 0.f, vyx = 0.f, vzz = 0.f;
      float2 vd = make_float2(0.f, 0.f), vz = vd;
      struct Geo {
        float2 d01;
        float d2, r2;
      };
      // nearest image: the wrapped difference of the box fractions (it and
      // ANINT could choose differently only at |d| = L/2, beyond the cutoff);
      // packed FP32 pairs (fmul/ffma .f32x2) round each element as the
      // scalar instructions do
      auto geo = [&](const int4& pj) {
        Geo G;
        G.d01 = __fmul2_rn(make_float2((float)(int)((unsigned)pi.x - (unsigned)pj.x),
                                       (float)(int)((unsigned)pi.y - (unsigned)pj.y)),
                           uxy);
        G.d2 = (float)(int)((unsigned)pi.z - (unsigned)pj.z) * uz;
        G.r2 = __fmaf_rn(G.d2, G.d2, __fmaf_rn(G.d01.y, G.d01.y, G.d01.x * G.d01.x));
        return G;
      };
      // a pair at the cutoff: k_nb_near decides and computes it (beyond the
      // buffer, it has the step repeated with a larger one)
      auto near = [&](const Geo& G, int t) {
        if (!(G.r2 > rcut_lo && G.r2 < rcut_hi)) return;
        const unsigned k = atomicAdd(&sc->near_n[A.work], 1u);
        if (k < (unsigned)A.near_cap) A.near[k] = make_int4(s, t, A.idx[A.sorted[s]], A.idx[A.sorted[t]]);
      };
      // a pair's interpolation coefficients {F base, P base, dF, dP}, F scaled
      // by -2^32 (exact), its r and its weight u.  One that does not count
      // reads a row of zeros, so that it adds nothing anywhere
      auto look = [&](float r2, bool in, int wj, float& r, float& u) -> float4 {
        if (UNI) {
          r2 = in ? r2 : r2_none;  // in the zero row that ends every table
          r = r2 * rsqrt_norm(r2);
          const float rb = r * inv;  // r / bin
          const int ni = (int)rb;
          u = rb - (float)ni;
          const int t = (int)(__byte_perm(pk.x, pk.y, wj & 0x7) & 0xffu);
          return tco[t * urows + ni];
        }
        r2 = in ? r2 : 1.f;
        r = r2 * rsqrt_norm(r2);
        const int4 pt = pti[wj & 0xffff];
        const float rb = r * __int_as_float(pt.z);
        int ni = (int)rb;
        // a missing table (all-zero descriptor) or a distance beyond the table
        // stops the step with an error; the row read stays inside the array
        // (it holds at least two rows), so no branch is needed here
        err |= !in || pt.w ? 0u : (unsigned)EB_MISSING_TABLE;
        err |= in && ni > pt.y ? (unsigned)EB_TABLE_RANGE : 0u;
        ni = min(ni, pt.y);
        u = rb - (float)ni;
        return in ? tco[pt.x + ni] : make_float4(0.f, 0.f, 0.f, 0.f);
      };
      auto pair = [&](const Geo& G, bool in, int t, int wj, const float4& co, float r, float u) {
        // linear interpolation between rows ni and ni + 1 (NONBONDED_FORCE.F90:66-74)
        const float fs = __fmaf_rn(co.z, u, co.x), vij = __fmaf_rn(co.w, u, co.y);
        if (MIXED) {
          const int lj = wj >> 16;
          em += (!i_bead || lj == 2) ? vij : 0.f;
          e3 += (i_bead && lj == 3) ? vij : 0.f;
        } else {
          em += vij;
        }
        // j's share in fixed point, round(-f * 2^32): fs * d equals the
        // product f_c * -2^32 exactly (scaling by a power of two), and
        // round-to-nearest is symmetric, so i's share is exactly its negation.
        // |f component| <= |fij| r (to rounding): one test keeps every
        // component in range
        fmax = max_nan(fmax, fabsf(fs) * r);
        const float sx = fs * G.d01.x, sy = fs * G.d01.y, sz = fs * G.d2;
        const long long qx = __float2ll_rn(sx), qy = __float2ll_rn(sy), qz = __float2ll_rn(sz);
        fi0 -= qx; fi1 -= qy; fi2 -= qz;
        if (in) {
          unsigned long long* fj = (unsigned long long*)A.fsort + fs_at(t);
          atomicAdd(fj, (unsigned long long)qx);
          atomicAdd(fj + 32, (unsigned long long)qy);
          atomicAdd(fj + 64, (unsigned long long)qz);
        }
        vd = __ffma2_rn(make_float2(sx, sy), G.d01, vd);
        vz = __ffma2_rn(make_float2(sz, sz), G.d01, vz);
        vyx = __fmaf_rn(sy, G.d01.x, vyx);
        vzz = __fmaf_rn(sz, G.d2, vzz);
      };
      // two rows per iteration, in step: both positions are gathered before
      // either distance, both table rows before either force, and the next
      // two entries are on their way meanwhile.  Entries are read once per
      // launch: loaded evict-first (__ldcs), so that the streamed list does
      // not push the positions and force sums it points into out of L2
      for (int it = b0; it < b1; it += 2) {
        const int4 p0 = pos[(unsigned)t0];
        const int4 p1 = pos[(unsigned)t1];
        const bool v0 = left > 0, v1 = left > T;
        left -= 2 * T;
        e += 64;
        const int n0 = left > 0 ? __ldcs(e) : 0;
        const int n1 = left > T ? __ldcs(e + 32) : 0;
        const Geo g0 = geo(p0), g1 = geo(p1);
        const bool in0 = v0 && g0.r2 <= rcut_lo, in1 = v1 && g1.r2 <= rcut_lo;
        if ((g0.r2 > rcut_lo && g0.r2 < rcut_hi) || (g1.r2 > rcut_lo && g1.r2 < rcut_hi)) {
          if (v0) near(g0, t0);
          if (v1) near(g1, t1);
        }
        if (in0 || in1) {
          float r_0, u_0, r_1, u_1;
          const float4 c0 = look(g0.r2, in0, p0.w, r_0, u_0);
          const float4 c1 = look(g1.r2, in1, p1.w, r_1, u_1);
          pair(g0, in0, t0, p0.w, c0, r_0, u_0);
          pair(g1, in1, t1, p1.w, c1, r_1, u_1);
        }
        t0 = n0;
        t1 = n1;
      }
      // the group's sums, 2^-24 fixed point; |.| of each stays below 2^39
      float big;
      if (MIXED) {
        la[(li == 1 ? 0 : (i_bead ? 1 : 2)) * NT] += fix24(em, 1.f);
        la[2 * NT] += fix24(e3, 1.f);
        big = max_nan(fabsf(em), fabsf(e3));
      } else {
        la[0] += fix24(em, 1.f);
        big = fabsf(em);
      }
      const float vir[6] = {vd.x, vd.y, vzz, vyx, vz.x, vz.y};
      float bigv = 0.f;
#pragma unroll
      for (int k = 0; k < 6; ++k) {
        la[(NE + k) * NT] += fix24(vir[k], -0x1p-32f);
        bigv = max_nan(bigv, fabsf(vir[k]));
      }
      if (!(big < 0x1p39f && bigv < 0x1p71f)) err |= (unsigned)EB_FIXED;
    }
#pragma unroll
    for (int o = T / 2; o > 0; o >>= 1) {
      fi0 += __shfl_down_sync(0xffffffffu, fi0, o, T);
      fi1 += __shfl_down_sync(0xffffffffu, fi1, o, T);
      fi2 += __shfl_down_sync(0xffffffffu, fi2, o, T);
    }
    if (mine && q == 0) {
      unsigned long long* fo = (unsigned long long*)A.fsort + fs_at(s);
      atomicAdd(fo, (unsigned long long)fi0);
      atomicAdd(fo + 32, (unsigned long long)fi1);
      atomicAdd(fo + 64, (unsigned long long)fi2);
    }
  };
  NbUnits<float> seq(A, bk, U, &s_next);
  int u = seq.next();
  Head h{-1, 0, 0};
  if (u >= 0) h = head(u);
  while (h.u >= 0) {
    u = seq.next();
    Head hn{-1, 0, 0};
    if (u >= 0) hn = head(u);
    unit(h);
    h = hn;
  }
  if (!(fmax < kFixLimScaled)) err |= (unsigned)EB_FIXED;
  if (err) atomicOr(&sc->err, err);
  nb_block_sums<NE, NT>(A, lacc);
}

// NONBONDED_FORCE.F90:45-104 over slice lists (k_list_build_slices), FP32
// force path.  A warp takes a unit of `rows` rows of one slice: its 32 lanes
// take 32 entries of the slice's list at a time, and each lane evaluates the
// pairs of its entry's neighbour with the (up to four) particles of its mask,
// holding the four particles' positions in registers.  The pair arithmetic,
// cutoff handling, error bits, fixed-point conversion and energy/virial
// grouping are those of k_nonbonded_f32, so every pair's force
// contribution is the same integer and the force sums are bit for bit those
// of the per-particle form.  What changes is what a pair costs in memory
// traffic: one list entry, one position gather and one set of three j-force
// atomics serve all the pairs of an entry, and the slice's i-forces are
// summed over the warp once per unit (a butterfly that leaves each of the
// twelve sums on one pair of lanes) before one atomic each.
template <bool SMEM, bool MIXED, bool B>
__global__ void __launch_bounds__(256, 3) k_nonbonded_slices(__grid_constant__ const NBArgs<float> A0,
                                                             const NBArgs<float>* const* tab, const BlockMap bm) {
  constexpr int NE = MIXED ? 3 : 1;  // energy sums per lane
  pdl_wait();
  pdl_trigger();
  const Blk bk = blk<B>(bm);
  __shared__ NBArgs<float> s_args;
  if (B) stage_args(&s_args, tab[bk.sys]);
  const NBArgs<float>& A = B ? s_args : A0;
  Scalars* sc = A.sc;
  if (nb_idle(A)) return;
  extern __shared__ unsigned char smem_raw[];
  long long* lacc = (long long*)smem_raw;  // [NE + 6][256] sums of each lane
  const int4* ptab = A.ptab;
  const float4* tco = A.tcoef;
  {
    unsigned char* p = smem_raw + nb_acc_bytes(MIXED, 256);
    if (SMEM) {
      int4* s_ptab = (int4*)p;       p += sizeof(int4) * A.ntype * A.ntype;
      float4* s_co = (float4*)p;
      for (int k = threadIdx.x; k < A.nrows; k += blockDim.x) s_co[k] = A.tcoef[k];
      for (int k = threadIdx.x; k < A.ntype * A.ntype; k += blockDim.x) s_ptab[k] = A.ptab[k];
      ptab = s_ptab; tco = s_co;
    }
  }
#pragma unroll
  for (int k = 0; k < NE + 6; ++k) lacc[k * 256 + threadIdx.x] = 0;
  __syncthreads();
  const float ux = (float)(sc->box[0] * 0x1p-32), uy = (float)(sc->box[1] * 0x1p-32), uz = (float)(sc->box[2] * 0x1p-32);
  const float2 uxy = make_float2(ux, uy);
  const int4* pos = A.posq;
  const int lane = threadIdx.x & 31;
  unsigned err = 0;
  const int rows = A.rows;
  const int U = nb_units_per_slice(A);
  long long* la = lacc + threadIdx.x;
  // each warp's slice: the positions of its four particles, read from shared
  // memory by the pair passes (held in registers they push the kernel past
  // its 80-register bound into spills)
  __shared__ int4 s_pi[8][kUSlots];
  auto unit = [&](int u) {
    const int g = u / U;
    const int r0 = (u - g * U) * rows;
    const int w = min(A.slice_w[g], A.w_cap);
    if (r0 >= w) return;
    const int r1 = min(w, r0 + rows);
    const int s0 = kUSlots * g;
    int4* pi = s_pi[threadIdx.x >> 5];
    if (lane < kUSlots) pi[lane] = s0 + lane < A.n ? pos[s0 + lane] : make_int4(0, 0, 0, 0);
    __syncwarp();
    const int* ent = A.entries + (long long)g * A.w_cap * 32 + lane;
    long long fi[kUSlots][3];
#pragma unroll
    for (int k = 0; k < kUSlots; ++k) fi[k][0] = fi[k][1] = fi[k][2] = 0;
    // energies and virials: FP32 over kEnergyRows rows, then fixed point
    for (int b0 = r0; b0 < r1; b0 += kEnergyRows) {
      const int b1 = min(r1, b0 + kEnergyRows);
      // V_NB(1), V_NB(2), V_NB(3) terms (MIXED); e1 alone otherwise.  The
      // virials are summed scaled by -2^32 (exact: a power of two).
      float e1 = 0.f, e2 = 0.f, e3 = 0.f;
      float2 v03 = make_float2(0.f, 0.f), v15 = v03, v24 = v03;
      auto entry = [&](int e, const int4& pj) {
        const int t = (int)((unsigned)e & kUSlotMask);
        const unsigned m = (unsigned)e >> 28;
        const int wj = pj.w;
        const int tj = wj & 0xffff, lj = wj >> 16;
        long long qj0 = 0, qj1 = 0, qj2 = 0;
        bool hit = false;
#pragma unroll
        for (int k = 0; k < kUSlots; ++k) {
          if (!((m >> k) & 1u)) continue;
          const int4 pik = pi[k];
          const float2 d01 = __fmul2_rn(make_float2((float)(int)((unsigned)pik.x - (unsigned)pj.x),
                                                    (float)(int)((unsigned)pik.y - (unsigned)pj.y)),
                                        uxy);
          const float d0 = d01.x, d1 = d01.y;
          const float d2 = (float)(int)((unsigned)pik.z - (unsigned)pj.z) * uz;
          const float r2 = __fmaf_rn(d2, d2, __fmaf_rn(d1, d1, d0 * d0));
          if (!(r2 < A.rcut_hi)) continue;
          if (r2 > A.rcut_lo) {  // at the cutoff: k_nb_near decides and computes it
            const unsigned kk = atomicAdd(&sc->near_n[A.work], 1u);
            if (kk < (unsigned)A.near_cap)
              A.near[kk] = make_int4(s0 + k, t, A.idx[A.sorted[s0 + k]], A.idx[A.sorted[t]]);
            continue;  // beyond the buffer: k_nb_near has the step repeated with a larger one
          }
          const int wi = pik.w;
          const int ti = wi & 0xffff, li = wi >> 16;
          const int4 pt = ptab[ti * A.ntype + tj];
          const float r = r2 * rsqrtf(r2);
          const float rb = r * __int_as_float(pt.z);  // r / bin
          int ni = (int)rb;
          err |= pt.w ? 0u : (unsigned)EB_MISSING_TABLE;
          err |= ni > pt.y ? (unsigned)EB_TABLE_RANGE : 0u;
          ni = min(ni, pt.y);
          const float uu = rb - (float)ni;
          const float4 co = tco[pt.x + ni];  // {F base, P base, dF, dP}
          const float2 fv = __ffma2_rn(make_float2(co.z, co.w), make_float2(uu, uu), make_float2(co.x, co.y));
          const float fs = fv.x, vij = fv.y;  // F scaled by -2^32
          if (MIXED) {
            // V_NB(1) for an atom i, V_NB(3) for a site i or a bead i with a
            // site j, V_NB(2) for two beads
            if (li == 1) e1 += vij;
            else if (li == 3 || lj == 3) e3 += vij;
            else if (lj == 2) e2 += vij;
          } else {
            e1 += vij;
          }
          err |= fabsf(fs) * r < kFixLimScaled ? 0u : (unsigned)EB_FIXED;
          const float2 sxy = __fmul2_rn(make_float2(fs, fs), d01);
          const float sx = sxy.x, sy = sxy.y, sz = fs * d2;
          const long long qx = __float2ll_rn(sx), qy = __float2ll_rn(sy), qz = __float2ll_rn(sz);
          fi[k][0] -= qx; fi[k][1] -= qy; fi[k][2] -= qz;
          qj0 += qx; qj1 += qy; qj2 += qz;
          hit = true;
          v03 = __ffma2_rn(sxy, make_float2(d0, d0), v03);
          v15 = __ffma2_rn(make_float2(sy, sz), make_float2(d1, d1), v15);
          v24 = __ffma2_rn(make_float2(sz, sz), make_float2(d2, d0), v24);
        }
        if (hit) {
          unsigned long long* fj = (unsigned long long*)A.fsort + fs_at(t);
          atomicAdd(fj, (unsigned long long)qj0);
          atomicAdd(fj + 32, (unsigned long long)qj1);
          atomicAdd(fj + 64, (unsigned long long)qj2);
        }
      };
      // two rows per iteration: both entry loads and both position gathers
      // in flight before either is evaluated; entries are read once per
      // launch (evict-first), empty ones (mask 0) point at slot 0
      for (int it = b0; it < b1; it += 2) {
        const bool has1 = it + 1 < b1;
        const int ea = __ldcs(ent + it * 32);
        const int eb = has1 ? __ldcs(ent + (it + 1) * 32) : 0;
        const int4 pa = pos[(unsigned)ea & kUSlotMask];
        const int4 pb = pos[(unsigned)eb & kUSlotMask];
        entry(ea, pa);
        if (has1) entry(eb, pb);
      }
      la[0] += fixq<24>(e1, err);
      if (MIXED) {
        la[256] += fixq<24>(e2, err);
        la[2 * 256] += fixq<24>(e3, err);
      }
      {
        const float vir[6] = {v03.x, v15.x, v24.x, v03.y, v24.y, v15.y};
#pragma unroll
        for (int k = 0; k < 6; ++k) la[(NE + k) * 256] += fixq<24>(vir[k] * -0x1p-32f, err);
      }
    }
    // the twelve i-force sums over the warp: at each level a lane keeps one
    // half of its values and adds the partner's share of that half, which
    // leaves sum 8 b4 + 4 b3 + 2 b2 + b1 (b: the lane's bits) on lanes 2m, 2m+1
    long long v[16];
#pragma unroll
    for (int k = 0; k < kUSlots; ++k)
#pragma unroll
      for (int c = 0; c < 3; ++c) v[3 * k + c] = fi[k][c];
#pragma unroll
    for (int k = 12; k < 16; ++k) v[k] = 0;
#pragma unroll
    for (int h = 8, o = 16; h >= 1; h >>= 1, o >>= 1) {
      const bool up = (lane & o) != 0;
#pragma unroll
      for (int j = 0; j < h; ++j) {
        const long long send = up ? v[j] : v[j + h];
        const long long keep = up ? v[j + h] : v[j];
        v[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
    }
    const long long tot = v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
    const int vi = ((lane >> 4) & 1) * 8 + ((lane >> 3) & 1) * 4 + ((lane >> 2) & 1) * 2 + ((lane >> 1) & 1);
    if (!(lane & 1) && vi < 3 * kUSlots && tot != 0) {
      const int s = s0 + vi / 3;
      if (s < A.n) atomicAdd((unsigned long long*)A.fsort + fs_at(s) + 32 * (vi % 3), (unsigned long long)tot);
    }
    __syncwarp();  // pi is rewritten by the next unit
  };
  __shared__ int s_next;
  if (threadIdx.x == 0) s_next = 0;
  __syncthreads();
  NbUnits<float> seq(A, bk, U, &s_next);
  for (int u = seq.next(); u >= 0; u = seq.next()) unit(u);
  if (err) atomicOr(&sc->err, err);
  nb_block_sums<NE, 256>(A, lacc);
}

// Whether the pair of particles gi, gj (FP32 r^2 = r2) lies inside the cutoff as
// the FP64 path decides it: the same fold of the FP64 state into the box
// (SHIFT), nearest image and sum of squares as k_positions<double> and
// k_nonbonded<double>.  FP32 rounding of r^2 (a relative ~5e-7) would
// otherwise take pairs that sit at the cutoff in or out against that path,
// each a jump of F(rc) r_c in the force (1.3e-5 of the largest force on the
// 40,000-bead melt).  A pair with a virtual site keeps the FP32 decision: its
// FP64 position is not kept on this path.
__device__ bool inside_as_fp64(const NBArgs<float>& A, const Scalars* sc, int gi, int gj, float r2) {
  if (gi >= A.natoms || gj >= A.natoms) return r2 < A.rcutsq;
  double b[3], bi[3], b2[3];
  box_of<double>(sc, b, bi, b2);
  double ri[3], rj[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    ri[c] = A.S[3 * (size_t)gi + c];
    rj[c] = A.S[3 * (size_t)gj + c];
  }
  fold3<double>(ri, b2);
  fold3<double>(rj, b2);
  double d[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    d[c] = ri[c] - rj[c];
    d[c] = d[c] - r_round(d[c] * bi[c]) * b[c];
  }
  double q = d[0] * d[0];
  q = q + d[1] * d[1];
  q = q + d[2] * d[2];
  return q < (double)A.rcutsq;
}

// A pair the FP32 kernel left at the cutoff: decided as the FP64 path decides
// it (inside_as_fp64) and, when inside, computed with the FP32 kernel's pair
// arithmetic.  force(c, q): i's share of component c in fixed point; term(k,
// q): V_NB(1..3) and the six virial terms, k = 0..8.
template <typename Force, typename Term>
__device__ __forceinline__ void near_pair(const NBArgs<float>& A, const int4& nk, float ux, float uy, float uz,
                                          unsigned& err, Force&& force, Term&& term) {
  const int4 pi = A.posq[nk.x], pj = A.posq[nk.y];
  const float d0 = (float)(int)((unsigned)pi.x - (unsigned)pj.x) * ux;
  const float d1 = (float)(int)((unsigned)pi.y - (unsigned)pj.y) * uy;
  const float d2 = (float)(int)((unsigned)pi.z - (unsigned)pj.z) * uz;
  const float r2 = __fmaf_rn(d2, d2, __fmaf_rn(d1, d1, d0 * d0));
  if (!inside_as_fp64(A, A.sc, nk.z, nk.w, r2)) return;
  const int ti = pi.w & 0xffff, li = pi.w >> 16, tj = pj.w & 0xffff, lj = pj.w >> 16;
  const int4 pt = A.ptab[ti * A.ntype + tj];
  if (!pt.w) { err |= EB_MISSING_TABLE; return; }
  const float r = r2 * rsqrtf(r2);
  const float ib = __int_as_float(pt.z);
  const int ni = (int)(r * ib);
  if (ni > pt.y) { err |= EB_TABLE_RANGE; return; }
  const int row = pt.x + ni;
  const float alpha = (r - A.tx[row]) * ib;
  const float2 a0 = ((const float2*)A.tfp)[row], a1 = ((const float2*)A.tfp)[row + 1];
  const float fij = __fmaf_rn(a1.x - a0.x, alpha, a0.x);
  const float vij = __fmaf_rn(a1.y - a0.y, alpha, a0.y);
  if (!(fabsf(fij) * r < 0.99f * kFixMax)) { err |= EB_FIXED; return; }
  const float fx = fij * d0, fy = fij * d1, fz = fij * d2;
  force(0, __float2ll_rn(fx * kFixScale));
  force(1, __float2ll_rn(fy * kFixScale));
  force(2, __float2ll_rn(fz * kFixScale));
  // V_NB(1) for an atom i, V_NB(2) for two beads, V_NB(3) with a site
  if (li == 1 || li == 3 || lj == 3 || lj == 2) term(li == 1 ? 0 : (li == 3 || lj == 3 ? 2 : 1), fixq<24>(vij, err));
  term(3, fixq<24>(fx * d0, err));
  term(4, fixq<24>(fy * d1, err));
  term(5, fixq<24>(fz * d2, err));
  term(6, fixq<24>(fy * d0, err));
  term(7, fixq<24>(fz * d0, err));
  term(8, fixq<24>(fz * d1, err));
}

// More pairs came at the cutoff than their buffer holds: record the need and
// abort the step, which the host repeats with a larger buffer (as for the
// Verlet-list storage).  Other threads of the launch may still be reading the
// count: it stays as it is (the host clears it), so that whoever reads it takes
// the same branch, and that branch leaves without a barrier, since a thread
// that finds the skip flag raised has already left.
__device__ __forceinline__ void near_overflow(Scalars* sc, int work, unsigned n) {
  sc->need_near[work] = (int)n;
  sc->abort = 1;
  sc->skip = 1;
}

// The pairs at the cutoff of a list too long for k_nb_collect to take them
// along (CollectArgs::nb): their forces to the slot-ordered sums, their energy
// and virial terms to the system's fixed-point sums.  One block per system and
// list; the block clears the list's pair count for the next launch.
template <bool B>
__global__ void __launch_bounds__(256) k_nb_near(__grid_constant__ const NBArgs<float> A0,
                                                 const NBArgs<float>* const* tab, const BlockMap bm) {
  pdl_wait();
  pdl_trigger();
  const Blk bk = blk<B>(bm);
  const NBArgs<float>& A = B ? *tab[bk.sys] : A0;
  Scalars* sc = A.sc;
  if (A.near_in_collect || nb_idle(A)) return;
  const unsigned n = sc->near_n[A.work];
  if (n > (unsigned)A.near_cap) {
    if (threadIdx.x == 0) near_overflow(sc, A.work, n);
    return;
  }
  __shared__ long long red[9 + 9 * 8];
  long long acc[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  const float ux = (float)(sc->box[0] * 0x1p-32), uy = (float)(sc->box[1] * 0x1p-32), uz = (float)(sc->box[2] * 0x1p-32);
  unsigned err = 0;
  for (unsigned k = threadIdx.x; k < n; k += blockDim.x) {
    const int4 nk = A.near[k];
    unsigned long long* fsi = (unsigned long long*)A.fsort + fs_at(nk.x);
    unsigned long long* fsj = (unsigned long long*)A.fsort + fs_at(nk.y);
    near_pair(
        A, nk, ux, uy, uz, err,
        [&](int c, long long f) {
          atomicAdd(fsi + 32 * c, (unsigned long long)f);
          atomicAdd(fsj + 32 * c, (unsigned long long)(-f));
        },
        [&](int t, long long e) {
#pragma unroll
          for (int c = 0; c < 9; ++c) acc[c] += c == t ? e : 0;
        });
  }
  if (err) atomicOr(&sc->err, err);
  block_sums<9>(acc, red);
  if (threadIdx.x < 9 && red[threadIdx.x] != 0)
    atomicAdd(&sc->nbacc[A.work][threadIdx.x], (unsigned long long)red[threadIdx.x]);
  __syncthreads();
  if (threadIdx.x == 0) sc->near_n[A.work] = 0u;
}

// Per-slot forces of both lists into the global-order nonbonded force
// array; the bead list's MTS history is saved (MTS_SAVEFORCE, explicit steps)
// or used for the extrapolation F = F3 + (m-3)/2 (F3 - F1) (MTS_APPROX,
// MTS_LOOP.f90:176).  The slot buffer is cleared for the next step.
template <typename R>
struct CollectArgs {
  Scalars* sc;
  int n;                         // slots in this list
  int mts;                       // 1 for the bead list of an MTS run
  const int* sorted;             // slot -> A
  const int* idx;                // A -> global id
  typename Prec<R>::acc_t* fsort;
  typename Prec<R>::acc_t* fnb;  // (3,NITEMS) global order
  typename Prec<R>::acc_t* mtsf; // [3][n][3] by A
  // FP32 path, lists of one slot per thread: the list's nonbonded arguments on
  // the device, whose pairs at the cutoff this kernel takes along; null where
  // k_nb_near has done them
  const NBArgs<float>* nb;
  int work;
};

template <typename R, bool B>
__global__ void __launch_bounds__(256, 4) k_nb_collect(__grid_constant__ const CollectArgs<R> C0, const CollectArgs<R>* const* tab,
                             const BlockMap bm) {
  using P = Prec<R>;
  pdl_wait();
  const Blk bk = blk<B>(bm);
  const CollectArgs<R>& C = B ? *tab[bk.sys] : C0;
  Scalars* sc = C.sc;
  if (sc->skip) return;
  const int m = sc->mts_m;
  const bool explicit_step = !C.mts || (m >= 1 && m <= 3);
  // The pairs at the cutoff (a few per 10,000 particles): every block goes
  // through the list of them and computes those with a slot of its own, so
  // that no launch of its own stands between the nonbonded kernel and this
  // one.  k_finalize clears the count.
  __shared__ unsigned long long s_near[3][256];
  unsigned near_n = 0;
  if constexpr (sizeof(R) == 4) {
    if (C.nb && explicit_step) near_n = sc->near_n[C.work];
    if (near_n > 0) {
      const NBArgs<float>& A = *C.nb;
      if (near_n > (unsigned)A.near_cap) {
        if (bk.b == 0 && threadIdx.x == 0) near_overflow(sc, C.work, near_n);
        return;
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) s_near[c][threadIdx.x] = 0ull;
      __syncthreads();
      const float ux = (float)(sc->box[0] * 0x1p-32), uy = (float)(sc->box[1] * 0x1p-32),
                  uz = (float)(sc->box[2] * 0x1p-32);
      for (unsigned k = threadIdx.x; k < near_n; k += blockDim.x) {
        const int4 nk = A.near[k];
        const bool own_i = (nk.x >> 8) == bk.b, own_j = (nk.y >> 8) == bk.b;
        if (!own_i && !own_j) continue;
        unsigned err = 0;
        near_pair(
            A, nk, ux, uy, uz, err,
            [&](int c, long long f) {
              if (own_i) atomicAdd(&s_near[c][nk.x & 255], (unsigned long long)f);
              if (own_j) atomicAdd(&s_near[c][nk.y & 255], (unsigned long long)(-f));
            },
            [&](int t, long long e) {
              if (own_i && e != 0) atomicAdd(&sc->nbacc[C.work][t], (unsigned long long)e);
            });
        if (own_i && err) atomicOr(&sc->err, err);
      }
      __syncthreads();
    }
  }
  for (int s = bk.b * blockDim.x + threadIdx.x; s < C.n; s += bk.g * blockDim.x) {
    const int a = C.sorted[s];
    const int gi = C.idx[a];
    if (explicit_step) {
      // all three loads before the first store (the arrays may alias as far
      // as the compiler knows)
      typename P::acc_t v[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) v[c] = C.fsort[fs_at(s) + 32 * c];
      if (sizeof(R) == 4 && near_n > 0)
#pragma unroll
        for (int c = 0; c < 3; ++c) v[c] += (typename P::acc_t)s_near[c][threadIdx.x];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        C.fnb[3 * (size_t)gi + c] = v[c];
        if (C.mts) C.mtsf[((size_t)(m - 1) * C.n + a) * 3 + c] = v[c];
        C.fsort[fs_at(s) + 32 * c] = 0;
      }
    } else {
      const double coef = (double)(m - 3) * 0.5;
      double f3[3], f1[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        f3[c] = P::get(C.mtsf[((size_t)2 * C.n + a) * 3 + c]);
        f1[c] = P::get(C.mtsf[((size_t)0 * C.n + a) * 3 + c]);
      }
#pragma unroll
      for (int c = 0; c < 3; ++c)
        C.fnb[3 * (size_t)gi + c] = (typename P::acc_t)P::from_double(f3[c] + coef * (f3[c] - f1[c]), &sc->err);
    }
  }
}

template <typename R>
struct DistArgs {
  Scalars* sc;
  typename Prec<R>::acc_t* F[2];  // nonbonded / bonded forces (3,NITEMS)
  int natoms, nvirta;
  const int* vnum;
  const int* vmem;
  const float* vcoef;
};

// DISTRIBUTE_VSFORCE.f90:27-37: F(atom) += F(vs) * VIRT_MASSCOEFF; F(vs) = 0,
// on the nonbonded (which = 0) or bonded (which = 1) forces.
template <typename R, bool B>
__global__ void k_distribute(__grid_constant__ const DistArgs<R> D0, const DistArgs<R>* const* tab, const BlockMap bm,
                             int which) {
  pdl_wait();
  pdl_trigger();
  using P = Prec<R>;
  const Blk bk = blk<B>(bm);
  const DistArgs<R>& D = B ? *tab[bk.sys] : D0;
  Scalars* sc = D.sc;
  if (sc->skip) return;
  typename P::acc_t* F = D.F[which];
  const int natoms = D.natoms, nvirta = D.nvirta;
  const int* vnum = D.vnum;
  const int* vmem = D.vmem;
  const float* vcoef = D.vcoef;
  // 16 lanes per site (half a warp), one member each (VIRT_NUMATOMS <= 15)
  const int hl = threadIdx.x & 15;
  const unsigned half = 0xffffu << (threadIdx.x & 16);
  const int h0 = (bk.b * blockDim.x + threadIdx.x) >> 4, nh = (bk.g * blockDim.x) >> 4;
  for (int v = h0; v < nvirta; v += nh) {
    const size_t vs = (size_t)(natoms + v);
    double f[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) f[c] = P::get(F[3 * vs + c]);
    if (hl < vnum[v]) {
      const int j = vmem[v * 15 + hl];
      const double cf = (double)vcoef[v * 15 + hl];
#pragma unroll
      for (int c = 0; c < 3; ++c) P::add(&F[3 * (size_t)j + c], P::from_double(f[c] * cf, &sc->err));
    }
    __syncwarp(half);  // the site's 16 lanes have read F(vs)
    if (hl == 0)
#pragma unroll
      for (int c = 0; c < 3; ++c) F[3 * vs + c] = 0;
  }
}

// --------------------------------------------------------------- bonded
template <typename A>
struct BondedArgs {
  Scalars* sc;
  const double* su;                // unwrapped positions (3,NITEMS), FP64
  typename Prec<A>::acc_t* fb;     // bonded forces (3,NITEMS)
  int nb, na, nt, no;
  const int4* bonds;               // i, j, table, label
  const int4* angles;              // i, j, k, table | label<<24
  const int4* tors;                // i, j, k, l
  const int2* tors_t;              // table, label
  const int4* oops;
  const int2* oops_t;
  // tables: rows {X, F, P, 0}; table t starts at off[t]
  const float4* tb; const int* tb_off; const int* tb_ndat; const float* tb_bin;
  const float4* ta; const int* ta_off; const int* ta_ndat; const float* ta_bin;
  const float4* tt; const int* tt_off; const int* tt_ndat; const float* tt_bin;
  const float4* to; const int* to_off; const int* to_ndat; const float* to_bin;
  float r2d;
  double* part;   // 12 per block: V_BOND(3), V_ANGLE(3), V_TORSION(3), V_OOP(3)
  int part_stride;
};

template <typename R>
__device__ __forceinline__ R lerp_mixed(R y0, R y1, R alpha) {
  // y0*(1.0D0-alpha) + alpha*y1 with the FP64 promotion of BONDS.inc:36-40
  return (R)((double)y0 * (1.0 - (double)alpha) + (double)(alpha * y1));
}

template <typename A>
__device__ __forceinline__ void addf(typename Prec<A>::acc_t* F, int i, const double* f, unsigned* err) {
  using P = Prec<A>;
  P::add(&F[3 * (size_t)i + 0], P::from_double(f[0], err));
  P::add(&F[3 * (size_t)i + 1], P::from_double(f[1], err));
  P::add(&F[3 * (size_t)i + 2], P::from_double(f[2], err));
}

// Two shares of one particle's force, sa * a + sb * b (signs +-1), each rounded
// to the accumulator on its own and added in one update per component.
template <typename A>
__device__ __forceinline__ void addf2(typename Prec<A>::acc_t* F, int i, const double* a, const double* b, double sa,
                                      double sb, unsigned* err) {
  using P = Prec<A>;
#pragma unroll
  for (int c = 0; c < 3; ++c)
    P::add(&F[3 * (size_t)i + c], P::from_double(sa * a[c], err) + P::from_double(sb * b[c], err));
}

// BONDS.inc:3-57, ANGLES.inc:2-75, TORSIONS.inc:1-152, OUTOFPLANES.inc:1-141
// with one thread per term; the four term kinds share the grid.  The bonded
// geometry is evaluated in FP64 on both paths: acos near straight angles and
// trans dihedrals amplifies REAL*4 rounding (about 1e-5 of the largest force
// in a strained chain), while the terms are few; the forces are summed in the
// path's accumulator (64-bit fixed point on the FP32 path).  Lengths and sines
// that only scale a force are divided by through one reciprocal each (an angle
// had 20 FP64 divisions, a torsion 27, of ~20 instructions; now 6 and 18).
// Every cosine keeps the reference's divisions: the arc cosine amplifies its
// rounding near straight angles and planar dihedrals, and a torsion's two bond
// angles enter 1/sqrt(1 - cos^2), which does so by 1/sin^2 near straight ones
// (with two reciprocals in their place forces were off by 3e-6 of the largest at
// 1e-5 rad).  A particle's two
// shares of a term are added in one update.
template <typename A, bool BA>
__global__ void __launch_bounds__(256) k_bonded(__grid_constant__ const BondedArgs<A> B0, const BondedArgs<A>* const* tab,
                                                const BlockMap bm) {
  using R = double;
  const Blk bk = blk<BA>(bm);
  const BondedArgs<A>& B = BA ? *tab[bk.sys] : B0;
  Scalars* sc = B.sc;
  __shared__ double red[12 + 12 * 8];
  double acc[12];
#pragma unroll
  for (int k = 0; k < 12; ++k) acc[k] = 0.0;
  unsigned long long overext = 0;
  unsigned* err = &sc->err;
  const R* S = B.su;
  const int total = sc->skip ? 0 : B.nb + B.na + B.nt + B.no;
  auto pos = [&](int i, R* o) { o[0] = S[3 * (size_t)i]; o[1] = S[3 * (size_t)i + 1]; o[2] = S[3 * (size_t)i + 2]; };
  for (int u = bk.b * blockDim.x + threadIdx.x; u < total; u += bk.g * blockDim.x) {
    if (u < B.nb) {  // -------------------------------- bond
      const int4 e = B.bonds[u];
      R ri[3], rj[3], d[3];
      pos(e.x, ri); pos(e.y, rj);
      for (int c = 0; c < 3; ++c) d[c] = ri[c] - rj[c];
      R rsq = d[0] * d[0] + d[1] * d[1];
      rsq = rsq + d[2] * d[2];
      const R rij = r_sqrt(rsq);
      const int t = e.z;
      const float4* T = B.tb + B.tb_off[t];
      const R bin = (R)B.tb_bin[t];
      int k = fint((rij - (R)T[0].x) / bin);  // the quotient: a length of whole bins decides the count below
      if (k > B.tb_ndat[t]) { ++overext; k = B.tb_ndat[t]; }
      else if (k < 0) k = 0;
      const float4 r0 = T[k], r1 = T[k + 1];
      const R alpha = (rij - (R)r0.x) / bin;
      const R fij = lerp_mixed<R>((R)r0.y, (R)r1.y, alpha);
      const R vij = lerp_mixed<R>((R)r0.z, (R)r1.z, alpha);
      acc[e.w - 1] += (double)vij;
      R f[3], mf[3];
      for (int c = 0; c < 3; ++c) { f[c] = fij * d[c]; mf[c] = -f[c]; }
      addf<A>(B.fb, e.x, f, err);
      addf<A>(B.fb, e.y, mf, err);
    } else if (u < B.nb + B.na) {  // ---------------- angle
      const int4 e = B.angles[u - B.nb];
      const int t = e.w & 0xffffff, lab = e.w >> 24;
      R ri[3], rj[3], rk[3], ij[3], kj[3];
      pos(e.x, ri); pos(e.y, rj); pos(e.z, rk);
      for (int c = 0; c < 3; ++c) { ij[c] = ri[c] - rj[c]; kj[c] = rk[c] - rj[c]; }
      const R rij = r_sqrt((ij[0] * ij[0] + ij[1] * ij[1]) + ij[2] * ij[2]);
      const R rkj = r_sqrt((kj[0] * kj[0] + kj[1] * kj[1]) + kj[2] * kj[2]);
      const R iij = (R)1 / rij, ikj = (R)1 / rkj;
      R ct = ((ij[0] * kj[0] + ij[1] * kj[1]) + ij[2] * kj[2]) / rij / rkj;
      ct = ct > (R)1 ? (R)1 : (ct < (R)-1 ? (R)-1 : ct);  // rounding of a straight angle (the oracle clamps too)
      const R theta = r_acos(ct) * (R)B.r2d;
      R m[3];
      m[0] = -(ij[1] * kj[2] - ij[2] * kj[1]);
      m[1] = -(-ij[0] * kj[2] + ij[2] * kj[0]);
      m[2] = -(ij[0] * kj[1] - ij[1] * kj[0]);
      const R rm = r_sqrt((m[0] * m[0] + m[1] * m[1]) + m[2] * m[2]);
      const R irm = (R)1 / rm;
      for (int c = 0; c < 3; ++c) m[c] = m[c] * irm;
      R nn[3], ss[3];
      nn[0] = (m[1] * ij[2] - m[2] * ij[1]) * iij;
      nn[1] = (-m[0] * ij[2] + m[2] * ij[0]) * iij;
      nn[2] = (m[0] * ij[1] - m[1] * ij[0]) * iij;
      ss[0] = -(m[1] * kj[2] - m[2] * kj[1]) * ikj;
      ss[1] = -(-m[0] * kj[2] + m[2] * kj[0]) * ikj;
      ss[2] = -(m[0] * kj[1] - m[1] * kj[0]) * ikj;
      const float4* T = B.ta + B.ta_off[t];
      const R bin = (R)B.ta_bin[t];
      int k = fint(theta / bin);
      if (k < 0 || k > B.ta_ndat[t] + 1) { atomicOr(err, EB_TABLE_RANGE); continue; }
      R fijk, vijk;
      const float4 r0 = T[k];
      if (theta == (R)180.0) {
        fijk = (R)r0.y; vijk = (R)r0.z;
      } else {
        const float4 r1 = T[k + 1];
        const R alpha = (theta - (R)r0.x) / bin;
        fijk = lerp_mixed<R>((R)r0.y, (R)r1.y, alpha);
        vijk = lerp_mixed<R>((R)r0.z, (R)r1.z, alpha);
      }
      acc[3 + lab - 1] += (double)vijk;
      R fI[3], fK[3], mI[3], mK[3];
      for (int c = 0; c < 3; ++c) {
        fI[c] = fijk * nn[c] * iij;
        fK[c] = fijk * ss[c] * ikj;
        mI[c] = -fI[c]; mK[c] = -fK[c];
      }
      addf<A>(B.fb, e.x, fI, err);
      addf<A>(B.fb, e.z, fK, err);
      addf2<A>(B.fb, e.y, mK, mI, (R)1, (R)1, err);
    } else if (u < B.nb + B.na + B.nt) {  // -------- torsion
      const int q = u - B.nb - B.na;
      const int4 e = B.tors[q];
      const int2 tl = B.tors_t[q];
      R ri[3], rj[3], rk[3], rl[3], ij[3], jk[3], kl[3];
      pos(e.x, ri); pos(e.y, rj); pos(e.z, rk); pos(e.w, rl);
      for (int c = 0; c < 3; ++c) { ij[c] = ri[c] - rj[c]; jk[c] = rj[c] - rk[c]; kl[c] = rk[c] - rl[c]; }
      R rij = r_sqrt((ij[0] * ij[0] + ij[1] * ij[1]) + ij[2] * ij[2]);
      const R rjk = r_sqrt((jk[0] * jk[0] + jk[1] * jk[1]) + jk[2] * jk[2]);
      R rkl = r_sqrt((kl[0] * kl[0] + kl[1] * kl[1]) + kl[2] * kl[2]);
      const R ijk = (R)1 / rjk;
      R m[3], nn[3], cosm = 0, isinm = 0, cotanm = 0, cosn = 0, isinn = 0, cotann = 0, iij = 0, ikl = 0;
      auto crossm = [&]() {
        m[0] = ij[1] * jk[2] - ij[2] * jk[1];
        m[1] = -ij[0] * jk[2] + ij[2] * jk[0];
        m[2] = ij[0] * jk[1] - ij[1] * jk[0];
      };
      auto crossn = [&]() {
        nn[0] = jk[1] * kl[2] - jk[2] * kl[1];
        nn[1] = -jk[0] * kl[2] + jk[2] * kl[0];
        nn[2] = jk[0] * kl[1] - jk[1] * kl[0];
      };
      crossm();
      R rm = r_sqrt((m[0] * m[0] + m[1] * m[1]) + m[2] * m[2]);
      if (rm == (R)0) {  // TORSIONS.inc:47-60: perturb collinear i-j-k
        ij[0] = ri[0] * (R)0.99f - rj[0];
        rij = r_sqrt((ij[0] * ij[0] + ij[1] * ij[1]) + ij[2] * ij[2]);
        crossm();
        rm = r_sqrt((m[0] * m[0] + m[1] * m[1]) + m[2] * m[2]);
      }
      if (rm > (R)0 || rm == (R)0) {
        for (int c = 0; c < 3; ++c) m[c] = m[c] / rm;
        iij = (R)1 / rij;
        cosm = ((ij[0] * jk[0] + ij[1] * jk[1]) + ij[2] * jk[2]) / rij / rjk;
        isinm = (R)1 / r_sqrt((R)1 - cosm * cosm);
        cotanm = cosm * isinm;
      }
      crossn();
      R rn = r_sqrt((nn[0] * nn[0] + nn[1] * nn[1]) + nn[2] * nn[2]);
      if (rn == (R)0) {  // TORSIONS.inc:75-88
        kl[0] = rk[0] - rl[0] * (R)0.99f;
        rkl = r_sqrt((kl[0] * kl[0] + kl[1] * kl[1]) + kl[2] * kl[2]);
        crossn();
        rn = r_sqrt((nn[0] * nn[0] + nn[1] * nn[1]) + nn[2] * nn[2]);
      }
      if (rn > (R)0 || rn == (R)0) {
        for (int c = 0; c < 3; ++c) nn[c] = nn[c] / rn;
        ikl = (R)1 / rkl;
        cosn = ((jk[0] * kl[0] + jk[1] * kl[1]) + jk[2] * kl[2]) / rjk / rkl;
        isinn = (R)1 / r_sqrt((R)1 - cosn * cosn);
        cotann = cosn * isinn;
      }
      R cost = (m[0] * nn[0] + m[1] * nn[1]) + m[2] * nn[2];
      const R signt = -((m[0] * kl[0] + m[1] * kl[1]) + m[2] * kl[2]);
      if (cost > (R)1.0) cost = (R)1.0;
      else if (cost < (R)-1.0) cost = (R)-1.0;
      R phi = r_acos(cost) * (R)B.r2d;
      if (signt < (R)0) phi = (R)360.0 - phi;
      const int t = tl.x;
      const float4* T = B.tt + B.tt_off[t];
      const R bin = (R)B.tt_bin[t];
      const int k = fint(phi / bin);
      if (k < 0 || k > B.tt_ndat[t]) { atomicOr(err, EB_TORSION); continue; }
      R fijkl, vijkl;
      const float4 r0 = T[k];
      if (phi == (R)360.0) {
        fijkl = (R)r0.y; vijkl = (R)r0.z;
      } else {
        const float4 r1 = T[k + 1];
        const R alpha = (phi - (R)r0.x) / bin;
        fijkl = (R)r0.y * ((R)1.0 - alpha) + alpha * (R)r1.y;
        vijkl = (R)r0.z * ((R)1.0 - alpha) + alpha * (R)r1.z;
      }
      acc[6 + tl.y - 1] += (double)vijkl;
      R f1[3], f4[3], f12[3];
      for (int c = 0; c < 3; ++c) {
        f1[c] = -(fijkl * m[c] * isinm * iij);
        f4[c] = fijkl * nn[c] * isinn * ikl;
        f12[c] = fijkl * (cotanm * m[c] + cotann * nn[c]) * ijk;
      }
      addf<A>(B.fb, e.x, f1, err);
      addf<A>(B.fb, e.w, f4, err);
      addf2<A>(B.fb, e.y, f1, f12, (R)-1, (R)1, err);
      addf2<A>(B.fb, e.z, f4, f12, (R)-1, (R)-1, err);
    } else {  // ------------------------------------------ out of plane
      const int q = u - B.nb - B.na - B.nt;
      const int4 e = B.oops[q];
      const int2 tl = B.oops_t[q];
      R ri[3], rj[3], rk[3], rl[3], ij[3], jk[3], kl[3];
      pos(e.x, ri); pos(e.y, rj); pos(e.z, rk); pos(e.w, rl);
      for (int c = 0; c < 3; ++c) { ij[c] = ri[c] - rj[c]; jk[c] = rk[c] - rj[c]; kl[c] = rk[c] - rl[c]; }
      const R rij = r_sqrt((ij[0] * ij[0] + ij[1] * ij[1]) + ij[2] * ij[2]);
      const R rjk = r_sqrt((jk[0] * jk[0] + jk[1] * jk[1]) + jk[2] * jk[2]);
      const R rkl = r_sqrt((kl[0] * kl[0] + kl[1] * kl[1]) + kl[2] * kl[2]);
      R m[3], nn[3], mn[3];
      m[0] = ij[1] * jk[2] - ij[2] * jk[1];
      m[1] = -ij[0] * jk[2] + ij[2] * jk[0];
      m[2] = ij[0] * jk[1] - ij[1] * jk[0];
      const R rm = r_sqrt((m[0] * m[0] + m[1] * m[1]) + m[2] * m[2]);
      for (int c = 0; c < 3; ++c) m[c] = m[c] / rm;
      const R cm = ((ij[0] * jk[0] + ij[1] * jk[1]) + ij[2] * jk[2]) / rij / rjk;
      const R sm = r_sqrt((R)1 - cm * cm);
      const R ctm = cm / sm;
      nn[0] = jk[1] * kl[2] - jk[2] * kl[1];
      nn[1] = -jk[0] * kl[2] + jk[2] * kl[0];
      nn[2] = jk[0] * kl[1] - jk[1] * kl[0];
      const R rn = r_sqrt((nn[0] * nn[0] + nn[1] * nn[1]) + nn[2] * nn[2]);
      for (int c = 0; c < 3; ++c) nn[c] = nn[c] / rn;
      const R cn = ((jk[0] * kl[0] + jk[1] * kl[1]) + jk[2] * kl[2]) / rjk / rkl;
      const R sn = r_sqrt((R)1 - cn * cn);
      const R ctn = cn / sn;
      R cost = (m[0] * nn[0] + m[1] * nn[1]) + m[2] * nn[2];
      mn[0] = m[1] * nn[2] - m[2] * nn[1];
      mn[1] = -m[0] * nn[2] + m[2] * nn[0];
      mn[2] = m[0] * nn[1] - m[1] * nn[0];
      const R sgn = copysign((R)1.0, (mn[0] * jk[0] + mn[1] * jk[1]) + mn[2] * jk[2]);
      const R eps = (R)1.0e-7f;
      if (cost > (R)1.0 + eps || cost < -((R)1.0 + eps)) { atomicOr(err, EB_OOP); continue; }
      if (cost > (R)1.0) cost = (R)1.0;
      else if (cost < (R)-1.0) cost = (R)-1.0;
      R phi = r_acos(cost);
      phi = sgn * phi;
      phi = phi * (R)B.r2d;
      const R phit = (R)180.0 + phi;
      const int t = tl.x;
      const float4* T = B.to + B.to_off[t];
      const R bin = (R)B.to_bin[t];
      int k = fint(r_round(phit / bin));
      if (k < 0 || k > B.to_ndat[t]) { atomicOr(err, EB_OOP); continue; }
      R alpha = r_abs(r_abs(phi) - r_abs((R)T[k].x)) / bin;
      if (alpha > (R)1.0) {
        k = k + 1;
        alpha = r_abs(r_abs(phi) - r_abs((R)T[k].x)) / bin;
      }
      const float4 r0 = T[k], r1 = T[k + 1];
      const R fijkl = (R)r0.y * ((R)1.0 - alpha) + alpha * (R)r1.y;
      const R vijkl = (R)r0.z * ((R)1.0 - alpha) + alpha * (R)r1.z;
      acc[9 + tl.y - 1] += (double)vijkl;
      R f1[3], f4[3], f12[3], a[3];
      for (int c = 0; c < 3; ++c) {
        f1[c] = fijkl * m[c] / sm / rij;
        f4[c] = -(fijkl * nn[c] / sn / rkl);
        f12[c] = fijkl * (ctm * m[c] + ctn * nn[c]) / rjk;
      }
      addf<A>(B.fb, e.x, f1, err);
      addf<A>(B.fb, e.w, f4, err);
      for (int c = 0; c < 3; ++c) a[c] = -f1[c];
      addf<A>(B.fb, e.y, a, err);
      addf<A>(B.fb, e.y, f12, err);
      for (int c = 0; c < 3; ++c) a[c] = -f4[c];
      addf<A>(B.fb, e.z, a, err);
      for (int c = 0; c < 3; ++c) a[c] = -f12[c];
      addf<A>(B.fb, e.z, a, err);
    }
  }
  if (overext) atomicAdd(&sc->bond_overext, overext);
  block_sums<12>(acc, red);
  if (threadIdx.x < 12) B.part[threadIdx.x * B.part_stride + bk.b] = red[threadIdx.x];
}

// ------------------------------------------------------------ integration
template <typename R>
struct MoveArgs {
  Scalars* sc;
  int natoms;
  double* S;  // (3,NATOMS) unwrapped, FP64 state
  double* V;  // (3,NATOMS)
  typename Prec<R>::acc_t* fnb;
  typename Prec<R>::acc_t* fb;
  const int* tbits;         // label in bits 16.. (1 atom, 2 bead)
  const double* mass;       // per particle
  const double* invmass;    // per particle
  double dt;
  int update;               // 0: bonded virial only (force stage without MOVE)
  double* part;             // 18 per block
  int part_stride;
};

// MOVE.F90:32-88 (leap-frog with Berendsen factors per class) and the
// bonded virial sum of NEW_FORCE.F90:73-80, which uses the positions before
// the update.  Partials: PTK(6) atoms, PTK(6) beads, bonded virial(6).  The
// bonded forces are folded into the nonbonded array (fnb becomes the total
// force FXYZ of the step) and cleared for the next step.
template <typename R, bool B>
__global__ void __launch_bounds__(256, 3) k_move(__grid_constant__ const MoveArgs<R> M0, const MoveArgs<R>* const* tab,
                                              const BlockMap bm) {
  using P = Prec<R>;
  pdl_wait();
  pdl_trigger();
  const Blk bk = blk<B>(bm);
  const MoveArgs<R>& M = B ? *tab[bk.sys] : M0;
  Scalars* sc = M.sc;
  __shared__ double red[18 + 18 * 8];
  double acc[18];
#pragma unroll
  for (int k = 0; k < 18; ++k) acc[k] = 0.0;
  const double lam0 = sc->lam[0], lam1 = sc->lam[1];
  const int nrun = sc->skip ? 0 : M.natoms;
  for (int i = bk.b * blockDim.x + threadIdx.x; i < nrun; i += bk.g * blockDim.x) {
    // every load of the particle is issued before its first store: the
    // arrays may alias as far as the compiler knows, so a store between two
    // loads would make each wait for the one before
    double s[3], v[3], fb[3], f[3];
    typename P::acc_t qb[3], qn[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      s[c] = M.S[3 * (size_t)i + c];
      v[c] = M.V[3 * (size_t)i + c];
      qb[c] = M.fb[3 * (size_t)i + c];
      qn[c] = M.fnb[3 * (size_t)i + c];
    }
    int tb = 0;
    double m = 0.0, im = 0.0;
    if (M.update) { tb = M.tbits[i]; m = M.mass[i]; im = M.invmass[i]; }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      fb[c] = P::get(qb[c]);
      f[c] = P::get(qn[c]) + fb[c];
      M.fnb[3 * (size_t)i + c] = qn[c] + qb[c];
      M.fb[3 * (size_t)i + c] = 0;
    }
    acc[12] += fb[0] * s[0];
    acc[13] += fb[1] * s[1];
    acc[14] += fb[2] * s[2];
    acc[15] += fb[1] * s[0];
    acc[16] += fb[2] * s[0];
    acc[17] += fb[2] * s[1];
    if (!M.update) continue;
    const int cls = (tb >> 16) == 2 ? 1 : 0;
    const double lam = cls ? lam1 : lam0;
    double vt[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double vn = (v[c] + M.dt * f[c] * im) * lam;
      M.V[3 * (size_t)i + c] = vn;
      M.S[3 * (size_t)i + c] = s[c] + M.dt * vn;
      vt[c] = 0.5 * (vn + v[c]);
    }
    // both classes' sums, the other class's term zero (an index by class would
    // put the sums into local memory)
    const double ma = cls ? 0.0 : m, mb = cls ? m : 0.0;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const double x = vt[k < 3 ? k : (k < 5 ? 0 : 1)], y = vt[k < 3 ? k : (k == 3 ? 1 : 2)];
      acc[k] += ma * x * y;
      acc[6 + k] += mb * x * y;
    }
  }
  block_sums<18>(acc, red);
  if (threadIdx.x < 18) M.part[threadIdx.x * M.part_stride + bk.b] = red[threadIdx.x];
}

// Initial kinetic energies (main.F90:179-195).  Partials: EK atoms, EK beads.
__global__ void k_kinetic(int natoms, const double* V, const int* tbits, const double* mass, double* part, int stride) {
  __shared__ double red[2 + 2 * 8];
  double acc[2] = {0.0, 0.0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < natoms; i += gridDim.x * blockDim.x) {
    const double* v = V + 3 * (size_t)i;
    acc[(tbits[i] >> 16) == 2 ? 1 : 0] += mass[i] * ((v[0] * v[0] + v[1] * v[1]) + v[2] * v[2]);
  }
  block_sums<2>(acc, red);
  if (threadIdx.x < 2) part[threadIdx.x * stride + blockIdx.x] = red[threadIdx.x];
}

struct MomArgs {
  Scalars* sc;
  int natoms, halt_drift;
  double* V;
  const double* mass;
  const double* invmass;
  double* part;  // 3 per block, nblocks blocks
  int nblocks;
};

// MOMENTUM.f90:14-29 in FP64 on steps that are multiples of HALT_DRIFT
// (NEW_LOOP.F90:108-114): partial sums of m v, then the removal.
template <bool B>
__global__ void k_mom_sum(__grid_constant__ const MomArgs A0, const MomArgs* const* tab, const BlockMap bm) {
  const Blk bk = blk<B>(bm);
  const MomArgs& A = B ? *tab[bk.sys] : A0;
  const Scalars* sc = A.sc;
  if (sc->skip || sc->step % A.halt_drift != 0) return;
  __shared__ double red[3 + 3 * 8];
  double acc[3] = {0.0, 0.0, 0.0};
  for (int i = bk.b * blockDim.x + threadIdx.x; i < A.natoms; i += bk.g * blockDim.x)
    for (int c = 0; c < 3; ++c) acc[c] += A.V[3 * (size_t)i + c] * A.mass[i];
  block_sums<3>(acc, red);
  if (threadIdx.x < 3) A.part[threadIdx.x * A.nblocks + bk.b] = red[threadIdx.x];
}

template <bool B>
__global__ void k_mom_apply(__grid_constant__ const MomArgs A0, const MomArgs* const* tab, const BlockMap bm) {
  const Blk bk = blk<B>(bm);
  const MomArgs& A = B ? *tab[bk.sys] : A0;
  const Scalars* sc = A.sc;
  if (sc->skip || sc->step % A.halt_drift != 0) return;
  __shared__ double tot[3];
  if (threadIdx.x < 32) {
    for (int c = 0; c < 3; ++c) {
      double s = 0.0;
      for (int b = threadIdx.x; b < A.nblocks; b += 32) s += A.part[c * A.nblocks + b];
      s = warp_sum(s);
      if (threadIdx.x == 0) tot[c] = s / (double)A.natoms;
    }
  }
  __syncthreads();
  for (int i = bk.b * blockDim.x + threadIdx.x; i < A.natoms; i += bk.g * blockDim.x)
    for (int c = 0; c < 3; ++c) A.V[3 * (size_t)i + c] -= tot[c] * A.invmass[i];
}

// SCALEBP.f90:37-39: positions scaled with the box on the steps the
// barostat changed it.
template <typename R, bool B>
__global__ void k_scale_positions(__grid_constant__ const MoveArgs<R> M0, const MoveArgs<R>* const* tab,
                                  const BlockMap bm) {
  const Blk bk = blk<B>(bm);
  const MoveArgs<R>& M = B ? *tab[bk.sys] : M0;
  const Scalars* sc = M.sc;
  if (sc->skip) return;
  const double miu = sc->miu;
  if (miu == 1.0) return;
  for (int i = bk.b * blockDim.x + threadIdx.x; i < M.natoms; i += bk.g * blockDim.x)
    for (int c = 0; c < 3; ++c) M.S[3 * (size_t)i + c] *= miu;
}

// ------------------------------------------------------------- reductions
struct FinalArgs {
  Scalars* sc;
  int fixed;                         // nonbonded accumulators in fixed point (FP32 path)
  const double* p_b; int g_b;        // bonded partials (12 x g_b)
  const double* p_mv; int g_mv;      // move partials (18 x g_mv)
  int mts;                           // MTS run
  int move;                          // 1: full step (kinetic part, thermostat, barostat)
  int ensemble;
  double temp_in, fac, pfac, pressure, mktemp, mktemp_atom, mktemp_bead;
  ObsD* ring; int ring_cap;
};

// Sum of g partials by one warp: each lane adds its own in increasing order
// (p[lane], p[lane+32], ...), then the lanes are summed.  Eight loads per lane
// are issued before they are added, so the warp waits for memory once per
// eight rather than once per partial; the order of the additions is the same.
__device__ double wsum(const double* p, int g) {
  double s = 0.0;
  for (int b0 = threadIdx.x & 31; b0 < g; b0 += 8 * 32) {
    double v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = b0 + 32 * k < g ? p[b0 + 32 * k] : 0.0;
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (b0 + 32 * k < g) s += v[k];
  }
  return warp_sum(s);
}

// Deterministic reduction of all partials into the observables, the MTS
// auxiliary history (MTS_SAVEAUXS / MTS_LOADAUXS), the thermostat factors of
// the next step and the barostat window (SCALEBP.f90:18-41).  The
// nonbonded accumulators are read and cleared for the next step.
template <bool B>
__global__ void k_finalize(__grid_constant__ const FinalArgs F0, const FinalArgs* const* tab, const BlockMap bm) {
  pdl_wait();
  pdl_trigger();
  const Blk bk = blk<B>(bm);
  const FinalArgs& F = B ? *tab[bk.sys] : F0;
  Scalars* sc = F.sc;
  __shared__ double q[64];
  if (sc->skip) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  // what warp 0 needs of the scalars after the sums, on its way meanwhile
  const int m = sc->mts_m, step = sc->step, stop_at = sc->stop_at, iavp = sc->iavp, ring_base = sc->ring_base;
  const unsigned err = sc->err;
  const unsigned long long overext = sc->bond_overext, clamps = sc->cell_clamps;
  double box[3];
  for (int c = 0; c < 3; ++c) box[c] = sc->box[c];
  const double prev = ((const double*)&sc->obs)[lane];
  double h3 = 0.0, h1 = 0.0;  // MTS history of bead sum `lane`: V_NB(1..3), PT11..PT23
  if (F.mts && lane < 9) {
    h3 = lane < 3 ? sc->mts_vnb[2][lane] : sc->mts_pt[lane - 3][2];
    h1 = lane < 3 ? sc->mts_vnb[0][lane] : sc->mts_pt[lane - 3][0];
  }
  // q[0..8] atom NB, q[9..17] bead NB, q[18..29] bonded, q[30..47] move
  if (threadIdx.x < 18) {
    unsigned long long* p = &sc->nbacc[threadIdx.x / 9][threadIdx.x % 9];
    const unsigned long long v = *p;
    q[threadIdx.x] = F.fixed ? (double)(long long)v * kEnInv : __longlong_as_double((long long)v);
    *p = 0ull;
  }
  for (int k = 18 + warp; k < 48; k += nw) {
    double v;
    if (k < 30) v = wsum(F.p_b + (size_t)(k - 18) * F.g_b, F.g_b);
    else v = wsum(F.p_mv + (size_t)(k - 30) * F.g_mv, F.g_mv);
    if (lane == 0) q[k] = v;
  }
  __syncthreads();
  if (warp) return;
  // lane c < 9: sum c of both lists, 0..2 the energies and 3..8 the virial
  double sum = 0.0;
  if (lane < 9) {
    double bead = q[9 + lane];
    if (F.mts) {
      if (m >= 1 && m <= 3) {
        // PT23 is not saved (MTS_LOOP.f90:193-199)
        if (lane < 3) sc->mts_vnb[m - 1][lane] = bead;
        else if (lane < 8) sc->mts_pt[lane - 3][m - 1] = bead;
      } else {
        bead = h3 + (double)(m - 3) * 0.5 * (h3 - h1);
      }
    }
    sum = q[lane] + bead;
    if (lane >= 3) sum = sum + q[42 + lane - 3];
  }
  double ek[2] = {0.0, 0.0}, temp[3] = {0.0, 0.0, 0.0};
  if (F.move) {
    // MOVE.F90:90-115
    if (lane >= 3 && lane < 9) {
      sum += q[30 + lane - 3] + q[36 + lane - 3];
      sum /= box[0] * box[1] * box[2];
    }
    ek[0] = 0.5 * (q[30] + q[31] + q[32]);
    ek[1] = 0.5 * (q[36] + q[37] + q[38]);
    temp[0] = (ek[0] + ek[1]) * F.mktemp;
    temp[1] = ek[0] * F.mktemp_atom;
    temp[2] = ek[1] * F.mktemp_bead;
    if (lane < 2) {
      const double t = lane == 0 ? temp[1] : temp[2];
      (lane == 0 ? sc->temp_atom : sc->temp_bead) = t;
      if (F.ensemble == 1 || F.ensemble == 2)  // MOVE.F90:32-38, for the next step
        sc->lam[lane] = sqrt(1.0 + F.fac * ((F.temp_in / t) - 1.0));
    }
    if (F.ensemble == 2) {  // SCALEBP.f90:18-41
      const double p3 = __shfl_sync(0xffffffffu, sum, 3), p4 = __shfl_sync(0xffffffffu, sum, 4),
                   p5 = __shfl_sync(0xffffffffu, sum, 5);
      int iv = iavp + 1;
      if (iv > 10) iv -= 10;
      const double now = (p3 + p4 + p5) / 3.0;
      if (lane == 0) {
        sc->iavp = iv;
        sc->sp[iv - 1] = now;
      }
      if (step % 10 == 0) {
        double avp = 0.0;
        for (int i = 0; i < 10; ++i) avp += i == iv - 1 ? now : sc->sp[i];
        const double p = avp / 10.0;
        const double miu = pow(1.0 + (p - F.pressure) * F.pfac, 1.0 / 3.0);
        for (int c = 0; c < 3; ++c) box[c] *= miu;
        if (lane == 0) sc->miu = miu;
        if (lane < 3) {
          const double b = lane == 0 ? box[0] : (lane == 1 ? box[1] : box[2]);
          sc->box[lane] = b;
          sc->boxinv[lane] = 1.0 / b;
          sc->box2[lane] = b / 2.0;
          const float bf = (float)b;
          sc->boxf[lane] = bf;
          sc->boxinvf[lane] = 1.0f / bf;
          sc->box2f[lane] = bf / 2.0f;
        }
      }
    }
  }
  // the observables, one 8-byte field per lane (a force stage keeps the
  // kinetic part of the step before)
  __shared__ double ob[32];
  ob[lane] = prev;
  __syncwarp();
  if (F.move && lane < 5) ob[lane] = lane < 2 ? ek[lane & 1] : temp[lane - 2];
  if (lane < 3) ob[5 + lane] = sum;
  if (lane < 12) ob[8 + lane] = q[18 + lane];
  if (lane >= 3 && lane < 9) ob[20 + lane - 3] = sum;
  if (lane < 3) ob[26 + lane] = lane == 0 ? box[0] : (lane == 1 ? box[1] : box[2]);
  if (lane == 29) ob[29] = __longlong_as_double((long long)overext);
  if (lane == 30) ob[30] = __longlong_as_double((long long)clamps);
  if (lane == 31) ob[31] = __longlong_as_double((long long)(((unsigned long long)err << 32) | (unsigned)step));
  __syncwarp();
  static_assert(sizeof(ObsD) == 32 * sizeof(double), "one field per lane");
  ((double*)&sc->obs)[lane] = ob[lane];
  if (lane == 0) sc->done = step >= stop_at;
  if (lane < 2) sc->near_n[lane] = 0u;
  const int slot = step - ring_base;
  if (F.ring && slot >= 0 && slot < F.ring_cap) ((double*)&F.ring[slot])[lane] = ob[lane];
}

// Step counter, observable ring base and step limit of the next run.
__global__ void k_set_counter(Scalars* sc, int step_before, int ring_base, int last) {
  sc->step = step_before;
  sc->ring_base = ring_base;
  sc->skip = 0;
  sc->stop_at = last;
  sc->done = step_before >= last ? 1 : 0;
}

// What the host reads after a batch's run, of every system in one copy.
struct BatchStat {
  int abort, step;
  unsigned err, pad;
  ObsD obs;
};
__global__ void k_batch_stat(const Scalars* const* scs, BatchStat* out) {
  const Scalars* sc = scs[blockIdx.x];
  BatchStat& o = out[blockIdx.x];
  for (int k = threadIdx.x; k < (int)(sizeof(ObsD) / 8); k += blockDim.x)
    ((double*)&o.obs)[k] = ((const double*)&sc->obs)[k];
  if (threadIdx.x == 0) {
    o.abort = sc->abort;
    o.step = sc->step;
    o.err = sc->err;
  }
}

// Initial temperatures and Berendsen factors (main.F90:174-195).
__global__ void k_init_temps(const double* part, int g, Scalars* sc, double mktemp, double mktemp_atom,
                             double mktemp_bead, double temp_in, double fac, int ensemble) {
  __shared__ double q[2];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp < 2) {
    double v = wsum(part + (size_t)warp * g, g);
    if (lane == 0) q[warp] = v;
  }
  __syncthreads();
  if (threadIdx.x) return;
  ObsD& o = sc->obs;
  o.ek[0] = 0.5 * q[0];
  o.ek[1] = 0.5 * q[1];
  o.temp = (o.ek[0] + o.ek[1]) * mktemp;
  o.temp_atom = o.ek[0] * mktemp_atom;
  o.temp_bead = o.ek[1] * mktemp_bead;
  sc->temp_atom = o.temp_atom;
  sc->temp_bead = o.temp_bead;
  if (ensemble == 1 || ensemble == 2) {
    sc->lam[0] = sqrt(1.0 + fac * ((temp_in / o.temp_atom) - 1.0));
    sc->lam[1] = sqrt(1.0 + fac * ((temp_in / o.temp_bead) - 1.0));
  } else {
    sc->lam[0] = sc->lam[1] = 1.0;
  }
}

}  // namespace ibg
