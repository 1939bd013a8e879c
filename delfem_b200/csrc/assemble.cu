// Element assembly into the block-CRS matrix and the residual, and the
// Dirichlet elimination, on the device.
//
// Reference element loops (one element at a time, Mearge scatter-add):
//   AddLinearSystem_Poisson2D_P1            src/femeqn/eqn_poisson.cpp:49-125
//   AddLinSys_LinearSolid2D_Static_P1       src/femeqn/eqn_linear_solid2d.cpp:505-598
//   AddLinSys_LinearSolid3D_Static_P1       src/femeqn/eqn_linear_solid3d.cpp:241-334
//   AddLinearSystem_Helmholtz2D_P1          src/femeqn/eqn_helmholtz.cpp:51-137
//   AddLinearSystem_SommerfeltRadiationBC2D_B1  src/femeqn/eqn_helmholtz.cpp:437-512
//   CMatDia_BlkCrs::Mearge                  src/matvec/matdia_blkcrs.cpp:165-258
//   CMatDia_BlkCrs::SetBoundaryCondition    src/matvec/matdia_blkcrs.cpp:261-343
//   CBCFlag::SetZeroToBCDof                 include/delfem/matvec/bcflag_blk.h:102-129
//
// Gather formulation: a group of lanes owns a node (a block row): a warp for
// tetrahedra (24 elements around a node of a box), 8 lanes for triangles (6).
// Its lanes compute the element-matrix rows of as many surrounding elements at
// once (ascending order, from a node->element adjacency built at mesh set-up)
// into shared memory and list, for every slot of the row, the contributions it
// gets in element order; then the row's values are dealt to the lanes one by
// one (value v of the row's contiguous run to lane v mod L, the diagonal
// block last), each adding its contributions in that order.  Each value
// therefore receives the same additions in the same order as in the
// reference's sequential scatter, and with this file compiled without FMA
// contraction (-fmad=false) the assembled values are bit-identical.
//
// What bounds it is latency: four dependent reads per node (adjacency,
// elements, coordinates) and the chains of FP64 operations of its elements'
// geometry, which each of their nodes computes, at 20 warps per SM (registers
// and shared memory allow no more).  On the 200x40x40 box the issue slots are
// 50% busy, shared memory 62%, the FP64 pipe 23%, DRAM 5%.  A lane per slot that looked through
// all contributions for its own took 2.48 ms on the 200x40x40 box (337,881
// nodes, 371 MB of values): 96 comparisons and the 24 additions of the diagonal
// block in one lane, while the others waited.
#include <algorithm>
#include <new>

#include "dfm_internal.h"

struct dfm_mesh_s {
  dfm_ctx ctx = nullptr;
  int ndim = 2;
  unsigned nnode = 0, nnoel = 3, nelem = 0, nbar = 0;
  double* d_coord = nullptr;
  int* d_elem = nullptr;
  int* d_bar = nullptr;
  unsigned* d_esup_ptr = nullptr;  // node -> elements (ascending)
  unsigned* d_esup = nullptr;
  unsigned* d_bsup_ptr = nullptr;  // node -> boundary bars (ascending)
  unsigned* d_bsup = nullptr;
  std::vector<int> h_elem;         // host copies for the pattern
  std::vector<unsigned> h_esup_ptr, h_esup;
};

namespace dfm {

constexpr int kAsmWarps = 4;  // warps (nodes) per CTA

// ---------------------------------------------------- element geometry (ref. order)
DFM_DEVINL double tri_area(const double* p0, const double* p1, const double* p2) {
  return 0.5 * ((p1[0] - p0[0]) * (p2[1] - p0[1]) - (p2[0] - p0[0]) * (p1[1] - p0[1]));
}
DFM_DEVINL void tri_dldx(double d[3][2], const double* p0, const double* p1, const double* p2) {
  const double area = tri_area(p0, p1, p2);
  const double tmp1 = 0.5 / area;
  d[0][0] = tmp1 * (p1[1] - p2[1]);
  d[1][0] = tmp1 * (p2[1] - p0[1]);
  d[2][0] = tmp1 * (p0[1] - p1[1]);
  d[0][1] = tmp1 * (p2[0] - p1[0]);
  d[1][1] = tmp1 * (p0[0] - p2[0]);
  d[2][1] = tmp1 * (p1[0] - p0[0]);
}
DFM_DEVINL double tet_volume(const double* p0, const double* p1, const double* p2, const double* p3) {
  double v = (p1[0] - p0[0]) * ((p2[1] - p0[1]) * (p3[2] - p0[2]) - (p3[1] - p0[1]) * (p2[2] - p0[2]))
           - (p1[1] - p0[1]) * ((p2[0] - p0[0]) * (p3[2] - p0[2]) - (p3[0] - p0[0]) * (p2[2] - p0[2]))
           + (p1[2] - p0[2]) * ((p2[0] - p0[0]) * (p3[1] - p0[1]) - (p3[0] - p0[0]) * (p2[1] - p0[1]));
  v *= 0.1666666666666;  // the reference's truncated 1/6 (include/delfem/femeqn/ker_emat_tet.h:32-40)
  return v;
}
DFM_DEVINL void tet_dldx(double d[4][3], const double* p0, const double* p1, const double* p2, const double* p3) {
  const double vol = tet_volume(p0, p1, p2, p3);
  const double t = 1.0 / (vol * 6.0);
  d[0][0] = -t * ((p2[1] - p1[1]) * (p3[2] - p1[2]) - (p3[1] - p1[1]) * (p2[2] - p1[2]));
  d[0][1] = +t * ((p2[0] - p1[0]) * (p3[2] - p1[2]) - (p3[0] - p1[0]) * (p2[2] - p1[2]));
  d[0][2] = -t * ((p2[0] - p1[0]) * (p3[1] - p1[1]) - (p3[0] - p1[0]) * (p2[1] - p1[1]));
  d[1][0] = +t * ((p3[1] - p2[1]) * (p0[2] - p2[2]) - (p0[1] - p2[1]) * (p3[2] - p2[2]));
  d[1][1] = -t * ((p3[0] - p2[0]) * (p0[2] - p2[2]) - (p0[0] - p2[0]) * (p3[2] - p2[2]));
  d[1][2] = +t * ((p3[0] - p2[0]) * (p0[1] - p2[1]) - (p0[0] - p2[0]) * (p3[1] - p2[1]));
  d[2][0] = -t * ((p0[1] - p3[1]) * (p1[2] - p3[2]) - (p1[1] - p3[1]) * (p0[2] - p3[2]));
  d[2][1] = +t * ((p0[0] - p3[0]) * (p1[2] - p3[2]) - (p1[0] - p3[0]) * (p0[2] - p3[2]));
  d[2][2] = -t * ((p0[0] - p3[0]) * (p1[1] - p3[1]) - (p1[0] - p3[0]) * (p0[1] - p3[1]));
  d[3][0] = +t * ((p1[1] - p0[1]) * (p2[2] - p0[2]) - (p2[1] - p0[1]) * (p1[2] - p0[2]));
  d[3][1] = -t * ((p1[0] - p0[0]) * (p2[2] - p0[2]) - (p2[0] - p0[0]) * (p1[2] - p0[2]));
  d[3][2] = +t * ((p1[0] - p0[0]) * (p2[1] - p0[1]) - (p2[0] - p0[0]) * (p1[1] - p0[1]));
}

// ------------------------------------------------ element kinds (row `a` only)
// entry a of three without an indexed (local-memory) array
DFM_DEVINL double pick3(int a, double v0, double v1, double v2) { return a == 0 ? v0 : a == 1 ? v1 : v2; }

struct AsmParams {
  double p[6];          // kind parameters (alpha,source | lambda,myu,rho,g.. | wave_length)
  const double* coef;   // per-element multiplier or nullptr
  const double* u;      // current field or nullptr (res += f_e - K_e u_e)
};

enum { K_POISSON = 0, K_SOLID2D = 1, K_SOLID3D = 2, K_HELM = 3, K_SOMMER = 4 };

template <int KIND> struct Kind;

// Poisson P1 triangle, b = 1
template <> struct Kind<K_POISSON> {
  static constexpr int NNO = 3, NDIM = 2, BW = 1, RW = 1;  // block width (doubles), residual width
  DFM_DEVINL static void row(const AsmParams& P, unsigned e, const int* no, const double* X, int a, double* blk,
                             double* res) {
    const double *p0 = X + 2 * no[0], *p1 = X + 2 * no[1], *p2 = X + 2 * no[2];
    const double area = tri_area(p0, p1, p2);
    double d[3][2];
    tri_dldx(d, p0, p1, p2);
    const double alpha = P.coef ? P.p[0] * P.coef[e] : P.p[0];
    const double a0 = pick3(a, d[0][0], d[1][0], d[2][0]), a1 = pick3(a, d[0][1], d[1][1], d[2][1]);
    double em[3];
    for (int c = 0; c < 3; c++) em[c] = alpha * area * (a0 * d[c][0] + a1 * d[c][1]);
    for (int c = 0; c < 3; c++) blk[c] = em[c];
    double r = P.p[1] * area * 0.33333333333333333;
    if (P.u)
      for (int c = 0; c < 3; c++) r -= em[c] * P.u[no[c]];
    res[0] = r;
  }
};

// linear solid P1 triangle, b = 2 (plane stress via lambda*)
template <> struct Kind<K_SOLID2D> {
  static constexpr int NNO = 3, NDIM = 2, BW = 4, RW = 2;
  DFM_DEVINL static void row(const AsmParams& P, unsigned e, const int* no, const double* X, int a, double* blk,
                             double* res) {
    const double *p0 = X + 2 * no[0], *p1 = X + 2 * no[1], *p2 = X + 2 * no[2];
    const double lambda = P.coef ? P.p[0] * P.coef[e] : P.p[0];
    const double myu = P.coef ? P.p[1] * P.coef[e] : P.p[1];
    const double area = tri_area(p0, p1, p2);
    double d[3][2];
    tri_dldx(d, p0, p1, p2);
    const double a0 = pick3(a, d[0][0], d[1][0], d[2][0]), a1 = pick3(a, d[0][1], d[1][1], d[2][1]);
    double em[3][4];
    for (int c = 0; c < 3; c++) {
      em[c][0] = area * (lambda + myu) * a0 * d[c][0];
      em[c][1] = area * (lambda * a0 * d[c][1] + myu * d[c][0] * a1);
      em[c][2] = area * (lambda * a1 * d[c][0] + myu * d[c][1] * a0);
      em[c][3] = area * (lambda + myu) * a1 * d[c][1];
      const double dtmp1 = (a1 * d[c][1] + a0 * d[c][0]) * area * myu;
      em[c][0] += dtmp1;
      em[c][3] += dtmp1;
    }
    for (int c = 0; c < 3; c++)
      for (int q = 0; q < 4; q++) blk[c * 4 + q] = em[c][q];
    double r0 = area * P.p[2] * P.p[3] * 0.33333333333333333;
    double r1 = area * P.p[2] * P.p[4] * 0.33333333333333333;
    if (P.u)
      for (int c = 0; c < 3; c++) {
        const double* uc = P.u + 2 * no[c];
        r0 -= em[c][0] * uc[0] + em[c][1] * uc[1];
        r1 -= em[c][2] * uc[0] + em[c][3] * uc[1];
      }
    res[0] = r0;
    res[1] = r1;
  }
};

// linear solid P1 tetrahedron, b = 3
template <> struct Kind<K_SOLID3D> {
  static constexpr int NNO = 4, NDIM = 3, BW = 9, RW = 3;
  DFM_DEVINL static void row(const AsmParams& P, unsigned, const int* no, const double* X, int a, double* blk,
                             double* res) {
    const double *p0 = X + 3 * no[0], *p1 = X + 3 * no[1], *p2 = X + 3 * no[2], *p3 = X + 3 * no[3];
    const double lambda = P.p[0], myu = P.p[1];
    const double vol = tet_volume(p0, p1, p2, p3);
    double d[4][3];
    tet_dldx(d, p0, p1, p2, p3);
    double da[3];
    for (int r = 0; r < 3; r++) da[r] = a == 3 ? d[3][r] : pick3(a, d[0][r], d[1][r], d[2][r]);
    for (int c = 0; c < 4; c++) {
      double m[9];
      for (int r = 0; r < 3; r++)
        for (int s = 0; s < 3; s++) m[r * 3 + s] = vol * (lambda * da[r] * d[c][s] + myu * d[c][r] * da[s]);
      const double dtmp1 = da[0] * d[c][0] + da[1] * d[c][1] + da[2] * d[c][2];
      m[0] += vol * myu * dtmp1;
      m[4] += vol * myu * dtmp1;
      m[8] += vol * myu * dtmp1;
      for (int q = 0; q < 9; q++) blk[c * 9 + q] = m[q];
    }
    for (int r = 0; r < 3; r++) {
      double v = vol * P.p[2] * P.p[3 + r] * 0.25;
      if (P.u)
        for (int c = 0; c < 4; c++) {
          const double* uc = P.u + 3 * no[c];
          const double* m = blk + c * 9 + r * 3;
          v -= m[0] * uc[0] + m[1] * uc[1] + m[2] * uc[2];
        }
      res[r] = v;
    }
  }
};

// Helmholtz P1 triangle, complex b = 1 (blocks and residual as (re, im))
template <> struct Kind<K_HELM> {
  static constexpr int NNO = 3, NDIM = 2, BW = 2, RW = 2;
  DFM_DEVINL static void row(const AsmParams& P, unsigned, const int* no, const double* X, int a, double* blk,
                             double* res) {
    const double *p0 = X + 2 * no[0], *p1 = X + 2 * no[1], *p2 = X + 2 * no[2];
    const double area = tri_area(p0, p1, p2);
    double d[3][2];
    tri_dldx(d, p0, p1, p2);
    double em[3];
    const double a0 = pick3(a, d[0][0], d[1][0], d[2][0]), a1 = pick3(a, d[0][1], d[1][1], d[2][1]);
    for (int c = 0; c < 3; c++) em[c] = area * (a0 * d[c][0] + a1 * d[c][1]);
    const double k = 2 * 3.1416 / P.p[0];  // the reference's truncated pi (eqn_helmholtz.cpp:113)
    const double tmp_val = k * k * area / 12.0;
    for (int c = 0; c < 3; c++) em[c] = c == a ? em[c] - tmp_val : em[c];
    for (int c = 0; c < 3; c++) em[c] -= tmp_val;
    for (int c = 0; c < 3; c++) {
      blk[2 * c] = em[c];
      blk[2 * c + 1] = 0.0;
    }
    double rr = 0.0, ri = 0.0;
    if (P.u)
      for (int c = 0; c < 3; c++) {  // res -= em * u (complex, em real)
        const double ur = P.u[2 * no[c]], ui = P.u[2 * no[c] + 1];
        const double pr = em[c] * ur - 0.0 * ui, pi = em[c] * ui + 0.0 * ur;
        rr -= pr;
        ri -= pi;
      }
    res[0] = rr;
    res[1] = ri;
  }
};

// Sommerfeld radiation condition on a boundary bar, complex b = 1
template <> struct Kind<K_SOMMER> {
  static constexpr int NNO = 2, NDIM = 2, BW = 2, RW = 2;
  DFM_DEVINL static void row(const AsmParams& P, unsigned, const int* no, const double* X, int a, double* blk,
                             double* res) {
    const double *c0 = X + 2 * no[0], *c1 = X + 2 * no[1];
    const double elen = sqrt((c0[0] - c1[0]) * (c0[0] - c1[0]) + (c0[1] - c1[1]) * (c0[1] - c1[1]));
    const double k = 2 * 3.1416 / P.p[0];
    const double s1 = k / 6.0 * elen, s2 = -1 / (2.0 * elen * k);
    const double t1r = s1 * 0.0, t1i = s1 * 1.0, t2r = s2 * 0.0, t2i = s2 * 1.0;
    const double dr = 2 * t1r + t2r, di = 2 * t1i + t2i;  // tmp_val1*2 + tmp_val2
    const double orr = t1r - t2r, oi = t1i - t2i;         // tmp_val1 - tmp_val2
    for (int c = 0; c < 2; c++) {
      blk[2 * c] = (c == a) ? dr : orr;
      blk[2 * c + 1] = (c == a) ? di : oi;
    }
    double rr = 0.0, ri = 0.0;
    if (P.u)
      for (int c = 0; c < 2; c++) {
        const double er = blk[2 * c], ei = blk[2 * c + 1];
        const double ur = P.u[2 * no[c]], ui = P.u[2 * no[c] + 1];
        rr -= er * ur - ei * ui;
        ri -= er * ui + ei * ur;
      }
    res[0] = rr;
    res[1] = ri;
  }
};

// A node group's share of shared memory.  ST: doubles of an element's row (NNO
// blocks), odd so that the lanes' stores spread over the banks.
constexpr int kAsmSlots = 64;  // slots of a row (off-diagonal blocks and the diagonal)
template <int NNO, int BW, int RW, int L>
struct AsmShared {
  static constexpr int ST = (NNO * BW) | 1;
  double blk[L * ST], res[L * RW];
  unsigned col[kAsmSlots], mask[kAsmSlots];  // the row's columns; the elements that contribute to a slot
  unsigned short start[kAsmSlots], pos[L * NNO];  // a slot's contributions: offsets into blk in element order
  unsigned count;
};

// One batch of up to L elements of one kind around node i (row slots s0..s1,
// the diagonal block last).  first: the row's values start at zero, else they
// continue from what this lane stored before.  Every lane of the warp takes
// part, with nb == 0 where its group has no elements left.
template <int KIND, int L, typename SH>
DFM_DEVINL void gather_batch(const AsmParams& P, unsigned i, unsigned eb, unsigned nb, const unsigned* lst,
                             const int* elem, const double* X, unsigned nslot, SH& sh, bool first, double* diag,
                             double* off, double& racc, unsigned sub) {
  using K = Kind<KIND>;
  constexpr int NNO = K::NNO, BW = K::BW, RW = K::RW;
  for (unsigned j = sub; j < nslot; j += L) sh.mask[j] = 0;
  if (sub == 0) sh.count = 0;
  __syncwarp();
  unsigned t[NNO];
#pragma unroll
  for (int c = 0; c < NNO; c++) t[c] = kAsmSlots;
  if (sub < nb) {
    const unsigned e = lst[eb + sub];
    int no[NNO];
    int a = 0;
#pragma unroll
    for (int c = 0; c < NNO; c++) {
      no[c] = elem[(size_t)e * NNO + c];
      if ((unsigned)no[c] == i) a = c;
    }
    K::row(P, e, no, X, a, sh.blk + sub * SH::ST, sh.res + sub * RW);
#pragma unroll
    for (int c = 0; c < NNO; c++) {
      if (c == a) {
        t[c] = nslot - 1;
        continue;
      }
      unsigned lo = 0, hi = nslot - 1;  // ascending columns
      while (lo < hi) {
        const unsigned m = (lo + hi) >> 1;
        if (sh.col[m] < (unsigned)no[c]) lo = m + 1; else hi = m;
      }
      if (lo < nslot - 1 && sh.col[lo] == (unsigned)no[c]) {  // not in the pattern: skipped, as in Mearge
        t[c] = lo;
        atomicOr(&sh.mask[lo], 1u << sub);
      }
    }
  }
  if (sub == 0) sh.mask[nslot - 1] = nb >= 32u ? 0xffffffffu : (1u << nb) - 1u;
  __syncwarp();
  for (unsigned j = sub; j < nslot; j += L) sh.start[j] = (unsigned short)atomicAdd(&sh.count, __popc(sh.mask[j]));
  __syncwarp();
#pragma unroll
  for (int c = 0; c < NNO; c++)
    if (t[c] < kAsmSlots)
      sh.pos[sh.start[t[c]] + __popc(sh.mask[t[c]] & ((1u << sub) - 1u))] = (unsigned short)(sub * SH::ST + c * BW);
  __syncwarp();
  if (nb) {
    const unsigned nv = nslot * BW;
    for (unsigned v = sub; v < nv; v += L) {
      const unsigned j = v / BW, q = v - j * BW;
      double* o = j == nslot - 1 ? diag + q : off + v;
      const unsigned n = __popc(sh.mask[j]);
      const unsigned short* pos = sh.pos + sh.start[j];
      double acc = first ? 0.0 : *o;  // SetZero
#pragma unroll 4
      for (unsigned k = 0; k < n; k++) acc += sh.blk[pos[k] + q];
      *o = acc;
    }
    if (sub < RW)
      for (unsigned k = 0; k < nb; k++) racc += sh.res[k * RW + sub];
  }
  __syncwarp();
}

// Lanes per node of an element kind.
template <int KIND>
struct AsmLanes {
  static constexpr int L = Kind<KIND>::NNO == 4 ? 32 : 8;
};

template <int KIND, int KIND2>
__global__ void __launch_bounds__(32 * kAsmWarps, 5)
k_assemble(unsigned N, const unsigned* __restrict__ rowptr, const unsigned* __restrict__ colind, double* diag,
           double* off, double* rhs, AsmParams P, const double* __restrict__ X, const int* __restrict__ elem,
           const unsigned* __restrict__ esup_ptr, const unsigned* __restrict__ esup, AsmParams P2,
           const int* __restrict__ elem2, const unsigned* __restrict__ esup2_ptr, const unsigned* __restrict__ esup2,
           const double* __restrict__ load) {
  using K = Kind<KIND>;
  constexpr int NNO = K::NNO, BW = K::BW, RW = K::RW, L = AsmLanes<KIND>::L;
  using SH = AsmShared<NNO, BW, RW, L>;
  __shared__ SH s_sh[kAsmWarps * 32 / L];
  const unsigned g = threadIdx.x / L, sub = threadIdx.x % L;
  SH& sh = s_sh[g];
  const unsigned ng = kAsmWarps * 32 / L;
  for (unsigned i0 = blockIdx.x * ng; i0 < N; i0 += gridDim.x * ng) {
    const unsigned i = i0 + g;
    const bool have = i < N;
    const unsigned s0 = have ? rowptr[i] : 0u, s1 = have ? rowptr[i + 1] : 0u, nslot = s1 - s0 + 1;
    for (unsigned j = sub; j + 1 < nslot; j += L) sh.col[j] = colind[s0 + j];
    double* od = diag + (size_t)(have ? i : 0u) * BW;
    double* oo = off + (size_t)s0 * BW;
    const unsigned e0 = have ? esup_ptr[i] : 0u, e1 = have ? esup_ptr[i + 1] : 0u;
    double racc = 0.0;  // component sub of the residual (SetVectorZero)
    bool first = true;
    for (unsigned eb = e0; __any_sync(0xffffffffu, eb < e1); eb += L) {
      const unsigned nb = eb < e1 ? min((unsigned)L, e1 - eb) : 0u;
      gather_batch<KIND, L>(P, i, eb, nb, esup, elem, X, nslot, sh, first, od, oo, racc, sub);
      first = first && nb == 0;
    }
    if (KIND2 >= 0 && esup2_ptr) {  // second element array after the first (Helmholtz bars)
      using K2 = Kind<(KIND2 >= 0 ? KIND2 : KIND)>;
      static_assert(K2::BW == BW && K2::RW == RW && K2::NNO <= NNO, "element kinds of one system share the block width");
      const unsigned f0 = have ? esup2_ptr[i] : 0u, f1 = have ? esup2_ptr[i + 1] : 0u;
      for (unsigned eb = f0; __any_sync(0xffffffffu, eb < f1); eb += L) {
        const unsigned nb = eb < f1 ? min((unsigned)L, f1 - eb) : 0u;
        gather_batch<(KIND2 >= 0 ? KIND2 : KIND), L>(P2, i, eb, nb, esup2, elem2, X, nslot, sh, first, od, oo, racc,
                                                     sub);
        first = first && nb == 0;
      }
    }
    if (have && first) {  // a node of no element
      for (unsigned v = sub; v < nslot * BW; v += L) (v / BW == nslot - 1 ? od[v % BW] : oo[v]) = 0.0;
    }
    if (have && sub < RW)  // nodal loads after all element contributions
      rhs[(size_t)i * RW + sub] = load ? racc + load[(size_t)i * RW + sub] : racc;
    __syncwarp();
  }
}

// Dirichlet elimination: rows and columns of fixed DOFs zeroed, diagonal 1,
// residual zeroed.  8 lanes per block row: a lane takes the row's blocks lane,
// lane + 8, ... and stores only the entries that a flag zeroes, so the pass
// reads the columns and the flags and not the matrix.  (A thread per stored
// entry that searched its row took 611 us on the 200x40x40 box, 41 M entries.)
template <int B>
__global__ void __launch_bounds__(256)
k_dirichlet(unsigned N, const unsigned* __restrict__ rowptr, const unsigned* __restrict__ colind,
            const int* __restrict__ flags, double* diag, double* off, double* rhs) {
  constexpr unsigned BB = B * B, L = 8;
  const unsigned sub = threadIdx.x % L;
  auto bits = [&](unsigned n) {
    unsigned m = 0;
#pragma unroll
    for (int c = 0; c < B; c++) m |= (__ldg(flags + (size_t)n * B + c) != 0 ? 1u : 0u) << c;
    return m;
  };
  for (unsigned i = (blockIdx.x * blockDim.x + threadIdx.x) / L; i < N; i += gridDim.x * blockDim.x / L) {
    const unsigned s0 = __ldg(rowptr + i), s1 = __ldg(rowptr + i + 1), fr = bits(i);
    for (unsigned s = s0 + sub; s < s1; s += L) {
      const unsigned fc = bits(__ldg(colind + s));
      if (fr | fc) {
#pragma unroll
        for (int r = 0; r < B; r++)
#pragma unroll
          for (int c = 0; c < B; c++)
            if ((fr >> r & 1u) || (fc >> c & 1u)) off[(size_t)s * BB + r * B + c] = 0.0;
      }
    }
    if (sub == 0 && fr) {
#pragma unroll
      for (int r = 0; r < B; r++) {
#pragma unroll
        for (int c = 0; c < B; c++)
          if ((fr >> r & 1u) || (fr >> c & 1u))
            diag[(size_t)i * BB + r * B + c] = r == c && (fr >> r & 1u) ? 1.0 : 0.0;
        if (rhs && (fr >> r & 1u)) rhs[(size_t)i * B + r] = 0.0;
      }
    }
  }
}

// Adjoint element kernel: grad_e = -lambda_e^T (dK_e/dcoef_e) u_e, where the
// element matrix is linear in its coefficient (K_e = coef_e K_e^0, K_e^0 the
// matrix at the base constants P.p, as the assembly computes it).
template <int KIND>
__global__ void k_coef_grad(unsigned nelem, AsmParams P, const double* __restrict__ X, const int* __restrict__ elem,
                            const double* __restrict__ lam, const double* __restrict__ u, double* __restrict__ grad) {
  using K = Kind<KIND>;
  constexpr int NNO = K::NNO, BW = K::BW, RW = K::RW;
  for (unsigned e = blockIdx.x * blockDim.x + threadIdx.x; e < nelem; e += gridDim.x * blockDim.x) {
    int no[NNO];
#pragma unroll
    for (int c = 0; c < NNO; c++) no[c] = elem[(size_t)e * NNO + c];
    double g = 0.0;
#pragma unroll
    for (int a = 0; a < NNO; a++) {
      double blk[NNO * BW], res[RW];
      K::row(P, e, no, X, a, blk, res);
#pragma unroll
      for (int r = 0; r < RW; r++) {
        double v = 0.0;  // (K_e^0 u_e) at node a, component r
#pragma unroll
        for (int c = 0; c < NNO; c++)
#pragma unroll
          for (int s = 0; s < RW; s++) v += blk[c * BW + r * RW + s] * u[(size_t)no[c] * RW + s];
        g += lam[(size_t)no[a] * RW + r] * v;
      }
    }
    grad[e] = -g;
  }
}

static void node_adjacency(unsigned nnode, unsigned nnoel, unsigned nelem, const int* elem, std::vector<unsigned>& ptr,
                           std::vector<unsigned>& lst) {
  ptr.assign(nnode + 1, 0);
  for (size_t k = 0; k < (size_t)nelem * nnoel; k++) ptr[elem[k] + 1]++;
  for (unsigned i = 0; i < nnode; i++) ptr[i + 1] += ptr[i];
  lst.assign(ptr[nnode], 0);
  std::vector<unsigned> fill(ptr.begin(), ptr.end() - 1);
  for (unsigned e = 0; e < nelem; e++)
    for (unsigned k = 0; k < nnoel; k++) lst[fill[elem[(size_t)e * nnoel + k]]++] = e;
}

template <typename T>
static int up(T** d, const T* h, size_t n, cudaStream_t s) {
  DFM_CUDA_TRY(cudaMalloc((void**)d, sizeof(T) * std::max<size_t>(n, 1)));
  if (n) DFM_CUDA_TRY(cudaMemcpyAsync(*d, h, sizeof(T) * n, cudaMemcpyHostToDevice, s));
  return DFM_OK;
}

template <int KIND, int KIND2>
static int launch_asm(dfm_mesh G, dfm_mat A, const AsmParams& P, const AsmParams& P2, const double* load,
                      double* rhs) {
  if (A->N == 0) return DFM_OK;
  const unsigned nodes = kAsmWarps * 32 / AsmLanes<KIND>::L;  // per CTA
  const int grid = std::max(1, (int)std::min<unsigned>((A->N + nodes - 1) / nodes, (unsigned)A->ctx->nsm * 32u));
  k_assemble<KIND, KIND2><<<grid, 32 * kAsmWarps, 0, A->ctx->stream>>>(
      A->N, A->d_rowptr, A->d_colind, A->d_diag, A->d_off, rhs, P, G->d_coord, G->d_elem, G->d_esup_ptr, G->d_esup,
      P2, G->d_bar, KIND2 >= 0 ? G->d_bsup_ptr : nullptr, G->d_bsup, load);
  DFM_CUDA_TRY(cudaGetLastError());
  DFM_CUDA_TRY(cudaStreamSynchronize(A->ctx->stream));
  return take_code(A->ctx);
}

static bool rows_fit(dfm_mat A) { return A->max_row + 1 <= (unsigned)kAsmSlots; }

}  // namespace dfm

using namespace dfm;

extern "C" {

int dfm_mesh_create(dfm_ctx c, int ndim, unsigned nnode, const double* coord, unsigned nnoel, unsigned nelem,
                    const int* elem, unsigned nbar, const int* bar, dfm_mesh* out) {
  if (!c || !out || !coord || (nelem && !elem) || (nbar && !bar)) return DFM_ERR_INVALID;
  *out = nullptr;
  if (!((ndim == 2 && nnoel == 3) || (ndim == 3 && nnoel == 4))) return DFM_ERR_UNSUPPORTED;
  for (size_t k = 0; k < (size_t)nelem * nnoel; k++)
    if (elem[k] < 0 || (unsigned)elem[k] >= nnode) return DFM_ERR_INVALID;
  for (size_t k = 0; k < (size_t)nbar * 2; k++)
    if (bar[k] < 0 || (unsigned)bar[k] >= nnode) return DFM_ERR_INVALID;
  dfm_mesh G = new (std::nothrow) dfm_mesh_s();
  if (!G) return DFM_ERR_NOMEM;
  G->ctx = c;
  ctx_retain(c);
  G->ndim = ndim;
  G->nnode = nnode;
  G->nnoel = nnoel;
  G->nelem = nelem;
  G->nbar = nbar;
  std::vector<unsigned> ep, el, bp, bl;
  node_adjacency(nnode, nnoel, nelem, elem, ep, el);
  node_adjacency(nnode, 2, nbar, bar, bp, bl);
  cudaStream_t s = c->stream;
  int rc = up(&G->d_coord, coord, (size_t)nnode * ndim, s);
  if (!rc) rc = up(&G->d_elem, elem, (size_t)nelem * nnoel, s);
  if (!rc) rc = up(&G->d_bar, bar, (size_t)nbar * 2, s);
  if (!rc) rc = up(&G->d_esup_ptr, ep.data(), ep.size(), s);
  if (!rc) rc = up(&G->d_esup, el.data(), el.size(), s);
  if (!rc) rc = up(&G->d_bsup_ptr, bp.data(), bp.size(), s);
  if (!rc) rc = up(&G->d_bsup, bl.data(), bl.size(), s);
  if (!rc && cudaStreamSynchronize(s) != cudaSuccess) rc = DFM_ERR_CUDA;
  if (rc) {
    dfm_mesh_destroy(G);
    return rc;
  }
  G->h_elem.assign(elem, elem + (size_t)nelem * nnoel);
  G->h_esup_ptr.swap(ep);
  G->h_esup.swap(el);
  *out = G;
  return DFM_OK;
}

// Block pattern of the mesh: node i's row lists every other node sharing an
// element with it, ascending (CMatDia_BlkCrs::AddPattern over the field's
// element connectivity, src/matvec/matdia_blkcrs.cpp:346-505).
int dfm_mesh_pattern(dfm_mesh G, unsigned* rowptr, unsigned* colind, size_t* ncrs) {
  if (!G || !ncrs) return DFM_ERR_INVALID;
  const unsigned n = G->nnode, nno = G->nnoel;
  std::vector<unsigned> mark(n, 0xffffffffu), row;
  size_t total = 0;
  if (rowptr) rowptr[0] = 0;
  for (unsigned i = 0; i < n; i++) {
    row.clear();
    for (unsigned k = G->h_esup_ptr[i]; k < G->h_esup_ptr[i + 1]; k++) {
      const int* no = G->h_elem.data() + (size_t)G->h_esup[k] * nno;
      for (unsigned a = 0; a < nno; a++) {
        const unsigned j = (unsigned)no[a];
        if (j != i && mark[j] != i) {
          mark[j] = i;
          row.push_back(j);
        }
      }
    }
    std::sort(row.begin(), row.end());
    if (colind) std::copy(row.begin(), row.end(), colind + total);
    total += row.size();
    if (total > 0xffffffffull) return DFM_ERR_UNSUPPORTED;
    if (rowptr) rowptr[i + 1] = (unsigned)total;
  }
  *ncrs = total;
  return DFM_OK;
}

int dfm_mesh_destroy(dfm_mesh G) {
  if (!G) return DFM_OK;
  cudaStreamSynchronize(G->ctx->stream);
  cudaFree(G->d_coord);
  cudaFree(G->d_elem);
  cudaFree(G->d_bar);
  cudaFree(G->d_esup_ptr);
  cudaFree(G->d_esup);
  cudaFree(G->d_bsup_ptr);
  cudaFree(G->d_bsup);
  dfm_ctx c = G->ctx;
  delete G;
  ctx_release(c);
  return DFM_OK;
}

int dfm_assemble_poisson2d(dfm_mesh G, dfm_mat A, double alpha, double source, const double* elem_coef,
                           const double* u, const double* load, double* rhs) {
  if (!G || !A || !rhs || G->ndim != 2 || A->b != 1 || A->vt != DFM_REAL || G->nnode != A->N) return DFM_ERR_INVALID;
  if (!rows_fit(A)) return DFM_ERR_UNSUPPORTED;
  AsmParams P = {{alpha, source, 0, 0, 0, 0}, elem_coef, u};
  return launch_asm<K_POISSON, -1>(G, A, P, P, load, rhs);
}

int dfm_assemble_solid2d(dfm_mesh G, dfm_mat A, double lambda, double myu, double rho, double gx, double gy,
                         const double* elem_coef, const double* u, const double* load, double* rhs) {
  if (!G || !A || !rhs || G->ndim != 2 || A->b != 2 || A->vt != DFM_REAL || G->nnode != A->N) return DFM_ERR_INVALID;
  if (!rows_fit(A)) return DFM_ERR_UNSUPPORTED;
  AsmParams P = {{lambda, myu, rho, gx, gy, 0}, elem_coef, u};
  return launch_asm<K_SOLID2D, -1>(G, A, P, P, load, rhs);
}

int dfm_assemble_solid3d(dfm_mesh G, dfm_mat A, double lambda, double myu, double rho, double gx, double gy,
                         double gz, const double* u, const double* load, double* rhs) {
  if (!G || !A || !rhs || G->ndim != 3 || A->b != 3 || A->vt != DFM_REAL || G->nnode != A->N) return DFM_ERR_INVALID;
  if (!rows_fit(A)) return DFM_ERR_UNSUPPORTED;
  AsmParams P = {{lambda, myu, rho, gx, gy, gz}, nullptr, u};
  return launch_asm<K_SOLID3D, -1>(G, A, P, P, load, rhs);
}

int dfm_assemble_helmholtz2d(dfm_mesh G, dfm_mat A, double wave_length, const double* u, const double* load,
                             double* rhs) {
  if (!G || !A || !rhs || G->ndim != 2 || A->vt != DFM_COMPLEX || G->nnode != A->N) return DFM_ERR_INVALID;
  if (!rows_fit(A)) return DFM_ERR_UNSUPPORTED;
  AsmParams P = {{wave_length, 0, 0, 0, 0, 0}, nullptr, u};
  if (G->nbar) return launch_asm<K_HELM, K_SOMMER>(G, A, P, P, load, rhs);
  return launch_asm<K_HELM, -1>(G, A, P, P, load, rhs);
}

int dfm_coef_grad_poisson2d(dfm_mesh G, double alpha, const double* lam, const double* u, double* grad) {
  if (!G || !lam || !u || !grad || G->ndim != 2) return DFM_ERR_INVALID;
  if (G->nelem == 0) return DFM_OK;
  AsmParams P = {{alpha, 0, 0, 0, 0, 0}, nullptr, nullptr};
  const int grid = (int)std::min<unsigned>((G->nelem + 255) / 256, (unsigned)G->ctx->nsm * 8);
  k_coef_grad<K_POISSON><<<grid, 256, 0, G->ctx->stream>>>(G->nelem, P, G->d_coord, G->d_elem, lam, u, grad);
  DFM_CUDA_TRY(cudaGetLastError());
  DFM_CUDA_TRY(cudaStreamSynchronize(G->ctx->stream));
  return DFM_OK;
}

int dfm_coef_grad_solid2d(dfm_mesh G, double lambda, double myu, const double* lam, const double* u,
                          double* grad) {
  if (!G || !lam || !u || !grad || G->ndim != 2) return DFM_ERR_INVALID;
  if (G->nelem == 0) return DFM_OK;
  AsmParams P = {{lambda, myu, 0, 0, 0, 0}, nullptr, nullptr};
  const int grid = (int)std::min<unsigned>((G->nelem + 255) / 256, (unsigned)G->ctx->nsm * 8);
  k_coef_grad<K_SOLID2D><<<grid, 256, 0, G->ctx->stream>>>(G->nelem, P, G->d_coord, G->d_elem, lam, u, grad);
  DFM_CUDA_TRY(cudaGetLastError());
  DFM_CUDA_TRY(cudaStreamSynchronize(G->ctx->stream));
  return DFM_OK;
}

int dfm_apply_dirichlet(dfm_mat A, const int* flags, double* rhs) {
  if (!A || !flags || A->vt != DFM_REAL) return DFM_ERR_INVALID;
  if (A->N == 0) return DFM_OK;
  const int grid = (int)std::min<size_t>(((size_t)A->N * 8 + 255) / 256, (size_t)A->ctx->nsm * 16);
  cudaStream_t s = A->ctx->stream;
  switch (A->b) {
    case 1: k_dirichlet<1><<<grid, 256, 0, s>>>(A->N, A->d_rowptr, A->d_colind, flags, A->d_diag, A->d_off, rhs); break;
    case 2: k_dirichlet<2><<<grid, 256, 0, s>>>(A->N, A->d_rowptr, A->d_colind, flags, A->d_diag, A->d_off, rhs); break;
    default: k_dirichlet<3><<<grid, 256, 0, s>>>(A->N, A->d_rowptr, A->d_colind, flags, A->d_diag, A->d_off, rhs);
  }
  DFM_CUDA_TRY(cudaGetLastError());
  DFM_CUDA_TRY(cudaStreamSynchronize(A->ctx->stream));
  return DFM_OK;
}

}  // extern "C"
