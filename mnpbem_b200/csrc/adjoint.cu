// Reverse-mode derivative of a functional of the BEM solution with respect to
// the face geometry: c = lambda^T (dA/dtheta) x for every geometry parameter
// theta at once, given the solution x = (sig1, h1 | sig2, h2) and the adjoint
// lambda = A^-T w (equation-space layout phi, a, alpha, De).  The reference has
// no gradients; the operator differentiated is the BEM operator of
// Garcia de Abajo & Howie Eqs. (19, 20) as assembled by the reference
// (mnpbem/greenfun/greenret_refined.py:654-867, compgreen_ret.py:192-272 and
// :376-400 for the closed-surface correction, bem_ret_iter.py:1362-1501 for the
// operator's structure).
//
// lambda^T A x = sum_ij  G1_ij CGa_ij + H1_ij CHa_ij - G2_ij CGb_ij - H2_ij CHb_ij
//   CGa_ij = sum_p [ lphi_i s1_j + la_i . h1_j - ik (n_i . lalpha_i) e1_j s1_j
//                    - ik lDe_i e1_j (n_i . h1_j) ]
//   CHa_ij = sum_p [ lalpha_i . h1_j + lDe_i e1_j s1_j ]      (b: s2, h2, e2)
// with G1 = G[r00] - G[r10], G2 = G[r11] - G[r01] (region terms of each
// particle block, wavenumber of the material filling them).  Far pairs:
//   G = a_j / d e^{ikd},  Gp = r phi(d) a_j,  F = n_i . Gp,
//   phi(d) = (ik - 1/d) e^{ikd} / d^2,  phi'(d) = e^{ikd} / d^2 (3/d^2 - 3ik/d - k^2)
// refined pairs: G = sum_m g_m (ik)^m e^{ikd}, Gp = sum_m f_m (ik)^m e^{ikd},
// whose coefficients g, f depend on the face nodes through the refinement
// quadrature: their derivatives are exact (reverse mode through the quadrature).
//
// Nothing n x n (x 3) is stored: the far pairs are swept by one warp per row
// (row-side gradients: pos_i, nvec_i) and one warp per column (pos_j, area_j),
// every Green value and derivative recomputed in registers.
//
// Output: complex cotangents (c = sum of lambda^T dA x contributions) for
// pos (n, 3), nvec (n, 3), area (n), tvec1 (n, 3), tvec2 (n, 3) and the face
// nodes (n, 9, 3); the caller chains them to the vertices.
#include "common.cuh"
#include "green_entry.cuh"

namespace bem200 {
namespace adj {

using ge::kEps;
using ge::kMaxMat;
using ge::kMaxOrder;
using ge::kTwoPi;
using ge::phase;

constexpr int kMaxPol = 4;

struct KTab {
  double re[kMaxMat], im[kMaxMat];
};

struct Args {
  int n, npol, npart, order;
  KTab kt;
  double k0;
  int eps_per_face;
  double2 e1s, e2s;
  const double2* e1d;
  const double2* e2d;
  const int32_t* pid;
  const int32_t* blk;  // (npart, npart, 4): r00, r10, r11, r01
  const uint64_t* closed_mask;
  const double* pos;
  const double* nvec;
  const double* area;
  const double* tvec1;
  const double* tvec2;
  const double* nodes;
  const int32_t* face_kind;
  const double* rules;
  int n28, n3, n4;
  long long nref;
  const int64_t* row_ptr;  // CSR of the refined pairs
  const int32_t* ref_row;
  const int32_t* ref_col;
  const int8_t* ref_kind;
  const int64_t* col_ptr;  // CSC: refined rows of every column
  const int32_t* csc_row;
  const double* g;     // (nref, order + 1)
  const double* f;     // (nref, 3, order + 1), after the closed-surface correction
  const double* corr;  // (n) closed-surface correction of each face (0 if open)
  // solution and adjoint
  const double2* W1;   // (n, 4p): s1 | h1
  const double2* W2;   // (n, 4p): s2 | h2
  const double2* lam;  // phi (n, p) | a (n, 3, p) | alpha (n, 3, p) | De (n, p)
  // outputs and scratch
  double2* gpos;
  double2* gnv;
  double2* garea;
  double2* gt1;
  double2* gt2;
  double2* gnodes;
  double2* ghat;   // (nref, order + 1)
  double2* fhat;   // (nref, 3, order + 1)
  double2* shat;   // (n): cotangent of the closed-surface sum S_j
  double2* chat;   // (n): cotangent of corr_j
  int64_t* diag_e; // (n): refined entry of the diagonal (j, j), or -1
};

__device__ __forceinline__ double2 cm(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cs(double2 a, double s) { return make_double2(a.x * s, a.y * s); }
__device__ __forceinline__ double2 ca(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 cneg(double2 a) { return make_double2(-a.x, -a.y); }
__device__ __forceinline__ void atomic_c(double2* p, double2 v) {
  atomicAdd(&p->x, v.x);
  atomicAdd(&p->y, v.y);
}
__device__ __forceinline__ double2 eps_of(const Args& A, int j, bool second) {
  if (!A.eps_per_face) return second ? A.e2s : A.e1s;
  return second ? A.e2d[j] : A.e1d[j];
}
__device__ __forceinline__ double2 wsum2(double2 v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
    v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
  }
  return v;
}

// operator weights of pair (i, j) for family a (s1, h1, e1) or b (s2, h2, e2):
// CG, CH and dCG/dn_i (explicit normal in the operator)
struct Weights {
  double2 CG, CH, dCGdn[3];
};

__device__ __forceinline__ Weights pair_weights(const Args& A, int i, int j, bool fam_b, const double (&ni)[3]) {
  const int p = A.npol;
  const long long np = (long long)A.n * p;
  const double2* W = (fam_b ? A.W2 : A.W1) + (long long)j * 4 * p;
  const double2 e = eps_of(A, j, fam_b);
  const double2 ik = make_double2(0.0, A.k0);
  const double2* lphi = A.lam + (long long)i * p;
  const double2* la = A.lam + np + (long long)i * 3 * p;
  const double2* lal = A.lam + 4 * np + (long long)i * 3 * p;
  const double2* lDe = A.lam + 7 * np + (long long)i * p;
  Weights w;
  w.CG = w.CH = make_double2(0, 0);
  w.dCGdn[0] = w.dCGdn[1] = w.dCGdn[2] = make_double2(0, 0);
  for (int q = 0; q < p; ++q) {
    const double2 s = W[q];
    const double2 es = cm(e, s);
    double2 nla = make_double2(0, 0), nh = make_double2(0, 0);
    double2 lah = make_double2(0, 0), lalh = make_double2(0, 0);
    const double2 ld = lDe[q];
    for (int c = 0; c < 3; ++c) {
      const double2 h = W[p + c * p + q];
      const double2 lac = la[c * p + q], lalc = lal[c * p + q];
      nla = ca(nla, cs(lalc, ni[c]));
      nh = ca(nh, cs(h, ni[c]));
      lah = ca(lah, cm(lac, h));
      lalh = ca(lalh, cm(lalc, h));
      // d/dn_ic of [-ik (n.lalpha) e s - ik lDe e (n.h)]
      const double2 dd = ca(cm(lalc, es), cm(ld, cm(e, h)));
      w.dCGdn[c] = ca(w.dCGdn[c], cneg(cm(ik, dd)));
    }
    double2 cg = ca(cm(lphi[q], s), lah);
    cg = ca(cg, cneg(cm(ik, cm(nla, es))));
    cg = ca(cg, cneg(cm(ik, cm(ld, cm(e, nh)))));
    w.CG = ca(w.CG, cg);
    w.CH = ca(w.CH, ca(lalh, cm(ld, es)));
  }
  return w;
}

// the four region terms: family (0: G1/H1, 1: G2/H2) and sign in lambda^T A x
__device__ __forceinline__ int term_fam(int t) { return t < 2 ? 0 : 1; }
__device__ __forceinline__ double term_sgn(int t) { return (t == 0 || t == 3) ? 1.0 : -1.0; }

// far-pair derivative pieces of one region term (wavenumber kr + i ki):
//   dpos = CG dG/dpos_i + CH dF/dpos_i,  dn = CH Gp,  Gv = G (for the explicit
//   normal terms), val = CG G + CH F (for the area derivative: d/da_j = val / a_j)
struct FarTerm {
  double2 dpos[3], dn[3], G, val;
};

__device__ __forceinline__ FarTerm far_term(double kr, double ki, double d, const double (&r)[3], double aj,
                                            const double (&ni)[3], double2 CG, double2 CH) {
  FarTerm o;
  double pr, pim;
  phase(kr, ki, d, pr, pim);
  const double2 ph = make_double2(pr, pim);
  const double id = 1.0 / d, id2 = id * id;
  const double2 ik = make_double2(-ki, kr);
  const double2 ikm = make_double2(-ki - id, kr);  // ik - 1/d
  const double2 G = cs(ph, aj * id);
  const double2 phi = cs(cm(ikm, ph), id2);        // (ik - 1/d) e^{ikd} / d^2
  // phi' = e^{ikd} / d^2 (3/d^2 - 3ik/d - k^2)
  const double2 k2 = cm(ik, ik);                   // -k^2
  const double2 fac = make_double2(3.0 * id2 - 3.0 * ik.x * id + k2.x, -3.0 * ik.y * id + k2.y);
  const double2 dphi = cs(cm(fac, ph), id2);
  const double ndr = ni[0] * r[0] + ni[1] * r[1] + ni[2] * r[2];
  const double2 F = cs(phi, ndr * aj);
  const double2 dGdd = cm(G, ikm);                 // dG/dd
  for (int c = 0; c < 3; ++c) {
    const double u = r[c] * id;                    // dd/dpos_i
    const double2 dF = ca(cs(phi, ni[c] * aj), cs(dphi, ndr * aj * u));
    o.dpos[c] = ca(cm(CG, cs(dGdd, u)), cm(CH, dF));
    o.dn[c] = cm(CH, cs(phi, r[c] * aj));
  }
  o.G = G;
  o.val = ca(cm(CG, G), cm(CH, F));
  return o;
}

// closed-surface far term a_i Fs_ij, Fs_ij = -(n_i . r) / d^3 a_j: derivatives
// with respect to pos_i (vector), n_i (vector), a_i and a_j
struct ClosedTerm {
  double dpos[3], dn[3], da_i, da_j;
};
__device__ __forceinline__ ClosedTerm closed_term(double d, const double (&r)[3], double ai, double aj,
                                                  const double (&ni)[3]) {
  ClosedTerm o;
  const double id = 1.0 / d, id3 = id * id * id, id5 = id3 * id * id;
  const double ndr = ni[0] * r[0] + ni[1] * r[1] + ni[2] * r[2];
  const double Fs = -ndr * id3 * aj;
  for (int c = 0; c < 3; ++c) {
    o.dpos[c] = ai * aj * (-ni[c] * id3 + 3.0 * ndr * r[c] * id5);
    o.dn[c] = -ai * aj * r[c] * id3;
  }
  o.da_i = Fs;
  o.da_j = ai * Fs / aj;
  return o;
}

__device__ __forceinline__ bool in_surf(const Args& A, int i, int j) {
  return (A.closed_mask[A.pid[j]] >> A.pid[i]) & 1ull;
}

// ------------------------------------------------------------ far pairs, rows
constexpr int kWarps = 4;

__global__ void __launch_bounds__(32 * kWarps) far_rows_kernel(Args A) {
  extern __shared__ uint32_t row_bits[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int i = blockIdx.x * kWarps + wid;
  const int words = (A.n + 31) >> 5;
  uint32_t* bits = row_bits + (size_t)wid * words;
  if (i >= A.n) return;
  for (int w = lane; w < words; w += 32) bits[w] = 0u;
  __syncwarp();
  for (long long e = A.row_ptr[i] + lane; e < A.row_ptr[i + 1]; e += 32) {
    const int j = A.ref_col[e];
    atomicOr(&bits[j >> 5], 1u << (j & 31));
  }
  __syncwarp();
  const int bi = A.pid[i];
  const double pix = A.pos[3 * i], piy = A.pos[3 * i + 1], piz = A.pos[3 * i + 2];
  const double ni[3] = {A.nvec[3 * i], A.nvec[3 * i + 1], A.nvec[3 * i + 2]};
  const double ai = A.area[i];
  double2 gp[3] = {make_double2(0, 0), make_double2(0, 0), make_double2(0, 0)};
  double2 gn[3] = {make_double2(0, 0), make_double2(0, 0), make_double2(0, 0)};
  double2 ga = make_double2(0, 0);
  for (int j = lane; j < A.n; j += 32) {
    if ((bits[j >> 5] >> (j & 31)) & 1u) continue;
    if (j == i) continue;
    const int bj = A.pid[j];
    const double r[3] = {pix - A.pos[3 * j], piy - A.pos[3 * j + 1], piz - A.pos[3 * j + 2]};
    const double d = fmax(sqrt(r[0] * r[0] + r[1] * r[1] + r[2] * r[2]), kEps);
    const double aj = A.area[j];
    const int* bm = A.blk + (bi * A.npart + bj) * 4;
    Weights wf[2];
    bool have[2] = {false, false};
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int m = bm[t];
      if (m <= 0) continue;
      const int fam = term_fam(t);
      if (!have[fam]) {
        wf[fam] = pair_weights(A, i, j, fam == 1, ni);
        have[fam] = true;
      }
      const FarTerm ft = far_term(A.kt.re[m - 1], A.kt.im[m - 1], d, r, aj, ni, wf[fam].CG, wf[fam].CH);
      const double sg = term_sgn(t);
      for (int c = 0; c < 3; ++c) {
        gp[c] = ca(gp[c], cs(ft.dpos[c], sg));
        gn[c] = ca(gn[c], cs(ca(ft.dn[c], cm(ft.G, wf[fam].dCGdn[c])), sg));
      }
    }
    if (in_surf(A, i, j)) {
      const double2 sh = A.shat[j];
      if (sh.x != 0.0 || sh.y != 0.0) {
        const ClosedTerm ct = closed_term(d, r, ai, aj, ni);
        for (int c = 0; c < 3; ++c) {
          gp[c] = ca(gp[c], cs(sh, ct.dpos[c]));
          gn[c] = ca(gn[c], cs(sh, ct.dn[c]));
        }
        ga = ca(ga, cs(sh, ct.da_i));
      }
    }
  }
  for (int c = 0; c < 3; ++c) {
    gp[c] = wsum2(gp[c]);
    gn[c] = wsum2(gn[c]);
  }
  ga = wsum2(ga);
  if (lane == 0) {
    for (int c = 0; c < 3; ++c) {
      A.gpos[3 * i + c] = ca(A.gpos[3 * i + c], gp[c]);
      A.gnv[3 * i + c] = ca(A.gnv[3 * i + c], gn[c]);
    }
    A.garea[i] = ca(A.garea[i], ga);
  }
}

// ------------------------------------------------------------ far pairs, columns
__global__ void __launch_bounds__(32 * kWarps) far_cols_kernel(Args A) {
  extern __shared__ uint32_t col_bits[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int j = blockIdx.x * kWarps + wid;
  const int words = (A.n + 31) >> 5;
  uint32_t* bits = col_bits + (size_t)wid * words;
  if (j >= A.n) return;
  for (int w = lane; w < words; w += 32) bits[w] = 0u;
  __syncwarp();
  for (long long e = A.col_ptr[j] + lane; e < A.col_ptr[j + 1]; e += 32) {
    const int i = A.csc_row[e];
    atomicOr(&bits[i >> 5], 1u << (i & 31));
  }
  __syncwarp();
  const int bj = A.pid[j];
  const double pjx = A.pos[3 * j], pjy = A.pos[3 * j + 1], pjz = A.pos[3 * j + 2];
  const double aj = A.area[j];
  const double2 sh = A.shat[j];
  double2 gp[3] = {make_double2(0, 0), make_double2(0, 0), make_double2(0, 0)};
  double2 ga = make_double2(0, 0);
  for (int i = lane; i < A.n; i += 32) {
    if ((bits[i >> 5] >> (i & 31)) & 1u) continue;
    if (i == j) continue;
    const int bi = A.pid[i];
    const double r[3] = {A.pos[3 * i] - pjx, A.pos[3 * i + 1] - pjy, A.pos[3 * i + 2] - pjz};
    const double d = fmax(sqrt(r[0] * r[0] + r[1] * r[1] + r[2] * r[2]), kEps);
    const double ni[3] = {A.nvec[3 * i], A.nvec[3 * i + 1], A.nvec[3 * i + 2]};
    const int* bm = A.blk + (bi * A.npart + bj) * 4;
    Weights wf[2];
    bool have[2] = {false, false};
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int m = bm[t];
      if (m <= 0) continue;
      const int fam = term_fam(t);
      if (!have[fam]) {
        wf[fam] = pair_weights(A, i, j, fam == 1, ni);
        have[fam] = true;
      }
      const FarTerm ft = far_term(A.kt.re[m - 1], A.kt.im[m - 1], d, r, aj, ni, wf[fam].CG, wf[fam].CH);
      const double sg = term_sgn(t);
      for (int c = 0; c < 3; ++c) gp[c] = ca(gp[c], cs(ft.dpos[c], -sg));  // d/dpos_j = -d/dpos_i
      ga = ca(ga, cs(ft.val, sg / aj));
    }
    if ((sh.x != 0.0 || sh.y != 0.0) && in_surf(A, i, j)) {
      const ClosedTerm ct = closed_term(d, r, A.area[i], aj, ni);
      for (int c = 0; c < 3; ++c) gp[c] = ca(gp[c], cs(sh, -ct.dpos[c]));
      ga = ca(ga, cs(sh, ct.da_j));
    }
  }
  for (int c = 0; c < 3; ++c) gp[c] = wsum2(gp[c]);
  ga = wsum2(ga);
  if (lane == 0) {
    for (int c = 0; c < 3; ++c) A.gpos[3 * j + c] = ca(A.gpos[3 * j + c], gp[c]);
    A.garea[j] = ca(A.garea[j], ga);
  }
}

// ------------------------------------------------------------ refined pairs
// Operator part: cotangents of the (corrected) coefficients g, f of entry e,
// the phase derivative (through d) and the normal derivatives.
__global__ void refined_op_kernel(Args A) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= A.nref) return;
  const int i = A.ref_row[e], j = A.ref_col[e];
  const int bi = A.pid[i], bj = A.pid[j];
  const bool diag = (bi == bj) && (i == j);
  const double r[3] = {A.pos[3 * i] - A.pos[3 * j], A.pos[3 * i + 1] - A.pos[3 * j + 1],
                       A.pos[3 * i + 2] - A.pos[3 * j + 2]};
  const double d = diag ? kEps : fmax(sqrt(r[0] * r[0] + r[1] * r[1] + r[2] * r[2]), kEps);
  const double ni[3] = {A.nvec[3 * i], A.nvec[3 * i + 1], A.nvec[3 * i + 2]};
  const int no = A.order + 1;
  const int* bm = A.blk + (bi * A.npart + bj) * 4;
  double2 gh[kMaxOrder + 1], fh[3][kMaxOrder + 1];
  for (int m = 0; m < no; ++m) {
    gh[m] = make_double2(0, 0);
    fh[0][m] = fh[1][m] = fh[2][m] = make_double2(0, 0);
  }
  double2 gp[3] = {make_double2(0, 0), make_double2(0, 0), make_double2(0, 0)};
  double2 gn[3] = {make_double2(0, 0), make_double2(0, 0), make_double2(0, 0)};
  Weights wf[2];
  bool have[2] = {false, false};
  for (int t = 0; t < 4; ++t) {
    const int mat = bm[t];
    if (mat <= 0) continue;
    const int fam = term_fam(t);
    if (!have[fam]) {
      wf[fam] = pair_weights(A, i, j, fam == 1, ni);
      have[fam] = true;
    }
    const double sg = term_sgn(t);
    const double kr = A.kt.re[mat - 1], ki = A.kt.im[mat - 1];
    const double2 ik = make_double2(-ki, kr);
    double pr, pim;
    phase(kr, ki, d, pr, pim);
    const double2 ph = make_double2(pr, pim);
    double2 ikm = make_double2(1, 0);  // (ik)^m
    double2 Sg = make_double2(0, 0), Sf[3] = {make_double2(0, 0), make_double2(0, 0), make_double2(0, 0)};
    const double2 CGs = cs(wf[fam].CG, sg), CHs = cs(wf[fam].CH, sg);
    for (int m = 0; m < no; ++m) {
      const double2 b = cm(ikm, ph);  // (ik)^m e^{ikd}
      gh[m] = ca(gh[m], cm(CGs, b));
      Sg = ca(Sg, cs(ikm, A.g[e * no + m]));
      for (int c = 0; c < 3; ++c) {
        fh[c][m] = ca(fh[c][m], cs(cm(CHs, b), ni[c]));
        Sf[c] = ca(Sf[c], cs(ikm, A.f[(e * 3 + c) * no + m]));
      }
      ikm = cm(ikm, ik);
    }
    const double2 G = cm(Sg, ph);
    double2 Gp[3];
    for (int c = 0; c < 3; ++c) Gp[c] = cm(Sf[c], ph);
    const double2 F = ca(ca(cs(Gp[0], ni[0]), cs(Gp[1], ni[1])), cs(Gp[2], ni[2]));
    if (!diag) {  // d/dd of e^{ikd}: ik times the value
      const double2 dv = cm(ik, ca(cm(CGs, G), cm(CHs, F)));
      for (int c = 0; c < 3; ++c) gp[c] = ca(gp[c], cs(dv, r[c] / d));
    }
    for (int c = 0; c < 3; ++c) gn[c] = ca(gn[c], ca(cm(CHs, Gp[c]), cm(G, cs(wf[fam].dCGdn[c], sg))));
  }
  for (int m = 0; m < no; ++m) {
    A.ghat[e * no + m] = gh[m];
    for (int c = 0; c < 3; ++c) A.fhat[(e * 3 + c) * no + m] = fh[c][m];
  }
  for (int c = 0; c < 3; ++c) {
    if (!diag) {
      atomic_c(&A.gpos[3 * i + c], gp[c]);
      atomic_c(&A.gpos[3 * j + c], cneg(gp[c]));
    }
    atomic_c(&A.gnv[3 * i + c], gn[c]);
  }
  if (diag) A.diag_e[j] = e;
}

// closed-surface correction of face j: corr_j = -2 pi - S_j / a_j, added as
// corr_j n_j to f[(j, j), :, 0].  chat_j = n_j . fhat[(j, j), :, 0]; the sum
// S_j gets the cotangent -chat_j / a_j; a_j and n_j get their direct parts.
__global__ void closed_prep_kernel(Args A) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= A.n) return;
  const long long e = A.diag_e[j];
  A.shat[j] = make_double2(0, 0);
  if (e < 0 || A.closed_mask[A.pid[j]] == 0) return;
  const int no = A.order + 1;
  const double nj[3] = {A.nvec[3 * j], A.nvec[3 * j + 1], A.nvec[3 * j + 2]};
  double2 ch = make_double2(0, 0);
  for (int c = 0; c < 3; ++c) {
    const double2 fh0 = A.fhat[(e * 3 + c) * no];
    ch = ca(ch, cs(fh0, nj[c]));
    A.gnv[3 * j + c] = ca(A.gnv[3 * j + c], cs(fh0, A.corr[j]));
  }
  const double aj = A.area[j];
  A.chat[j] = ch;
  A.shat[j] = cs(ch, -1.0 / aj);
  // corr_j = -2 pi - S_j / a_j with S_j / a_j = -2 pi - corr_j: d/da_j (direct) = S_j / a_j^2
  A.garea[j] = ca(A.garea[j], cs(ch, (-kTwoPi - A.corr[j]) / aj));
}

// refined entries of a closed surface's sum: S_j gets a_i n_i . f_e0 (the
// uncorrected coefficient) for the refined pairs (i, j) with i on j's surface
__global__ void refined_closed_kernel(Args A) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= A.nref) return;
  const int i = A.ref_row[e], j = A.ref_col[e];
  const double2 sh = A.shat[j];
  if ((sh.x == 0.0 && sh.y == 0.0) || !in_surf(A, i, j)) return;
  const int no = A.order + 1;
  const double ni[3] = {A.nvec[3 * i], A.nvec[3 * i + 1], A.nvec[3 * i + 2]};
  const double ai = A.area[i];
  const bool diag = (i == j);
  double f0[3], nf = 0.0;
  for (int c = 0; c < 3; ++c) {
    f0[c] = A.f[(e * 3 + c) * no] - (diag ? A.corr[j] * ni[c] : 0.0);
    nf += ni[c] * f0[c];
  }
  for (int c = 0; c < 3; ++c) {
    A.fhat[(e * 3 + c) * no] = ca(A.fhat[(e * 3 + c) * no], cs(sh, ai * ni[c]));
    atomic_c(&A.gnv[3 * i + c], cs(sh, ai * f0[c]));
  }
  atomic_c(&A.garea[i], cs(sh, nf));
}

// ------------------------------------------------------------ refinement coefficients
// Derivatives of the refinement coefficients g_m, f_cm of entry e with respect
// to its inputs, contracted with their cotangents: reverse mode through the
// refinement quadrature (the reference's _refine_diagonal / _refine_offdiagonal,
// mnpbem/greenfun/greenret_refined.py:122-516, with the rules of
// refine_integrals_kernel in green.cu).  Inputs: self terms (kind 2): pos_i, n_i,
// t1_i, t2_i and the nodes of face j; others: pos_i, pos_j and the nodes of
// face j.
//
// A quadrature point x = sum_c N_c node_c has the weight wf |px x py|, px and
// py the sums with the derivatives Dx_c, Dy_c of its shape functions (flat
// triangles: the two edges).  Its contribution to the contraction is w phi(v, ..),
// v = pos_i - x; the point's cotangents are -w dphi/dv for x and phi wf times the
// gradient of |px x py| for px, py.
//
// One warp per entry, one point per lane; the points' cotangents and shape
// functions go through shared memory, and lane 3 c + x then sums node c's
// component x over the points.  One evaluation of the quadrature replaces one
// dual-number evaluation per input coordinate (24 - 39 of them): FP64 bound.
constexpr int kPtVals = 18;    // complex cotangents of x, px, py
constexpr int kPtBasis = 27;   // N, Dx, Dy of up to 9 nodes
constexpr int kCoefWarps = 4;

struct Vec { double x, y, z; };
__device__ __forceinline__ Vec vsub(Vec a, Vec b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ Vec vcross(Vec a, Vec b) {
  return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
__device__ __forceinline__ double vdot(Vec a, Vec b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ Vec vload(const double* p) { return {p[0], p[1], p[2]}; }
__device__ __forceinline__ double2 cfma(double2 a, double s, double2 c) {
  return make_double2(fma(a.x, s, c.x), fma(a.y, s, c.y));
}

// node of the face behind shape function c of the current (sub-)element
__device__ __forceinline__ int sub_node(int fk, bool self, int s, int c) {
  if (self || fk == 0 || fk == 2) return c;
  if (fk == 1) return c == 0 ? 0 : c + s;                 // flat quad: triangles 0 1 2 and 0 2 3
  const unsigned m = s == 0 ? 0x854210u : 0x876032u;      // curved quad: 0 1 2 4 5 8 and 2 3 0 6 7 8
  return (m >> (4 * c)) & 15;
}

// shape functions at rule point q: number of nodes, weight factor; B[3 c .. 3 c + 2] = N, Dx, Dy
__device__ __forceinline__ double shape_at(const Args& A, int fk, bool self, int q, double* B, int stride) {
  const double* x3 = A.rules + 3 * A.n28;
  const double* x4 = x3 + 3 * A.n3;
  auto put = [&](int c, double N, double Dx, double Dy) {
    B[(3 * c) * stride] = N;
    B[(3 * c + 1) * stride] = Dx;
    B[(3 * c + 2) * stride] = Dy;
  };
  if (self && (fk == 1 || fk == 3)) {
    const double x = x4[q], y = x4[A.n4 + q], w = x4[2 * A.n4 + q];
    if (fk == 1) {
      put(0, 0.25 * (1 - x) * (1 - y), -0.25 * (1 - y), -0.25 * (1 - x));
      put(1, 0.25 * (1 + x) * (1 - y), 0.25 * (1 - y), -0.25 * (1 + x));
      put(2, 0.25 * (1 + x) * (1 + y), 0.25 * (1 + y), 0.25 * (1 + x));
      put(3, 0.25 * (1 - x) * (1 + y), -0.25 * (1 + y), 0.25 * (1 - x));
    } else {
      put(0, 0.25 * x * (x - 1) * y * (y - 1), 0.25 * (2 * x - 1) * y * (y - 1), 0.25 * x * (x - 1) * (2 * y - 1));
      put(1, 0.25 * x * (x + 1) * y * (y - 1), 0.25 * (2 * x + 1) * y * (y - 1), 0.25 * x * (x + 1) * (2 * y - 1));
      put(2, 0.25 * x * (x + 1) * y * (y + 1), 0.25 * (2 * x + 1) * y * (y + 1), 0.25 * x * (x + 1) * (2 * y + 1));
      put(3, 0.25 * x * (x - 1) * y * (y + 1), 0.25 * (2 * x - 1) * y * (y + 1), 0.25 * x * (x - 1) * (2 * y + 1));
      put(4, 0.5 * (1 - x * x) * y * (y - 1), -x * y * (y - 1), 0.5 * (1 - x * x) * (2 * y - 1));
      put(5, 0.5 * x * (x + 1) * (1 - y * y), 0.5 * (2 * x + 1) * (1 - y * y), -x * (x + 1) * y);
      put(6, 0.5 * (1 - x * x) * y * (y + 1), -x * y * (y + 1), 0.5 * (1 - x * x) * (2 * y + 1));
      put(7, 0.5 * x * (x - 1) * (1 - y * y), 0.5 * (2 * x - 1) * (1 - y * y), -x * (x - 1) * y);
      put(8, (1 - x * x) * (1 - y * y), -2 * x * (1 - y * y), -2 * (1 - x * x) * y);
    }
    return w;
  }
  const double* r = self ? x3 : A.rules;
  const int np = self ? A.n3 : A.n28;
  const double x = r[q], y = r[np + q], z = 1.0 - x - y;
  double w = 0.5 * r[2 * np + q];
  if (fk >= 2) {
    put(0, x * (2 * x - 1), 4 * x - 1, 0.0);
    put(1, y * (2 * y - 1), 0.0, 4 * y - 1);
    put(2, z * (2 * z - 1), -4 * z + 1, -4 * z + 1);
    put(3, 4 * x * y, 4 * y, 4 * x);
    put(4, 4 * y * z, -4 * y, 4 * (z - y));
    put(5, 4 * z * x, 4 * (z - x), -4 * x);
  } else {
    put(0, x, -1.0, -1.0);
    put(1, y, 1.0, 0.0);
    put(2, z, 0.0, 1.0);
  }
  return w;
}

__device__ __forceinline__ double wmax(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

__global__ void __launch_bounds__(32 * kCoefWarps) refine_coef_grad_kernel(Args A) {
  extern __shared__ double coef_smem[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const long long e = (long long)blockIdx.x * kCoefWarps + wid;
  if (e >= A.nref) return;
  constexpr int P = 33;  // pitch of a value over the lanes
  double* pv = coef_smem + wid * (kPtVals + kPtBasis) * P;  // [kPtVals][P] cotangents of this chunk's points
  double* pb = pv + kPtVals * P;                             // [kPtBasis][P] shape functions
  const int i = A.ref_row[e], j = A.ref_col[e], kind = A.ref_kind[e];
  const int no = A.order + 1;
  const int fk = A.face_kind[j];
  const bool self = (kind == 2);
  const bool quad = fk == 1 || fk == 3;
  const int nsub = !self && quad ? 2 : 1;
  const int nb = self ? (fk == 0 ? 3 : fk == 1 ? 4 : fk == 2 ? 6 : 9) : (fk >= 2 ? 6 : 3);
  const int npts = self ? (quad ? A.n4 : A.n3) : A.n28;
  const double* nodes = A.nodes + 27LL * j;
  const double2* gh = A.ghat + e * no;
  const double2* fh = A.fhat + e * 3 * no;
  const Vec pi = vload(A.pos + 3 * i);
  Vec pj{0, 0, 0}, ni{0, 0, 0}, t1{0, 0, 0}, t2{0, 0, 0}, u0{0, 0, 0};
  double r0 = 0.0, rfloor = 0.0;
  // point q of sub-element s: shape functions to shared memory, position, px, py
  auto point = [&](int s, int q, Vec& x, Vec& px, Vec& py) -> double {
    const double wf = shape_at(A, fk, self, q, pb + lane, P);
    x = px = py = Vec{0, 0, 0};
    for (int c = 0; c < nb; ++c) {
      const double* nd = nodes + 3 * sub_node(fk, self, s, c);
      const double N = pb[(3 * c) * P + lane], Dx = pb[(3 * c + 1) * P + lane], Dy = pb[(3 * c + 2) * P + lane];
      x = {fma(N, nd[0], x.x), fma(N, nd[1], x.y), fma(N, nd[2], x.z)};
      px = {fma(Dx, nd[0], px.x), fma(Dx, nd[1], px.y), fma(Dx, nd[2], px.z)};
      py = {fma(Dy, nd[0], py.x), fma(Dy, nd[1], py.y), fma(Dy, nd[2], py.z)};
    }
    return wf;
  };
  if (self) {
    ni = vload(A.nvec + 3 * i);
    t1 = vload(A.tvec1 + 3 * i);
    t2 = vload(A.tvec2 + 3 * i);
    double rmax = 0.0;
    for (int q = lane; q < npts; q += 32) {
      Vec x, px, py;
      point(0, q, x, px, py);
      const Vec v = vsub(pi, x);
      rmax = fmax(rmax, fmax(sqrt(vdot(v, v)), kEps));
    }
    rfloor = 1e-4 * wmax(rmax);
  } else {
    pj = vload(A.pos + 3 * j);
    const Vec d = vsub(pj, pi);
    r0 = sqrt(vdot(d, d));
    const double ir0 = r0 > 0 ? 1.0 / r0 : 0.0;
    u0 = {d.x * ir0, d.y * ir0, d.z * ir0};
  }
  const double2 zero = make_double2(0, 0);
  double2 gpi[3] = {zero, zero, zero};  // pos_i
  double2 gr0 = zero;                   // r0
  double2 gn[3] = {zero, zero, zero}, g1[3] = {zero, zero, zero}, g2[3] = {zero, zero, zero};  // n, t1, t2 (self)
  double2 gnode[2] = {zero, zero};      // lane 3 c + x: node of shape function c, per sub-element
  for (int s = 0; s < nsub; ++s) {
    for (int q0 = 0; q0 < npts; q0 += 32) {
      const int q = q0 + lane;
      double2 ct[9];
#pragma unroll
      for (int c = 0; c < 9; ++c) ct[c] = zero;
      if (q < npts) {
        Vec x, px, py;
        const double wf = point(s, q, x, px, py);
        const Vec nn = vcross(px, py);
        const double J = sqrt(vdot(nn, nn)), w = J * wf;
        const Vec v = vsub(pi, x);
        const double rv = sqrt(vdot(v, v));
        const double r = fmax(rv, kEps), ir = 1.0 / r;
        const double act = rv >= kEps ? ir : 0.0;  // dr / dv = v act
        double2 phi, dv[3];
        if (!self) {
          // phi = G ir - ir^3 v.P + ir^2 v.P', polynomials in dl = r - r0:
          // G = sum ghat_m dl^m / m!, P_c = sum fhat_cm dl^m / m!
          const double dl = r - r0, ir2 = ir * ir, ir3 = ir2 * ir;
          double2 G = zero, G1 = zero, p0[3], p1[3], p2[3];
#pragma unroll
          for (int c = 0; c < 3; ++c) p0[c] = p1[c] = p2[c] = zero;
          double t0 = 1.0, tm1 = 0.0, tm2 = 0.0;  // dl^m / m!, and one and two orders lower
          for (int m = 0; m < no; ++m) {
            const double2 a = gh[m];
            G = cfma(a, t0, G);
            G1 = cfma(a, tm1, G1);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
              const double2 f = fh[c * no + m];
              p0[c] = cfma(f, t0, p0[c]);
              p1[c] = cfma(f, tm1, p1[c]);
              p2[c] = cfma(f, tm2, p2[c]);
            }
            tm2 = tm1;
            tm1 = t0;
            t0 *= dl / (m + 1);
          }
          double2 s0 = zero, s1 = zero, s2 = zero;
          const double vv[3] = {v.x, v.y, v.z};
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            s0 = cfma(p0[c], vv[c], s0);
            s1 = cfma(p1[c], vv[c], s1);
            s2 = cfma(p2[c], vv[c], s2);
          }
          phi = ca(ca(cs(G, ir), cs(s0, -ir3)), cs(s1, ir2));
          const double2 pdl = ca(ca(cs(G1, ir), cs(s1, -ir3)), cs(s2, ir2));
          const double2 pr = ca(ca(cs(G, -ir2), cs(s0, 3.0 * ir2 * ir2)), cs(s1, -2.0 * ir3));
          const double2 rad = cs(ca(pdl, pr), act);
#pragma unroll
          for (int c = 0; c < 3; ++c) dv[c] = cfma(rad, vv[c], ca(cs(p0[c], -ir3), cs(p1[c], ir2)));
          gr0 = cfma(pdl, -w, gr0);
        } else {
          // phi = A + ndr n.FB + irr3 (in1 t1.FC + in2 t2.FC),  A = sum ghat_m r^(m-1) / m!,
          // FB = sum fhat_m (m-1) / m! r^(m-3),  FC = r^3 FB
          const double rr = fmax(r, rfloor), irr = 1.0 / rr, irr3 = irr * irr * irr;
          double2 a0 = zero, a1 = zero, b0[3], b1[3];
#pragma unroll
          for (int c = 0; c < 3; ++c) b0[c] = b1[c] = zero;
          double rm = 1.0, fact = 1.0;  // r^m, m!
          for (int m = 0; m < no; ++m) {
            if (m > 0) fact *= m;
            const double2 a = gh[m];
            a0 = cfma(a, rm * ir / fact, a0);
            a1 = cfma(a, (m - 1) * rm * ir * ir / fact, a1);
            const double cf = (m - 1) / fact;
#pragma unroll
            for (int c = 0; c < 3; ++c) {  // FC and its derivative
              const double2 f = fh[c * no + m];
              b0[c] = cfma(f, cf * rm, b0[c]);
              b1[c] = cfma(f, cf * m * rm * ir, b1[c]);
            }
            rm *= r;
          }
          const double ir3 = ir * ir * ir;
          const double nvv[3] = {ni.x, ni.y, ni.z}, t1v[3] = {t1.x, t1.y, t1.z}, t2v[3] = {t2.x, t2.y, t2.z};
          const double vv[3] = {v.x, v.y, v.z};
          const double ndr = vdot(ni, v), in1 = vdot(t1, v), in2 = vdot(t2, v);
          double2 B = zero, B1 = zero, C = zero, C1 = zero, D = zero, D1 = zero;
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const double2 fb = cs(b0[c], ir3);                               // FB
            const double2 fb1 = ca(cs(b1[c], ir3), cs(b0[c], -3.0 * ir3 * ir));  // FB'
            B = cfma(fb, nvv[c], B);
            B1 = cfma(fb1, nvv[c], B1);
            C = cfma(b0[c], t1v[c], C);
            C1 = cfma(b1[c], t1v[c], C1);
            D = cfma(b0[c], t2v[c], D);
            D1 = cfma(b1[c], t2v[c], D1);
          }
          const double2 tcd = ca(cs(C, in1), cs(D, in2));
          phi = ca(ca(a0, cs(B, ndr)), cs(tcd, irr3));
          double2 pr = ca(ca(a1, cs(B1, ndr)), cs(ca(cs(C1, in1), cs(D1, in2)), irr3));
          if (r >= rfloor) pr = cfma(tcd, -3.0 * irr3 * irr, pr);
          const double2 rad = cs(pr, act);
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            dv[c] = cfma(rad, vv[c], ca(cs(B, nvv[c]), cs(ca(cs(C, t1v[c]), cs(D, t2v[c])), irr3)));
            gn[c] = ca(gn[c], cs(ca(cs(B, vv[c]), cs(b0[c], ndr * ir3)), w));
            g1[c] = ca(g1[c], cs(ca(cs(C, vv[c]), cs(b0[c], in1)), w * irr3));
            g2[c] = ca(g2[c], cs(ca(cs(D, vv[c]), cs(b0[c], in2)), w * irr3));
          }
        }
        // cotangents of x, px, py
        const double iJ = J > 0 ? 1.0 / J : 0.0;
        const Vec un{nn.x * iJ, nn.y * iJ, nn.z * iJ};
        const Vec jx = vcross(py, un), jy = vcross(un, px);
        const double2 pj_ = cs(phi, wf);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          gpi[c] = cfma(dv[c], w, gpi[c]);
          ct[c] = cs(dv[c], -w);
        }
        ct[3] = cs(pj_, jx.x);
        ct[4] = cs(pj_, jx.y);
        ct[5] = cs(pj_, jx.z);
        ct[6] = cs(pj_, jy.x);
        ct[7] = cs(pj_, jy.y);
        ct[8] = cs(pj_, jy.z);
      }
#pragma unroll
      for (int c = 0; c < 9; ++c) {
        pv[(2 * c) * P + lane] = ct[c].x;
        pv[(2 * c + 1) * P + lane] = ct[c].y;
      }
      __syncwarp();
      if (lane < 3 * nb) {
        const int c = lane / 3, x = lane - 3 * c;
        const int np = min(32, npts - q0);
        double2 acc = gnode[s];
        for (int k = 0; k < np; ++k) {
          const double N = pb[(3 * c) * P + k], Dx = pb[(3 * c + 1) * P + k], Dy = pb[(3 * c + 2) * P + k];
          acc.x = fma(N, pv[(2 * x) * P + k], fma(Dx, pv[(2 * x + 6) * P + k], fma(Dy, pv[(2 * x + 12) * P + k], acc.x)));
          acc.y = fma(N, pv[(2 * x + 1) * P + k],
                      fma(Dx, pv[(2 * x + 7) * P + k], fma(Dy, pv[(2 * x + 13) * P + k], acc.y)));
        }
        gnode[s] = acc;
      }
      __syncwarp();
    }
  }
  if (lane < 3 * nb) {
    const int c = lane / 3, x = lane - 3 * c;
    for (int s = 0; s < nsub; ++s) atomic_c(&A.gnodes[27LL * j + 3 * sub_node(fk, self, s, c) + x], gnode[s]);
  }
  const double uu[3] = {u0.x, u0.y, u0.z};
  if (!self) gr0 = wsum2(gr0);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double2 g = wsum2(gpi[c]);
    if (lane == 0) {
      atomic_c(&A.gpos[3 * i + c], self ? g : cfma(gr0, -uu[c], g));  // d r0 / d pos_i = -u0
      if (!self) atomic_c(&A.gpos[3 * j + c], cs(gr0, uu[c]));
    }
    if (self) {
      const double2 a = wsum2(gn[c]), b = wsum2(g1[c]), d = wsum2(g2[c]);
      if (lane == 0) {
        atomic_c(&A.gnv[3 * i + c], a);
        atomic_c(&A.gt1[3 * i + c], b);
        atomic_c(&A.gt2[3 * i + c], d);
      }
    }
  }
}

}  // namespace adj
}  // namespace bem200

using namespace bem200;
using namespace bem200::adj;

static size_t al256(size_t b) { return (b + 255) & ~size_t(255); }

extern "C" {

size_t bem200_shape_gradient_workspace_size(int n, int64_t nref, int order) {
  const size_t no = (size_t)order + 1;
  const size_t nr = (size_t)(nref > 0 ? nref : 1);
  return al256(sizeof(double2) * nr * no) + al256(sizeof(double2) * nr * 3 * no) + 2 * al256(sizeof(double2) * n) +
         al256(sizeof(int64_t) * n);
}

int bem200_shape_gradient(int n, int npol, int npart, const int32_t* pid, const int32_t* blk_mat, int nmat,
                          const double* kmat_host, double k0, int eps_per_face, const double* eps1,
                          const double* eps2, const uint64_t* closed_mask, const double* pos, const double* nvec,
                          const double* tvec1, const double* tvec2, const double* area, const double* nodes,
                          const int32_t* face_kind, const double* rules, int n28, int n3, int n4, int64_t nref,
                          const int64_t* ref_row_ptr, const int32_t* ref_row, const int32_t* ref_col,
                          const int8_t* ref_kind, const int64_t* csc_col_ptr, const int32_t* csc_row, int order,
                          const double* g, const double* f, const double* corr, const void* W1, const void* W2,
                          const void* lam, void* grad, void* scratch, void* stream) {
  BEM_REQUIRE(n > 0 && npol > 0 && npart > 0 && pid && blk_mat && closed_mask && pos && nvec && tvec1 && tvec2 &&
                  area && nodes && face_kind && rules && corr && W1 && W2 && lam && grad && scratch && eps1 && eps2,
              BEM200_ERR_ARG, "shape_gradient: bad arguments");
  BEM_REQUIRE(npol <= kMaxPol, BEM200_ERR_UNSUPPORTED, "shape_gradient: at most %d polarisations", kMaxPol);
  BEM_REQUIRE(nmat > 0 && nmat <= kMaxMat && kmat_host, BEM200_ERR_ARG, "shape_gradient: 1 <= nmat <= %d", kMaxMat);
  BEM_REQUIRE(order >= 0 && order <= kMaxOrder, BEM200_ERR_ARG, "shape_gradient: order above %d", kMaxOrder);
  BEM_REQUIRE(nref > 0 && ref_row_ptr && ref_row && ref_col && ref_kind && csc_col_ptr && csc_row && g && f,
              BEM200_ERR_ARG, "shape_gradient: refinement tables missing (every mesh has refined self terms)");
  BEM_REQUIRE(n <= 8 * 48 * 1024 / kWarps, BEM200_ERR_UNSUPPORTED, "shape_gradient: n = %d faces is too many", n);
  cudaStream_t s = (cudaStream_t)stream;
  Args A;
  A.n = n;
  A.npol = npol;
  A.npart = npart;
  A.order = order;
  for (int m = 0; m < kMaxMat; ++m) {
    A.kt.re[m] = m < nmat ? kmat_host[2 * m] : 0.0;
    A.kt.im[m] = m < nmat ? kmat_host[2 * m + 1] : 0.0;
  }
  A.k0 = k0;
  A.eps_per_face = eps_per_face;
  if (eps_per_face) {
    A.e1d = (const double2*)eps1;
    A.e2d = (const double2*)eps2;
    A.e1s = A.e2s = make_double2(0, 0);
  } else {
    A.e1d = A.e2d = nullptr;
    A.e1s = make_double2(eps1[0], eps1[1]);
    A.e2s = make_double2(eps2[0], eps2[1]);
  }
  A.pid = pid;
  A.blk = blk_mat;
  A.closed_mask = closed_mask;
  A.pos = pos;
  A.nvec = nvec;
  A.area = area;
  A.tvec1 = tvec1;
  A.tvec2 = tvec2;
  A.nodes = nodes;
  A.face_kind = face_kind;
  A.rules = rules;
  A.n28 = n28;
  A.n3 = n3;
  A.n4 = n4;
  A.nref = nref;
  A.row_ptr = ref_row_ptr;
  A.ref_row = ref_row;
  A.ref_col = ref_col;
  A.ref_kind = ref_kind;
  A.col_ptr = csc_col_ptr;
  A.csc_row = csc_row;
  A.g = g;
  A.f = f;
  A.corr = corr;
  A.W1 = (const double2*)W1;
  A.W2 = (const double2*)W2;
  A.lam = (const double2*)lam;
  double2* gb = (double2*)grad;
  A.gpos = gb;
  A.gnv = gb + 3 * (size_t)n;
  A.garea = gb + 6 * (size_t)n;
  A.gt1 = gb + 7 * (size_t)n;
  A.gt2 = gb + 10 * (size_t)n;
  A.gnodes = gb + 13 * (size_t)n;
  const size_t no = (size_t)order + 1;
  const size_t nr = (size_t)(nref > 0 ? nref : 1);
  char* p = (char*)scratch;
  A.ghat = (double2*)p;   p += al256(sizeof(double2) * nr * no);
  A.fhat = (double2*)p;   p += al256(sizeof(double2) * nr * 3 * no);
  A.shat = (double2*)p;   p += al256(sizeof(double2) * n);
  A.chat = (double2*)p;   p += al256(sizeof(double2) * n);
  A.diag_e = (int64_t*)p;
  BEM_CUDA_CHECK(cudaMemsetAsync(grad, 0, sizeof(double2) * 40 * (size_t)n, s));
  BEM_CUDA_CHECK(cudaMemsetAsync(A.chat, 0, sizeof(double2) * n, s));
  BEM_CUDA_CHECK(cudaMemsetAsync(A.diag_e, 0xff, sizeof(int64_t) * n, s));  // -1
  refined_op_kernel<<<ceil_div(nref, 128), 128, 0, s>>>(A);
  BEM_LAUNCH_CHECK();
  closed_prep_kernel<<<ceil_div(n, 128), 128, 0, s>>>(A);
  BEM_LAUNCH_CHECK();
  const int smem = kWarps * ((n + 31) / 32) * (int)sizeof(uint32_t);
  BEM_CUDA_CHECK(set_kernel_attrs_once(far_rows_kernel, smem, false));
  BEM_CUDA_CHECK(set_kernel_attrs_once(far_cols_kernel, smem, false));
  far_rows_kernel<<<ceil_div(n, kWarps), 32 * kWarps, smem, s>>>(A);
  BEM_LAUNCH_CHECK();
  far_cols_kernel<<<ceil_div(n, kWarps), 32 * kWarps, smem, s>>>(A);
  BEM_LAUNCH_CHECK();
  refined_closed_kernel<<<ceil_div(nref, 128), 128, 0, s>>>(A);
  BEM_LAUNCH_CHECK();
  const int csm = kCoefWarps * (kPtVals + kPtBasis) * 33 * (int)sizeof(double);
  refine_coef_grad_kernel<<<ceil_div(nref, kCoefWarps), 32 * kCoefWarps, csm, s>>>(A);
  BEM_LAUNCH_CHECK();
  return BEM200_OK;
}

}  // extern "C"
