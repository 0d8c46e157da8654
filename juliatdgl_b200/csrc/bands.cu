// bands.cu — the order-parameter update of every band (gtdgl/src/bands.jl).
//
// One kernel per band stage: the gauge-link stencil of _band_row! (bands.jl:71-97) with the KWT update
// (kwt_update :135-140, kwt_update_rot :151-159), fused with the per-node epilogues that follow it in the
// reference — the rotating-frame rate or term (_frame_rate! :213-234, _frame_term! :274-286), the RKL/RKC
// combination (_combine! :425-430) and the final turn back (_frame_turn! :321-327).  The links of later RKL/RKC stages
// (_rotlinks!, _rotfrac!) are formed where a stage reads them; the other link rotations (_rot!, _advance_links!,
// _frame_links!, _link_rate!, :292-423) run as one kernel over the three link ranges.  The covariant Neumann ghosts of
// an intermediate stage (ghosts! :524-539) are formed in the next stage too, the step's final ones at the end of the
// step (k_finish, field.cu).
#include "common.cuh"
#include "merge.cuh"

namespace tdgl {

// The links a stage reads: the arrays as given (mode 0), or the rotated links of a later RKL/RKC stage formed from the
// step's links where the stencil reads them: (mode 1) V e^{iRc} with the per-step rate R of a rotating-frame band
// (_rotlinks!, bands.jl:311-316), (mode 2) V Q^c with Q = V conj(U) of a band without the frame (_rotfrac!, :409-423).
// The formulas are the link passes'.  Mode 2 replaces a pass per stage that read V and U and stored the result (144
// bytes a node, and a launch) by 48 more bytes a node in the stage.
struct LinkRot {
  int mode;
  double c;
  const cd *V[3], *U[3];
  const double *R[3];
};
__device__ __forceinline__ cd link_frac(cd v, cd u, double c);
// LR: the mode, fixed per kernel instance
template <int LR>
__device__ __forceinline__ cd link_at(const LinkRot &R, const cd *L, int ax, long long o) {
  if (LR == 0) return L[o];
  if (LR == 2) return link_frac(R.V[ax][o], R.U[ax][o], R.c);
  return cmul(R.V[ax][o], ccis_short(R.R[ax][o] * R.c));
}

struct StageArgs {
  cd *C;              // destination
  const cd *S;        // stage source
  int gfly;           // 1: S is an intermediate stage, whose ghosts are formed here (see nbp / nbm)
  BandPtrs G;         // every band at the start of the step (coupling)
  const cd *Lx, *Ly, *Lz;
  const double *f;
  tdgl_bandcoef cf;
  int mu, N, hard, rk;
  // epilogue
  int frame_rate;     // 1: first (sub)stage of a rotating-frame band: Ω from C and S, C ← C − iΩhS
  int frame_store;    // with frame_rate: store Ω only (noise: the rate is low-passed before it is applied)
  int frame_term;     // 1: later (sub)stage: C ← C − iΩhS
  int frame_rotterm;  // with frame_term: as the rotation C ← C e^{−iΩh} (noise, bands.jl:274-286)
  double h, wmax;
  double *Om;
  int combine;        // 1: C ← μC + νA
  int combine_log;    // with combine: C ← A exp(μ log(C/A)) (noise on a KWT band, bands.jl:439-445)
  double cmu, cnu;
  const cd *A;
  int turn;           // 1: C ← C e^{iΩ dt}
  double dt;
  Rng r;              // interior nodes
  Dim d;
  // material per region (bands.jl:53-68, 168-182): the node map, the tables (stage or full-step), τ for ρ
  const uint8_t *mat;
  const MatDev *mt;
  const double *tau[3];
  int mstage;
  const uint8_t *vac;   // a sculpted sample's vacuum nodes (bands.jl:103-124)
  LinkRot lr;           // how Lx, Ly, Lz are read
  const double *Th;     // the heat model's temperature field (null: none): ε = a − θ (bands.jl:33-35)
  double heat_a;
  const double *drag;   // the drag's full-step coefficients [µ][ν][x, y, z] (null: no drag), divided by ddiv
  double ddiv;          // the pass's divisor: n substeps, or the RKL/RKC weight q (_dragof, bands.jl:195-196)
};

__device__ __forceinline__ cd kwt_update(cd g, cd dd, double g2) {
  double a2 = cabs2(g);
  double q = 1 + g2 * a2;
  cd dp = rmul(sqrt(q), dd);
  return cadd(g, csub(dp, mulr(rmul(g2, g), cmul(cconj(g), dp).x / q)));
}

__device__ __forceinline__ cd kwt_update_rot(cd g, cd dd, double g2) {
  double a2 = cabs2(g);
  double q = 1 + g2 * a2;
  cd dp = rmul(sqrt(q), dd);
  cd Dl = csub(dp, mulr(rmul(g2, g), cmul(cconj(g), dp).x / q));
  if (!(a2 > 1e-24)) return cadd(g, Dl);
  double a = sqrt(a2);
  cd u = cdivr(g, a);
  cd w = cmul(cconj(u), Dl);
  return cmul(u, rmul(a + w.x, ccis(w.y / a)));
}

// _combine_log! (bands.jl:439-445): A exp(μ log(C/A)) where |A|² and |C|² exceed 1e-3, else μC + (1−μ)A.  C/A by
// the plain formula (Julia's is its robust complex division).
__device__ __forceinline__ cd combine_log(cd c, cd a, double mu) {
  if (!(cabs2(a) > 1e-3 && cabs2(c) > 1e-3)) return cadd(rmul(mu, c), rmul(1 - mu, a));
  const double dd = a.x * a.x + a.y * a.y;
  const cd z = mkc((c.x * a.x + c.y * a.y) / dd, (c.y * a.x - c.x * a.y) / dd);
  const cd w = rmul(mu, mkc(log(hypot(z.x, z.y)), atan2(z.y, z.x)));
  return cmul(a, rmul(exp(w.x), ccis(w.y)));
}

// _dif with the link weights ρ₊, ρ₋ (bands.jl:63-64): today's expression plus k((ρ₊−1)(v₊s₊−g) + (ρ₋−1)(v₋s₋−g))
__device__ __forceinline__ cd dif_mat(double rp, double rm, double k, cd vp, cd sp, cd vm, cd sm, cd g) {
  const cd a = cmul(vp, sp), b = cmul(vm, sm);
  return cadd(rmul(k, cadd(csub(a, rmul(2.0, g)), b)), rmul(k, cadd(rmul(rp - 1, csub(a, g)), rmul(rm - 1, csub(b, g)))));
}

template <bool MAT, bool VAC, int LR>
__device__ __forceinline__ void band_stage_b(const Blk bk, StageArgs const &A);
template <bool MAT, bool VAC, int LR>
__global__ void __launch_bounds__(256, (MAT || LR) ? 4 : 5) k_band_stage(StageArgs A) { band_stage_b<MAT, VAC, LR>(TDGL_BLK, A); }
#define TDGL_STAGE_MERGE(MAT, VAC, LR) \
  TDGL_MERGEABLE((k_band_stage<MAT, VAC, LR>), (band_stage_b<MAT, VAC, LR>), 256, 4, false)
TDGL_STAGE_MERGE(false, false, 0);
TDGL_STAGE_MERGE(true, false, 0);
TDGL_STAGE_MERGE(false, true, 0);
TDGL_STAGE_MERGE(true, true, 0);
TDGL_STAGE_MERGE(false, false, 1);
TDGL_STAGE_MERGE(true, false, 1);
TDGL_STAGE_MERGE(false, true, 1);
TDGL_STAGE_MERGE(true, true, 1);
TDGL_STAGE_MERGE(false, false, 2);
TDGL_STAGE_MERGE(true, false, 2);
TDGL_STAGE_MERGE(false, true, 2);
TDGL_STAGE_MERGE(true, true, 2);
template <bool MAT, bool VAC, int LR>
__device__ __forceinline__ void band_stage_b(const Blk bk, StageArgs const &A) {
  long long t = (long long)bk.x * blockDim.x + threadIdx.x;
  if (t >= A.r.n()) return;
  int i, j, k;
  rng_ijk(A.r, t, i, j, k);
  const Dim d = A.d;
  const long long o = d.at(i, j, k);
  const long long sx = 1, sy = d.n1, sz = (long long)d.n1 * d.n2;
  auto LX = [&](long long q) { return link_at<LR>(A.lr, A.Lx, 0, q); };
  auto LY = [&](long long q) { return link_at<LR>(A.lr, A.Ly, 1, q); };
  auto LZ = [&](long long q) { return link_at<LR>(A.lr, A.Lz, 2, q); };
  cd g = A.S[o];
  double fm = A.f[o];
  // the stage source at the next (nbp) and previous (nbm) node along an axis.  A node beside a face reads its ghost:
  // of an intermediate stage (gfly) the value ghosts! would have stored, L S of the node inside (which is this node) on
  // the low face and conj(L) S on the high one, with this stage's own links (the same product, the same bits).  The
  // stencil reads face points only, never edges.  This saves the ghost pass of every intermediate stage, a launch
  // between two stages that cannot overlap it.  With the links of mode 2, the clamped Ω faces and no copy at the end,
  // 40 steps went from 3318 to 2811 µs (12×8×4 cells), 4183 to 3782 (64×32×8), 8289 to 7893 (192×64×16), 10207 to
  // 6841 (101×37×9 with noise) and 252.9 to 250.0 ms (the 256×128×32 ramp).
  const Rng &rg = A.r;
  auto nbp = [&](int ax, long long s, cd l) {
    const bool edge = ax == 0 ? i == rg.i0 + rg.ni - 1 : ax == 1 ? j == rg.j0 + rg.nj - 1 : k == rg.k0 + rg.nk - 1;
    return A.gfly && edge ? cmul(cconj(l), g) : A.S[o + s];
  };
  auto nbm = [&](int ax, long long s, cd lc) {   // lc: the conjugate of the previous link
    const bool edge = ax == 0 ? i == rg.i0 : ax == 1 ? j == rg.j0 : k == rg.k0;
    return A.gfly && edge ? cmul(cconj(lc), g) : A.S[o - s];
  };
  cd v;
  if ((VAC && A.vac[o]) || (A.hard && fm == 0.0)) {
    v = mkc(0.0, 0.0);
  } else if (VAC) {   // _band_row_vac!: each neighbour with the mask of its link (τ, or ρ = τ·W with materials)
    const int mu = A.mu, m = MAT ? A.mat[o] - 1 : 0;
    const tdgl_bandcoef &cf = MAT ? (A.mstage ? A.mt->stage[mu][m] : A.mt->full[mu][m]) : A.cf;
    double wxp = A.tau[0][o], wxm = A.tau[0][o - sx], wyp = A.tau[1][o], wym = A.tau[1][o - sy], wzp = A.tau[2][o],
           wzm = A.tau[2][o - sz];
    if (MAT) {
      const double(*W)[TDGL_MAXMAT][TDGL_MAXMAT] = A.mt->W[mu];
      wxp *= W[0][m][A.mat[o + sx] - 1];
      wxm *= W[0][A.mat[o - sx] - 1][m];
      wyp *= W[1][m][A.mat[o + sy] - 1];
      wym *= W[1][A.mat[o - sy] - 1][m];
      wzp *= W[2][m][A.mat[o + sz] - 1];
      wzm *= W[2][A.mat[o - sz] - 1][m];
    }
    const cd lxp = LX(o), lxm = cconj(LX(o - sx)), lyp = LY(o), lym = cconj(LY(o - sy)), lzp = LZ(o), lzm = cconj(LZ(o - sz));
    cd tx = rmul(cf.kx, cadd(rmul(wxp, csub(cmul(lxp, nbp(0, sx, lxp)), g)), rmul(wxm, csub(cmul(lxm, nbm(0, sx, lxm)), g))));
    cd ty = rmul(cf.ky, cadd(rmul(wyp, csub(cmul(lyp, nbp(1, sy, lyp)), g)), rmul(wym, csub(cmul(lym, nbm(1, sy, lym)), g))));
    cd tz = rmul(cf.kz, cadd(rmul(wzp, csub(cmul(lzp, nbp(2, sz, lzp)), g)), rmul(wzm, csub(cmul(lzm, nbm(2, sz, lzm)), g))));
    cd acc = cadd(cadd(cadd(cadd(g, tx), ty), tz), mulr(rmul(cf.c, g), fm * cf.eps - cf.beta * cabs2(g)));
    for (int nu = 0; nu < A.N; nu++) {
      if (nu == mu) continue;
      acc = cadd(acc, rmul(cf.cpl[nu], A.G.p[nu][o]));
    }
    if (cf.gamma2 > 0) v = A.rk ? kwt_update_rot(g, csub(acc, g), cf.gamma2) : kwt_update(g, csub(acc, g), cf.gamma2);
    else v = acc;
    if (MAT && A.mt->absent[mu][m]) v = mkc(0.0, 0.0);
  } else if (MAT) {   // the node's material: its coefficients, ρ = τ·W of each link, Ψ = 0 where the band is absent
    const int m = A.mat[o] - 1, mu = A.mu;
    const tdgl_bandcoef &cf = A.mstage ? A.mt->stage[mu][m] : A.mt->full[mu][m];
    const double(*W)[TDGL_MAXMAT][TDGL_MAXMAT] = A.mt->W[mu];
    const int mxp = A.mat[o + sx] - 1, mxm = A.mat[o - sx] - 1, myp = A.mat[o + sy] - 1, mym = A.mat[o - sy] - 1,
              mzp = A.mat[o + sz] - 1, mzm = A.mat[o - sz] - 1;
    const cd vxp = LX(o), vxm = cconj(LX(o - sx));
    cd tx = dif_mat(A.tau[0][o] * W[0][m][mxp], A.tau[0][o - sx] * W[0][mxm][m], cf.kx, vxp, nbp(0, sx, vxp), vxm,
                    nbm(0, sx, vxm), g);
    const cd vyp = LY(o), vym = cconj(LY(o - sy));
    cd ty = dif_mat(A.tau[1][o] * W[1][m][myp], A.tau[1][o - sy] * W[1][mym][m], cf.ky, vyp, nbp(1, sy, vyp), vym,
                    nbm(1, sy, vym), g);
    const cd vzp = LZ(o), vzm = cconj(LZ(o - sz));
    cd tz = dif_mat(A.tau[2][o] * W[2][m][mzp], A.tau[2][o - sz] * W[2][mzm][m], cf.kz, vzp, nbp(2, sz, vzp), vzm,
                    nbm(2, sz, vzm), g);
    const double eps = A.Th ? A.mt->a[mu][m] - A.Th[o] : cf.eps;   // _anode: the material's a (bands.jl:65-66)
    cd nl = mulr(rmul(cf.c, g), fm * eps - cf.beta * cabs2(g));
    cd acc = cadd(cadd(cadd(cadd(g, tx), ty), tz), nl);
    for (int nu = 0; nu < A.N; nu++) {
      if (nu == mu) continue;
      acc = cadd(acc, rmul(cf.cpl[nu], A.G.p[nu][o]));
    }
    if (cf.gamma2 > 0) v = A.rk ? kwt_update_rot(g, csub(acc, g), cf.gamma2) : kwt_update(g, csub(acc, g), cf.gamma2);
    else v = acc;
    if (A.mt->absent[mu][m]) v = mkc(0.0, 0.0);
  } else {
    const tdgl_bandcoef &cf = A.cf;
    cd g2 = rmul(2.0, g);
    const cd vxp = LX(o), vxm = cconj(LX(o - sx));
    cd tx = rmul(cf.kx, cadd(csub(cmul(vxp, nbp(0, sx, vxp)), g2), cmul(vxm, nbm(0, sx, vxm))));
    const cd vyp = LY(o), vym = cconj(LY(o - sy));
    cd ty = rmul(cf.ky, cadd(csub(cmul(vyp, nbp(1, sy, vyp)), g2), cmul(vym, nbm(1, sy, vym))));
    const cd vzp = LZ(o), vzm = cconj(LZ(o - sz));
    cd tz = rmul(cf.kz, cadd(csub(cmul(vzp, nbp(2, sz, vzp)), g2), cmul(vzm, nbm(2, sz, vzm))));
    const double eps = A.Th ? A.heat_a - A.Th[o] : cf.eps;
    cd nl = mulr(rmul(cf.c, g), fm * eps - cf.beta * cabs2(g));
    cd acc = cadd(cadd(cadd(cadd(g, tx), ty), tz), nl);
    for (int nu = 0; nu < A.N; nu++) {
      if (nu == A.mu) continue;
      acc = cadd(acc, rmul(cf.cpl[nu], A.G.p[nu][o]));
    }
    if (A.drag)   // _drag (bands.jl:37-51): the lattice Laplacian of every other band on this pass's links
      for (int nu = 0; nu < A.N; nu++) {
        if (nu == A.mu) continue;
        const double *c3 = A.drag + 3 * (TDGL_MAXB * A.mu + nu);
        const double cx = c3[0] / A.ddiv, cy = c3[1] / A.ddiv, cz = c3[2] / A.ddiv;
        const cd *P = A.G.p[nu];
        const cd p2 = rmul(2.0, P[o]);
        const cd ex = rmul(cx, cadd(csub(cmul(vxp, P[o + sx]), p2), cmul(vxm, P[o - sx])));
        const cd ey = rmul(cy, cadd(csub(cmul(vyp, P[o + sy]), p2), cmul(vym, P[o - sy])));
        const cd ez = rmul(cz, cadd(csub(cmul(vzp, P[o + sz]), p2), cmul(vzm, P[o - sz])));
        acc = cadd(acc, cadd(cadd(ex, ey), ez));
      }
    if (cf.gamma2 > 0) v = A.rk ? kwt_update_rot(g, csub(acc, g), cf.gamma2) : kwt_update(g, csub(acc, g), cf.gamma2);
    else v = acc;
  }
  if (A.frame_rate) {
    double a2 = cabs2(g);
    double w = 0.0;
    if (a2 > 1e-3) {
      w = cmul(cconj(g), csub(v, g)).y / (a2 * A.h);
      w = w < -A.wmax ? -A.wmax : (w > A.wmax ? A.wmax : w);
    }
    A.Om[o] = w;
    if (!A.frame_store) v = cminus_i(v, w * A.h, g);
  } else if (A.frame_term) {
    v = A.frame_rotterm ? cmul(v, ccis(-(A.Om[o] * A.h))) : cminus_i(v, A.Om[o] * A.h, g);
  }
  if (A.combine) v = A.combine_log ? combine_log(v, A.A[o], A.cmu) : cadd(rmul(A.cmu, v), rmul(A.cnu, A.A[o]));
  if (A.turn) v = cmul(v, ccis(A.Om[o] * A.dt));
  A.C[o] = v;
}

// Link operations over the three link ranges of the band stencil (_rx, _ry, _rz, bands.jl:349-351).
enum LinkOp { LOP_ROT_INIT = 0, LOP_ADVANCE, LOP_FRAME_LINKS, LOP_LINK_RATE };

struct LinkArgs {
  int op;
  Rng r[3];
  Dim d;
  cd *L[3], *Rl[3];
  const cd *V[3], *U[3];
  double *Rr[3];
  const double *Om;
  Rng ri;       // the interior nodes, where Ω is stored
  double par;   // n (ROT_INIT), τ (FRAME_LINKS), dt (LINK_RATE)
};

// The per-link formulas (bands.jl:303-310 _link_rate!, :355-369 _rot!, :409-423 _rotfrac!), shared by the step's
// link passes and by tdgl_link_rotations.  −arg q of q = V conj(U), with the short series while Re q > 0 and
// |sin| <= 0.05:
__device__ __forceinline__ double link_angle(cd v, cd u) {
  const cd q = cmul(v, cconj(u));
  const double sf = -q.y;
  return (q.x > 0 && fabs(sf) <= 0.05) ? -(sf + sf * sf * sf / 6) : cangle(q);
}
// Q^{1/n}
__device__ __forceinline__ cd link_root(cd v, cd u, double n) {
  const cd q = cmul(v, cconj(u));
  const double sf = -q.y;
  if (q.x > 0 && fabs(sf) <= 0.05) {
    const double a = (sf + sf * sf * sf / 6) / n;
    const double a2 = a * a;
    return mkc(1 - a2 / 2, -a * (1 - a2 / 6));
  }
  return ccis(cangle(q) / n);
}
// V Q^c
__device__ __forceinline__ cd link_frac(cd v, cd u, double c) {
  const cd q = cmul(v, cconj(u));
  const double sf = -q.y;
  if (q.x > 0 && fabs(sf) <= 0.05) {
    const double a = (sf + sf * sf * sf / 6) * c;
    const double a2 = a * a;
    return cmul(v, mkc(1 - a2 / 2, -a * (1 - a2 / 6)));
  }
  return cmul(v, ccis(cangle(q) * c));
}

__device__ __forceinline__ void link_op_b(const Blk bk, LinkArgs const &A);
__global__ void __launch_bounds__(256, 5) k_link_op(LinkArgs A) { link_op_b(TDGL_BLK, A); }
TDGL_MERGEABLE(k_link_op, link_op_b, 256, 1, false);
__device__ __forceinline__ void link_op_b(const Blk bk, LinkArgs const &A) {
  long long t = (long long)bk.x * blockDim.x + threadIdx.x;
  int ax = 0;
  if (t >= A.r[0].n()) {
    t -= A.r[0].n();
    ax = 1;
    if (t >= A.r[1].n()) {
      t -= A.r[1].n();
      ax = 2;
      if (t >= A.r[2].n()) return;
    }
  }
  int i, j, k;
  rng_ijk(A.r[ax], t, i, j, k);
  const long long o = A.d.at(i, j, k);
  const int oi = ax == 0, oj = ax == 1, ok = ax == 2;
  // Ω along the link; a face point has the node inside (bands.jl:224-232: the copies x, then y, then z clamp each index)
  auto dOm = [&]() {
    return A.Om[om_at(A.d, A.ri, i + oi, j + oj, k + ok)] - A.Om[om_at(A.d, A.ri, i, j, k)];
  };
  switch (A.op) {
    case LOP_ROT_INIT: {
      const cd v = A.V[ax][o];
      A.L[ax][o] = v;
      A.Rl[ax][o] = link_root(v, A.U[ax][o], A.par);
      break;
    }
    case LOP_ADVANCE:
      A.L[ax][o] = cmul(A.L[ax][o], A.Rl[ax][o]);
      break;
    case LOP_FRAME_LINKS:
      A.L[ax][o] = cmul(A.L[ax][o], ccis_short(dOm() * A.par));
      break;
    case LOP_LINK_RATE:
      A.Rr[ax][o] = link_angle(A.V[ax][o], A.U[ax][o]) + dOm() * A.par;
      break;
  }
}

// X = 0 on the nodes outside the block (x1..x2+1 and so on)
__global__ void k_zero_outside(cd *X, Geo g) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= g.d.n()) return;
  const int i = 1 + (int)(t % g.d.n1), j = 1 + (int)((t / g.d.n1) % g.d.n2), k = 1 + (int)(t / ((long long)g.d.n1 * g.d.n2));
  if (i < g.x1 || i > g.x2 + 1 || j < g.y1 || j > g.y2 + 1 || k < g.z1 || k > g.z2 + 1) X[t] = mkc(0.0, 0.0);
}

namespace {

const int BS = 256;

Rng interior(const Geo &g) { return mkrng(g.x1 + 1, g.x2, g.y1 + 1, g.y2, g.z1 + 1, g.z2); }

void link_op(Ctx *ctx, int op, double par) {
  const Geo &g = ctx->g;
  LinkArgs A;
  A.op = op;
  A.r[0] = mkrng(g.x1, g.x2, g.y1, g.y2 + 1, g.z1, g.z2 + 1);
  A.r[1] = mkrng(g.x1, g.x2 + 1, g.y1, g.y2, g.z1, g.z2 + 1);
  A.r[2] = mkrng(g.x1, g.x2 + 1, g.y1, g.y2 + 1, g.z1, g.z2);
  A.d = g.d;
  for (int ax = 0; ax < 3; ax++) {
    A.L[ax] = ctx->L[ax]; A.Rl[ax] = ctx->Rl[ax]; A.V[ax] = ctx->V[ax]; A.U[ax] = ctx->U[ax]; A.Rr[ax] = ctx->Rr[ax];
  }
  A.Om = ctx->Om;
  A.ri = interior(g);
  A.par = par;
  long long n = A.r[0].n() + A.r[1].n() + A.r[2].n();
  static const double per[4] = {64, 48, 40, 48};   // compulsory bytes per link of each operation
  TDGL_LAUNCH(ctx, K_LINK, per[op] * n, k_link_op, nblk(n, BS), BS, 0, A);
}

StageArgs stage_base(Ctx *ctx, int mu, const tdgl_bandcoef &cf, double ddiv) {
  StageArgs A;
  memset(&A, 0, sizeof(A));
  for (int nu = 0; nu < ctx->N; nu++) A.G.p[nu] = ctx->G[nu];
  A.f = ctx->f;
  A.cf = cf;
  A.mu = mu;
  A.N = ctx->N;
  A.hard = ctx->P.hard;
  A.rk = ctx->P.noise_on;
  A.Om = ctx->Om;
  A.dt = ctx->P.dt;
  A.wmax = 0.5 / ctx->P.dt;
  A.r = interior(ctx->g);
  A.d = ctx->g.d;
  A.mat = ctx->mat;
  A.mt = ctx->mt;
  for (int ax = 0; ax < 3; ax++) A.tau[ax] = ctx->tau[ax];
  A.mstage = &cf == &ctx->P.bcs[mu];   // the stage table where the band's stage coefficients are in use
  A.vac = ctx->vac;
  A.drag = ctx->drag_c;
  A.ddiv = ddiv;
  A.Th = ctx->P.heat_on ? ctx->Th : nullptr;
  A.heat_a = ctx->P.heat_a[mu];
  return A;
}

// compulsory bytes per interior node: S, C, f, three links, the other bands, and the epilogue's A and Ω
double stage_bytes(const StageArgs &A) {
  double b = 16 + 16 + 8 + 48 + 16.0 * (A.N - 1);
  if (A.lr.mode == 1) b += 24;   // the rate R beside the links V
  if (A.lr.mode == 2) b += 48;   // the links U of the step before
  if (A.combine) b += 16;
  if (A.frame_rate || A.frame_term || A.turn) b += 8;
  if (A.mat || A.vac) b += 24 + 1;   // τ along the three axes, the node's material or vacuum flag
  if (A.drag) b += 16.0 * (A.N - 1);   // the other bands' neighbours come from the cache
  return b * (double)A.r.n();
}

void launch_stage(Ctx *ctx, const StageArgs &A) {
  const long long nb = nblk(A.r.n(), BS);
  const double by = stage_bytes(A);
#define TDGL_STAGE_LAUNCH(LR)                                                                        \
  do {                                                                                               \
    if (A.vac && A.mat) TDGL_LAUNCH(ctx, K_BAND, by, (k_band_stage<true, true, LR>), nb, BS, 0, A);   \
    else if (A.vac) TDGL_LAUNCH(ctx, K_BAND, by, (k_band_stage<false, true, LR>), nb, BS, 0, A);      \
    else if (A.mat) TDGL_LAUNCH(ctx, K_BAND, by, (k_band_stage<true, false, LR>), nb, BS, 0, A);      \
    else TDGL_LAUNCH(ctx, K_BAND, by, (k_band_stage<false, false, LR>), nb, BS, 0, A);               \
  } while (0)
  if (A.lr.mode == 2) TDGL_STAGE_LAUNCH(2);
  else if (A.lr.mode == 1) TDGL_STAGE_LAUNCH(1);
  else TDGL_STAGE_LAUNCH(0);
#undef TDGL_STAGE_LAUNCH
}

void band_euler(Ctx *ctx, int mu) {
  const bool noise = ctx->P.noise_on != 0;
  StageArgs A = stage_base(ctx, mu, ctx->P.bc[mu], 1.0);
  A.C = ctx->F[mu];
  A.S = ctx->G[mu];
  A.Lx = ctx->V[0]; A.Ly = ctx->V[1]; A.Lz = ctx->V[2];
  if (ctx->P.rotframe) {
    A.frame_rate = 1;
    A.frame_store = noise;
    A.h = ctx->P.dt;
    A.turn = !noise;
  }
  launch_stage(ctx, A);
  if (ctx->P.rotframe && noise) {   // the low-passed rate, its rotation, then the turn back (bands.jl:336-339)
    frame_smooth_rot(ctx, ctx->F[mu], ctx->P.dt);
    frame_rot(ctx, ctx->F[mu], -ctx->P.dt);
  }
}

void band_substeps(Ctx *ctx, int mu, int n) {
  const bool rot = ctx->P.rotframe != 0, ex = ctx->P.extrap != 0, noise = ctx->P.noise_on != 0;
  const cd *L[3] = {ctx->V[0], ctx->V[1], ctx->V[2]};
  if (ex) {
    link_op(ctx, LOP_ROT_INIT, (double)n);
    for (int ax = 0; ax < 3; ax++) L[ax] = ctx->L[ax];
  }
  const cd *src = ctx->G[mu];
  const double h = ctx->P.dt / n;
  for (int m = 1; m <= n; m++) {
    cd *dst = ((n - m) % 2 == 0) ? ctx->F[mu] : ctx->W;
    StageArgs A = stage_base(ctx, mu, ctx->P.bcs[mu], (double)n);
    A.C = dst;
    A.S = src;
    A.gfly = m > 1;
    A.Lx = L[0]; A.Ly = L[1]; A.Lz = L[2];
    A.h = h;
    if (rot) {
      if (m == 1) {
        A.frame_rate = 1;
        A.frame_store = noise;
      } else {
        A.frame_term = 1;
        A.frame_rotterm = noise;
      }
      if (m == n) A.turn = 1;
    }
    launch_stage(ctx, A);
    if (rot && noise && m == 1) frame_smooth_rot(ctx, dst, h);
    if (m < n) {
      if (ex) link_op(ctx, LOP_ADVANCE, 0.0);
      if (rot) link_op(ctx, LOP_FRAME_LINKS, h);
    }
    src = dst;
  }
}

void band_rkl(Ctx *ctx, int mu, int ns) {
  const tdgl_params &P = ctx->P;
  const bool kc = P.use_rkc[mu] != 0, rot = P.rotframe != 0, ex = P.extrap != 0, noise = P.noise_on != 0;
  const bool skq = skrock_band(ctx, mu), lg = noise && haskwt(ctx, mu);
  const double q = kc ? P.rkc_q[mu] : (double)(ns * (ns + 1) / 2);
  const double h = P.dt / q;
  const cd *L[3] = {ctx->V[0], ctx->V[1], ctx->V[2]};
  // the stages' destinations in turn, so that the last one is F[µ] (no copy at the end)
  const int off = (2 - (ns - 1) % 3 + 3) % 3;
  cd *ring[3] = {ctx->W, ctx->W2, ctx->F[mu]};
  auto dest = [&](int j) { return ring[(j - 1 + off) % 3]; };
  const cd *A_ = ctx->G[mu], *B = ctx->G[mu];
  cd *Cc = dest(1);
  // the links of stage j > 1 are the step's links rotated to the fraction c_{j−1} of the step, formed where the stage
  // reads them (no stored copy)
  LinkRot lr;
  memset(&lr, 0, sizeof(lr));
  for (int ax = 0; ax < 3; ax++) {
    lr.V[ax] = ctx->V[ax];
    lr.U[ax] = ctx->U[ax];
    lr.R[ax] = ctx->Rr[ax];
  }
  for (int j = 1; j <= ns; j++) {
    Cc = dest(j);
    const cd *src = B;
    if (j == 1 && skq) {   // SK-ROCK for the phase: K₁ = E(Ψⁿ e^{iν₁δθ}) e^{i(κ₁−ν₁)δθ} (bands.jl:482-488)
      sk_turn(ctx, dest(2), B, mu, P.rkc_sk[mu][0]);   // the second stage's destination is free until then
      src = dest(2);
    }
    StageArgs A = stage_base(ctx, mu, P.bcs[mu], q);
    A.C = Cc;
    A.S = src;
    A.gfly = j > 1 || skq;
    A.Lx = L[0]; A.Ly = L[1]; A.Lz = L[2];
    A.lr = lr;
    A.h = h;
    if (rot) {
      if (j == 1) {
        A.frame_rate = 1;
        A.frame_store = noise;
      } else {
        A.frame_term = 1;
        A.frame_rotterm = noise;
      }
    }
    if (j >= 2) {
      A.combine = 1;
      A.combine_log = lg;
      A.cmu = kc ? P.rkc_mu[mu][j - 1] : (double)(2 * j - 1) / j;
      A.cnu = kc ? P.rkc_nu[mu][j - 1] : (double)(1 - j) / j;
      A.A = A_;
    }
    const bool late_turn = j == ns && rot && j == 1 && noise;   // the turn follows the low-passed rate
    if (j == ns && rot && !late_turn) A.turn = 1;
    launch_stage(ctx, A);
    if (j == 1 && rot && noise) frame_smooth_rot(ctx, Cc, h);
    if (j == 1 && skq) sk_turn(ctx, Cc, Cc, mu, P.rkc_sk[mu][1] - P.rkc_sk[mu][0]);
    if (late_turn) frame_rot(ctx, Cc, -P.dt);
    if (rot && j == 1 && ex && ns > 1) link_op(ctx, LOP_LINK_RATE, P.dt);
    if (j < ns && ex) {
      lr.mode = rot ? 1 : 2;
      lr.c = kc ? P.rkc_c[mu][j - 1] : (double)(j * (j + 1)) / (double)(ns * (ns + 1));
    }
    A_ = B;
    B = Cc;
  }
}

}  // namespace

// The reference copies the last of an RKL/RKC band's buffers into F[µ] whole unless the stage count put it there: on
// the nodes outside the block, which no stage writes, F is then the buffer's zeros.  The stages here end in F[µ]
// themselves, so those nodes are cleared once, when a state came in from outside.
void clear_outside(Ctx *ctx) {
  const long long n = ctx->g.d.n();
  for (int mu = 0; mu < ctx->N; mu++)
    if (ctx->P.stages[mu] > 0 && (ctx->P.stages[mu] - 1) % 3 != 2) {
      k_zero_outside<<<nblk(n, BS), BS, 0, ctx->stream>>>(ctx->F[mu], ctx->g);
      ctx->launches++;
    }
}

struct BandOut {
  cd *p[TDGL_MAXB];
};

__device__ __forceinline__ void vacuum_zero_b(const Blk bk, BandOut const &F, int const &N, const uint8_t * const &vac, long long const &n);
__global__ void k_vacuum_zero(BandOut F, int N, const uint8_t *vac, long long n) { vacuum_zero_b(TDGL_BLK, F, N, vac, n); }
TDGL_MERGEABLE(k_vacuum_zero, vacuum_zero_b, 256, 1, false);
__device__ __forceinline__ void vacuum_zero_b(const Blk bk, BandOut const &F, int const &N, const uint8_t * const &vac, long long const &n) {
  const long long t = (long long)bk.x * blockDim.x + threadIdx.x;
  if (t >= n || !vac[t]) return;
  for (int mu = 0; mu < N; mu++) F.p[mu][t] = mkc(0.0, 0.0);
}

void vacuum_zero(Ctx *ctx) {
  BandOut F;
  for (int mu = 0; mu < ctx->N; mu++) F.p[mu] = ctx->F[mu];
  const long long n = ctx->g.d.n();
  TDGL_LAUNCH(ctx, K_GHOST, 1.0 * n, k_vacuum_zero, nblk(n, BS), BS, 0, F, ctx->N, ctx->vac, n);
}

static void use_ws(Ctx *ctx, const Ctx::BandWs &w) {
  ctx->W = w.W;
  ctx->W2 = w.W2;
  ctx->Om = w.Om;
  ctx->Oms = w.Oms;
  for (int ax = 0; ax < 3; ax++) {
    ctx->L[ax] = w.L[ax];
    ctx->Rl[ax] = w.Rl[ax];
    ctx->Rr[ax] = w.Rr[ax];
  }
}

// update_bands! (bands.jl:330-346).  Each band reads the state at the start of the step (its own Ψ and, for the
// coupling and the drag, the other bands' G) and writes only its F[µ]: band µ ≥ 1 runs on its own stream with its
// own workspaces, forked from the context's stream and joined back (parallel branches of a captured step).  When the
// launches are timed one by one the bands run in order on the one stream; the results are the same.
int update_bands(Ctx *ctx) {
  const bool par = ctx->N > 1 && ctx->branches && !ctx->prof.on && ctx->bstream[1];
  cudaStream_t main = ctx->stream;
  if (par) cudaEventRecord(ctx->bev[0], main);
  for (int mu = 0; mu < ctx->N; mu++) {
    if (par && mu > 0) {
      cudaStreamWaitEvent(ctx->bstream[mu], ctx->bev[0], 0);
      ctx->stream = ctx->bstream[mu];
    }
    use_ws(ctx, ctx->bws[par ? mu : 0]);
    int n = ctx->P.nsub[mu];
    if (ctx->P.stages[mu] > 0) band_rkl(ctx, mu, ctx->P.stages[mu]);
    else if (n == 1) band_euler(ctx, mu);
    else band_substeps(ctx, mu, n);
    if (par && mu > 0) {
      cudaEventRecord(ctx->bev[mu], ctx->bstream[mu]);
      ctx->stream = main;
    }
  }
  use_ws(ctx, ctx->bws[0]);
  if (par)
    for (int mu = 1; mu < ctx->N; mu++) cudaStreamWaitEvent(main, ctx->bev[mu], 0);
  return 0;
}

}  // namespace tdgl

// ---------------------------------------------------------------------------------------------- link rotations alone
// The step's per-link rotation formulas on caller arrays (the reference drives its device kernels the same way on
// manufactured links, gpu/TDGLGPU/test/test_link_rotations.jl:21-60).
namespace {
struct RotArgs {
  int op, ax, i0, j0, k0, ni, nj, nk;
  Dim d;
  const cd *V, *U;
  const double *Om;
  double par;
  cd *L, *R;
  double *Rr;
};
__global__ void k_rotations(RotArgs A) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)A.ni * A.nj * A.nk) return;
  const int i = A.i0 + (int)(t % A.ni), j = A.j0 + (int)((t / A.ni) % A.nj), k = A.k0 + (int)(t / ((long long)A.ni * A.nj));
  const long long o = A.d.at(i, j, k);
  if (A.op == 0) {
    A.L[o] = A.V[o];
    A.R[o] = tdgl::link_root(A.V[o], A.U[o], A.par);
  } else if (A.op == 1) {
    A.L[o] = tdgl::link_frac(A.V[o], A.U[o], A.par);
  } else {
    A.Rr[o] = tdgl::link_angle(A.V[o], A.U[o]) +
              (A.Om[A.d.at(i + (A.ax == 0), j + (A.ax == 1), k + (A.ax == 2))] - A.Om[o]) * A.par;
  }
}
}  // namespace

extern "C" int tdgl_link_rotations(int32_t op, int32_t n1, int32_t n2, int32_t n3, const int32_t *rng, int32_t ax,
                                   const double *V, const double *U, const double *Om, double par, double *L, double *R) {
  if (op < 0 || op > 2 || ax < 0 || ax > 2 || n1 < 1 || n2 < 1 || n3 < 1 || !rng || !V || !U) return TDGL_EINVAL;
  if ((op == 0 && (!L || !R)) || (op == 1 && !L) || (op == 2 && (!Om || !R))) return TDGL_EINVAL;
  const int oi = ax == 0, oj = ax == 1, ok = ax == 2;
  const bool rate = op == 2;
  // every point of the range, and its neighbour along ax for the rate, lies inside the arrays
  if (rng[0] < 1 || rng[2] < 1 || rng[4] < 1 || rng[1] + (rate ? oi : 0) > n1 || rng[3] + (rate ? oj : 0) > n2 ||
      rng[5] + (rate ? ok : 0) > n3 || rng[1] < rng[0] || rng[3] < rng[2] || rng[5] < rng[4])
    return TDGL_EINVAL;
  const size_t n = (size_t)n1 * n2 * n3;
  std::vector<void *> bufs;
  auto dev = [&](size_t bytes, const void *src) -> void * {
    void *p = nullptr;
    if (cudaMalloc(&p, bytes) != cudaSuccess) return nullptr;
    bufs.push_back(p);
    if (src) cudaMemcpy(p, src, bytes, cudaMemcpyHostToDevice);
    else cudaMemset(p, 0, bytes);
    return p;
  };
  RotArgs A;
  A.op = op; A.ax = ax;
  A.i0 = rng[0]; A.j0 = rng[2]; A.k0 = rng[4];
  A.ni = rng[1] - rng[0] + 1; A.nj = rng[3] - rng[2] + 1; A.nk = rng[5] - rng[4] + 1;
  A.d.n1 = n1; A.d.n2 = n2; A.d.n3 = n3;
  A.par = par;
  A.V = (const cd *)dev(n * sizeof(cd), V);
  A.U = (const cd *)dev(n * sizeof(cd), U);
  A.Om = rate ? (const double *)dev(n * sizeof(double), Om) : nullptr;
  A.L = op != 2 ? (cd *)dev(n * sizeof(cd), L) : nullptr;
  A.R = op == 0 ? (cd *)dev(n * sizeof(cd), R) : nullptr;
  A.Rr = rate ? (double *)dev(n * sizeof(double), R) : nullptr;
  int rc = TDGL_OK;
  if (!A.V || !A.U || (rate && (!A.Om || !A.Rr)) || (op != 2 && !A.L) || (op == 0 && !A.R)) rc = TDGL_ENOMEM;
  if (rc == TDGL_OK) {
    const long long cnt = (long long)A.ni * A.nj * A.nk;
    k_rotations<<<(unsigned)((cnt + 255) / 256), 256>>>(A);
    cudaError_t e = cudaDeviceSynchronize();
    if (e == cudaSuccess && A.L) e = cudaMemcpy(L, A.L, n * sizeof(cd), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess && A.R) e = cudaMemcpy(R, A.R, n * sizeof(cd), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess && A.Rr) e = cudaMemcpy(R, A.Rr, n * sizeof(double), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) rc = TDGL_ECUDA;
  }
  for (void *p : bufs) cudaFree(p);
  return rc;
}
