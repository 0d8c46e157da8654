// heat.cu — the heat model's temperature field (gtdgl/src/terms.jl: Heat, _band_heat, heat_step! with one material).
//
// The reference updates θ in place in lexicographic order: a node reads the new θ of its i−1, j−1 and k−1
// neighbours and the old θ of i+1, j+1 and k+1.  The same order on the device is a sweep over the planes
// i + j + k = s: every node of a plane depends only on the planes before it, so each plane's nodes are updated at
// once and the result is the reference's to the bit.
//
// The sweep is a chain of nx + ny + nz planes, so all that does not depend on the new θ is done before it by the whole
// GPU (k_heat_source): the dissipation, and the old θ and the source copied to arrays ordered by plane, where a
// plane's columns (j, k) are consecutive.  One block then takes the planes (k_heat_sweep), the new θ of the plane
// before in shared memory, and k_heat_store brings the result back.  What bounds the sweep is the latency of a plane:
// a block barrier, a shared load and the FP64 chain with a division.  When one block also computed the sources and
// read the grid's own arrays (a sector per thread and load), the heat model took 574 µs of a 683 µs step on 96×48×8
// cells; a step there takes 215 µs now.
#include <algorithm>
#include <cmath>

#include "common.cuh"

namespace tdgl {
namespace {

const int HT_THREADS = 1024, HT_BS = 256;
const size_t HT_SMEM = 200 * 1024;   // shared memory for the last two planes

struct HeatArgs {
  double *T;
  double *Q, *S;        // by plane: the old θ (then the new one) and the source, [(s − s0) mod nx][column] (one D_T)
  double *prev;         // the last two planes' new θ when they do not fit shared memory (2 × columns)
  BandPtrs G, F;
  const double *th[3], *ph[3], *f;
  int N, x1, x2, y1, y2, z1, z2;
  Dim d;
  double dt, dx2, dy2, dz2, DT, gam, eta, thb, cap, sig;
  int joule, margin;
  double Gam[TDGL_MAXB], gk[TDGL_MAXB];
  // materials (_heat_step_mat!, terms.jl:134-202): the node map, each material's Γ, γ̃, σn and D_T; uni: one D_T (the
  // in-place sweep), else R holds the field of the step before and every node is updated from it (Jacobi)
  const uint8_t *mat;
  double Gm[TDGL_MAXMAT][TDGL_MAXB], gkm[TDGL_MAXMAT][TDGL_MAXB], sigm[TDGL_MAXMAT], DTm[TDGL_MAXMAT];
  int uni;
  double *R;
  // normal fluids per band (qp_joule, exchange.jl): 1 two bands (δ in qmu[0]), 2 N fluids (μ_µ); 0 none
  int qp;
  const double *qmu[TDGL_MAXB];
  double qs[TDGL_MAXB], qsig, qGm[TDGL_MAXB][TDGL_MAXB];
};

// qp_joule (exchange.jl:391-399; N fluids :516-531): the Joule heat of the normal fluids beyond σn|E|² at node o,
// from this step's potentials; |∇·|² as the heat model takes |E|² (the mean over the two links of each axis)
__device__ double qp_joule(const HeatArgs &A, long long o, long long sx, long long sy, long long sz) {
  auto grad2 = [&](const double *m) {
    const double a0 = m[o + sx] - m[o], a1 = m[o] - m[o - sx], b0 = m[o + sy] - m[o], b1 = m[o] - m[o - sy],
                 c0 = m[o + sz] - m[o], c1 = m[o] - m[o - sz];
    return 0.5 * (a0 * a0 + a1 * a1) / A.dx2 + 0.5 * (b0 * b0 + b1 * b1) / A.dy2 + 0.5 * (c0 * c0 + c1 * c1) / A.dz2;
  };
  if (A.qp == 1) {
    const double d = A.qmu[0][o];
    return A.qsig * A.qs[0] * A.qs[1] * grad2(A.qmu[0]) + A.qGm[0][1] * (d * d);
  }
  double q = 0.0;
  for (int mu = 0; mu < A.N; mu++) q += A.qs[mu] * grad2(A.qmu[mu]);
  q *= A.qsig;
  for (int mu = 0; mu < A.N; mu++)
    for (int nu = mu + 1; nu < A.N; nu++) {
      const double e = A.qmu[mu][o] - A.qmu[nu][o];
      q += A.qGm[mu][nu] * (e * e);
    }
  return q;
}

__device__ __forceinline__ double band_heat(double Gam, double gk, cd g, cd f, double invdt2) {
  if (gk == 0) return Gam * (cabs2(csub(f, g)) * invdt2);
  const double g2 = gk * gk;
  const cd d = csub(f, g);
  const double r = cmul(cconj(g), d).x;
  return (Gam / sqrt(1 + g2 * cabs2(g))) * ((cabs2(d) + g2 * (r * r)) * invdt2);
}

// the heat released at the inner node o = (i, j, k): η((dissipation + σn|E|²) + the fluids' share), terms.jl:85-110
__device__ double heat_source(const HeatArgs &A, int i, long long o) {
  const Dim d = A.d;
  const long long sx = 1, sy = d.n1, sz = (long long)d.n1 * d.n2;
  const double invdt2 = 1 / (A.dt * A.dt);
  const double cx = invdt2 / A.dx2, cy = invdt2 / A.dy2, cz = invdt2 / A.dz2;
  const int m = A.mat ? A.mat[o] - 1 : 0;
  const bool in = A.x1 + A.margin < i && i < A.x2 + 1 - A.margin;
  double src = 0.0;
  if (in) {
    if (A.mat) {
      for (int mu = 0; mu < A.N; mu++) src += band_heat(A.Gm[m][mu], A.gkm[m][mu], A.G.p[mu][o], A.F.p[mu][o], invdt2);
    } else {
      src = band_heat(A.Gam[0], A.gk[0], A.G.p[0][o], A.F.p[0][o], invdt2);
      for (int mu = 1; mu < A.N; mu++) src += band_heat(A.Gam[mu], A.gk[mu], A.G.p[mu][o], A.F.p[mu][o], invdt2);
    }
  }
  if (!A.joule) return A.eta * src;
  const double sig = A.mat ? A.sigm[m] : A.sig;
  double e2 = 0.0, qj = 0.0;
  if (in && A.f[o] > 0) {
    if (A.qp) qj = qp_joule(A, o, sx, sy, sz);   // terms.jl:107-108
    const double a0 = A.th[0][o - sx] - A.ph[0][o - sx], a1 = A.th[0][o] - A.ph[0][o];
    const double b0 = A.th[1][o - sy] - A.ph[1][o - sy], b1 = A.th[1][o] - A.ph[1][o];
    const double c0 = A.th[2][o - sz] - A.ph[2][o - sz], c1 = A.th[2][o] - A.ph[2][o];
    const double ex = 0.5 * (a0 * a0 + a1 * a1) * cx, ey = 0.5 * (b0 * b0 + b1 * b1) * cy, ez = 0.5 * (c0 * c0 + c1 * c1) * cz;
    e2 = (ex + ey) + ez;
  }
  return A.eta * ((src + sig * e2) + qj);
}

// the update from the flux and the source (terms.jl:111-118)
__device__ __forceinline__ double heat_node(const HeatArgs &A, double q, double flux, double src) {
  const double acc = q + A.dt * (flux + src);
  double tn = (acc + A.dt * A.gam * A.thb) / (1 + A.dt * A.gam);
  if (tn < 0) tn = 0.0;
  else if (tn > A.cap) tn = A.cap;
  return tn;
}

// Every node of the block: a face takes the θ inside (copied x, then y, then z, terms.jl:70-78: each index clamped; the
// parameter check refuses a block without inner nodes); an inner node its source and old θ by plane, or, with D_T per
// material, a copy of the field (faces included) in R.
__global__ void __launch_bounds__(HT_BS) k_heat_source(const __grid_constant__ HeatArgs A) {
  const int nx1 = A.x2 + 2 - A.x1, ny1 = A.y2 + 2 - A.y1, nz1 = A.z2 + 2 - A.z1;
  const long long t = (long long)blockIdx.x * HT_BS + threadIdx.x;
  if (t >= (long long)nx1 * ny1 * nz1) return;
  const unsigned u = (unsigned)t, b = u / (unsigned)nx1, c = b / (unsigned)ny1;
  const int i = A.x1 + (int)(u - b * (unsigned)nx1), j = A.y1 + (int)(b - c * (unsigned)ny1), k = A.z1 + (int)c;
  const int ii = min(max(i, A.x1 + 1), A.x2), jj = min(max(j, A.y1 + 1), A.y2), kk = min(max(k, A.z1 + 1), A.z2);
  const long long o = A.d.at(i, j, k);
  const bool face = i != ii || j != jj || k != kk;
  const double q = A.T[A.d.at(ii, jj, kk)];   // no inner node changes here
  if (face) A.T[o] = q;
  if (!A.uni) A.R[o] = q;
  if (face) return;
  const double s = heat_source(A, i, o);
  if (!A.uni) {
    A.S[o] = s;
    return;
  }
  const int ny = A.y2 - A.y1, nz = A.z2 - A.z1;
  const long long w = (long long)(((i - A.x1 - 1) + (j - A.y1 - 1) + (k - A.z1 - 1)) % (A.x2 - A.x1)) * (ny * nz) +
                      (j - A.y1 - 1) + ny * (k - A.z1 - 1);
  A.Q[w] = q;
  A.S[w] = s;
}

// One D_T: the planes in order.  Plane s takes the slot s mod nx: a column (j, k) has its nx nodes in as many successive
// planes, so each node has its own entry and the arrays are as large as the block, whatever its shape.  Column (j, k) of
// plane s holds i = s − j − k, so the old θ of i+1, j+1 and k+1 are in plane s + 1 (columns c, c + 1, c + ny) and the new
// θ of i−1, j−1 and k−1 in plane s − 1 (c, c − 1, c − ny); beyond the block's inner nodes each is the node's own old θ
// (the face's copy).  P2: the squared spacings are powers of two, so a product by the reciprocal is the quotient's bits
// and the chain holds one division instead of two.
template <bool P2>
__global__ void __launch_bounds__(HT_THREADS) k_heat_sweep(const __grid_constant__ HeatArgs A) {
  extern __shared__ double hsh[];
  const int nx = A.x2 - A.x1, ny = A.y2 - A.y1, nz = A.z2 - A.z1, nc = ny * nz;   // inner nodes and columns
  double *buf = A.prev ? A.prev : hsh;
  const double rx = 1 / A.dx2, ry = 1 / A.dy2, rz = 1 / A.dz2;
  auto div = [](double v, double d, double r) { return P2 ? v * r : v / d; };
  const int ns = nx + ny + nz - 2;
  for (int s = 0, m = 0; s < ns; s++) {   // m = s mod nx
    const int mn = m + 1 < nx ? m + 1 : 0;
    const double *pv = buf + ((s + 1) & 1) * nc;
    double *nw = buf + (s & 1) * nc;
    for (int c = threadIdx.x; c < nc; c += blockDim.x) {
      const int k = c / ny, j = c - k * ny, i = s - j - k;
      if (i < 0 || i >= nx) continue;
      double *Qs = A.Q + (long long)m * nc + c;
      const double *Qn = A.Q + (long long)mn * nc + c;
      const double q = Qs[0];
      const double xp = i + 1 < nx ? Qn[0] : q, yp = j + 1 < ny ? Qn[1] : q, zp = k + 1 < nz ? Qn[ny] : q;
      const double src = A.S[(long long)m * nc + c];
      const double xm = i > 0 ? pv[c] : q, ym = j > 0 ? pv[c - 1] : q, zm = k > 0 ? pv[c - ny] : q;
      const double flux = A.DT * (div((xp - 2 * q) + xm, A.dx2, rx) + div((yp - 2 * q) + ym, A.dy2, ry) + div((zp - 2 * q) + zm, A.dz2, rz));
      const double tn = heat_node(A, q, flux, src);
      nw[c] = tn;
      Qs[0] = tn;
    }
    m = mn;
    __syncthreads();
  }
}

// the inner nodes' new θ from the planes (one D_T), or from the field of the step before at once (D_T per material)
__global__ void __launch_bounds__(HT_BS) k_heat_store(const __grid_constant__ HeatArgs A) {
  const int nx = A.x2 - A.x1, ny = A.y2 - A.y1, nz = A.z2 - A.z1;
  const long long t = (long long)blockIdx.x * HT_BS + threadIdx.x;
  if (t >= (long long)nx * ny * nz) return;
  const unsigned u = (unsigned)t, b = u / (unsigned)nx, k = b / (unsigned)ny;
  const int i = (int)(u - b * (unsigned)nx), j = (int)(b - k * (unsigned)ny);
  const long long o = A.d.at(A.x1 + 1 + i, A.y1 + 1 + j, A.z1 + 1 + (int)k);
  if (A.uni) {
    A.T[o] = A.Q[(long long)((i + j + (int)k) % nx) * (ny * nz) + j + ny * (int)k];
    return;
  }
  const long long sx = 1, sy = A.d.n1, sz = (long long)A.d.n1 * A.d.n2;
  const double *R = A.R;
  const double q = R[o], d0 = A.DTm[A.mat[o] - 1];
  auto dn = [&](long long on) {
    const double e = A.DTm[A.mat[on] - 1];
    return d0 == e ? d0 : 2 * d0 * e / (d0 + e);
  };
  const double flux = (dn(o + sx) * (R[o + sx] - q) + dn(o - sx) * (R[o - sx] - q)) / A.dx2 +
                      (dn(o + sy) * (R[o + sy] - q) + dn(o - sy) * (R[o - sy] - q)) / A.dy2 +
                      (dn(o + sz) * (R[o + sz] - q) + dn(o - sz) * (R[o - sz] - q)) / A.dz2;
  A.T[o] = heat_node(A, q, flux, A.S[o]);
}

__global__ void k_fill(double *a, double v, long long n) {
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
    a[t] = v;
}

}  // namespace

int heat_create(Ctx *ctx, const tdgl_materials *M) {
  const long long nn = ctx->g.d.n();
  int rc;
  if ((rc = dalloc(ctx, &ctx->Th, (size_t)nn))) return rc;
  if (M) {   // each material's values; D_T per material: a second field for the Jacobi update
    HeatMat &h = ctx->hm;
    h.nmat = M->nmat;
    bool uni = true;
    for (int m = 0; m < M->nmat; m++) {
      for (int mu = 0; mu < ctx->N; mu++) {
        h.G[m][mu] = M->gamma[m][mu];
        h.gk[m][mu] = M->gk[m][mu];
      }
      h.sig[m] = M->sigma_n[m];
      h.DT[m] = M->heat_DT[m];
      uni = uni && M->heat_DT[m] == ctx->P.heat_DT;
    }
    if (!uni && (rc = dalloc(ctx, &ctx->Th2, (size_t)nn))) return rc;
  }
  // the source (with D_T per material by node, else by plane beside the old θ), and the last two planes' θ where they do
  // not fit shared memory
  const Geo &g = ctx->g;
  const size_t nc = (size_t)(g.y2 - g.y1) * (g.z2 - g.z1);
  const size_t np = (size_t)(g.x2 - g.x1) * nc;
  if ((rc = dalloc(ctx, &ctx->heat_S, ctx->Th2 ? (size_t)nn : np))) return rc;
  if (!ctx->Th2 && (rc = dalloc(ctx, &ctx->heat_Q, np))) return rc;
  if (!ctx->Th2 && 2 * nc * sizeof(double) > HT_SMEM && (rc = dalloc(ctx, &ctx->heat_prev, 2 * nc))) return rc;
  smem_optin(k_heat_sweep<false>);
  smem_optin(k_heat_sweep<true>);
  TDGL_LAUNCH(ctx, K_HEAT, 8.0 * nn, k_fill, nblk(nn, 256), 256, 0, ctx->Th, ctx->P.heat_T, nn);
  return 0;
}

// heat_step! (terms.jl:58-130): after the bands, before the field increment (it reads θ − φ, the change of the link
// phases over the last step, which the fused supercurrent and field increment overwrites)
void heat_step(Ctx *ctx) {
  const tdgl_params &P = ctx->P;
  const Geo &g = ctx->g;
  HeatArgs A;
  A.T = ctx->Th;
  for (int mu = 0; mu < ctx->N; mu++) {
    A.G.p[mu] = ctx->G[mu];
    A.F.p[mu] = ctx->F[mu];
    A.Gam[mu] = P.heat_Gamma[mu];
    A.gk[mu] = P.heat_gk[mu];
  }
  for (int ax = 0; ax < 3; ax++) {
    A.th[ax] = ctx->th[ax];
    A.ph[ax] = ctx->ph[ax];
  }
  A.f = ctx->f;
  A.N = ctx->N;
  A.x1 = g.x1; A.x2 = g.x2; A.y1 = g.y1; A.y2 = g.y2; A.z1 = g.z1; A.z2 = g.z2;
  A.d = g.d;
  A.dt = P.dt;
  A.dx2 = g.dx * g.dx; A.dy2 = g.dy * g.dy; A.dz2 = g.dz * g.dz;
  A.DT = P.heat_DT; A.gam = P.heat_gamma_bath; A.eta = P.heat_eta; A.thb = P.heat_T; A.cap = P.heat_cap;
  A.sig = P.heat_sigma_n;
  A.joule = P.heat_joule;
  A.margin = P.heat_margin;
  A.mat = ctx->mat;
  A.uni = ctx->Th2 == nullptr;
  A.R = ctx->Th2;
  A.Q = ctx->heat_Q;
  A.S = ctx->heat_S;
  A.prev = ctx->heat_prev;
  A.qp = P.qp_on;
  qp_potentials(ctx, A.qmu);
  A.qsig = P.qp_sigma_n;
  for (int mu = 0; mu < TDGL_MAXB; mu++) {
    A.qs[mu] = P.qp_s[mu];
    for (int nu = 0; nu < TDGL_MAXB; nu++) A.qGm[mu][nu] = P.qp_Gm[mu][nu];
  }
  for (int m = 0; m < ctx->hm.nmat; m++) {
    for (int mu = 0; mu < ctx->N; mu++) {
      A.Gm[m][mu] = ctx->hm.G[m][mu];
      A.gkm[m][mu] = ctx->hm.gk[m][mu];
    }
    A.sigm[m] = ctx->hm.sig[m];
    A.DTm[m] = ctx->hm.DT[m];
  }
  const long long ni = (long long)(g.x2 - g.x1) * (g.y2 - g.y1) * (g.z2 - g.z1), nc = (long long)(g.y2 - g.y1) * (g.z2 - g.z1);
  const long long nb = (long long)(g.x2 + 2 - g.x1) * (g.y2 + 2 - g.y1) * (g.z2 + 2 - g.z1);
  TDGL_LAUNCH(ctx, K_HEAT, nb * (8.0 * 9 + 32.0 * ctx->N), k_heat_source, nblk(nb, HT_BS), HT_BS, 0, A);
  if (A.uni) {
    auto pow2 = [](double v) {
      int e;
      return std::frexp(v, &e) == 0.5 && std::isnormal(1 / v);
    };
    const int threads = (int)std::min<long long>(HT_THREADS, (nc + 31) / 32 * 32);
    const size_t smem = A.prev ? 0 : 2 * nc * sizeof(double);
    if (pow2(A.dx2) && pow2(A.dy2) && pow2(A.dz2)) TDGL_LAUNCH(ctx, K_HEAT, 32.0 * ni, k_heat_sweep<true>, 1, threads, smem, A);
    else TDGL_LAUNCH(ctx, K_HEAT, 32.0 * ni, k_heat_sweep<false>, 1, threads, smem, A);
  }
  TDGL_LAUNCH(ctx, K_HEAT, 16.0 * ni, k_heat_store, nblk(ni, HT_BS), HT_BS, 0, A);
}

int heat_carry(Ctx *ctx, double *host, bool up) {
  const size_t bytes = ctx->g.d.n() * sizeof(double);
  cudaError_t e = up ? cudaMemcpyAsync(ctx->Th, host, bytes, cudaMemcpyHostToDevice, ctx->stream)
                     : cudaMemcpyAsync(host, ctx->Th, bytes, cudaMemcpyDeviceToHost, ctx->stream);
  if (e != cudaSuccess) return set_err(ctx, TDGL_ECUDA, "heat carry copy", e);
  if ((e = cudaStreamSynchronize(ctx->stream)) != cudaSuccess) return set_err(ctx, TDGL_ECUDA, "heat carry", e);
  return 0;
}

}  // namespace tdgl
