// field.cu — the blocks of the step after the band update (gtdgl/src/field.jl).
//
//   k_current_increment  supercurrent! (:19-46) fused with field_increment! (:84-102): J on each link is computed,
//                        stored (the State carries it) and used at once for φ = θ + d1 τ J − s·Δh
//   k_scale              scale_increment! (gtdgl/src/implicit.jl:337-342)
//   k_finish             the end of the step in one launch: links! (:105-121), curl_h! (:124-137), field_bc!
//                        (:189-228) with _open_add! (gtdgl/src/openbc.jl:210-223), neumann! (:231-246) and advance!
//                        (:248-263; θ/φ and V/U swap by pointer)
#include "common.cuh"
#include "merge.cuh"

namespace tdgl {

namespace {
const int BS = 256;

struct CurArgs {
  BandPtrs G;
  const cd *V[3];
  const double *th[3], *tau[3];
  double *J[3], *ph[3];
  const double *h[3];
  double wa[3][TDGL_MAXB];
  int N;
  double d1, sxy, sxz, syx, syz, szx, szy;
  Rng r[3];
  Dim d;
  const uint8_t *mat;   // material per region: each band's link carries w_µ ρ_µ (field.jl:48-71)
  const MatDev *mt;
  const double *dnu;    // the drag matrix ν_µν [MAXB][MAXB] (null: no drag; field.jl:73-81)
};

__device__ __forceinline__ void current_increment_b(const Blk bk, CurArgs const &A);
__global__ void k_current_increment(CurArgs A) { current_increment_b(TDGL_BLK, A); }
TDGL_MERGEABLE(k_current_increment, current_increment_b, BS, 4, false);
__device__ __forceinline__ void current_increment_b(const Blk bk, CurArgs const &A) {
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
  const Dim d = A.d;
  const long long o = d.at(i, j, k);
  const long long sx = 1, sy = d.n1, sz = (long long)d.n1 * d.n2;
  const long long s = ax == 0 ? sx : ax == 1 ? sy : sz;
  const cd v = A.V[ax][o];
  double acc;
  if (A.mat) {   // ρ_µ = τ·W[µ][ax][a][b] of the link from node a to node b
    const int a = A.mat[o] - 1, b = A.mat[o + s] - 1;
    const double tv = A.tau[ax][o];
    acc = (A.wa[ax][0] * (tv * A.mt->W[0][ax][a][b])) * cmul(cmul(cconj(A.G.p[0][o]), v), A.G.p[0][o + s]).y;
    for (int mu = 1; mu < A.N; mu++)
      acc += (A.wa[ax][mu] * (tv * A.mt->W[mu][ax][a][b])) * cmul(cmul(cconj(A.G.p[mu][o]), v), A.G.p[mu][o + s]).y;
  } else {
    acc = A.wa[ax][0] * cmul(cmul(cconj(A.G.p[0][o]), v), A.G.p[0][o + s]).y;
    for (int mu = 1; mu < A.N; mu++) acc += A.wa[ax][mu] * cmul(cmul(cconj(A.G.p[mu][o]), v), A.G.p[mu][o + s]).y;
    if (A.dnu)   // _jdrag: Σ_{µ<η} ν_µη (Im(Ψµ* V Ψη[+e]) + Im(Ψη* V Ψµ[+e]))
      for (int mu = 0; mu < A.N; mu++)
        for (int eta = mu + 1; eta < A.N; eta++) {
          const double c = A.dnu[TDGL_MAXB * mu + eta];
          if (c == 0.0) continue;
          acc += c * (cmul(cmul(cconj(A.G.p[mu][o]), v), A.G.p[eta][o + s]).y +
                      cmul(cmul(cconj(A.G.p[eta][o]), v), A.G.p[mu][o + s]).y);
        }
  }
  A.J[ax][o] = acc;
  const double *hx = A.h[0], *hy = A.h[1], *hz = A.h[2];
  double p;
  if (ax == 0)
    p = ((A.th[0][o] + (A.d1 * A.tau[0][o]) * acc) - A.sxy * (hz[o] - hz[o - sy])) + A.sxz * (hy[o] - hy[o - sz]);
  else if (ax == 1)
    p = ((A.th[1][o] + (A.d1 * A.tau[1][o]) * acc) - A.syz * (hx[o] - hx[o - sz])) + A.syx * (hz[o] - hz[o - sx]);
  else
    p = ((A.th[2][o] + (A.d1 * A.tau[2][o]) * acc) - A.szx * (hy[o] - hy[o - sx])) + A.szy * (hx[o] - hx[o - sy]);
  A.ph[ax][o] = p;
}

struct ScaleArgs {
  const double *th[3], *D[3];
  double *ph[3];
  Rng r[3];
  Dim d;
};

__device__ __forceinline__ void scale_b(const Blk bk, ScaleArgs const &A);
__global__ void k_scale(ScaleArgs A) { scale_b(TDGL_BLK, A); }
TDGL_MERGEABLE(k_scale, scale_b, BS, 1, false);
__device__ __forceinline__ void scale_b(const Blk bk, ScaleArgs const &A) {
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
  A.ph[ax][o] = A.th[ax][o] + (A.ph[ax][o] - A.th[ax][o]) / A.D[ax][o];
}

// The end of the step, one item per thread over sixteen ranges (the items of one range are whole warps but for its
// ends): links U = e^{−iφ} (0..2), the curl on the inner plaquettes (3..5), the outer faces of h (6..14: per
// component the k faces, the j faces and the i faces), the block's nodes of every band (15).  No item reads what
// another writes: the faces of h are disjoint from the plaquettes of the curl, the ghosts take their links from φ
// (the same e^{−iφ}) and read nodes inside the block, which no item writes in F but to clear vacuum.  A vacuum node may
// hold Ψ ≠ 0 until the first step of an uploaded state has ended (an RKL/RKC combination keeps its share of it), so a
// ghost beside one could be formed before or after it is cleared: it does not matter where the ghost is vacuum too, as
// `sculpt` makes it; a sample with another ghost beside vacuum (vac_late) is cleared by a launch of its own afterwards.
// What bounds it on large grids: issue (63 %) and the latency of its loads (2.4 TB/s; the FP64 pipe, with a sincos per
// link, is at 10 %); on small ones it is one launch where the links with the
// curl, the faces of h, the ghosts of each band and the copy of advance! were N + 3, each waiting for the one before.
// 40 steps took 2709 µs instead of 2811 (12×8×4 cells), 3597 instead of 3782 (64×32×8), 7638 instead of 7893
// (192×64×16), 245.9 ms instead of 250.0 (the 256×128×32 ramp).  The registers are held to 40: with the
// ghosts' sincos inlined three times (110 registers) the links lost their occupancy and the 192×64×16 cycle took 8252 µs.
struct FinArgs {
  const double *ph[3];
  cd *U[3];
  double *h[3];
  double dx, dy, dz;
  Rng r[16];
  long long off[17];
  Dim d;
  // field_bc!
  const double *bar[6];     // hy_z, hy_y, hz_z, hz_y, hz_x, hy_x
  const double *oo[3], *on[3];
  const StepScal *cur;      // H, HJ and the ramp fraction of this step
  int bc, open;
  int Nx, Ny, Nz;
  // neumann! and advance!
  cd *G[TDGL_MAXB], *F[TDGL_MAXB];
  int N;
  int x1, x2, y1, y2, z1, z2;
  const uint8_t *vac;       // a sculpted sample: F = 0 on every vacuum node (range 15 is then the whole grid)
  int vac_late;             // leave F on the vacuum inside the block as it is (k_vacuum_zero follows)
};

// Shell of a box (a, b, c) split into k faces, j faces and i faces without overlap.
void shell(int a, int b, int c, Rng *r) {
  r[0] = mkrng(1, a, 1, b, 1, 1);
  if (c > 1) r[0].nk = 2;  // k = 1 and k = c: handled through a stride below
  r[1] = mkrng(1, a, 1, 1, 2, c - 1);
  if (b > 1) r[1].nj = 2;
  r[2] = mkrng(1, 1, 2, b - 1, 2, c - 1);
  if (a > 1) r[2].ni = 2;
}

}  // namespace

// k faces etc. are enumerated as index 1 and 2 of a two-element range; map 2 to the far face.
__device__ __forceinline__ int face_of(int x, int far) { return x == 2 ? far : x; }

void supercurrent_increment(Ctx *ctx) {
  const Geo &g = ctx->g;
  const tdgl_params &P = ctx->P;
  CurArgs A;
  for (int mu = 0; mu < ctx->N; mu++) A.G.p[mu] = ctx->G[mu];
  for (int ax = 0; ax < 3; ax++) {
    A.V[ax] = ctx->V[ax]; A.th[ax] = ctx->th[ax]; A.tau[ax] = ctx->tau[ax]; A.J[ax] = ctx->J[ax];
    A.ph[ax] = ctx->ph[ax]; A.h[ax] = ctx->h[ax];
    for (int mu = 0; mu < TDGL_MAXB; mu++) A.wa[ax][mu] = P.wa[ax][mu];
  }
  A.N = ctx->N;
  A.mat = ctx->mat;
  A.mt = ctx->mt;
  A.dnu = ctx->drag_nu;
  A.d1 = P.d1; A.sxy = P.sxy; A.sxz = P.sxz; A.syx = P.syx; A.syz = P.syz; A.szx = P.szx; A.szy = P.szy;
  A.r[0] = mkrng(1, g.Nx, 2, g.Ny, 2, g.Nz);
  A.r[1] = mkrng(2, g.Nx, 1, g.Ny, 2, g.Nz);
  A.r[2] = mkrng(2, g.Nx, 2, g.Ny, 1, g.Nz);
  A.d = g.d;
  long long n = A.r[0].n() + A.r[1].n() + A.r[2].n();
  // per link: V, θ, τ in, J and φ out; per node: every band once and the three h
  const double bytes = 48.0 * n + (16.0 * ctx->N + 24.0) * (double)g.d.n();
  TDGL_LAUNCH(ctx, K_CURINC, bytes, k_current_increment, nblk(n, BS), BS, 0, A);
}

void scale_increment(Ctx *ctx) {
  const Geo &g = ctx->g;
  ScaleArgs A;
  for (int ax = 0; ax < 3; ax++) {
    A.th[ax] = ctx->th[ax]; A.D[ax] = ctx->D[ax]; A.ph[ax] = ctx->ph[ax];
  }
  // every entry of the reference's link arrays (the broadcast over the whole array)
  A.r[0] = mkrng(1, g.Nx, 1, g.Ny + 1, 1, g.Nz + 1);
  A.r[1] = mkrng(1, g.Nx + 1, 1, g.Ny, 1, g.Nz + 1);
  A.r[2] = mkrng(1, g.Nx + 1, 1, g.Ny + 1, 1, g.Nz);
  A.d = g.d;
  long long n = A.r[0].n() + A.r[1].n() + A.r[2].n();
  TDGL_LAUNCH(ctx, K_SCALE, 32.0 * n, k_scale, nblk(n, BS), BS, 0, A);
}

void advance_swap(Ctx *ctx) {
  for (int ax = 0; ax < 3; ax++) {
    std::swap(ctx->th[ax], ctx->ph[ax]);
    std::swap(ctx->V[ax], ctx->U[ax]);
  }
  ctx->parity ^= 1;
}

// one face point of h: the sequence of field_bc!'s face writes (field.jl:189-228) and _open_add! (openbc.jl:210-223)
// as it ends at this point, so that the precedence of the overlapping `.=` statements needs no order of the threads
__device__ __forceinline__ void face_point(const FinArgs &A, int comp, int i, int j, int k) {
  const int Nx = A.Nx, Ny = A.Ny, Nz = A.Nz;
  const long long o = A.d.at(i, j, k);
  const double H = A.cur->H, HJ = A.cur->HJ, fr = A.cur->open_fr;
  double v = A.h[comp][o];
  if (comp == 2) {  // hz (Nx, Ny, Nz+1)
    if (k == 1 || k == Nz + 1 || i == 1 || i == Nx || j == 1 || j == Ny) v = H;
    if (A.bc != TDGL_BC_SLAB) {
      if (k == 1 || k == Nz + 1) v = H + HJ * A.bar[2][(j - 1) + (long long)Ny * (k == 1 ? 0 : 1)];
      if (j == 1 || j == Ny) v = H + HJ * A.bar[3][(j == 1 ? 0 : 1) + 2LL * (k - 1)];
      if (i == 1 || i == Nx) v = H + HJ * A.bar[4][(j - 1) + (long long)Ny * (k - 1)];
      if (A.open) {
        double oo = A.oo[2][o], nn = A.on[2][o];
        if ((j == 1 || j == Ny) && i >= 2 && i <= Nx - 1) v += oo + fr * (nn - oo);
        if (i == 1 || i == Nx) v += oo + fr * (nn - oo);
      }
    }
  } else if (comp == 0) {  // hx (Nx+1, Ny, Nz)
    if (i == 1 || i == Nx + 1 || j == 1 || j == Ny) v = 0.0;
    if (A.open && i >= 2 && i <= Nx && (j == 1 || j == Ny || k == 1 || k == Nz)) {
      double oo = A.oo[0][o], nn = A.on[0][o];
      v = oo + fr * (nn - oo);
    }
  } else {  // hy (Nx, Ny+1, Nz)
    if (j == 1 || j == Ny + 1) v = 0.0;
    if (A.bc == TDGL_BC_SLAB) {
      if (k == 1) v = -HJ;
      if (k == Nz) v = +HJ;
    } else {
      if (k == 1 || k == Nz) v = HJ * A.bar[0][(j - 1) + (long long)(Ny + 1) * (k == 1 ? 0 : 1)];
      if (j == 1 || j == Ny + 1) v = HJ * A.bar[1][(j == 1 ? 0 : 1) + 2LL * (k - 1)];
      if (i == 1 || i == Nx) v = HJ * A.bar[5][(j - 1) + (long long)(Ny + 1) * (k - 1)];
      if (A.open) {
        double oo = A.oo[1][o], nn = A.on[1][o];
        if ((k == 1 || k == Nz) && i >= 2 && i <= Nx - 1) v += oo + fr * (nn - oo);
        if (i == 1 || i == Nx) v += oo + fr * (nn - oo);
      }
    }
  }
  A.h[comp][o] = v;
}

// The three face passes of ghosts! (bands.jl:524-539) at the point o = (i, j, k) of the block's shell, every band: the
// writes that reach it in the reference's order (x faces, then y, then z).  An x-face point takes the x pass's link
// times the node inside; a y-face point the y pass over that (at the first column inside), a z-face point the z pass
// over both (at the first plane inside).  One pass at a time, through F[o], each link formed once for all bands by a
// single sincos site: the chain of up to three per band made the launch 9 µs on 12×8×4 cells (its cycle went from 2160
// to 1990 µs), and the kernel stays at 40 registers.
__device__ __forceinline__ void ghost_point(const FinArgs &A, int i, int j, int k, long long o) {
  const Dim d = A.d;
  const int ii = min(max(i, A.x1 + 1), A.x2), jj = min(max(j, A.y1 + 1), A.y2), kk = min(max(k, A.z1 + 1), A.z2);
  long long src = d.at(ii, jj, kk);   // the node inside, then the pass before
#pragma unroll 1
  for (int ax = 0; ax < 3; ax++) {
    const int at = ax == 0 ? i : ax == 1 ? j : k, lo = ax == 0 ? A.x1 : ax == 1 ? A.y1 : A.z1;
    const int hi = ax == 0 ? A.x2 : ax == 1 ? A.y2 : A.z2;
    if (at != lo && at != hi + 1) continue;
    const int e = at == lo ? lo : hi;   // the link along ax that ends on the face
    const long long q = ax == 0 ? d.at(e, jj, kk) : ax == 1 ? d.at(i, e, kk) : d.at(i, j, e);
    cd u = ccis(-A.ph[ax][q]);
    if (at != lo) u = cconj(u);
    for (int mu = 0; mu < A.N; mu++) A.F[mu][o] = cmul(u, A.F[mu][src]);
    src = o;
  }
  const bool vac = A.vac && A.vac[o];
  for (int mu = 0; mu < A.N; mu++) {
    const cd v = vac ? mkc(0.0, 0.0) : A.F[mu][o];
    if (vac) A.F[mu][o] = v;
    A.G[mu][o] = v;
  }
}

__device__ __forceinline__ void finish_b(const Blk bk, FinArgs const &A);
__global__ void __launch_bounds__(BS, 6) k_finish(const __grid_constant__ FinArgs A) { finish_b(TDGL_BLK, A); }
TDGL_MERGEABLE(k_finish, finish_b, BS, 6, false);
__device__ __forceinline__ void finish_b(const Blk bk, FinArgs const &A) {
  long long t = (long long)bk.x * blockDim.x + threadIdx.x;
  if (t >= A.off[16]) return;
  int q = 0;
  while (t >= A.off[q + 1]) q++;
  t -= A.off[q];
  int i, j, k;
  rng_ijk(A.r[q], t, i, j, k);
  const Dim d = A.d;
  if (q >= 6 && q < 15) {   // the shells list the far faces at index 2
    const int comp = (q - 6) / 3, part = (q - 6) % 3;
    const int far = part == 0 ? (comp == 2 ? A.Nz + 1 : A.Nz) : part == 1 ? (comp == 1 ? A.Ny + 1 : A.Ny)
                                                                          : (comp == 0 ? A.Nx + 1 : A.Nx);
    if (part == 0) k = face_of(k, far);
    else if (part == 1) j = face_of(j, far);
    else i = face_of(i, far);
    face_point(A, comp, i, j, k);
    return;
  }
  const long long o = d.at(i, j, k);
  const long long sx = 1, sy = d.n1, sz = (long long)d.n1 * d.n2;
  const double *px = A.ph[0], *py = A.ph[1], *pz = A.ph[2];
  if (q < 3) {
    A.U[q][o] = ccis(-A.ph[q][o]);
  } else if (q == 3) {
    A.h[0][o] = ((pz[o + sy] - pz[o]) - py[o + sz] + py[o]) / (A.dy * A.dz);
  } else if (q == 4) {
    A.h[1][o] = ((px[o + sz] - px[o]) - pz[o + sx] + pz[o]) / (A.dz * A.dx);
  } else if (q == 5) {
    A.h[2][o] = ((py[o + sx] - py[o]) - px[o + sy] + px[o]) / (A.dx * A.dy);
  } else {
    const bool block = i >= A.x1 && i <= A.x2 + 1 && j >= A.y1 && j <= A.y2 + 1 && k >= A.z1 && k <= A.z2 + 1;
    const bool shell = i == A.x1 || i == A.x2 + 1 || j == A.y1 || j == A.y2 + 1 || k == A.z1 || k == A.z2 + 1;
    if (block && shell) {
      ghost_point(A, i, j, k, o);
      return;
    }
    const bool vac = A.vac && A.vac[o];
    for (int mu = 0; mu < A.N; mu++) {
      if (vac && !A.vac_late) A.F[mu][o] = mkc(0.0, 0.0);
      if (block) A.G[mu][o] = vac ? mkc(0.0, 0.0) : A.F[mu][o];   // outside the block: with vacuum only
    }
  }
}

// links!, curl_h!, field_bc! (H, HJ and the ramp fraction from ctx->ss_cur), neumann! and advance!
void finish_step(Ctx *ctx) {
  const Geo &g = ctx->g;
  FinArgs A;
  memset(&A, 0, sizeof(A));
  for (int ax = 0; ax < 3; ax++) {
    A.ph[ax] = ctx->ph[ax]; A.U[ax] = ctx->U[ax]; A.h[ax] = ctx->h[ax];
  }
  A.dx = g.dx; A.dy = g.dy; A.dz = g.dz;
  A.r[0] = mkrng(1, g.Nx, 2, g.Ny, 2, g.Nz);
  A.r[1] = mkrng(2, g.Nx, 1, g.Ny, 2, g.Nz);
  A.r[2] = mkrng(2, g.Nx, 2, g.Ny, 1, g.Nz);
  A.r[3] = mkrng(2, g.Nx, 2, g.Ny - 1, 2, g.Nz - 1);
  A.r[4] = mkrng(2, g.Nx - 1, 2, g.Ny, 2, g.Nz - 1);
  A.r[5] = mkrng(2, g.Nx - 1, 2, g.Ny - 1, 2, g.Nz);
  const int shp[3][3] = {{g.Nx + 1, g.Ny, g.Nz}, {g.Nx, g.Ny + 1, g.Nz}, {g.Nx, g.Ny, g.Nz + 1}};
  for (int c = 0; c < 3; c++) shell(shp[c][0], shp[c][1], shp[c][2], &A.r[6 + 3 * c]);
  for (int q = 0; q < 6; q++) A.bar[q] = ctx->bar[q];
  A.cur = ctx->ss_cur;
  A.bc = ctx->P.selffield_bc;
  A.open = A.bc == TDGL_BC_OPEN;
  if (A.open) open_face_args(ctx, A.oo, A.on);
  A.Nx = g.Nx; A.Ny = g.Ny; A.Nz = g.Nz;
  for (int mu = 0; mu < ctx->N; mu++) {
    A.G[mu] = ctx->G[mu];
    A.F[mu] = ctx->F[mu];
  }
  A.N = ctx->N;
  A.x1 = g.x1; A.x2 = g.x2; A.y1 = g.y1; A.y2 = g.y2; A.z1 = g.z1; A.z2 = g.z2;
  A.vac = ctx->vac;
  A.vac_late = ctx->vac_late;
  A.r[15] = ctx->vac ? mkrng(1, g.Nx + 1, 1, g.Ny + 1, 1, g.Nz + 1) : mkrng(g.x1, g.x2 + 1, g.y1, g.y2 + 1, g.z1, g.z2 + 1);
  A.off[0] = 0;
  for (int q = 0; q < 16; q++) A.off[q + 1] = A.off[q] + A.r[q].n();
  A.d = g.d;
  const double nl = (double)A.off[3], nh = (double)(A.off[6] - A.off[3]), nf = (double)(A.off[15] - A.off[6]);
  const double bytes = 24.0 * nl + 8.0 * nh + (A.open ? 32.0 : 16.0) * nf + 32.0 * ctx->N * A.r[15].n();
  TDGL_LAUNCH(ctx, K_LINKSCURL, bytes, k_finish, nblk(A.off[16], BS), BS, 0, A);
  if (ctx->vac_late) vacuum_zero(ctx);
  advance_swap(ctx);
}

}  // namespace tdgl
