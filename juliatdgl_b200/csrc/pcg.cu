// pcg.cu — the insulating-padding field solve on the device (gtdgl/src/implicit.jl:106-446).
//
// (D + aK)Δ = φₑ − θ on the coupled links by preconditioned conjugate gradients, the separable inverse of
// (I + aK) as the preconditioner (in FP32 with pcg_f32, then with the flexible β = r·(z − z_old)/rz_old), the
// warm start and the extrapolated first guess 2xₙ − xₙ₋₁ of pcg_fast (_implicit_curl_fast! :376-446), the
// zero-source update (_pcg_zero_update! :251-271), and φ = θ + (φₑ − θ)/D on the decoupled links.
//
// Iterates, residuals and dot products are FP64; z is held in the precision the preconditioner computes it in.  Every
// vector is a plane-major node-shaped array per component (sep.cu), zero outside the ranges, so the vector kernels are
// flat loops.  A·p forms the new direction p = z + βp and the curl of p on the fly (no plaquette arrays).  Dot products
// are deterministic: a fixed grid of block partial sums reduced by one block in a fixed order.  The loop runs on the device: α, β and the convergence test (‖r‖ ≤ tol·‖b‖) are computed by
// the reduction kernels, and once the test passes every later kernel of the iteration returns at once; the host
// launches iterations in batches and reads the flag between batches only.
#include <algorithm>
#include <climits>
#include <cmath>

#define TDGL_PDL   // every kernel launched from this file begins with pdl_enter()
#include "common.cuh"
#include "pcg.cuh"

namespace tdgl {

Rng sep_range(const Geo &g, int ax);
void to_planes(Ctx *ctx, const double *const *a, const double *const *b, double *const *out);
void from_planes(Ctx *ctx, const double *const *in, const double *const *base, double *const *out);

static const int STR_BLOCKS = 1184;  // at most 8 × 148 SMs: full occupancy for the streaming kernels
static const int BATCH = 4;          // iterations between two reads of the convergence flag

struct PcgDev {
  double *P[2][3] = {}, *Q[3] = {}, *x[3] = {}, *r[3] = {}, *b[3] = {}, *xprev[3] = {}, *Dp[3] = {};
  void *z[2][3] = {};                           // z and the z before (FP32 with the FP32 preconditioner)
  uint8_t *Dc[3] = {};                          // σ_l/σ_n as codes into Dt (null: more than 256 values)
  double *Dt = nullptr;
  double *part = nullptr;                       // partial sums (two per block)
  cudaStream_t side = nullptr;                  // the x update beside the preconditioner
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
  int xblocks = 1;                              // grid of the kernels beside the preconditioner (2 per SM at most)
  double *sc = nullptr;                         // device scalars SC_*
  int *ic = nullptr;                            // device flags IC_*
  double *host_sc = nullptr;                    // pinned copies
  int *host_ic = nullptr;
  long long *stat = nullptr, *host_stat = nullptr;   // ST_* (device, pinned copy)
  long long noconv_seen = 0;                    // ST_NOCONV at the last status read
  long long tcwait_seen = 0;                    // ST_TCWAIT at the last status read
  bool warm = false, have2 = false;
  long long n;                                  // node count (per component array)
  int sblocks = STR_BLOCKS;                     // grid of the streaming kernels for this size
  int tj = 1, tk = 1, ntj = 1, ntk = 1, chunk = 1, nchunk = 1;   // A·p: tile, tiles along j and k, planes per block
};

namespace {
const int BS = 256;

struct Vec3 {
  double *p[3];
};
struct CVec3 {
  const double *p[3];
};
struct F3 {                  // FP32 copy of a vector (p[0] null: none)
  float *p[3];
};

// partial sums of a·b and a·c (c may be null) over the three component arrays
template <class T>
struct ZVec3 {
  const T *p[3];
};
template <class T>
__global__ void __launch_bounds__(256, 8) k_dot2(CVec3 a, ZVec3<T> b, ZVec3<T> c, int use_c, long long n, double *part, const int *ic, Fold F) {
  tdgl::pdl_enter();
  if (ic && ic[IC_DONE]) return;
  __shared__ double sh[32];
  double s1 = 0.0, s2 = 0.0;
  // unrolled: the loads of several entries in flight per thread (the sums keep their order)
  for (int cc = 0; cc < 3; cc++)
#pragma unroll 2
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
      const double av = a.p[cc][t];
      s1 += av * (double)b.p[cc][t];
      if (use_c) s2 += av * (double)c.p[cc][t];
    }
  double r1 = block_sum(s1, sh);
  __syncthreads();
  double r2 = block_sum(s2, sh);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = r1;
    part[gridDim.x + blockIdx.x] = r2;
  }
  __syncthreads();
  fold_last(F, part, sh);
}

// Q = D P + a curl curl P on the ranges (implicit.jl:212-235), the plaquette fields computed on the fly, with the
// partial sums of P·Q, over the box i ∈ 2..Nx, j ∈ 2..Ny, k ∈ 2..Nz.  With DIR the direction is formed here too,
// P = z + βP (the solve's first iteration, ic[IC_ITERS] = 0: P = z), from the old P into the other buffer.
//
// What bounds it: latency at 20 warps per SM (fixed-latency chains, the barrier of each plane, shared memory; its loads
// wait no more, and it moves its compulsory bytes at 2.4 TB/s).  A block takes a tile of tj × tk columns (tj ≤ 24 rows of
// the unit-stride axis; both split evenly), a column per thread, and marches over `chunk` planes i.  A thread reads its
// own column (and one element of the tile's halo) straight into registers two planes ahead, forms P, and leaves it in
// shared memory for its neighbours: three planes in turn, so that one barrier a plane suffices.  The plaquettes of plane
// i − 1 that plane i needs are the thread's own, kept in registers.  Each plane is read once per tile with a halo of one
// row and column.  The conductivities are a byte per link where they have at most 256 values (padding, materials), looked
// up in shared memory.  One thread per node reading its 36 neighbours through L1 fetched each plane several times from L2,
// and the direction was a pass of its own: 57 + 24 µs on the 256×128×32 ramp, 78 + 31 on 97 × 287 × 95 unknowns a
// component; this kernel takes 48 and 61.  320 threads: with more, the registers of two blocks per SM do not hold the
// planes ahead (352 threads: 70 µs); 24 rows: the halo of a nearly square tile is the smallest.
struct ApplyArgs {
  const double *P[3];
  const void *Z[3];
  double *Pn[3];
  const double *D[3];
  const uint8_t *Dc[3];
  const double *Dt;
  double *Q[3];
  double sxy, sxz, syx, syz, szx, szy, iyz, izx, ixy;
  int Nx, Ny, Nz, n2, n3;
  int tj, tk, ntj, ntk, chunk;
  const double *sc;
  double *part;
  const int *ic;
  int gated;
  Fold F;
};
const int AP_T = 320;
// the tile's halo, three components of one element each, must not outnumber the threads: tj + tk ≤ AP_T / 6 − 2
const int AP_TJ = 24, AP_SUM = AP_T / 6 - 2;

__host__ __device__ constexpr size_t apply_smem(int tj, int tk) {   // three planes of P; the conductivity table
  return ((size_t)9 * (tj + 2) * (tk + 2) + 256) * sizeof(double);
}

// what a thread reads of a plane ahead of its use: its own column's old P and z, and its halo element's
template <class TZ>
struct ApRaw {
  double p[3], hp;
  TZ z[3], hz;
};

template <class TZ, bool DIR>
__global__ void __launch_bounds__(AP_T, 2) k_apply(const __grid_constant__ ApplyArgs A) {
  tdgl::pdl_enter();
  if (A.gated && A.ic[IC_DONE]) return;
  __shared__ double sh[32];
  extern __shared__ __align__(16) double apsm[];
  const int Nx = A.Nx, Ny = A.Ny, Nz = A.Nz, W = A.tj + 2, E = W * (A.tk + 2), nc = A.tj * A.tk;
  double *const tab = apsm, *const ps = apsm + 256;     // P: [plane in turn][component][E]
  const int tid = threadIdx.x;
  const int bj = blockIdx.x % A.ntj, bk = (blockIdx.x / A.ntj) % A.ntk, bi = blockIdx.x / (A.ntj * A.ntk);
  const int j0 = 2 + bj * A.tj, k0 = 2 + bk * A.tk;                 // the tile's first node
  const int i0 = 2 + bi * A.chunk, i1 = min(Nx, i0 + A.chunk - 1);   // the block's planes
  const int si = A.n2 * A.n3;                                        // (the context's node counts fit 32 bits)
  const bool coded = A.Dc[0] != nullptr;
  if (coded)
    for (int t = tid; t < 256; t += AP_T) tab[t] = A.Dt[t];
  const bool first = DIR && A.ic[IC_ITERS] == 0;
  const double beta = DIR && !first ? A.sc[SC_BETA] : 0.0;
  // this thread's column, and its halo element (a row of W below and above the tile, then the two columns beside it)
  const int jj = 1 + tid % A.tj, kk = 1 + tid / A.tj, j = j0 - 1 + jj, k = k0 - 1 + kk;
  const bool in = tid < nc && j <= A.n2 && k <= A.n3, act = tid < nc && j <= Ny && k <= Nz;
  const int e0 = jj + W * kk, oc = (j - 1) + A.n2 * (k - 1);
  const int H = E - nc, hc = tid / H, h = tid - hc * H;
  const int hj = h < 2 * W ? h % W : (h - 2 * W) / A.tk * (A.tj + 1);
  const int hk = h < 2 * W ? h / W * (A.tk + 1) : 1 + (h - 2 * W) % A.tk;
  const bool ring = hc < 3, hin = ring && j0 - 1 + hj <= A.n2 && k0 - 1 + hk <= A.n3;
  const int he = hj + W * hk, ho = (j0 + hj - 2) + A.n2 * (k0 + hk - 2);
  const double *const hP = A.P[ring ? hc : 0];
  const TZ *const hZ = (const TZ *)A.Z[ring ? hc : 0];
  auto load = [&](ApRaw<TZ> &R, int i) {
    if (i > i1 + 1) return;
    const int pl = si * (i - 1);
#pragma unroll
    for (int c = 0; c < 3; c++) {
      R.p[c] = in ? A.P[c][pl + oc] : 0.0;
      if (DIR) R.z[c] = in ? ((const TZ *)A.Z[c])[pl + oc] : TZ(0);
    }
    R.hp = hin ? hP[pl + ho] : 0.0;
    if (DIR) R.hz = hin ? hZ[pl + ho] : TZ(0);
  };
  auto dir = [&](double p, TZ z) { return !DIR ? p : first ? (double)z : (double)z + beta * p; };
  // plane i from its raw values: P into v, shared memory and (the block's own planes) memory
  auto enter = [&](const ApRaw<TZ> &R, int i, double *slot, double (&v)[3]) {
#pragma unroll
    for (int c = 0; c < 3; c++) v[c] = dir(R.p[c], R.z[c]);
    if (tid < nc) {
#pragma unroll
      for (int c = 0; c < 3; c++) slot[c * E + e0] = v[c];
    }
    if (ring) slot[hc * E + he] = dir(R.hp, R.hz);
    if (DIR && act && i >= i0 && i <= i1) {
      const int o = si * (i - 1) + oc;
#pragma unroll
      for (int c = 0; c < 3; c++) A.Pn[c][o] = v[c];
    }
  };
  unsigned cd[3] = {0, 0, 0};
  double Dv[3] = {0.0, 0.0, 0.0};
  auto conduct = [&](int i) {   // the conductivities of plane i, a plane ahead
    if (!act || i < i0 || i > i1) return;
    const int o = si * (i - 1) + oc;
#pragma unroll
    for (int c = 0; c < 3; c++) {
      if (coded) cd[c] = A.Dc[c][o];
      else Dv[c] = A.D[c][o];
    }
  };
  const bool ky = k <= Nz - 1, jy = j <= Ny - 1;   // plaquettes beside this node exist
  const bool kp = k >= 3, jp = j >= 3;             // and before it
  double hyp = 0.0, hzp = 0.0, sx = 0.0, sy = 0.0, sz = 0.0;
  double v0[3], v1[3];
  double *s0 = ps, *s1 = ps + 3 * E, *s2 = ps + 6 * E;
  ApRaw<TZ> R0, R1;
  load(R0, i0 - 1);
  load(R1, i0);
  enter(R0, i0 - 1, s0, v0);
  load(R0, i0 + 1);
  auto step = [&](int i, ApRaw<TZ> &R) {   // plane i, plane i + 1 in R
    enter(R, i + 1, s1, v1);
    load(R, i + 3);
    double d[3];
#pragma unroll
    for (int c = 0; c < 3; c++) d[c] = coded ? 0.0 : Dv[c];
    unsigned dc[3] = {cd[0], cd[1], cd[2]};
    conduct(i + 1);
    __syncthreads();   // plane i + 1 is there for all; the slot written next was last read before this barrier
    if (act) {
      if (coded) {
#pragma unroll
        for (int c = 0; c < 3; c++) d[c] = tab[dc[c]];
      }
      const double *px = s0 + e0, *py = px + E, *pz = py + E, *qy = s1 + E + e0, *qz = qy + E;
      const double x0 = v0[0], y0 = v0[1], z0 = v0[2];
      // the plaquette areas as reciprocals: nine FP64 divisions per node were half of this kernel's instructions (the
      // operator differs from the reference's division by at most an ulp per plaquette field)
      double hy0 = 0.0, hz0 = 0.0;
      if (i >= 2 && i <= Nx - 1) {
        if (ky) hy0 = ((px[W] - x0) - v1[2] + z0) * A.izx;
        if (jy) hz0 = ((v1[1] - y0) - px[1] + x0) * A.ixy;
      }
      if (i >= i0) {
        const int o = si * (i - 1) + oc;
        if (i <= Nx - 1) {
          const double pm = px[-1], pw = px[-W];
          const double hzm = jp ? ((qy[-1] - py[-1]) - x0 + pm) * A.ixy : 0.0;
          const double hym = kp ? ((x0 - pw) - qz[-W] + pz[-W]) * A.izx : 0.0;
          const double q = d[0] * x0 + A.sxy * (hz0 - hzm) - A.sxz * (hy0 - hym);
          A.Q[0][o] = q;
          sx += x0 * q;
        }
        const double hx0 = ky && jy ? ((pz[1] - z0) - py[W] + y0) * A.iyz : 0.0;
        if (jy) {
          const double hxm = kp ? ((pz[1 - W] - pz[-W]) - y0 + py[-W]) * A.iyz : 0.0;
          const double q = d[1] * y0 + A.syz * (hx0 - hxm) - A.syx * (hz0 - hzp);
          A.Q[1][o] = q;
          sy += y0 * q;
        }
        if (ky) {
          const double hxm = jp ? ((z0 - pz[-1]) - py[W - 1] + py[-1]) * A.iyz : 0.0;
          const double q = d[2] * z0 + A.szx * (hy0 - hyp) - A.szy * (hx0 - hxm);
          A.Q[2][o] = q;
          sz += z0 * q;
        }
      }
      hyp = hy0;
      hzp = hz0;
    }
#pragma unroll
    for (int c = 0; c < 3; c++) v0[c] = v1[c];
    double *s = s0;
    s0 = s1;
    s1 = s2;
    s2 = s;
  };
  for (int i = i0 - 1; i <= i1; i += 2) {
    step(i, R1);
    if (i + 1 <= i1) step(i + 1, R0);
  }
  const double r = block_sum((sx + sy) + sz, sh);
  if (tid == 0) {
    A.part[blockIdx.x] = r;
    A.part[gridDim.x + blockIdx.x] = 0.0;
  }
  __syncthreads();
  fold_last(A.F, A.part, sh);
}

// The distinct values of the conductivities as a table of at most 256, and each entry's place in it: an open-addressed
// set of bit patterns (a value takes its hash's slot or a later one).  The first pass (no codes) fills the set and stops
// once a value found no place (*bad): with more values than places every further link would walk the whole set for
// nothing.  The second, when all have one, writes the codes.
const unsigned long long DT_FREE = 0xfff8dead0000beefULL;   // no value a conductivity has (a NaN with this payload)
__global__ void k_dtab_clear(unsigned long long *tab, int *bad) {
  tdgl::pdl_enter();
  tab[threadIdx.x] = DT_FREE;
  if (threadIdx.x == 0) *bad = 0;
}
__global__ void k_dtab(CVec3 D, long long n, unsigned long long *tab, uint8_t *c0, uint8_t *c1, uint8_t *c2, int *bad) {
  tdgl::pdl_enter();
  uint8_t *code[3] = {c0, c1, c2};
  for (int c = 0; c < 3 && !*(volatile int *)bad; c++)
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
      const unsigned long long v = (unsigned long long)__double_as_longlong(D.p[c][t]);
      unsigned h = (unsigned)((v ^ (v >> 29) ^ (v >> 47)) * 0x9e3779b1u) >> 24;
      int left = 256;
      for (; left > 0; left--, h = (h + 1) & 255) {
        unsigned long long w = *(volatile unsigned long long *)(tab + h);
        if (w == DT_FREE) w = atomicCAS(tab + h, DT_FREE, v);
        if (w == DT_FREE || w == v) break;
      }
      if (left == 0 || v == DT_FREE) {
        *(volatile int *)bad = 1;
        return;
      }
      if (c0) code[c][t] = (uint8_t)h;
      else if (*(volatile int *)bad) return;
    }
}

// r = b − Q (and its FP32 copy when given), partial r·r
__global__ void __launch_bounds__(256, 8) k_residual(Vec3 r, CVec3 b, CVec3 Q, long long n, double *part, F3 r32, Fold F) {
  tdgl::pdl_enter();
  __shared__ double sh[32];
  double s = 0.0;
  for (int c = 0; c < 3; c++)
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
      const double v = b.p[c][t] - Q.p[c][t];
      r.p[c][t] = v;
      if (r32.p[0]) r32.p[c][t] = (float)v;
      s += v * v;
    }
  const double rr = block_sum(s, sh);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = rr;
    part[gridDim.x + blockIdx.x] = 0.0;
  }
  __syncthreads();
  fold_last(F, part, sh);
}

// r −= αQ (and r's FP32 copy when given), partial r·r; the convergence test folded in (x: k_update_x)
__global__ void __launch_bounds__(256, 8) k_update(Vec3 r, CVec3 Q, long long n, const double *sc, double *part, const int *ic,
                         F3 r32, Fold F) {
  tdgl::pdl_enter();
  if (ic[IC_DONE]) return;
  __shared__ double sh[32];
  const double alpha = sc[SC_ALPHA];
  double s = 0.0;
  for (int c = 0; c < 3; c++)
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
      const double v = r.p[c][t] - alpha * Q.p[c][t];
      r.p[c][t] = v;
      if (r32.p[0]) r32.p[c][t] = (float)v;
      s += v * v;
    }
  const double rr = block_sum(s, sh);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = rr;
    part[gridDim.x + blockIdx.x] = 0.0;
  }
  __syncthreads();
  fold_last(F, part, sh);
}

// x += αP once per iteration that ran A·p (IC_ITERS counts those; IC_XDONE is where the x updates stand), so also
// in the iteration whose r update met the tolerance and set IC_DONE.  It may run beside the preconditioner (on
// another stream): nothing there changes IC_ITERS, α, P or x.  Four entries per thread in flight.
__global__ void __launch_bounds__(256) k_update_x(Vec3 x, CVec3 P, long long n, const double *sc, int *ic) {
  tdgl::pdl_enter();
  __shared__ int run, last;
  const int it = ic[IC_ITERS];
  if (threadIdx.x == 0) run = ic[IC_XDONE] != it;
  __syncthreads();
  if (!run) return;
  const double alpha = sc[SC_ALPHA];
  const long long S = (long long)gridDim.x * blockDim.x;
  for (int c = 0; c < 3; c++) {
    double *__restrict__ xp = x.p[c];
    const double *__restrict__ pp = P.p[c];
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    for (; t + 3 * S < n; t += 4 * S) {
      double xv[4], pv[4];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        xv[u] = xp[t + u * S];
        pv[u] = pp[t + u * S];
      }
#pragma unroll
      for (int u = 0; u < 4; u++) xp[t + u * S] = xv[u] + alpha * pv[u];
    }
    for (; t < n; t += S) xp[t] += alpha * pp[t];
  }
  if (threadIdx.x == 0) {   // the last block to finish records the update (every block has read IC_XDONE by then)
    __threadfence();
    last = atomicAdd(&ic[IC_XCNT], 1) == (int)gridDim.x - 1;
  }
  __syncthreads();
  if (last && threadIdx.x == 0) {
    ic[IC_XDONE] = it;
    ic[IC_XCNT] = 0;
  }
}

// x ← 2x − xprev, xprev ← x (pcg_fast's extrapolated guess, implicit.jl:394-398)
__global__ void __launch_bounds__(256, 8) k_extrap(Vec3 x, Vec3 xp, long long n) {
  tdgl::pdl_enter();
  for (int c = 0; c < 3; c++)   // per component (no 64-bit division of the flat index)
    for (long long u = (long long)blockIdx.x * blockDim.x + threadIdx.x; u < n; u += (long long)gridDim.x * blockDim.x) {
      const double v = x.p[c][u];
      x.p[c][u] = 2 * v - xp.p[c][u];
      xp.p[c][u] = v;
    }
}

// The first guess of a settled solve, decided on the device (implicit.jl:381-398 and _pcg_zero_update! :251-271):
// with ‖b‖ = 0 the solution is x = 0 (the extrapolation keeps xₙ as xₙ₋₁) and the solve is done; otherwise, with
// the extrapolated guess, x ← 2xₙ − xₙ₋₁ and xₙ₋₁ ← xₙ.
__global__ void __launch_bounds__(256, 8) k_guess(Vec3 x, Vec3 xp, long long n, const double *sc, int *ic, int extrap) {
  tdgl::pdl_enter();
  const bool zero = sc[SC_BB] == 0.0;
  if (zero && blockIdx.x == 0 && threadIdx.x == 0) ic[IC_DONE] = 1;
  if (!zero && !extrap) return;
  for (int c = 0; c < 3; c++)   // per component (no 64-bit division of the flat index)
    for (long long u = (long long)blockIdx.x * blockDim.x + threadIdx.x; u < n; u += (long long)gridDim.x * blockDim.x) {
      const double v = x.p[c][u];
      const double w = zero ? 0.0 : 2 * v - xp.p[c][u];   // xₙ₋₁ read before it becomes xₙ
      if (extrap) xp.p[c][u] = v;
      x.p[c][u] = w;
    }
}

// the loop's condition in a captured step: go on while the solve is not done and maxit is not reached
__global__ void k_loop_enter(cudaGraphConditionalHandle h, const int *ic, int maxit) {
  tdgl::pdl_enter();
  if (threadIdx.x == 0) cudaGraphSetConditional(h, (!ic[IC_DONE] && ic[IC_LAUNCHED] < maxit) ? 1u : 0u);
}
__global__ void k_loop_turn(cudaGraphConditionalHandle h, int *ic, long long *stat, int batch, int maxit) {
  tdgl::pdl_enter();
  if (threadIdx.x == 0) {
    ic[IC_LAUNCHED] += batch;
    stat[ST_TURNS] += 1;
    cudaGraphSetConditional(h, (!ic[IC_DONE] && ic[IC_LAUNCHED] < maxit) ? 1u : 0u);
  }
}

// the statistics of one solve (done: the zero-source update, which has no iterations)
__global__ void k_finish(const int *ic, long long *stat, int done) {
  tdgl::pdl_enter();
  if (threadIdx.x == 0) {
    const int it = ic[IC_ITERS];
    stat[ST_TOTAL] += it;
    stat[ST_LAST] = it;
    if (!done && !ic[IC_DONE]) stat[ST_NOCONV] += 1;
  }
}

CVec3 cv(double *const *p) {
  CVec3 v;
  for (int c = 0; c < 3; c++) v.p[c] = p[c];
  return v;
}
Vec3 vv(double *const *p) {
  Vec3 v;
  for (int c = 0; c < 3; c++) v.p[c] = p[c];
  return v;
}

// z is FP32 with the FP32 preconditioner of the fast PCG
bool zfloat(Ctx *ctx) { return ctx->P.pcg_f32 != 0; }

Fold fold(Ctx *ctx, int mode, int flexible = 0) {
  Fold F;
  F.mode = mode;
  F.flexible = flexible;
  F.tol = ctx->P.pcg_tol;
  F.sc = ctx->pcg->sc;
  F.ic = ctx->pcg->ic;
  return F;
}
// a·b (and a·c) folded into the scalars of `mode`
template <class T>
ZVec3<T> zv(const void *const *p) {
  ZVec3<T> v;
  for (int c = 0; c < 3; c++) v.p[c] = p ? (const T *)p[c] : nullptr;
  return v;
}
template <class T>
void dot2(Ctx *ctx, double *const *a, const void *const *b, const void *const *c, bool gated, int mode, int flexible = 0) {
  PcgDev *S = ctx->pcg;
  TDGL_LAUNCH(ctx, K_PCG_DOT, (8.0 + (c ? 2 : 1) * sizeof(T)) * 3 * S->n, k_dot2<T>, S->sblocks, BS, 0, cv(a), zv<T>(b),
              zv<T>(c ? c : b), c ? 1 : 0, S->n, S->part, gated ? S->ic : nullptr, fold(ctx, mode, flexible));
}
// r·z (and r·z_old) in z's precision
void dot_z(Ctx *ctx, const void *const *z, const void *const *zold, int mode, int flexible, bool gated) {
  PcgDev *S = ctx->pcg;
  if (zfloat(ctx)) dot2<float>(ctx, S->r, z, zold, gated, mode, flexible);
  else dot2<double>(ctx, S->r, z, zold, gated, mode, flexible);
}
void read_back(Ctx *ctx) {
  PcgDev *S = ctx->pcg;
  cudaMemcpyAsync(S->host_sc, S->sc, SC_N * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream);
  cudaMemcpyAsync(S->host_ic, S->ic, IC_N * sizeof(int), cudaMemcpyDeviceToHost, ctx->stream);
  cudaStreamSynchronize(ctx->stream);
}

// Q = A P, folded into the scalars of `mode`; with z also P = z + βP from the buffer pold into pnew first
void apply_A(Ctx *ctx, double *const *P, const void *const *z, double *const *pnew, bool gated, int mode) {
  PcgDev *S = ctx->pcg;
  const Geo &g = ctx->g;
  const tdgl_params &Pp = ctx->P;
  ApplyArgs A;
  memset(&A, 0, sizeof(A));
  for (int c = 0; c < 3; c++) {
    A.P[c] = P[c];
    A.Z[c] = z ? z[c] : nullptr;
    A.Pn[c] = pnew ? pnew[c] : nullptr;
    A.D[c] = S->Dp[c];
    A.Dc[c] = S->Dc[c];
    A.Q[c] = S->Q[c];
  }
  A.Dt = S->Dt;
  A.sxy = Pp.sxy; A.sxz = Pp.sxz; A.syx = Pp.syx; A.syz = Pp.syz; A.szx = Pp.szx; A.szy = Pp.szy;
  A.iyz = 1.0 / (g.dy * g.dz); A.izx = 1.0 / (g.dz * g.dx); A.ixy = 1.0 / (g.dx * g.dy);
  A.Nx = g.Nx; A.Ny = g.Ny; A.Nz = g.Nz; A.n2 = g.Ny + 1; A.n3 = g.Nz + 1;
  A.tj = S->tj; A.tk = S->tk; A.ntj = S->ntj; A.ntk = S->ntk; A.chunk = S->chunk;
  A.sc = S->sc;
  A.part = S->part;
  A.ic = S->ic;
  A.gated = gated;
  A.F = fold(ctx, mode);
  const double nbox = (double)(g.Nx - 1) * (g.Ny - 1) * (g.Nz - 1), zb = zfloat(ctx) ? 4 : 8;
  const double bytes = 3 * nbox * (8 + 8 + (S->Dc[0] ? 1 : 8) + (z ? 8 + zb : 0));
  const int grid = S->ntj * S->ntk * S->nchunk;
  if (!z) TDGL_LAUNCH(ctx, K_PCG_Q, bytes, (k_apply<float, false>), grid, AP_T, apply_smem(S->tj, S->tk), A);
  else if (zfloat(ctx)) TDGL_LAUNCH(ctx, K_PCG_Q, bytes, (k_apply<float, true>), grid, AP_T, apply_smem(S->tj, S->tk), A);
  else TDGL_LAUNCH(ctx, K_PCG_Q, bytes, (k_apply<double, true>), grid, AP_T, apply_smem(S->tj, S->tk), A);
}

int copy3(Ctx *ctx, double *const *dst, double *const *src) {
  for (int c = 0; c < 3; c++)
    TDGL_CUDA(cudaMemcpyAsync(dst[c], src[c], ctx->pcg->n * sizeof(double), cudaMemcpyDeviceToDevice, ctx->stream));
  return 0;
}

}  // namespace

int pcg_create(Ctx *ctx) {
  const Geo &g = ctx->g;
  PcgDev *S = new PcgDev();
  ctx->pcg = S;
  S->n = g.d.n();
  if (S->n > INT_MAX / 2) return set_err(ctx, TDGL_EINVAL, "grid too large for the PCG solve (32-bit node indices)");
  // a small grid takes fewer blocks (at least 4 entries per thread): the full grid's fixed cost of 1184 blocks and
  // their partial sums would dominate its microsecond kernels and crowd out concurrent contexts
  const long long per = (long long)BS * 4;
  S->sblocks = (int)std::min<long long>(STR_BLOCKS, std::max<long long>(1, (3 * S->n + per - 1) / per));
  int rc;
  double **vecs[8] = {S->P[0], S->P[1], S->Q, S->x, S->r, S->b, S->xprev, S->Dp};
  for (int q = 0; q < 8; q++)
    for (int c = 0; c < 3; c++)
      if ((rc = dalloc(ctx, &vecs[q][c], S->n))) return rc;
  const size_t zn = ((size_t)S->n * (zfloat(ctx) ? 4 : 8) + 7) / 8;
  for (int q = 0; q < 2; q++)
    for (int c = 0; c < 3; c++)
      if ((rc = dalloc(ctx, (double **)&S->z[q][c], zn))) return rc;
  int dev = 0, nsm = 148;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    nsm = 148;
  // A·p: tiles of at most AP_TJ rows and AP_T columns, split evenly; as many planes per block as leave one wave of two
  // blocks per SM (a block also reads the plane before and after its own)
  const int nj = g.Ny - 1, nk = g.Nz - 1, ni = g.Nx - 1;
  S->ntj = (nj + AP_TJ - 1) / AP_TJ;
  S->tj = (nj + S->ntj - 1) / S->ntj;
  const int tkm = std::max(1, std::min(AP_SUM - S->tj, AP_T / S->tj));
  S->ntk = (nk + tkm - 1) / tkm;
  S->tk = (nk + S->ntk - 1) / S->ntk;
  const int tiles = S->ntj * S->ntk, cols = std::max(1, 2 * nsm / tiles);
  S->chunk = std::max(1, (ni + cols - 1) / cols);
  S->nchunk = (ni + S->chunk - 1) / S->chunk;
  smem_optin(k_apply<float, false>);
  smem_optin(k_apply<float, true>);
  smem_optin(k_apply<double, true>);
  if ((rc = dalloc(ctx, &S->part, 2 * (size_t)std::max(STR_BLOCKS, tiles * S->nchunk)))) return rc;
  // two blocks per SM at most: they fit beside a preconditioner transform block on every SM
  S->xblocks = std::min(S->sblocks, 2 * nsm);
  TDGL_CUDA(cudaStreamCreateWithFlags(&S->side, cudaStreamNonBlocking));
  TDGL_CUDA(cudaEventCreateWithFlags(&S->ev_fork, cudaEventDisableTiming));
  TDGL_CUDA(cudaEventCreateWithFlags(&S->ev_join, cudaEventDisableTiming));
  if ((rc = dalloc(ctx, &S->sc, SC_N))) return rc;
  if ((rc = dalloc(ctx, &S->ic, IC_N))) return rc;
  if ((rc = dalloc(ctx, &S->stat, ST_N))) return rc;
  if (cudaMallocHost(&S->host_sc, SC_N * sizeof(double)) != cudaSuccess) return set_err(ctx, TDGL_ENOMEM, "cudaMallocHost");
  if (cudaMallocHost(&S->host_ic, IC_N * sizeof(int)) != cudaSuccess) return set_err(ctx, TDGL_ENOMEM, "cudaMallocHost");
  if (cudaMallocHost(&S->host_stat, ST_N * sizeof(long long)) != cudaSuccess) return set_err(ctx, TDGL_ENOMEM, "cudaMallocHost");
  // σ_l/σ_n on the ranges, plane-major, for A·p
  const double *D[3] = {ctx->D[0], ctx->D[1], ctx->D[2]};
  to_planes(ctx, D, nullptr, S->Dp);
  // as byte codes where they have at most 256 values
  if ((rc = dalloc(ctx, &S->Dt, 256))) return rc;
  CVec3 dv = cv(S->Dp);
  k_dtab_clear<<<1, 256, 0, ctx->stream>>>((unsigned long long *)S->Dt, S->ic);
  k_dtab<<<S->sblocks, BS, 0, ctx->stream>>>(dv, S->n, (unsigned long long *)S->Dt, nullptr, nullptr, nullptr, S->ic);
  int bad = 0;
  TDGL_CUDA(cudaMemcpyAsync(&bad, S->ic, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  TDGL_CUDA(cudaStreamSynchronize(ctx->stream));
  if (bad) return 0;
  uint8_t *code[3];
  for (int c = 0; c < 3; c++)
    if ((rc = dalloc(ctx, &code[c], S->n))) return rc;
  k_dtab<<<S->sblocks, BS, 0, ctx->stream>>>(dv, S->n, (unsigned long long *)S->Dt, code[0], code[1], code[2], S->ic);
  for (int c = 0; c < 3; c++) S->Dc[c] = code[c];
  TDGL_CUDA(cudaGetLastError());
  return 0;
}

void pcg_destroy(Ctx *ctx) {
  if (ctx->pcg) {
    if (ctx->pcg->host_sc) cudaFreeHost(ctx->pcg->host_sc);
    if (ctx->pcg->host_ic) cudaFreeHost(ctx->pcg->host_ic);
    if (ctx->pcg->host_stat) cudaFreeHost(ctx->pcg->host_stat);
    if (ctx->pcg->side) cudaStreamDestroy(ctx->pcg->side);
    if (ctx->pcg->ev_fork) cudaEventDestroy(ctx->pcg->ev_fork);
    if (ctx->pcg->ev_join) cudaEventDestroy(ctx->pcg->ev_join);
    delete ctx->pcg;
    ctx->pcg = nullptr;
  }
}

static void read_stat(Ctx *ctx) {
  PcgDev *S = ctx->pcg;
  cudaMemcpyAsync(S->host_stat, S->stat, ST_N * sizeof(long long), cudaMemcpyDeviceToHost, ctx->stream);
  cudaStreamSynchronize(ctx->stream);
}

int pcg_iters(Ctx *ctx, long long *total) {
  if (!ctx->pcg) {
    if (total) *total = 0;
    return 0;
  }
  read_stat(ctx);
  if (total) *total = ctx->pcg->host_stat[ST_TOTAL];
  return (int)ctx->pcg->host_stat[ST_LAST];
}

int pcg_take_status(Ctx *ctx) {
  if (!ctx->pcg) return 0;
  read_stat(ctx);
  PcgDev *S = ctx->pcg;
  const long long nc = S->host_stat[ST_NOCONV], tw = S->host_stat[ST_TCWAIT];
  const bool any = nc > S->noconv_seen, tc = tw > S->tcwait_seen;
  S->noconv_seen = nc;
  S->tcwait_seen = tw;
  if (tc) return set_err(ctx, TDGL_ECUDA, "preconditioner transform: a wait on the tensor cores ran out");
  return any ? TDGL_ENOCONV : 0;
}

long long *pcg_stat_tc(Ctx *ctx) { return ctx->pcg ? ctx->pcg->stat + ST_TCWAIT : nullptr; }

void pcg_regions(Ctx *ctx, Regions &r) {
  PcgDev *S = ctx->pcg;
  for (int c = 0; c < 3; c++) {
    r.push_back({S->x[c], S->n * sizeof(double)});
    r.push_back({S->xprev[c], S->n * sizeof(double)});
  }
}

void pcg_flags(Ctx *ctx, int *warm, int *have2, bool set) {
  PcgDev *S = ctx->pcg;
  if (set) {
    S->warm = *warm != 0;
    S->have2 = *have2 != 0;
  } else {
    *warm = S->warm;
    *have2 = S->have2;
  }
}

bool pcg_steady(Ctx *ctx) {
  PcgDev *S = ctx->pcg;
  const bool ext = (ctx->P.pcg_fast || ctx->P.pcg_f32) && ctx->P.pcg_extrap;
  return S->warm && (!ext || S->have2);
}

// The buffers of an iteration: z and the z before, p and the p before; each pair alternates.
struct Bufs {
  const void *z[2][3];
  double *p[2][3];
  void swap(int which) {
    for (int c = 0; c < 3; c++) {
      if (which == 0) std::swap(z[0][c], z[1][c]);
      else std::swap(p[0][c], p[1][c]);
    }
  }
};

// One PCG iteration (implicit.jl:416-437 with the flexible β of :299-305): p = z + βp, q = Ap, α; x, r; z = M⁻¹r; β.
// Every kernel returns at once after the convergence flag is set.  In: z[0] is M⁻¹r, p[0] the old direction; out the
// same for the next one.
static void iteration(Ctx *ctx, Bufs &B, bool flex, F3 r32, bool r32_ready, double wb32) {
  PcgDev *S = ctx->pcg;
  apply_A(ctx, B.p[0], B.z[0], B.p[1], true, 3);
  B.swap(1);
  TDGL_LAUNCH(ctx, K_PCG_UPD, (24.0 + wb32) * 3 * S->n, k_update, S->sblocks, BS, 0, vv(S->r), cv(S->Q), S->n, S->sc,
              S->part, S->ic, r32, fold(ctx, 5));
  // x += αP needs nothing the preconditioner computes: it runs on a second stream beside its compute-bound transforms
  // (one parallel branch of a captured loop), joined before β.  When the launches are timed one by one, the same
  // kernels run in the same order on the one stream.
  const bool side = ctx->branches && !ctx->prof.on;
  cudaStream_t main = ctx->stream;
  if (side) {
    cudaEventRecord(S->ev_fork, main);
    cudaStreamWaitEvent(S->side, S->ev_fork, 0);
    ctx->stream = S->side;
  }
  TDGL_LAUNCH(ctx, K_PCG_XUPD, 24.0 * 3 * S->n, k_update_x, S->xblocks, BS, 0, vv(S->x), cv(B.p[0]), S->n, S->sc, S->ic);
  if (side) {
    ctx->stream = main;
    cudaEventRecord(S->ev_join, S->side);
  }
  B.swap(0);   // the new z takes the older buffer
  sep_apply(ctx, S->r, (void *const *)B.z[0], zfloat(ctx), S->ic, r32_ready);
  if (side) cudaStreamWaitEvent(main, S->ev_join, 0);
  dot_z(ctx, B.z[0], flex ? B.z[1] : nullptr, 4, flex, true);
}

static Bufs bufs(PcgDev *S) {
  Bufs B;
  for (int q = 0; q < 2; q++)
    for (int c = 0; c < 3; c++) {
      B.z[q][c] = S->z[q][c];
      B.p[q][c] = S->P[q][c];
    }
  return B;
}

// The loop of a captured step: a conditional WHILE node whose body is BATCH iterations and the kernel that updates
// the condition (the device decides when the solve is done, as the host did between batches).
static int loop_graph(Ctx *ctx, Bufs &B, bool flex, F3 r32, bool r32_ready, double wb32) {
  PcgDev *S = ctx->pcg;
  const int maxit = ctx->P.pcg_maxit;
  cudaStreamCaptureStatus cs;
  cudaGraph_t cg;
  const cudaGraphNode_t *deps;
  size_t nd;
  cudaGraphConditionalHandle h;
  TDGL_CUDA(cudaStreamGetCaptureInfo(ctx->stream, &cs, nullptr, &cg, &deps, &nd));
  TDGL_CUDA(cudaGraphConditionalHandleCreate(&h, cg, 0, cudaGraphCondAssignDefault));
  TDGL_LAUNCH(ctx, K_PCG_FINAL, 0.0, k_loop_enter, 1, 32, 0, h, S->ic, maxit);
  TDGL_CUDA(cudaStreamGetCaptureInfo(ctx->stream, &cs, nullptr, &cg, &deps, &nd));
  cudaGraphNodeParams np = {cudaGraphNodeTypeConditional};   // aggregate initialisation: the rest zero
  np.conditional.handle = h;
  np.conditional.type = cudaGraphCondTypeWhile;
  np.conditional.size = 1;
  cudaGraphNode_t node;
  TDGL_CUDA(cudaGraphAddNode(&node, cg, deps, nd, &np));
  cudaGraph_t body = np.conditional.phGraph_out[0];
  TDGL_CUDA(cudaStreamUpdateCaptureDependencies(ctx->stream, &node, 1, cudaStreamSetCaptureDependencies));
  cudaStream_t main = ctx->stream;
  ctx->stream = ctx->cap_stream;
  cudaError_t e = cudaStreamBeginCaptureToGraph(ctx->stream, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal);
  if (e == cudaSuccess) {
    for (int q = 0; q < BATCH; q++) iteration(ctx, B, flex, r32, r32_ready, wb32);
    TDGL_LAUNCH(ctx, K_PCG_FINAL, 0.0, k_loop_turn, 1, 32, 0, h, S->ic, S->stat, BATCH, maxit);
    cudaGraph_t out = nullptr;
    e = cudaStreamEndCapture(ctx->stream, &out);
  }
  ctx->stream = main;
  if (e != cudaSuccess) return set_err(ctx, TDGL_ECUDA, "capture of the PCG loop", e);
  return 0;
}

// A settled solve (warm start, extrapolation history present): every decision on the device, so that the same
// launches serve every step and the step can be captured.
static int pcg_settled(Ctx *ctx) {
  PcgDev *S = ctx->pcg;
  const tdgl_params &P = ctx->P;
  const bool fast = P.pcg_fast || P.pcg_f32, f32 = P.pcg_f32 != 0, ext = fast && P.pcg_extrap;
  int rc;
  to_planes(ctx, ctx->ph, ctx->th, S->b);
  scale_increment(ctx);
  dot2<double>(ctx, S->b, (const void *const *)S->b, nullptr, false, 0);
  TDGL_CUDA(cudaMemsetAsync(S->ic, 0, IC_N * sizeof(int), ctx->stream));
  TDGL_LAUNCH(ctx, K_PCG_EXTRAP, (ext ? 32.0 : 0.0) * 3 * S->n, k_guess, S->sblocks, BS, 0, vv(S->x), vv(S->xprev), S->n,
              S->sc, S->ic, ext ? 1 : 0);
  apply_A(ctx, S->x, nullptr, nullptr, false, -1);
  F3 r32 = {{nullptr, nullptr, nullptr}};
  float *const *r32p = fast && f32 ? sep_r32(ctx) : nullptr;
  if (r32p)
    for (int c = 0; c < 3; c++) r32.p[c] = r32p[c];
  const double wb32 = r32p ? 4.0 : 0.0;
  TDGL_LAUNCH(ctx, K_PCG_RES, (24.0 + wb32) * 3 * S->n, k_residual, S->sblocks, BS, 0, vv(S->r), cv(S->b), cv(S->Q), S->n,
              S->part, r32, fold(ctx, 1));
  const bool flex = fast && f32;
  Bufs B = bufs(S);
  sep_apply(ctx, S->r, (void *const *)B.z[0], zfloat(ctx), S->ic, r32p != nullptr);
  dot_z(ctx, B.z[0], nullptr, 2, 0, true);
  if (ctx->capturing) {
    if ((rc = loop_graph(ctx, B, flex, r32, r32p != nullptr, wb32))) return rc;
  } else {
    int launched = 0;
    while (launched < P.pcg_maxit) {
      const int nb_it = std::min(BATCH, P.pcg_maxit - launched);
      for (int q = 0; q < nb_it; q++) iteration(ctx, B, flex, r32, r32p != nullptr, wb32);
      launched += nb_it;
      read_back(ctx);
      if (S->host_ic[IC_DONE]) break;
    }
  }
  TDGL_LAUNCH(ctx, K_PCG_FINAL, 0.0, k_finish, 1, 32, 0, S->ic, S->stat, 0);
  from_planes(ctx, S->x, ctx->th, ctx->ph);
  return 0;
}

// The solve of implicit.jl:279-446.  Until the warm start has settled (the first steps, or after the carry was
// reset) the host takes the decisions of the reference's loop from read-back scalars; afterwards pcg_settled.
int pcg_implicit(Ctx *ctx) {
  if (pcg_steady(ctx)) return pcg_settled(ctx);
  PcgDev *S = ctx->pcg;
  const tdgl_params &P = ctx->P;
  const bool fast = P.pcg_fast || P.pcg_f32, f32 = P.pcg_f32 != 0;
  int rc;
  // b = φₑ − θ on the ranges, then φ = θ + (φₑ − θ)/D on every link (implicit.jl:381-388)
  to_planes(ctx, ctx->ph, ctx->th, S->b);
  scale_increment(ctx);
  dot2<double>(ctx, S->b, (const void *const *)S->b, nullptr, false, 0);
  TDGL_CUDA(cudaMemsetAsync(S->ic, 0, IC_N * sizeof(int), ctx->stream));
  read_back(ctx);
  const double nb = std::sqrt(S->host_sc[SC_BB]);
  if (nb == 0) {
    // _pcg_zero_update! (implicit.jl:251-271)
    if (fast) {
      if (S->warm && P.pcg_extrap) {
        if ((rc = copy3(ctx, S->xprev, S->x))) return rc;
        S->have2 = true;
      } else {
        S->have2 = false;
      }
    }
    for (int c = 0; c < 3; c++) TDGL_CUDA(cudaMemsetAsync(S->x[c], 0, S->n * sizeof(double), ctx->stream));
    S->warm = true;
    TDGL_LAUNCH(ctx, K_PCG_FINAL, 0.0, k_finish, 1, 32, 0, S->ic, S->stat, 1);
    from_planes(ctx, S->x, ctx->th, ctx->ph);
    return 0;
  }
  if (!S->warm) {
    sep_apply(ctx, S->b, (void *const *)S->x, false, nullptr);
    S->have2 = false;
  } else if (fast && P.pcg_extrap) {
    if (S->have2) {
      TDGL_LAUNCH(ctx, K_PCG_EXTRAP, 32.0 * 3 * S->n, k_extrap, S->sblocks, BS, 0, vv(S->x), vv(S->xprev), S->n);
    } else {
      if ((rc = copy3(ctx, S->xprev, S->x))) return rc;
      S->have2 = true;
    }
  }
  S->warm = true;
  apply_A(ctx, S->x, nullptr, nullptr, false, -1);
  F3 r32 = {{nullptr, nullptr, nullptr}};
  float *const *r32p = fast && f32 ? sep_r32(ctx) : nullptr;
  if (r32p)
    for (int c = 0; c < 3; c++) r32.p[c] = r32p[c];
  const double wb32 = r32p ? 4.0 : 0.0;   // bytes per entry of the FP32 copy
  TDGL_LAUNCH(ctx, K_PCG_RES, (24.0 + wb32) * 3 * S->n, k_residual, S->sblocks, BS, 0, vv(S->r), cv(S->b), cv(S->Q), S->n,
              S->part, r32, fold(ctx, 1));
  read_back(ctx);
  const double tol = P.pcg_tol * nb;
  if (std::sqrt(S->host_sc[SC_RR]) > tol) {
    const bool flex = fast && f32;
    Bufs B = bufs(S);
    sep_apply(ctx, S->r, (void *const *)B.z[0], zfloat(ctx), nullptr, r32p != nullptr);
    dot_z(ctx, B.z[0], nullptr, 2, 0, false);
    int launched = 0;
    while (launched < P.pcg_maxit) {
      const int nb_it = std::min(BATCH, P.pcg_maxit - launched);
      for (int q = 0; q < nb_it; q++) iteration(ctx, B, flex, r32, r32p != nullptr, wb32);
      launched += nb_it;
      read_back(ctx);
      if (S->host_ic[IC_DONE]) break;
    }
  }
  TDGL_LAUNCH(ctx, K_PCG_FINAL, 0.0, k_finish, 1, 32, 0, S->ic, S->stat, 0);
  from_planes(ctx, S->x, ctx->th, ctx->ph);
  return 0;
}

bool pcg_graphable(Ctx *ctx) { return ctx->P.pcg_maxit % BATCH == 0; }

static int carry_xfer(Ctx *ctx, double *const *pm, double *host, bool up) {
  return up ? pm_from_packed_host(ctx, pm, host) : pm_to_packed_host(ctx, pm, host);
}

int pcg_set_carry(Ctx *ctx, const tdgl_carry_view *v) {
  PcgDev *S = ctx->pcg;
  int rc;
  if (v->pcg_x && (rc = carry_xfer(ctx, S->x, v->pcg_x, true))) return rc;
  if (v->pcg_xprev && (rc = carry_xfer(ctx, S->xprev, v->pcg_xprev, true))) return rc;
  S->warm = v->pcg_warm != 0;
  S->have2 = v->pcg_have2 != 0;
  return 0;
}

int pcg_get_carry(Ctx *ctx, const tdgl_carry_view *v) {
  PcgDev *S = ctx->pcg;
  int rc;
  if (v->pcg_x && (rc = carry_xfer(ctx, S->x, v->pcg_x, false))) return rc;
  if (v->pcg_xprev && (rc = carry_xfer(ctx, S->xprev, v->pcg_xprev, false))) return rc;
  const_cast<tdgl_carry_view *>(v)->pcg_warm = S->warm;
  const_cast<tdgl_carry_view *>(v)->pcg_have2 = S->have2;
  return 0;
}

}  // namespace tdgl
