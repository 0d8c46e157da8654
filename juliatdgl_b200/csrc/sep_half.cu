// sep_half.cu — the FP32 preconditioner's mirror-halved plane transforms (the operator of k_half32, sep.cu) for planes
// too large for one block: four launches a direction for the three components.
//
//   forward   k_pair (points → class entries X), k_hgemm<ROW_F> (O1 = W1ᵀ X along y), k_hgemm<COL_F> (along z, the
//             modes written in order)
//   inverse   k_hgemm<ROW_I> (the modes read in class order), k_hgemm<COL_I>, k_unpair (class entries → points)
//
// Per plane: X (n1 × n2, class order, column-major), O1 (JP × n2), O2 (JP × (C0 + C1), in X's buffer).
#include <algorithm>

#define TDGL_PDL   // every kernel launched from this file begins with pdl_enter()
#include "common.cuh"
#include "sep.cuh"

namespace tdgl {
namespace {

// C(m, n) = Σ_k W[k][m] D(n, k) for the half blocks of one component and class: m the outputs along the transformed
// axis, n the points of all planes along the other axis, end to end (a plane's extent need not be a multiple of the
// tile), k in index order (fma from 0).  Both axes, both directions and all components and classes (blk.z) of a
// direction's product are one launch.
//
// What bounds it: the operands' shared-memory loads and issue (43 to 58 % of the cycles issue, at 13 to 15 warps per
// SM).  A block takes bm outputs (⌈h / 64⌉ equal tiles, rounded to 8: 48 for h = 144, 40 for 73) of HG_N = 128 points,
// 8 × 8 outputs a thread, so four 128-bit shared loads (six wavefronts a warp) feed 64 multiply-adds; three stages of
// 16 k in flight by cp.async (40 KB a block: registers and shared memory both leave five blocks of 96 threads per SM).
// The loads along k are element by element (class rows start at any column), so their places are constants and their
// predicates one byte count: 96 µs for the row product of 95 planes of 287 × 95 points instead of 111.  Before, each
// component and class had its own launch of 48 × 96 tiles without prefetching: 36 launches of 25 µs per PCG iteration
// there, two blocks per SM each.
enum HMode { ROW_F, ROW_I, COL_F, COL_I };
const int HG_N = 128, HG_K = 16, HG_ST = 3, HG_WS = 64, HG_DS = HG_N + 12;

struct HGroup {
  const float *W;   // [K][ldw], columns beyond the block zero up to ldw (a multiple of 8)
  const float *D;
  float *C;
  int ldw, K, M;    // M: outputs to write (rows: ldw, the padding included; columns: the block's own)
  int N;            // points, all planes
  int bm;           // outputs per block
  // geometry
  int n1, n2, hS1, hD1, hS2, R0, JP;
  int cls;          // the class (0 even, 1 odd)
  int d_off, d_q, c_off, c_q;   // a component's arrays hold fewer than 2^31 entries (sep_create checks)
  int d_ld, c_ld;
};
struct HGroups {
  HGroup g[6];
  const int *done;
};

// n bytes (4 or 0) from g, the rest zero
__device__ __forceinline__ void cpa4(unsigned s, const float *g, int n) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(s), "l"(g), "r"(n) : "memory");
}
__device__ __forceinline__ void cpa16(float *s, const float *g, bool ok) {
  const int n = ok ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(s)), "l"(g), "r"(n) : "memory");
}

// NT: the block's threads (2 bm), a constant so that the loads' places in shared memory are
template <int MODE, int NT>
__global__ void __launch_bounds__(NT, NT > 96 ? 4 : 5) k_hgemm(const __grid_constant__ HGroups P) {
  tdgl::pdl_enter();
  if (P.done && *P.done) return;
  const HGroup &G = P.g[blockIdx.z];
  const int m0 = blockIdx.y * G.bm, n0 = blockIdx.x * HG_N;
  if (m0 >= G.M || n0 >= G.N) return;
  constexpr bool ROW = MODE == ROW_F || MODE == ROW_I;
  __shared__ __align__(16) float Ws[HG_ST][HG_K][HG_WS];
  __shared__ __align__(16) float Ds[HG_ST][HG_K][HG_DS];
  __shared__ int dbase[HG_DS], cbase[HG_N];   // where point n's data and results start (cbase −1: no result)
  const int tid = threadIdx.x;
  constexpr int nt = NT;
  for (int t = tid; t < HG_DS; t += nt) {   // beyond the tile or the points: the first point's data, read for nothing
    const int n = t < HG_N && n0 + t < G.N ? n0 + t : n0;
    int db, cb = -1;
    {
      if (ROW) {   // n = (plane q, column c in class order)
        const int q = n / G.n2, c = n - q * G.n2;
        if (MODE == ROW_F) db = G.d_off + q * G.d_q + (G.cls ? G.hS1 : 0) + G.n1 * c;
        else db = G.d_off + q * G.d_q + G.cls + G.d_ld * (c < G.hS2 ? 2 * c : 2 * (c - G.hS2) + 1);
        cb = G.c_off + q * G.c_q + (G.cls ? G.R0 : 0) + G.JP * c;
      } else {     // n = (plane q, row r of O1)
        const int q = n / G.JP, r = n - q * G.JP;
        db = G.d_off + q * G.d_q + r + G.JP * (G.cls ? G.hS2 : 0);
        if (MODE == COL_F) {   // row r is mode 2r (even class) or 2(r − R0) + 1; the padding rows have none
          const bool odd = r >= G.R0;
          const int p = odd ? r - G.R0 : r;
          if (p < (odd ? G.hD1 : G.hS1)) cb = G.c_off + q * G.c_q + 2 * p + odd;
        } else {
          cb = G.c_off + q * G.c_q + r;
        }
      }
    }
    dbase[t] = db;
    if (t < HG_N) cbase[t] = n0 + t < G.N ? cb : -1;
  }
  __syncthreads();
  const int bm4 = G.bm / 4, nk = (G.K + HG_K - 1) / HG_K;
  auto load = [&](int kt) {
    const int s = kt % HG_ST, k0 = kt * HG_K;
    for (int e = tid; e < HG_K * bm4; e += nt) {
      const int k = e / bm4, m = 4 * (e - k * bm4);
      const bool ok = k0 + k < G.K && m0 + m < G.ldw;
      cpa16(&Ws[s][k][m], ok ? G.W + (long long)(k0 + k) * G.ldw + m0 + m : G.W, ok);
    }
    if (ROW) {   // consecutive lanes along k; NT / 16 points at a time (the last ones beyond the tile, into the padding)
      const int k = tid % HG_K;
      const float *src = G.D + (k0 + k < G.K ? (MODE == ROW_F ? k0 + k : 2 * (k0 + k)) : 0);
      const int nb = k0 + k < G.K ? 4 : 0;
      const unsigned dst = (unsigned)__cvta_generic_to_shared(&Ds[s][k][tid / HG_K]);
      const int *db = dbase + tid / HG_K;
      constexpr int DN = NT / HG_K, U = (HG_N + DN - 1) / DN;
      static_assert(U * DN <= HG_DS, "the last points' padding");
#pragma unroll
      for (int u = 0; u < U; u++) cpa4(dst + 4 * DN * u, src + db[DN * u], nb);
    } else {     // consecutive lanes along the rows, four at a time (JP and the tiles are multiples of 4)
      const int n = 4 * (tid % (HG_N / 4)), b = dbase[n];
      for (int k = tid / (HG_N / 4); k < HG_K; k += nt / (HG_N / 4)) {
        const bool ok = k0 + k < G.K;
        cpa16(&Ds[s][k][n], ok ? G.D + b + G.JP * (k0 + k) : G.D, ok);
      }
    }
  };
  const int tn = tid % 16, tm = tid / 16;
  float acc[8][8];
#pragma unroll
  for (int a = 0; a < 8; a++)
#pragma unroll
    for (int b = 0; b < 8; b++) acc[a][b] = 0.f;
#pragma unroll
  for (int s = 0; s < HG_ST - 1; s++) {
    if (s < nk) load(s);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  }
  for (int kt = 0; kt < nk; kt++) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(HG_ST - 2) : "memory");
    __syncthreads();   // stage kt has landed for every thread, and stage kt − 1 is free again
    if (kt + HG_ST - 1 < nk) load(kt + HG_ST - 1);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    const int s = kt % HG_ST;
    const float *wp = &Ws[s][0][8 * tm], *dp = &Ds[s][0][4 * tn];
#pragma unroll 4
    for (int k = 0; k < HG_K; k++) {
      const float4 w0 = *reinterpret_cast<const float4 *>(wp + k * HG_WS);
      const float4 w1 = *reinterpret_cast<const float4 *>(wp + k * HG_WS + 4);
      const float4 d0 = *reinterpret_cast<const float4 *>(dp + k * HG_DS);
      const float4 d1 = *reinterpret_cast<const float4 *>(dp + k * HG_DS + HG_N / 2);
      const float wv[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
      const float dv[8] = {d0.x, d0.y, d0.z, d0.w, d1.x, d1.y, d1.z, d1.w};
#pragma unroll
      for (int a = 0; a < 8; a++)
#pragma unroll
        for (int b = 0; b < 8; b++) acc[a][b] = fmaf(wv[a], dv[b], acc[a][b]);
    }
  }
  const int m = m0 + 8 * tm;
#pragma unroll
  for (int h = 0; h < 2; h++) {   // the thread's points 4 tn .. + 3 and 64 + 4 tn .. + 3
    const int n = h * (HG_N / 2) + 4 * tn;
    if (ROW) {
#pragma unroll
      for (int b = 0; b < 4; b++) {
        const int cb = cbase[n + b];
        if (cb < 0 || m >= G.M) continue;
        float *c = G.C + cb + m;
        *reinterpret_cast<float4 *>(c) = make_float4(acc[0][4 * h + b], acc[1][4 * h + b], acc[2][4 * h + b], acc[3][4 * h + b]);
        *reinterpret_cast<float4 *>(c + 4) = make_float4(acc[4][4 * h + b], acc[5][4 * h + b], acc[6][4 * h + b], acc[7][4 * h + b]);
      }
    } else {
#pragma unroll
      for (int a = 0; a < 8; a++) {
        if (m + a >= G.M) continue;
        if (MODE == COL_F) {
#pragma unroll
          for (int b = 0; b < 4; b++) {
            const int cb = cbase[n + b];
            if (cb >= 0) G.C[cb + G.c_ld * (2 * (m + a) + G.cls)] = acc[a][4 * h + b];
          }
        } else if (cbase[n] >= 0) {
          *reinterpret_cast<float4 *>(G.C + cbase[n] + G.JP * (m + a)) =
              make_float4(acc[a][4 * h], acc[a][4 * h + 1], acc[a][4 * h + 2], acc[a][4 * h + 3]);
        }
      }
    }
  }
}

// the four points of each mirror quadrant (p, qc) → its class entries SS, SD, DS, DD (blk.y: the plane, blk.z: the
// component; consecutive lanes on consecutive p)
struct PairArgs {
  const double *in[3];
  float *X[3];
  long long xps;
  HalfMulti M;
};
__global__ void __launch_bounds__(256) k_pair(const __grid_constant__ PairArgs P) {
  tdgl::pdl_enter();
  if (P.M.done && *P.M.done) return;
  const HalfArgs &A = P.M.c[blockIdx.z];
  const int q = blockIdx.y;
  if (q >= A.nplanes) return;
  const HalfGeo G(A.n1, A.n2);
  const int n1 = A.n1, n2 = A.n2, e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= G.hS1 * G.hS2) return;
  const int qc = e / G.hS1, p = e - qc * G.hS1, pp = n1 - 1 - p, qq = n2 - 1 - qc;
  const double *in = P.in[blockIdx.z] + A.in_base + q * A.in_ps + A.in_j0 + (long long)A.in_ld * A.in_k0;
  float *x = P.X[blockIdx.z] + q * P.xps;
  const bool rp = pp != p, cp = qq != qc;
  const float a = (float)in[p + (long long)A.in_ld * qc];
  const float b = rp ? (float)in[pp + (long long)A.in_ld * qc] : 0.f;
  const float c = cp ? (float)in[p + (long long)A.in_ld * qq] : 0.f;
  const float d = rp && cp ? (float)in[pp + (long long)A.in_ld * qq] : 0.f;
  const float s0 = a + c, s1 = b + d, d0 = a - c, d1 = b - d;
  x[p + (long long)n1 * qc] = s0 + s1;
  if (cp) x[p + (long long)n1 * (G.hS2 + qc)] = d0 + d1;
  if (rp) {
    x[G.hS1 + p + (long long)n1 * qc] = s0 - s1;
    if (cp) x[G.hS1 + p + (long long)n1 * (G.hS2 + qc)] = d0 - d1;
  }
}

// the class entries of each mirror quadrant → its four points
__global__ void __launch_bounds__(256) k_unpair(const __grid_constant__ PairArgs P) {
  tdgl::pdl_enter();
  if (P.M.done && *P.M.done) return;
  const HalfArgs &A = P.M.c[blockIdx.z];
  const int q = blockIdx.y;
  if (q >= A.nplanes) return;
  const HalfGeo G(A.n1, A.n2);
  const int n1 = A.n1, n2 = A.n2, JP = G.JP, e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= G.hS1 * G.hS2) return;
  const int qc = e / G.hS1, p = e - qc * G.hS1, pp = n1 - 1 - p, qq = n2 - 1 - qc;
  const float *o2 = P.X[blockIdx.z] + q * P.xps;
  float *out = (float *)A.out + A.out_base + q * A.out_ps + A.out_j0 + (long long)A.out_ld * A.out_k0;
  const bool rp = pp != p, cp = qq != qc;
  const float ee = o2[p + (long long)JP * qc];
  const float eo = cp ? o2[p + (long long)JP * (G.C0 + qc)] : 0.f;
  const float oe = rp ? o2[G.R0 + p + (long long)JP * qc] : 0.f;
  const float oo = rp && cp ? o2[G.R0 + p + (long long)JP * (G.C0 + qc)] : 0.f;
  const float s0 = ee + oe, s1 = eo + oo, d0 = ee - oe, d1 = eo - oo;
  const long long oq = (long long)A.out_ld * qc, oqq = (long long)A.out_ld * qq;
  out[oq + p] = s0 + s1;
  if (rp) out[oq + pp] = d0 + d1;
  if (cp) {
    out[oqq + p] = s0 - s1;
    if (rp) out[oqq + pp] = d0 - d1;
  }
}

// outputs per block: equal tiles of at most 64, a multiple of 8; at least 16, so that a block holds a whole warp (the
// loads along the rows take 32 threads a row)
int tile_of(int h) {
  const int nt = std::max(1, (h + 63) / 64);
  return std::max(16, rup8((h + nt - 1) / nt));
}

template <int MODE>
void launch(Ctx *ctx, HGroups &P, KCat cat, double bytes) {
  int gx = 0, gy = 0, bm = 16;
  for (HGroup &g : P.g) bm = std::max(bm, tile_of(g.M));   // one block shape for every group
  for (HGroup &g : P.g) {
    g.bm = bm;
    if (g.M <= 0 || g.N <= 0) continue;
    gx = std::max(gx, (g.N + HG_N - 1) / HG_N);
    gy = std::max(gy, (g.M + bm - 1) / bm);
  }
  if (!gx) return;
  const dim3 grid(gx, gy, 6);
  switch (bm) {   // 16, 24, ... 64
    case 16: TDGL_LAUNCH(ctx, cat, bytes, (k_hgemm<MODE, 32>), grid, 32, 0, P); break;
    case 24: TDGL_LAUNCH(ctx, cat, bytes, (k_hgemm<MODE, 48>), grid, 48, 0, P); break;
    case 32: TDGL_LAUNCH(ctx, cat, bytes, (k_hgemm<MODE, 64>), grid, 64, 0, P); break;
    case 40: TDGL_LAUNCH(ctx, cat, bytes, (k_hgemm<MODE, 80>), grid, 80, 0, P); break;
    case 48: TDGL_LAUNCH(ctx, cat, bytes, (k_hgemm<MODE, 96>), grid, 96, 0, P); break;
    case 56: TDGL_LAUNCH(ctx, cat, bytes, (k_hgemm<MODE, 112>), grid, 112, 0, P); break;
    default: TDGL_LAUNCH(ctx, cat, bytes, (k_hgemm<MODE, 128>), grid, 128, 0, P); break;
  }
}

}  // namespace

HalfWork half_work(int ny, int nz) {   // plane strides of X / O2 and O1 (the largest component's)
  const HalfGeo G(ny, nz);
  HalfWork w;
  w.x_ps = (std::max((long long)ny * nz, (long long)G.JP * (G.C0 + G.C1)) + 3) & ~3LL;
  w.o_ps = (long long)G.JP * nz;
  return w;
}

void half_large(Ctx *ctx, const HalfMulti &M, bool fwd, const double *const *in64, const HalfWork &w) {
  const KCat cat = fwd ? K_TX32 : K_TX32I;
  double pts = 0;
  int ge = 0, gq = 0;
  PairArgs Q;
  Q.M = M;
  Q.xps = w.x_ps;
  HGroups R, C;
  memset(&R, 0, sizeof(R));
  memset(&C, 0, sizeof(C));
  R.done = C.done = M.done;
  for (int c = 0; c < 3; c++) {
    const HalfArgs &A = M.c[c];
    const HalfGeo G(A.n1, A.n2);
    pts += (double)A.n1 * A.n2 * A.nplanes;
    ge = std::max(ge, G.hS1 * G.hS2);
    gq = std::max(gq, A.nplanes);
    Q.in[c] = in64 ? in64[c] : nullptr;
    Q.X[c] = w.x[c];
    const float *W1[2] = {A.W1, A.W1 + (size_t)G.hS1 * G.R0}, *W2[2] = {A.W2, A.W2 + (size_t)G.hS2 * G.C0};
    const int h1[2] = {G.hS1, G.hD1}, Rr[2] = {G.R0, G.R1}, h2[2] = {G.hS2, G.hD2}, Cw[2] = {G.C0, G.C1};
    for (int a = 0; a < 2; a++) {
      HGroup &r = R.g[2 * c + a], &k = C.g[2 * c + a];
      r.n1 = k.n1 = A.n1; r.n2 = k.n2 = A.n2; r.hS1 = k.hS1 = G.hS1; r.hD1 = k.hD1 = G.hD1; r.hS2 = k.hS2 = G.hS2;
      r.R0 = k.R0 = G.R0; r.JP = k.JP = G.JP; r.cls = k.cls = a;
      r.W = W1[a]; r.ldw = Rr[a]; r.K = h1[a]; r.M = h1[a] > 0 ? Rr[a] : 0; r.N = A.n2 * A.nplanes;
      r.D = fwd ? w.x[c] : A.in;
      r.d_off = fwd ? 0 : A.in_base + A.in_j0 + (long long)A.in_ld * A.in_k0;
      r.d_q = fwd ? w.x_ps : A.in_ps;
      r.d_ld = A.in_ld;
      r.C = w.o[c]; r.c_off = 0; r.c_q = w.o_ps;
      k.W = W2[a]; k.ldw = Cw[a]; k.K = h2[a]; k.M = h2[a]; k.N = G.JP * A.nplanes;
      k.D = w.o[c]; k.d_off = 0; k.d_q = w.o_ps;
      k.C = fwd ? (float *)A.out : w.x[c];
      k.c_off = fwd ? A.out_base + A.out_j0 + (long long)A.out_ld * A.out_k0 : (long long)G.JP * (a ? G.C0 : 0);
      k.c_q = fwd ? A.out_ps : w.x_ps;
      k.c_ld = A.out_ld;
    }
  }
  const dim3 gp((ge + 255) / 256, gq, 3);
  if (fwd) {
    TDGL_LAUNCH(ctx, cat, 12.0 * pts, k_pair, gp, 256, 0, Q);
    launch<ROW_F>(ctx, R, cat, 8.0 * pts);
    launch<COL_F>(ctx, C, cat, 8.0 * pts);
  } else {
    launch<ROW_I>(ctx, R, cat, 8.0 * pts);
    launch<COL_I>(ctx, C, cat, 8.0 * pts);
    TDGL_LAUNCH(ctx, cat, 8.0 * pts, k_unpair, gp, 256, 0, Q);
  }
}

}  // namespace tdgl
