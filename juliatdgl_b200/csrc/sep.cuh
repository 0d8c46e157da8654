// sep.cuh — what the FP32 preconditioner's plane transforms share (sep.cu: the SIMT kernel, the line solve and
// the host side; sep_tc.cu: the tensor-core kernel).
#pragma once
#include "common.cuh"

#include <vector>

namespace tdgl {

__host__ __device__ inline int rup8(int n) { return (n + 7) & ~7; }
__host__ __device__ inline int rup16(int n) { return (n + 15) & ~15; }

const int P32_KPAD = 52;   // row length of k_half32's X
__host__ __device__ inline int p32_ks(int KO) { return 4 * ((KO / 4) | 1); }

// The class geometry of a mirror-halved transform of n1 × n2 planes: hS = ⌈n/2⌉ even and hD = ⌊n/2⌋ odd modes per
// axis, padded to 8 (R along y, C along z).
struct HalfGeo {
  int hS1, hD1, hS2, hD2, R0, R1, C0, C1, JP, KP, KS, XR;
  __host__ __device__ HalfGeo(int n1, int n2) {
    hS1 = (n1 + 1) / 2; hD1 = n1 / 2; hS2 = (n2 + 1) / 2; hD2 = n2 / 2;
    R0 = rup8(hS1); R1 = rup8(hD1); C0 = rup8(hS2); C1 = rup8(hD2);
    JP = R0 + R1; KP = rup8(n2); KS = p32_ks(C0 + C1); XR = n1 > JP ? n1 : JP;
  }
  __host__ __device__ size_t wfloats() const {
    return (size_t)hS1 * R0 + (size_t)hD1 * R1 + (size_t)hS2 * C0 + (size_t)hD2 * C1;
  }
  __host__ __device__ size_t slot(int n1, int n2) const {   // one plane's XO, O1 and Stg, rounded to 16 bytes
    return ((size_t)XR * P32_KPAD + (size_t)KP * JP + (size_t)n1 * n2 + 3) & ~(size_t)3;
  }
};

// One component's planes for a mirror-halved transform: plane q of the input is in[in_base + q·in_ps + (in_j0 + j)
// + in_ld·(in_k0 + k)] (j < n1, k < n2), likewise the output.
struct HalfArgs {
  const float *in;
  long long in_base, in_ps;
  int in_ld, in_j0, in_k0;
  int n1, n2;                  // points (= modes) along the row axis (y) and the column axis (z)
  const float *W1, *W2;        // SIMT: the half blocks of each axis: [E | O], row-major (in, out), rows padded to 8
  const float *T1, *T2;        // tensor cores: the half blocks as MMA operand images (tc_images), null if absent
  void *out;
  long long out_base, out_ps;
  int out_ld, out_j0, out_k0;
  int nplanes;
};
// The three components (x, y and z links) in one launch.
struct HalfMulti {
  HalfArgs c[3];
  int ncomp;
  const int *done;             // skip when the PCG has converged (null: always run)
};

// The same transforms for planes too large for one block (sep_half.cu): a direction of the three components through X /
// O2 and O1 buffers per component; in64: the FP64 points of the forward direction.
struct HalfWork {
  float *x[3] = {nullptr, nullptr, nullptr}, *o[3] = {nullptr, nullptr, nullptr};
  long long x_ps = 0, o_ps = 0;   // plane strides
};
HalfWork half_work(int ny, int nz);
void half_large(Ctx *ctx, const HalfMulti &M, bool fwd, const double *const *in64, const HalfWork &w);

// Tensor-core operand images of the mirror half blocks of a basis B(p, m) (point p, mode m) with np points:
// E = B(p, 2m) for p, m < hS = ⌈np/2⌉ and O = B(p, 2m+1) for p, m < hD = ⌊np/2⌋.  Four images [class a][hi, lo],
// each R = rup16(hS) rows (outputs) × K = rup8(hS) columns (inputs), zero outside the block, laid out K-major
// without swizzle: element (o, i) at float (o % 8)·4 + (o / 8)·8K + (i % 4) + (i / 4)·32.  Forward (points →
// modes): element (o, i) = H_a(i, o); inverse (modes → points): H_a(o, i).  hi is the value rounded to TF32, lo the
// remainder rounded to TF32 (umma::split_tf32).
void tc_images(int np, const double *B, int ldB, std::vector<float> &fwd, std::vector<float> &inv);

// The tensor-core transform (sep_tc.cu): whether it takes planes up to n1 × n2, and the launch (one direction for
// the three components; `err` counts blocks whose tensor-core waits ran out).
extern int g_sm_count;   // SMs of the device (set by sep_create)
bool half_tc_fits(int n1, int n2);
void half_tc(Ctx *ctx, const HalfMulti &M, bool fwd, long long *err);
void half_tc_init();

}  // namespace tdgl
