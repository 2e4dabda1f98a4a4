// tfm.cuh -- FP64 transform algebra for the registration path, usable on the
// host and on the device.
//
// On the device a whole aligned quad of lanes calls together, all four active with
// the same arguments: functions that take three angles' sines, cosines or arc
// tangents (sincos3, atan2_3, and through them euler_zxy_matrix, euler_zxy_angles,
// quat_euler_angles, tfm_set_params, tfm_set_matrix, tfm_compose, tfm_inverse and
// the fits of a rigid transform) share them out over the quad's lanes by shuffles,
// which a lone thread or a partial quad would leave waiting.  The LTS solve runs
// so in one warp (lts.cu).
//
// It restates the semantics the reference relies on:
//   * itk::MatrixOffsetTransformBase: y = M (x - c) + c + t = M x + offset,
//     offset = t + c - M c; SetCenter/SetTranslation keep t and recompute the
//     offset; SetMatrix recomputes the offset then the matrix parameters;
//     Compose(other, pre) (pre: self(other(x)), else other(self(x))) keeps the
//     centre and recomputes the translation; GetInverse keeps the centre.
//   * itk::Euler3DTransform (ComputeZYX off): R = Rz Rx Ry, parameters
//     (ax, ay, az, tx, ty, tz); SetMatrix requires |M M^T - I| <= 1e-10 and
//     re-derives the matrix from the extracted angles.
//   * itk::AffineTransform: parameters = matrix row-major + translation.
//   * vnl_quaternion (x, y, z, r): rotation matrix, rotation_euler_angles
//     (R = Rz Ry Rx), axis(), angle(), (axis, angle) constructor.
//   * src/mirorr/vnl_utils.h: Denman-Beavers square root (:46-95) and
//     orthogonalize = U V^T of the SVD (:124-135).
#pragma once

#include <math.h>

// Every loop over matrix entries has constant bounds and is unrolled on the
// device, and every index is a constant then, so that the compiler can hold the
// matrices in registers (an index known only at run time would put them into local
// memory).  The classic solve's all fit; the symmetric one, at 128 registers a
// thread, spills 1.3 to 1.4 KB of them.
#ifdef __CUDACC__
#define MB2_HD __host__ __device__ inline
#define MB2_UNROLL _Pragma("unroll")
#else
#define MB2_HD inline
#define MB2_UNROLL
#endif

namespace mb2 {

enum { KIND_RIGID = 0, KIND_AFFINE = 1 };

// ---- small dense matrices (row-major) ------------------------------------
MB2_HD void m3_mul(const double *a, const double *b, double *o) {
  double r[9];
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) {
      double s = 0.0;
      for (int k = 0; k < 3; ++k) s += a[3 * i + k] * b[3 * k + j];
      r[3 * i + j] = s;
    }
  for (int i = 0; i < 9; ++i) o[i] = r[i];
}
MB2_HD void m3_vec(const double *a, const double *v, double *o) {
  double r[3];
  for (int i = 0; i < 3; ++i) r[i] = a[3 * i] * v[0] + a[3 * i + 1] * v[1] + a[3 * i + 2] * v[2];
  o[0] = r[0]; o[1] = r[1]; o[2] = r[2];
}
MB2_HD void m3_transpose(const double *a, double *o) {
  double r[9];
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) r[3 * j + i] = a[3 * i + j];
  for (int i = 0; i < 9; ++i) o[i] = r[i];
}
MB2_HD void m3_identity(double *o) {
  for (int i = 0; i < 9; ++i) o[i] = (i % 4 == 0) ? 1.0 : 0.0;
}
MB2_HD double m3_det(const double *a) {
  return a[0] * (a[4] * a[8] - a[5] * a[7]) - a[1] * (a[3] * a[8] - a[5] * a[6]) +
         a[2] * (a[3] * a[7] - a[4] * a[6]);
}

// Gauss-Jordan inverse with partial pivoting; returns false when singular.
// The pivot row is found by comparisons in row order and brought up by
// selects on constant indices.
template <int N>
MB2_HD bool mn_inverse(const double *a, double *o) {
  double m[N][2 * N];
  MB2_UNROLL
  for (int i = 0; i < N; ++i)
    MB2_UNROLL
    for (int j = 0; j < N; ++j) {
      m[i][j] = a[N * i + j];
      m[i][N + j] = (i == j) ? 1.0 : 0.0;
    }
  MB2_UNROLL
  for (int c = 0; c < N; ++c) {
    int p = c;
    double best = fabs(m[c][c]);
    MB2_UNROLL
    for (int r = c + 1; r < N; ++r)
      if (fabs(m[r][c]) > best) { best = fabs(m[r][c]); p = r; }
    if (best == 0.0) return false;
    MB2_UNROLL
    for (int r = c + 1; r < N; ++r)
      MB2_UNROLL
      for (int j = 0; j < 2 * N; ++j) {
        const double u = m[c][j], v = m[r][j];
        m[c][j] = p == r ? v : u;
        m[r][j] = p == r ? u : v;
      }
    const double inv = 1.0 / m[c][c];
    MB2_UNROLL
    for (int j = 0; j < 2 * N; ++j) m[c][j] *= inv;
    MB2_UNROLL
    for (int r = 0; r < N; ++r) {
      if (r == c) continue;
      const double f = m[r][c];
      MB2_UNROLL
      for (int j = 0; j < 2 * N; ++j) m[r][j] -= f * m[c][j];
    }
  }
  MB2_UNROLL
  for (int i = 0; i < N; ++i)
    MB2_UNROLL
    for (int j = 0; j < N; ++j) o[N * i + j] = m[i][N + j];
  return true;
}

template <int N>
MB2_HD void mn_mul(const double *a, const double *b, double *o) {
  double r[N * N];
  for (int i = 0; i < N; ++i)
    for (int j = 0; j < N; ++j) {
      double s = 0.0;
      for (int k = 0; k < N; ++k) s += a[N * i + k] * b[N * k + j];
      r[N * i + j] = s;
    }
  for (int i = 0; i < N * N; ++i) o[i] = r[i];
}

// 1 / sqrt(x) for x in [1e-36, 1e36]: on the device a single-precision seed
// and two Newton steps y (3 - x y^2) / 2 (the seed's error of 2^-22 squares
// twice), without the branches that would keep two of them from overlapping.
MB2_HD double inv_sqrt(double x) {
#ifdef __CUDA_ARCH__
  double y = (double)rsqrtf((float)x);
  const double hx = 0.5 * x;
  MB2_UNROLL
  for (int i = 0; i < 2; ++i) {
    const double e = fma(-hx * y, y, 0.5);
    y = fma(y, e, y);
  }
  return y;
#else
  return 1.0 / sqrt(x);
#endif
}

// One Jacobi rotation of the symmetric matrix a (upper triangle) in the plane
// (P, Q), accumulated into the columns of v.
template <int N, int P, int Q>
MB2_HD void jacobi_rotate(double *a, double *v) {
  const double apq = a[N * P + Q], app = a[N * P + P], aqq = a[N * Q + Q];
  // with d = aqq - app and e = 2 apq the smaller angle has cos 2x = |d| r and
  // |sin 2x| = |e| r, r = 1 / sqrt(d^2 + e^2); its sign is positive when d = 0
  // or d and e agree.  c = sqrt((1 + cos 2x) / 2) and w = 1 / c, so a rotation
  // is two reciprocal square roots and no division.
  // An entry below 1e-18 (of a matrix scaled to a largest entry of about one) is
  // taken as zero.
  const double d = aqq - app, e = 2.0 * apq, h2 = d * d + e * e;
  const bool skip = !(fabs(apq) > 1e-18);
  const double r = inv_sqrt(skip ? 1.0 : h2), x = 0.5 + 0.5 * (fabs(d) * r), w = inv_sqrt(x);
  const double neg = (d != 0.0 && (d > 0.0) != (e > 0.0)) ? -0.5 : 0.5;
  const double c = skip ? 1.0 : x * w;
  const double s = skip ? 0.0 : neg * (fabs(e) * r) * w;
  const double t = s * w;
  a[N * P + P] = app - t * apq;
  a[N * Q + Q] = aqq + t * apq;
  a[N * P + Q] = 0.0;
  MB2_UNROLL
  for (int k = 0; k < N; ++k) {
    if (k == P || k == Q) continue;
    double &akp = a[k < P ? N * k + P : N * P + k], &akq = a[k < Q ? N * k + Q : N * Q + k];
    const double x = akp, y = akq;
    akp = c * x - s * y;
    akq = s * x + c * y;
  }
  MB2_UNROLL
  for (int k = 0; k < N; ++k) {
    const double x = v[N * k + P], y = v[N * k + Q];
    v[N * k + P] = c * x - s * y;
    v[N * k + Q] = s * x + c * y;
  }
}

// Cyclic Jacobi eigen-decomposition of a symmetric NxN matrix (N = 3 or 4).
// On return w[] holds eigenvalues in ascending order and column k of v is the
// eigenvector of w[k].  For N = 4 a sweep takes the planes in three pairs of
// disjoint ones, whose angles depend on different entries: the reciprocal square
// roots of a pair overlap.
template <int N>
MB2_HD void jacobi_eigen(const double *a_in, double *w, double *v) {
  static_assert(N == 3 || N == 4, "3x3 or 4x4");
  double a[N * N], u[N * N], big = 0.0;
  MB2_UNROLL
  for (int i = 0; i < N * N; ++i) big = fmax(big, fabs(a_in[i]));
  // scaled by a power of two (exactly) to a largest entry in [1/2, 1)
  int ex = 0;
  if (big > 1e-300 && big < 1e300) frexp(big, &ex);
  const double down = ldexp(1.0, -ex), up = ldexp(1.0, ex);
  MB2_UNROLL
  for (int i = 0; i < N * N; ++i) {
    a[i] = a_in[i] * down;
    u[i] = (i % (N + 1) == 0) ? 1.0 : 0.0;
  }
  for (int sweep = 0; sweep < 64; ++sweep) {
    double off = 0.0, diag = 0.0;
    MB2_UNROLL
    for (int i = 0; i < N; ++i) {
      diag += a[N * i + i] * a[N * i + i];
      MB2_UNROLL
      for (int j = i + 1; j < N; ++j) off += a[N * i + j] * a[N * i + j];
    }
    if (off <= 1e-32 * diag || off == 0.0) break;
    if constexpr (N == 4) {
      jacobi_rotate<N, 0, 1>(a, u);
      jacobi_rotate<N, 2, 3>(a, u);
      jacobi_rotate<N, 0, 2>(a, u);
      jacobi_rotate<N, 1, 3>(a, u);
      jacobi_rotate<N, 0, 3>(a, u);
      jacobi_rotate<N, 1, 2>(a, u);
    } else {
      jacobi_rotate<N, 0, 1>(a, u);
      jacobi_rotate<N, 0, 2>(a, u);
      jacobi_rotate<N, 1, 2>(a, u);
    }
  }
  double d[N];
  MB2_UNROLL
  for (int i = 0; i < N; ++i) d[i] = a[N * i + i] * up;
  // sort ascending (exchanges of columns)
  MB2_UNROLL
  for (int i = 0; i < N; ++i)
    MB2_UNROLL
    for (int j = i + 1; j < N; ++j) {
      const bool sw = d[j] < d[i];
      const double x = d[i], y = d[j];
      d[i] = sw ? y : x;
      d[j] = sw ? x : y;
      MB2_UNROLL
      for (int k = 0; k < N; ++k) {
        const double p = u[N * k + i], q = u[N * k + j];
        u[N * k + i] = sw ? q : p;
        u[N * k + j] = sw ? p : q;
      }
    }
  MB2_UNROLL
  for (int i = 0; i < N; ++i) w[i] = d[i];
  MB2_UNROLL
  for (int i = 0; i < N * N; ++i) v[i] = u[i];
}

// Orthogonal polar factor U V^T of a (non-singular) 3x3 matrix:
// M (M^T M)^(-1/2), computed from the eigen-decomposition of M^T M.
MB2_HD void orthogonalize3(const double *m, double *o) {
  double mt[9], mtm[9], w[3], v[9], l[3];
  m3_transpose(m, mt);
  m3_mul(mt, m, mtm);
  jacobi_eigen<3>(mtm, w, v);
  MB2_UNROLL
  for (int k = 0; k < 3; ++k) l[k] = w[k] > 0.0 ? 1.0 / sqrt(w[k]) : 0.0;
  double isq[9];
  MB2_UNROLL
  for (int i = 0; i < 3; ++i)
    MB2_UNROLL
    for (int j = 0; j < 3; ++j) {
      double s = 0.0;
      MB2_UNROLL
      for (int k = 0; k < 3; ++k) s += v[3 * i + k] * l[k] * v[3 * j + k];
      isq[3 * i + j] = s;
    }
  m3_mul(m, isq, o);
}

// Inverse of a homogeneous affine 4x4 matrix [A t; 0 0 0 1] (row-major):
// [A^-1, -A^-1 t; 0 0 0 1], with A^-1 from its cofactors.  False when A is
// singular.
MB2_HD bool affine4_inverse(const double *m, double *o) {
  const double a = m[0], b = m[1], c = m[2], d = m[4], e = m[5], f = m[6];
  const double g = m[8], h = m[9], k = m[10];
  const double c00 = e * k - f * h, c01 = f * g - d * k, c02 = d * h - e * g;
  const double det = a * c00 + b * c01 + c * c02;
  if (det == 0.0) return false;
  const double r = 1.0 / det;
  double ia[9];
  ia[0] = c00 * r; ia[1] = (c * h - b * k) * r; ia[2] = (b * f - c * e) * r;
  ia[3] = c01 * r; ia[4] = (a * k - c * g) * r; ia[5] = (c * d - a * f) * r;
  ia[6] = c02 * r; ia[7] = (b * g - a * h) * r; ia[8] = (a * e - b * d) * r;
  for (int i = 0; i < 3; ++i) {
    o[4 * i + 0] = ia[3 * i + 0];
    o[4 * i + 1] = ia[3 * i + 1];
    o[4 * i + 2] = ia[3 * i + 2];
    o[4 * i + 3] = -(ia[3 * i + 0] * m[3] + ia[3 * i + 1] * m[7] + ia[3 * i + 2] * m[11]);
  }
  o[12] = 0.0; o[13] = 0.0; o[14] = 0.0; o[15] = 1.0;
  return true;
}

// Denman-Beavers square root of a homogeneous affine 4x4 matrix
// (vnl_utils.h:46-95) with EPS = 1e-14, MAX_ITER = 50 as called from
// itkSymMirorrRegistrationMethod.txx.  Every iterate keeps the last row
// 0 0 0 1, so the inverses are the affine ones.
MB2_HD void matrix_sqrt4(const double *m, double *y_out) {
  double y[16], z[16], iy[16], iz[16];
  MB2_UNROLL
  for (int i = 0; i < 16; ++i) { y[i] = m[i]; z[i] = (i % 5 == 0) ? 1.0 : 0.0; }
  double dd = 1.7976931348623157e308;
  int it = 0;
  while (dd > 1e-14 && it < 50) {
    affine4_inverse(z, iz);
    affine4_inverse(y, iy);
    MB2_UNROLL
    for (int i = 0; i < 12; ++i) {
      const double ny = 0.5 * (y[i] + iz[i]), nz = 0.5 * (z[i] + iy[i]);
      y[i] = ny;
      z[i] = nz;
    }
    ++it;
    // y y - m over the first three rows (the last ones are 0 0 0 1)
    dd = 0.0;
    MB2_UNROLL
    for (int i = 0; i < 3; ++i)
      MB2_UNROLL
      for (int j = 0; j < 4; ++j) {
        double d = y[4 * i] * y[j] + y[4 * i + 1] * y[4 + j] + y[4 * i + 2] * y[8 + j];
        if (j == 3) d += y[4 * i + 3];
        const double e = fabs(d - m[4 * i + j]);
        if (e > dd) dd = e;
      }
  }
  MB2_UNROLL
  for (int i = 0; i < 16; ++i) y_out[i] = y[i];
}

// ---- Euler3D (Z*X*Y) -------------------------------------------------------
// Three angles at once.  On the device the four lanes of an aligned quad call
// these together with the same arguments and each takes one angle: the time of
// one evaluation instead of three in a row.
MB2_HD void sincos3(const double *ang, double *s, double *c) {
#ifdef __CUDA_ARCH__
  const unsigned lane = threadIdx.x & 31u, quad = 0xFu << (lane & 28u);
  const double x = (lane & 3u) == 0 ? ang[0] : ((lane & 3u) == 1 ? ang[1] : ang[2]);
  double sv, cv;
  sincos(x, &sv, &cv);
  MB2_UNROLL
  for (int k = 0; k < 3; ++k) {
    s[k] = __shfl_sync(quad, sv, k, 4);
    c[k] = __shfl_sync(quad, cv, k, 4);
  }
#else
  for (int k = 0; k < 3; ++k) { s[k] = sin(ang[k]); c[k] = cos(ang[k]); }
#endif
}
MB2_HD void atan2_3(const double *y, const double *x, double *ang) {
#ifdef __CUDA_ARCH__
  const unsigned lane = threadIdx.x & 31u, quad = 0xFu << (lane & 28u);
  const double yy = (lane & 3u) == 0 ? y[0] : ((lane & 3u) == 1 ? y[1] : y[2]);
  const double xx = (lane & 3u) == 0 ? x[0] : ((lane & 3u) == 1 ? x[1] : x[2]);
  const double a = atan2(yy, xx);
  MB2_UNROLL
  for (int k = 0; k < 3; ++k) ang[k] = __shfl_sync(quad, a, k, 4);
#else
  for (int k = 0; k < 3; ++k) ang[k] = atan2(y[k], x[k]);
#endif
}

MB2_HD void euler_zxy_matrix(const double *ang, double *o) {
  double s3[3], c3[3];
  sincos3(ang, s3, c3);
  const double cx = c3[0], sx = s3[0], cy = c3[1], sy = s3[1], cz = c3[2], sz = s3[2];
  double rx[9] = {1, 0, 0, 0, cx, -sx, 0, sx, cx};
  double ry[9] = {cy, 0, sy, 0, 1, 0, -sy, 0, cy};
  double rz[9] = {cz, -sz, 0, sz, cz, 0, 0, 0, 1};
  double t[9];
  m3_mul(rz, rx, t);
  m3_mul(t, ry, o);
}

MB2_HD void euler_zxy_angles(const double *m, double *ang) {
  double s = m[7];
  if (s > 1.0) s = 1.0;
  if (s < -1.0) s = -1.0;
  ang[0] = asin(s);
  const double a = cos(ang[0]);
  const bool regular = fabs(a) > 0.00005;
  const double y[3] = {0.0, regular ? -m[6] / a : m[3], regular ? -m[1] / a : 0.0};
  const double x[3] = {1.0, regular ? m[8] / a : m[0], regular ? m[4] / a : 1.0};
  double t[3];
  atan2_3(y, x, t);
  ang[1] = t[1];
  ang[2] = regular ? t[2] : 0.0;
}

// ---- transform -------------------------------------------------------------
struct Tfm {
  int kind;
  double M[9];
  double off[3];
  double c[3];
  double t[3];
  double ang[3];
};

MB2_HD void tfm_identity(Tfm &a, int kind) {
  a.kind = kind;
  m3_identity(a.M);
  for (int i = 0; i < 3; ++i) { a.off[i] = 0; a.c[i] = 0; a.t[i] = 0; a.ang[i] = 0; }
}
MB2_HD void tfm_compute_offset(Tfm &a) {
  double mc[3];
  m3_vec(a.M, a.c, mc);
  for (int i = 0; i < 3; ++i) a.off[i] = a.t[i] + a.c[i] - mc[i];
}
MB2_HD void tfm_compute_translation(Tfm &a) {
  double mc[3];
  m3_vec(a.M, a.c, mc);
  for (int i = 0; i < 3; ++i) a.t[i] = a.off[i] - a.c[i] + mc[i];
}
MB2_HD void tfm_compute_matrix_params(Tfm &a) {
  if (a.kind == KIND_RIGID) {
    euler_zxy_angles(a.M, a.ang);
    euler_zxy_matrix(a.ang, a.M);
  }
}
MB2_HD void tfm_set_center(Tfm &a, const double *c) {
  for (int i = 0; i < 3; ++i) a.c[i] = c[i];
  tfm_compute_offset(a);
}
MB2_HD void tfm_set_translation(Tfm &a, const double *t) {
  for (int i = 0; i < 3; ++i) a.t[i] = t[i];
  tfm_compute_offset(a);
}
// Returns false (and leaves the transform unchanged) when a rigid transform is
// given a matrix that is not orthogonal within 1e-10.
MB2_HD bool tfm_set_matrix(Tfm &a, const double *m) {
  if (a.kind == KIND_RIGID) {
    double mt[9], p[9];
    m3_transpose(m, mt);
    m3_mul(m, mt, p);
    for (int i = 0; i < 9; ++i) {
      double d = p[i] - ((i % 4 == 0) ? 1.0 : 0.0);
      if (fabs(d) > 1e-10) return false;
    }
  }
  for (int i = 0; i < 9; ++i) a.M[i] = m[i];
  tfm_compute_offset(a);
  tfm_compute_matrix_params(a);
  return true;
}
MB2_HD int tfm_nparams(const Tfm &a) { return a.kind == KIND_RIGID ? 6 : 12; }
MB2_HD void tfm_params(const Tfm &a, double *p) {
  if (a.kind == KIND_RIGID) {
    for (int i = 0; i < 3; ++i) { p[i] = a.ang[i]; p[3 + i] = a.t[i]; }
  } else {
    for (int i = 0; i < 9; ++i) p[i] = a.M[i];
    for (int i = 0; i < 3; ++i) p[9 + i] = a.t[i];
  }
}
MB2_HD void tfm_set_params(Tfm &a, const double *p) {
  if (a.kind == KIND_RIGID) {
    for (int i = 0; i < 3; ++i) { a.ang[i] = p[i]; a.t[i] = p[3 + i]; }
    euler_zxy_matrix(a.ang, a.M);
  } else {
    for (int i = 0; i < 9; ++i) a.M[i] = p[i];
    for (int i = 0; i < 3; ++i) a.t[i] = p[9 + i];
  }
  tfm_compute_offset(a);
}
MB2_HD void tfm_compose(Tfm &a, const Tfm &o, bool pre) {
  double nm[9], noff[3];
  if (pre) {
    m3_vec(a.M, o.off, noff);
    for (int i = 0; i < 3; ++i) noff[i] += a.off[i];
    m3_mul(a.M, o.M, nm);
  } else {
    m3_vec(o.M, a.off, noff);
    for (int i = 0; i < 3; ++i) noff[i] += o.off[i];
    m3_mul(o.M, a.M, nm);
  }
  for (int i = 0; i < 9; ++i) a.M[i] = nm[i];
  for (int i = 0; i < 3; ++i) a.off[i] = noff[i];
  tfm_compute_translation(a);
  tfm_compute_matrix_params(a);
}
MB2_HD bool tfm_inverse(const Tfm &a, Tfm &o) {
  double mi[9];
  if (!mn_inverse<3>(a.M, mi)) return false;
  o.kind = a.kind;
  for (int i = 0; i < 3; ++i) { o.c[i] = a.c[i]; o.ang[i] = 0; }
  for (int i = 0; i < 9; ++i) o.M[i] = mi[i];
  double v[3];
  m3_vec(mi, a.off, v);
  for (int i = 0; i < 3; ++i) o.off[i] = -v[i];
  tfm_compute_translation(o);
  tfm_compute_matrix_params(o);
  return true;
}
MB2_HD void tfm_apply(const Tfm &a, const double *x, double *y) {
  for (int i = 0; i < 3; ++i) {
    double s = 0.0;
    for (int j = 0; j < 3; ++j) s += a.M[3 * i + j] * x[j];
    y[i] = s + a.off[i];
  }
}
// itkTransformUtils.h:22-35
MB2_HD void tfm_center_to_origin(Tfm &a) {
  double off[3] = {a.off[0], a.off[1], a.off[2]};
  double z[3] = {0, 0, 0};
  tfm_set_center(a, z);
  tfm_set_translation(a, off);
}
// itkTransformUtils.h:42-57
MB2_HD void tfm_update_center(Tfm &a, const double *c2) {
  tfm_center_to_origin(a);
  double ic[3] = {-c2[0], -c2[1], -c2[2]};
  tfm_set_center(a, ic);
  double off[3] = {a.off[0], a.off[1], a.off[2]};
  tfm_set_center(a, c2);
  tfm_set_translation(a, off);
}

// ---- vnl_quaternion (x, y, z, r) --------------------------------------------
MB2_HD void quat_rotation(const double *q, double *r) {
  double x = q[0], y = q[1], z = q[2], w = q[3];
  double rt[9];
  double x2 = x * x, y2 = y * y, z2 = z * z, r2 = w * w;
  double xy = x * y, yz = y * z, zx = z * x, rx = w * x, ry = w * y, rz = w * z;
  rt[0] = r2 + x2 - y2 - z2;
  rt[4] = r2 - x2 + y2 - z2;
  rt[8] = r2 - x2 - y2 + z2;
  rt[1] = 2 * (xy + rz);
  rt[2] = 2 * (zx - ry);
  rt[5] = 2 * (yz + rx);
  rt[3] = 2 * (xy - rz);
  rt[6] = 2 * (zx + ry);
  rt[7] = 2 * (yz - rx);
  m3_transpose(rt, r);
}
MB2_HD void quat_euler_angles(const double *q, double *ang) {
  double r[9], rt[9];
  quat_rotation(q, r);
  m3_transpose(r, rt);
  double xy = sqrt(rt[0] * rt[0] + rt[1] * rt[1]);
  const bool regular = xy > 2.220446049250313e-16 * 8.0;
  const double y[3] = {regular ? rt[5] : -rt[7], -rt[2], rt[1]};
  const double x[3] = {regular ? rt[8] : rt[4], xy, rt[0]};
  atan2_3(y, x, ang);
  if (!regular) ang[2] = 0.0;
}
MB2_HD void quat_axis_angle(const double *q, double *axis, double *angle) {
  double mag = sqrt(q[0] * q[0] + q[1] * q[1] + q[2] * q[2]);
  *angle = 2.0 * atan2(mag, q[3]);
  if (mag == 0.0) { axis[0] = 0; axis[1] = 0; axis[2] = 1; }
  else { axis[0] = q[0] / mag; axis[1] = q[1] / mag; axis[2] = q[2] / mag; }
}
MB2_HD void quat_from_axis_angle(const double *axis, double angle, double *q) {
  double a = angle * 0.5, s = sin(a);
  q[0] = s * axis[0]; q[1] = s * axis[1]; q[2] = s * axis[2]; q[3] = cos(a);
}

// Horn's quaternion from the moments of centred point pairs.  Z is the 6x6
// second-moment matrix of z = (a0,a1,a2,b0,b1,b2) with a = initial - mean,
// b = moved - mean.  The per-point matrix Q of CalculateRigidQuaternion
// (itkMirorrRegistrationMethod.txx:1063-1106) is linear in z, so
// sum Q^T Q = sum_i C_i^T Z C_i over its coefficient vectors.  Returns the
// eigenvector of the smallest eigenvalue as (x, y, z, r).
MB2_HD void horn_quaternion(const double *Z, double *q) {
  // tot = sum over the subset of Q^T Q, Q the 4x4 matrix of one pair whose
  // entries are +-1 times the six centred coordinates z_k: entry (j, l) is
  // sum_i sum_{a,b} c(i,j,a) c(i,l,b) Z[a][b] over the non-zero coefficients
  // c (all +-1), written out term by term in that order (i, then a, then b),
  // so every entry is the same sequence of additions as the coefficient form
  double tot[16];
  {  // entry (0, 0)
    double s = 0.0;
    s += Z[0]; s -= Z[3]; s -= Z[18]; s += Z[21]; s += Z[7]; s -= Z[10]; s -= Z[25]; s += Z[28];
    s += Z[14]; s -= Z[17]; s -= Z[32]; s += Z[35];
    tot[0] = s;
  }
  {  // entry (0, 1)
    double s = 0.0;
    s -= Z[8]; s -= Z[11]; s += Z[26]; s += Z[29]; s += Z[13]; s += Z[16]; s -= Z[31];
    s -= Z[34];
    tot[1] = s;
  }
  {  // entry (0, 2)
    double s = 0.0;
    s += Z[2]; s += Z[5]; s -= Z[20]; s -= Z[23]; s -= Z[12]; s -= Z[15]; s += Z[30];
    s += Z[33];
    tot[2] = s;
  }
  {  // entry (0, 3)
    double s = 0.0;
    s -= Z[1]; s -= Z[4]; s += Z[19]; s += Z[22]; s += Z[6]; s += Z[9]; s -= Z[24]; s -= Z[27];
    tot[3] = s;
  }
  {  // entry (1, 0)
    double s = 0.0;
    s -= Z[13]; s += Z[16]; s -= Z[31]; s += Z[34]; s += Z[8]; s -= Z[11]; s += Z[26];
    s -= Z[29];
    tot[4] = s;
  }
  {  // entry (1, 1)
    double s = 0.0;
    s += Z[0]; s -= Z[3]; s -= Z[18]; s += Z[21]; s += Z[14]; s += Z[17]; s += Z[32];
    s += Z[35]; s += Z[7]; s += Z[10]; s += Z[25]; s += Z[28];
    tot[5] = s;
  }
  {  // entry (1, 2)
    double s = 0.0;
    s += Z[1]; s -= Z[4]; s -= Z[19]; s += Z[22]; s -= Z[6]; s -= Z[9]; s -= Z[24]; s -= Z[27];
    tot[6] = s;
  }
  {  // entry (1, 3)
    double s = 0.0;
    s += Z[2]; s -= Z[5]; s -= Z[20]; s += Z[23]; s -= Z[12]; s -= Z[15]; s -= Z[30];
    s -= Z[33];
    tot[7] = s;
  }
  {  // entry (2, 0)
    double s = 0.0;
    s += Z[12]; s -= Z[15]; s += Z[30]; s -= Z[33]; s -= Z[2]; s += Z[5]; s -= Z[20];
    s += Z[23];
    tot[8] = s;
  }
  {  // entry (2, 1)
    double s = 0.0;
    s += Z[6]; s -= Z[9]; s -= Z[24]; s += Z[27]; s -= Z[1]; s -= Z[4]; s -= Z[19]; s -= Z[22];
    tot[9] = s;
  }
  {  // entry (2, 2)
    double s = 0.0;
    s += Z[7]; s -= Z[10]; s -= Z[25]; s += Z[28]; s += Z[14]; s += Z[17]; s += Z[32];
    s += Z[35]; s += Z[0]; s += Z[3]; s += Z[18]; s += Z[21];
    tot[10] = s;
  }
  {  // entry (2, 3)
    double s = 0.0;
    s += Z[8]; s -= Z[11]; s -= Z[26]; s += Z[29]; s -= Z[13]; s -= Z[16]; s -= Z[31];
    s -= Z[34];
    tot[11] = s;
  }
  {  // entry (3, 0)
    double s = 0.0;
    s -= Z[6]; s += Z[9]; s -= Z[24]; s += Z[27]; s += Z[1]; s -= Z[4]; s += Z[19]; s -= Z[22];
    tot[12] = s;
  }
  {  // entry (3, 1)
    double s = 0.0;
    s += Z[12]; s -= Z[15]; s -= Z[30]; s += Z[33]; s -= Z[2]; s -= Z[5]; s -= Z[20];
    s -= Z[23];
    tot[13] = s;
  }
  {  // entry (3, 2)
    double s = 0.0;
    s += Z[13]; s -= Z[16]; s -= Z[31]; s += Z[34]; s -= Z[8]; s -= Z[11]; s -= Z[26];
    s -= Z[29];
    tot[14] = s;
  }
  {  // entry (3, 3)
    double s = 0.0;
    s += Z[14]; s -= Z[17]; s -= Z[32]; s += Z[35]; s += Z[7]; s += Z[10]; s += Z[25];
    s += Z[28]; s += Z[0]; s += Z[3]; s += Z[18]; s += Z[21];
    tot[15] = s;
  }
  double ev[4], vec[16];
  jacobi_eigen<4>(tot, ev, vec);
  q[0] = vec[4 * 1 + 0];
  q[1] = vec[4 * 2 + 0];
  q[2] = vec[4 * 3 + 0];
  q[3] = vec[4 * 0 + 0];
}

// ---- LTS steps ---------------------------------------------------------------
// Working state of one LTS fit (one OptimizeTransform call).
struct LtsState {
  int kind;
  int symmetric;
  double lts_keep;
  Tfm tfm;        // m_Transform
  Tfm t12f, t12b; // half-space transforms (symmetric)
  Tfm fin;        // final_transform (classic) / final_transformF (symmetric)
  Tfm finb;       // final_transformB (symmetric)
  double rc[3];
  double last_params[12];
  double fraction;
  double delta, last_delta;
  int iter;       // completed inner iterations
  int running;    // 1 while the while-condition holds
  int failed;
};

MB2_HD bool lts_continue(const LtsState &s) {
  return s.delta > 1e-3 && (s.iter - 1) < 100 && fabs(s.delta - s.last_delta) > 1e-3;
}

MB2_HD void lts_begin(LtsState &s) {
  for (int i = 0; i < 3; ++i) s.rc[i] = s.tfm.c[i];
  tfm_identity(s.fin, s.kind);
  tfm_set_center(s.fin, s.rc);
  tfm_identity(s.finb, s.kind);
  tfm_set_center(s.finb, s.rc);
  tfm_params(s.fin, s.last_params);
  s.fraction = 1.0;
  s.last_delta = 0.0;
  s.delta = 1.0;
  s.iter = 0;
  s.running = 1;
  s.failed = 0;
}

// Least-squares affine A = Cov(y, x) Cov(x, x)^-1 with x the initial and y the
// moved points (back: the other way), skipping the inverse when
// |det Cov(x, x)| < 1e-4 (itkMirorrRegistrationMethod.txx:871-883).  zn: the
// second moments divided by the subset's size.
MB2_HD void affine_ls_n(const double *zn, bool back, double *rot) {
  double oxy[9], oxx[9];
  MB2_UNROLL
  for (int r = 0; r < 3; ++r)
    MB2_UNROLL
    for (int c = 0; c < 3; ++c) {
      oxy[3 * r + c] = back ? zn[6 * r + 3 + c] : zn[6 * (3 + r) + c];
      oxx[3 * r + c] = back ? zn[6 * (3 + r) + 3 + c] : zn[6 * r + c];
    }
  MB2_UNROLL
  for (int i = 0; i < 9; ++i) rot[i] = oxy[i];
  if (fabs(m3_det(oxx)) >= 1e-4) {
    double inv[9];
    if (mn_inverse<3>(oxx, inv)) m3_mul(oxy, inv, rot);
  }
}

// One inner iteration of the classic fit, after the subset moments are known
// (itkMirorrRegistrationMethod.txx:841-998): T (whose centre is the previous
// subset's barycentre) from the subset; np: the new parameters.  im, mm: the
// subset's barycentres; Z, zn: its second moments, and those divided by its
// size.
MB2_HD void classic_fit(Tfm &T, const double *im, const double *mm, const double *Z,
                        const double *zn, double *np) {
  double mfc[3], ifc[3], rot[9], ri[3];
  MB2_UNROLL
  for (int i = 0; i < 3; ++i) { mfc[i] = mm[i] - T.c[i]; ifc[i] = im[i] - T.c[i]; }
  if (T.kind == KIND_AFFINE) {
    affine_ls_n(zn, false, rot);
    m3_vec(rot, ifc, ri);
    MB2_UNROLL
    for (int i = 0; i < 9; ++i) np[i] = rot[i];
    MB2_UNROLL
    for (int i = 0; i < 3; ++i) np[9 + i] = mfc[i] - ri[i];
  } else {
    double q[4], ang[3];
    horn_quaternion(Z, q);
    quat_rotation(q, rot);
    m3_vec(rot, ifc, ri);
    quat_euler_angles(q, ang);
    MB2_UNROLL
    for (int i = 0; i < 3; ++i) { np[i] = ang[i]; np[3 + i] = mfc[i] - ri[i]; }
  }
  tfm_set_center(T, im);
  tfm_set_params(T, np);
}

MB2_HD void half_step(const double *K, const double *trans, double *m12) {
  double m[16];
  for (int i = 0; i < 16; ++i) m[i] = 0.0;
  for (int r = 0; r < 3; ++r) {
    for (int c = 0; c < 3; ++c) m[4 * r + c] = K[3 * r + c];
    m[4 * r + 3] = trans[r];
  }
  m[15] = 1.0;
  matrix_sqrt4(m, m12);
}

// One inner iteration of the symmetric fit (itkSymMirorrRegistrationMethod.txx:865-1432),
// in stages that each work on one half (forward h = 0, backward h = 1) and see
// the other half's result of the stage before: the device runs the two halves
// on two lane groups at once, exchanging by shuffles.
//   sym_fit      the half's least-squares fit in T; inv: T's inverse matrix
//   sym_mean     T's matrix averaged with the other half's inverse; T moved to
//                centre 0; iT: its inverse
//   sym_half     the matrix and translation averaged with the other half's iT,
//                then the half-way square root m12
//   sym_finish   T from the square root

// im, mm: the subset's barycentres; Z, zn: its second moments, and those
// divided by its size; np: the new parameters (meaningful for h = 0).
MB2_HD void sym_fit(Tfm &T, int h, const double *im, const double *mm, const double *Z,
                    const double *zn, double *np, double *inv) {
  double tr[3], p[12];
  MB2_UNROLL
  for (int i = 0; i < 3; ++i) tr[i] = h ? -(mm[i] - im[i]) : mm[i] - im[i];
  if (T.kind == KIND_AFFINE) {
    double rot[9];
    affine_ls_n(zn, h != 0, rot);
    MB2_UNROLL
    for (int i = 0; i < 9; ++i) np[i] = p[i] = rot[i];
    MB2_UNROLL
    for (int i = 0; i < 3; ++i) np[9 + i] = p[9 + i] = tr[i];
  } else {
    double q[4], ang[3], axis[3], angle, qh[4], ah[3];
    horn_quaternion(Z, q);
    quat_euler_angles(q, ang);
    quat_axis_angle(q, axis, &angle);
    quat_from_axis_angle(axis, h ? -angle : angle, qh);
    quat_euler_angles(qh, ah);
    MB2_UNROLL
    for (int i = 0; i < 3; ++i) {
      np[i] = ang[i];
      np[3 + i] = tr[i];
      p[i] = ah[i];
      p[3 + i] = tr[i];
    }
  }
  tfm_set_center(T, h ? mm : im);
  tfm_set_params(T, p);
  MB2_UNROLL
  for (int i = 0; i < 9; ++i) inv[i] = 0.0;
  mn_inverse<3>(T.M, inv);
}

// T's matrix set to K (affine: the half's own mean; rigid: the orthogonalised
// forward mean, transposed for the backward half).  Returns whether a rigid T
// took it.
MB2_HD bool sym_mean(Tfm &T, int h, const double *K) {
  double k[9];
  if (T.kind == KIND_AFFINE) {
    MB2_UNROLL
    for (int i = 0; i < 9; ++i) k[i] = K[i];
  } else {
    double o[9];
    orthogonalize3(K, o);
    MB2_UNROLL
    for (int r = 0; r < 3; ++r)
      MB2_UNROLL
      for (int c = 0; c < 3; ++c) k[3 * r + c] = h ? o[3 * c + r] : o[3 * r + c];
  }
  return tfm_set_matrix(T, k);
}

MB2_HD void sym_to_origin(Tfm &T, Tfm &iT) {
  const double off[3] = {T.off[0], T.off[1], T.off[2]};
  const double zero[3] = {0, 0, 0};
  tfm_set_center(T, zero);
  tfm_set_translation(T, off);
  tfm_identity(iT, T.kind);
  tfm_inverse(T, iT);
}

MB2_HD void sym_half(const Tfm &T, const double *oM, const double *ot, double *m12) {
  double K[9], t[3];
  MB2_UNROLL
  for (int i = 0; i < 9; ++i) K[i] = (T.M[i] + oM[i]) / 2.0;
  if (T.kind == KIND_RIGID) {
    double o[9];
    orthogonalize3(K, o);
    MB2_UNROLL
    for (int i = 0; i < 9; ++i) K[i] = o[i];
  }
  MB2_UNROLL
  for (int i = 0; i < 3; ++i) t[i] = (T.t[i] + ot[i]) / 2.0;
  half_step(K, t, m12);
}

// T's matrix from the square root, and whether T took it; with reorth, the
// orthogonalised one (SymMirorrRegistrationMethod re-orthogonalises both halves
// when one is rejected, :1327-1342).
MB2_HD bool sym_finish(Tfm &T, const double *m12, bool reorth) {
  double k[9];
  MB2_UNROLL
  for (int r = 0; r < 3; ++r)
    MB2_UNROLL
    for (int c = 0; c < 3; ++c) k[3 * r + c] = m12[4 * r + c];
  if (reorth) {
    double o[9];
    orthogonalize3(k, o);
    MB2_UNROLL
    for (int i = 0; i < 9; ++i) k[i] = o[i];
  }
  return tfm_set_matrix(T, k);
}

// The loop's parameter change; the symmetric method compares with the last
// parameters, the classic one with the identity's throughout.
MB2_HD void lts_delta(LtsState &s, const double *np) {
  double d = 0.0;
  MB2_UNROLL
  for (int i = 0; i < 12; ++i)
    if (i < 6 || s.kind == KIND_AFFINE) {
      const double e = s.last_params[i] - np[i];
      d += e * e;
      if (s.symmetric) s.last_params[i] = np[i];
    }
  s.last_delta = s.delta;
  s.delta = d;
}

// After the inner loop: m_Transform->Compose(final, true) (classic) or the
// half-space composition (symmetric, itkSymMirorrRegistrationMethod.txx:1452-1462).
MB2_HD void lts_finish(LtsState &s) {
  if (!s.symmetric) {
    tfm_compose(s.tfm, s.fin, true);
  } else {
    tfm_compose(s.t12f, s.fin, true);
    tfm_compose(s.t12b, s.finb, true);
    Tfm ib;
    tfm_inverse(s.t12b, ib);
    tfm_identity(s.tfm, s.tfm.kind);
    tfm_compose(s.tfm, ib, true);
    tfm_compose(s.tfm, s.t12f, false);
  }
}

// ComputeHalfSpaceTransforms (itkSymMirorrRegistrationMethod.txx:139-201).
MB2_HD void half_space(const Tfm &t, Tfm &f, Tfm &b) {
  double m[16], mi[16], m12[16], im12[16];
  for (int i = 0; i < 16; ++i) m[i] = 0.0;
  for (int r = 0; r < 3; ++r) {
    for (int c = 0; c < 3; ++c) m[4 * r + c] = t.M[3 * r + c];
    m[4 * r + 3] = t.t[r];
  }
  m[15] = 1.0;
  matrix_sqrt4(m, m12);
  affine4_inverse(m, mi);
  matrix_sqrt4(mi, im12);
  tfm_identity(f, t.kind);
  tfm_identity(b, t.kind);
  double k3[9], l3[9];
  for (int r = 0; r < 3; ++r)
    for (int c = 0; c < 3; ++c) { k3[3 * r + c] = m12[4 * r + c]; l3[3 * r + c] = im12[4 * r + c]; }
  if (!tfm_set_matrix(f, k3)) { double o[9]; orthogonalize3(k3, o); tfm_set_matrix(f, o); }
  if (!tfm_set_matrix(b, l3)) { double o[9]; orthogonalize3(l3, o); tfm_set_matrix(b, o); }
  double tf[3] = {m12[3], m12[7], m12[11]}, tb[3] = {im12[3], im12[7], im12[11]};
  tfm_set_translation(f, tf);
  tfm_set_translation(b, tb);
}

}  // namespace mb2
