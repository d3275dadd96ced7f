// Largest eigenpair of a symmetric 3x3 matrix in FP64 by cyclic Jacobi rotations (Golub & Van Loan,
// "Matrix Computations", Algorithm 8.5.3). Replaces gsl_eigen_symmv + sort (src/parameter_order.cpp:19-37),
// which the reference uses to get S (largest eigenvalue of Q) and the director (its eigenvector).
//
// The rotations are written out for the three index pairs, so the matrix lives in registers (indexed by loop variables
// it went to local memory, and one thread's solve took 5 us of every measured sweep), and only the upper triangle is
// kept: t = h sgn(d) / (|d| + sqrt(d^2 + h^2)) with d = a_qq - a_pp, h = 2 a_pq is the book's tangent with one division.
#pragma once
#include <math.h>

namespace mcl {

// One rotation in the plane (p, q); r is the third axis. Symmetric entries: diagonal app, aqq, off-diagonal apq, arp,
// arq; vp, vq are the eigenvector columns.
__host__ __device__ inline void jacobi_rotate(double &app, double &aqq, double &apq, double &arp, double &arq,
                                              double (&vp)[3], double (&vq)[3]) {
  if (apq == 0) return;
  const double d = aqq - app, h = 2 * apq;
  const double t = d == 0 ? 1.0 : (d > 0 ? h : -h) / (fabs(d) + sqrt(d * d + h * h));
#ifdef __CUDA_ARCH__
  const double c = rsqrt(t * t + 1);
#else
  const double c = 1 / sqrt(t * t + 1);
#endif
  const double s = t * c;
  if (d == 0) {  // t = 1: the general form of the diagonal update
    const double m = 0.5 * (app + aqq);
    app = m - apq;
    aqq = m + apq;
  } else {
    app -= t * apq;
    aqq += t * apq;
  }
  apq = 0;
  const double rp = arp, rq = arq;
  arp = c * rp - s * rq;
  arq = s * rp + c * rq;
  for (int k = 0; k < 3; k++) {
    const double a = vp[k], b = vq[k];
    vp[k] = c * a - s * b;
    vq[k] = s * a + c * b;
  }
}

__host__ __device__ inline double largest_eigen3(const double q6[6], double vec[3]) {
  double a00 = q6[0], a01 = q6[1], a02 = q6[2], a11 = q6[3], a12 = q6[4], a22 = q6[5];
  double v0[3] = {1, 0, 0}, v1[3] = {0, 1, 0}, v2[3] = {0, 0, 1};
  for (int sweep = 0; sweep < 50; sweep++) {
    const double off = a01 * a01 + a02 * a02 + a12 * a12;
    const double dg = a00 * a00 + a11 * a11 + a22 * a22;
    if (off == 0 || off <= 1e-34 * dg) break;
    jacobi_rotate(a00, a11, a01, a02, a12, v0, v1);
    jacobi_rotate(a00, a22, a02, a01, a12, v0, v2);
    jacobi_rotate(a11, a22, a12, a01, a02, v1, v2);
  }
  const bool one = a11 > a00;
  double best = one ? a11 : a00;
  const bool two = a22 > best;
  if (two) best = a22;
  for (int k = 0; k < 3; k++) vec[k] = two ? v2[k] : (one ? v1[k] : v0[k]);
  return best;
}

}  // namespace mcl
