// Element work with 8 lanes per element ("octet"): lane t is the element's node
// with the natural-coordinate sign bits t and its Gauss point with the same
// bits.  Nodal values become values or reference derivatives at the Gauss
// points, and Gauss-point terms become nodal sums, by exchanges along the three
// bits (the trilinear shape functions are a tensor product), 6 shuffled doubles
// a field; a lane then loads one node and holds one Gauss point, instead of
// every thread loading all 8 nodes or walking through all 8 points.
#pragma once

#include <cuda_runtime.h>

#include "c3d8_device.cuh"
#include "rows.cuh"

namespace ufc {
namespace {

constexpr unsigned kAllLanes = 0xffffffffu;
constexpr double kGaussOwn = 0.5 + 0.5 * 0.57735026918962576451;    // (1 + g) / 2: node and Gauss point on one side
constexpr double kGaussOther = 0.5 - 0.5 * 0.57735026918962576451;  // (1 - g) / 2

struct Octet {
  double s0, s1, s2;  // half the lane's signs: +-1/2
  __device__ __forceinline__ explicit Octet(int t)
      : s0(t & 1 ? 0.5 : -0.5), s1(t & 2 ? 0.5 : -0.5), s2(t & 4 ? 0.5 : -0.5) {}

  // d v / d (xi, eta, zeta) at the lane's Gauss point of the field with nodal value v
  __device__ __forceinline__ void gradient(double v, double& d0, double& d1, double& d2) const {
    double o = __shfl_xor_sync(kAllLanes, v, 1);
    const double D = s0 * (v - o), I = kGaussOwn * v + kGaussOther * o;
    o = __shfl_xor_sync(kAllLanes, I, 2);
    const double oD = __shfl_xor_sync(kAllLanes, D, 2);
    const double IE = s1 * (I - o), II = kGaussOwn * I + kGaussOther * o, DI = kGaussOwn * D + kGaussOther * oD;
    const double a = __shfl_xor_sync(kAllLanes, II, 4), b = __shfl_xor_sync(kAllLanes, IE, 4),
                 c = __shfl_xor_sync(kAllLanes, DI, 4);
    d2 = s2 * (II - a);
    d1 = kGaussOwn * IE + kGaussOther * b;
    d0 = kGaussOwn * DI + kGaussOther * c;
  }

  // The transpose: sum over the Gauss points of dN/d(xi, eta, zeta) . F at the lane's node
  __device__ __forceinline__ double divergence(double f0, double f1, double f2) const {
    const double a = __shfl_xor_sync(kAllLanes, f2, 4), b = __shfl_xor_sync(kAllLanes, f1, 4),
                 c = __shfl_xor_sync(kAllLanes, f0, 4);
    const double C = s2 * (f2 + a), A = kGaussOwn * f1 + kGaussOther * b, B = kGaussOwn * f0 + kGaussOther * c;
    // interpolation of C and derivative of A share an exchange: what the other lane needs of both
    const double P = kGaussOwn * C + s1 * A + __shfl_xor_sync(kAllLanes, kGaussOther * C - s1 * A, 2);
    const double Q = kGaussOwn * B + kGaussOther * __shfl_xor_sync(kAllLanes, B, 2);
    return kGaussOwn * P + s0 * Q + __shfl_xor_sync(kAllLanes, kGaussOther * P - s0 * Q, 1);
  }

  // Extrapolation of Gauss-point values to the lane's node: the inverse of the
  // trilinear interpolation, prod_d (1 + sqrt(3) s_d,node s_d,gp) / 2.
  __device__ __forceinline__ double extrapolate(double v) const {
    constexpr double own = 0.5 + 0.5 * 1.7320508075688772935, other = 0.5 - 0.5 * 1.7320508075688772935;
    v = own * v + other * __shfl_xor_sync(kAllLanes, v, 1);
    v = own * v + other * __shfl_xor_sync(kAllLanes, v, 2);
    return own * v + other * __shfl_xor_sync(kAllLanes, v, 4);
  }

  // J^-1 (inv[3 i + d] = d xi_d / d x_i) and det J at the lane's Gauss point from its node's coordinates.
  __device__ __forceinline__ double jacobian(const double X[3], double inv[9]) const {
    double J[9];  // J[3 d + i] = d x_i / d xi_d
#pragma unroll
    for (int i = 0; i < 3; ++i) gradient(X[i], J[i], J[3 + i], J[6 + i]);
    const double c0 = J[4] * J[8] - J[5] * J[7], c3 = J[5] * J[6] - J[3] * J[8], c6 = J[3] * J[7] - J[4] * J[6];
    const double det = J[0] * c0 + J[1] * c3 + J[2] * c6;
    const double id = 1.0 / det;
    inv[0] = c0 * id;
    inv[1] = (J[2] * J[7] - J[1] * J[8]) * id;
    inv[2] = (J[1] * J[5] - J[2] * J[4]) * id;
    inv[3] = c3 * id;
    inv[4] = (J[0] * J[8] - J[2] * J[6]) * id;
    inv[5] = (J[2] * J[3] - J[0] * J[5]) * id;
    inv[6] = c6 * id;
    inv[7] = (J[1] * J[6] - J[0] * J[7]) * id;
    inv[8] = (J[0] * J[4] - J[1] * J[3]) * id;
    return det;
  }

  // Voigt strain (engineering shear) at the lane's Gauss point of the displacement u of its node.
  __device__ __forceinline__ void strain(const double inv[9], const double u[3], double e[6]) const {
    double H[9];  // H[3 i + j] = d u_i / d x_j
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      double d0, d1, d2;
      gradient(u[i], d0, d1, d2);
#pragma unroll
      for (int j = 0; j < 3; ++j) H[3 * i + j] = inv[3 * j] * d0 + inv[3 * j + 1] * d1 + inv[3 * j + 2] * d2;
    }
    e[0] = H[0];
    e[1] = H[4];
    e[2] = H[8];
    e[3] = H[1] + H[3];
    e[4] = H[5] + H[7];
    e[5] = H[6] + H[2];
  }

  // Nodal forces sum_gp w B^T s of the lane's node, s the Voigt stress at its Gauss point.
  __device__ __forceinline__ void nodal_force(const double inv[9], double w, const double s[6], double f[3]) const {
    const int V[3][3] = {{0, 3, 5}, {3, 1, 4}, {5, 4, 2}};
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const double a = w * s[V[i][0]], b = w * s[V[i][1]], c = w * s[V[i][2]];
      f[i] = divergence(a * inv[0] + b * inv[3] + c * inv[6], a * inv[1] + b * inv[4] + c * inv[7],
                        a * inv[2] + b * inv[5] + c * inv[8]);
    }
  }
};

}  // namespace
}  // namespace ufc
