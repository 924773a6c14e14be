// chem_implicit.cuh — the point-implicit chemistry systems of mechanisms whose
// structure is known at build time (mech_h2air9.cuh), in registers.
//
// (d I - dt J) x = b with J = d omega / d(rho Y), restricted to the NA species
// that take part in reactions: an inert species' row and column hold only its
// diagonal. The generic form (chem.cuh: chemistry_rates, chemistry_jacobian,
// lu_factor) walks stoichiometric tables in runtime loops and keeps the rates,
// the n_spec^2 matrix and the pivots in local memory; here every index is a
// literal, so the matrix lives in registers, each reaction touches the entries
// of its own species, and a pivot other than the diagonal is a branch that
// (d I - dt J) seldom takes. Bound by FP64 issue at 8 warps per SM (255
// registers): DPLUR's first pass with the factorisation of 64 x 60 x 48
// cells took 826 us with the generic form, 172 with this one; a sweep, which solves with
// the stored factors, 158 and 132.
#pragma once
#include <utility>

#include "mech_h2air9.cuh"

namespace ostc {

// f(integral_constant<0>) .. f(integral_constant<N-1>): the elimination's outer loop, whose
// inner bounds depend on the step, as literals (left to the unroller, the matrix went to
// local memory)
template <class F, int... I>
__device__ __forceinline__ void static_for(F &&f, std::integer_sequence<int, I...>) {
  (f(std::integral_constant<int, I>{}), ...);
}

// LU factors of A in place with partial pivoting (the largest magnitude of the
// column, the first of equals, as lu_factor); unit lower factor, and the
// reciprocals of the pivots on the diagonal. Returns the pivot rows, 4 bits
// each.
template <int N>
__device__ __forceinline__ unsigned lu_factor_reg(double (&A)[N][N]) {
  static_assert(N <= 8, "pivot rows of four bits in one word");
  unsigned piv = 0;
  static_for([&](auto step) {
    constexpr int n = decltype(step)::value;
    int ik = n;
    double best = fabs(A[n][n]);
#pragma unroll
    for (int m = n + 1; m < N; ++m) {
      if (fabs(A[m][n]) > best) {
        best = fabs(A[m][n]);
        ik = m;
      }
    }
    piv |= (unsigned)ik << (4 * n);
    if (ik != n) {
#pragma unroll
      for (int m = n + 1; m < N; ++m) {
        if (ik == m) {
#pragma unroll
          for (int t = 0; t < N; ++t) {
            const double mid = A[m][t];
            A[m][t] = A[n][t];
            A[n][t] = mid;
          }
        }
      }
    }
    const double inv = 1.0 / A[n][n];
    A[n][n] = inv;
#pragma unroll
    for (int m = n + 1; m < N; ++m) {
      A[m][n] *= inv;
#pragma unroll
      for (int t = n + 1; t < N; ++t) A[m][t] -= A[m][n] * A[n][t];
    }
  }, std::make_integer_sequence<int, N>{});
  return piv;
}

// the pivots of a factorisation that kept every diagonal
template <int N>
__host__ __device__ constexpr unsigned lu_no_pivots() {
  unsigned p = 0;
  for (int n = 0; n < N; ++n) p |= (unsigned)n << (4 * n);
  return p;
}

// b <- A^-1 b with the factors and pivots of lu_factor_reg
template <int N>
__device__ __forceinline__ void lu_apply_reg(const double (&A)[N][N], unsigned piv, double (&b)[N]) {
  if (piv != lu_no_pivots<N>()) {
#pragma unroll
    for (int n = 0; n < N; ++n) {
      const int ik = (piv >> (4 * n)) & 15;
#pragma unroll
      for (int m = n + 1; m < N; ++m) {
        if (ik == m) {
          const double mid = b[m];
          b[m] = b[n];
          b[n] = mid;
        }
      }
    }
  }
#pragma unroll
  for (int m = 1; m < N; ++m)
#pragma unroll
    for (int t = 0; t < m; ++t) b[m] -= A[m][t] * b[t];
#pragma unroll
  for (int m = N - 1; m >= 0; --m) {
#pragma unroll
    for (int t = m + 1; t < N; ++t) b[m] -= A[m][t] * b[t];
    b[m] *= A[m][m];
  }
}

// A <- d I - dt J over the active species from the sensitivities Z (in place);
// columns of absent species (Y_n <= 1e-25) hold their diagonal alone
__device__ __forceinline__ void implicit_matrix(double (&Z)[mech_h2air9::NA][mech_h2air9::NA], double rho,
                                                const double *Y, double dt, double d) {
  using namespace mech_h2air9;
#pragma unroll
  for (int n = 0; n < NA; ++n) {
    const double y = Y[active(n)];
    const double s = y > 1e-25 ? 1e3 * dt / (rho * y) : 0.0;
#pragma unroll
    for (int m = 0; m < NA; ++m) {
      const double a = -c_p.mw[active(m)] * (s * Z[m][n]);
      Z[m][n] = m == n ? d + a : a;
    }
  }
}

// (d I - dt J) b = b in place for the species right-hand side b[NS]
__device__ __forceinline__ void h2air9_implicit_solve(double rho, double T, const double *Y, double dt, double *b) {
  using namespace mech_h2air9;
  double wd[NA], Z[NA][NA], x[NA];
  production_jacobian(rho, T, Y, wd, Z);
  implicit_matrix(Z, rho, Y, dt, 1.0);
#pragma unroll
  for (int m = 0; m < NA; ++m) x[m] = b[active(m)];
  const unsigned piv = lu_factor_reg<NA>(Z);
  lu_apply_reg<NA>(Z, piv, x);
#pragma unroll
  for (int m = 0; m < NA; ++m) b[active(m)] = x[m];
}

}  // namespace ostc
