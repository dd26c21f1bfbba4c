// Prolate spheroidal wave function psi_{alpha,0}(c, nu), normalised to 1 at
// nu = 0 and zero for |nu| >= 1: the grdsf() of yandasoft's gridders
// (askap/gridding/SphFuncVisGridder.h:101, constructed as
// SpheroidalFunction(pi*support, alpha) at SphFuncVisGridder.cc:47).  The
// class itself is in the un-vendored base-scimath library; the method is the
// Legendre-series eigenvector expansion that the reference documents in
// apps/gridderExperiments.cc:180-260.
#pragma once
#include <vector>

namespace yg {

// The Legendre series of a Spheroidal as plain numbers, passed by value to the
// kernel that evaluates it: P_l^m by the upward recurrence
// P_l = a[l - m - 2] (x P_{l-1} - b[l - m - 2] P_{l-2}).
struct SphSeries {
  static constexpr int kTerms = 16;
  int m = 0, nterms = 0;
  double alpha = 0, sum0 = 1;
  double coeff[kTerms] = {};
  double pmm[2] = {};                    // P_k^k from P_{k-1}^{k-1}: -pmm[k - 1] sqrt(1 - x^2), k = 1..m
  double a[2 * kTerms] = {}, b[2 * kTerms] = {};
};

class Spheroidal {
 public:
  Spheroidal(double c, double alpha, int nterms = 16);
  double operator()(double nu) const;
  SphSeries series_tables() const;

 private:
  double series(double eta) const;
  double alpha_;
  int m_;
  int nterms_;
  std::vector<double> coeffs_;
  double sum0_;
};

}  // namespace yg
