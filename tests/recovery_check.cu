// Device check of the building blocks of the primitive recovery, run by test_recovery_gpu.py:
//   quotient, root: div_fast and sqrt_fast against CUDA's division and square root (which are
//     correctly rounded), in units in the last place, over their operands' ranges, and what they
//     give outside them;
//   solver: energy_from_conserved_n on states whose Newton divisors leave the range of div_fast, and
//     c_s^2 at every energy.
// Prints one line per check and the number of failures.
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include <random>
#include <vector>

#include "gvh_physics.cuh"

using namespace gvh;

__global__ void quotient(int n, const double *a, const double *b, double *fast, double *ieee) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  fast[i] = div_fast(a[i], b[i]);
  ieee[i] = a[i] / b[i];
}
__global__ void root(int n, const double *a, double *fast, double *ieee) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  fast[i] = sqrt_fast(a[i]);
  ieee[i] = sqrt(a[i]);
}
// state i: guess g[i], M0, M, Pi
__global__ void solve(int n, const double *s, double *e, int *bad) {
  eos_table_load<EOS_QCD>();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const GuessEos g = guess_eos<EOS_QCD>(s[4 * i]);
  double m0[1] = {s[4 * i + 1]}, m[1] = {s[4 * i + 2]}, pi[1] = {s[4 * i + 3]}, r[1];
  bool b = false;
  energy_from_conserved_n<EOS_QCD, 1>(g, m0, m, pi, r, b);
  e[i] = r[0];
  bad[i] = b;
}
// c_s^2 of a cell, and with the IEEE division
__global__ void guess(int n, const double *e, double *fast, double *ieee) {
  eos_table_load<EOS_QCD>();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  fast[i] = guess_cs2<EOS_QCD>(guess_eos<EOS_QCD>(e[i]));
  ieee[i] = sound_speed2<EOS_QCD>(e[i]);
}

template <class T>
struct Dev {
  T *p = nullptr;
  size_t n;
  explicit Dev(size_t n_) : n(n_) { cudaMalloc(&p, n * sizeof(T)); }
  explicit Dev(const std::vector<T> &v) : Dev(v.size()) { cudaMemcpy(p, v.data(), n * sizeof(T), cudaMemcpyHostToDevice); }
  std::vector<T> get() const {
    std::vector<T> v(n);
    cudaMemcpy(v.data(), p, n * sizeof(T), cudaMemcpyDeviceToHost);
    return v;
  }
  ~Dev() { cudaFree(p); }
};

static int64_t ordered(double x) {  // consecutive doubles are consecutive integers
  int64_t k;
  memcpy(&k, &x, 8);
  return k < 0 ? INT64_MIN - k : k;
}
static double ulps(double a, double b) {
  if (isnan(a) || isnan(b)) return isnan(a) && isnan(b) ? 0 : INFINITY;
  return fabs((double)ordered(a) - (double)ordered(b));
}

static int failures = 0;
static void check(const char *what, bool ok, double value) {
  printf("%s %s %g\n", ok ? "ok" : "FAIL", what, value);
  failures += !ok;
}

static std::vector<double> run_quotient(const std::vector<double> &a, const std::vector<double> &b,
                                        std::vector<double> *ieee = nullptr) {
  Dev<double> da(a), db(b), f(a.size()), q(a.size());
  quotient<<<(int)((a.size() + 255) / 256), 256>>>((int)a.size(), da.p, db.p, f.p, q.p);
  if (ieee) *ieee = q.get();
  return f.get();
}
static std::vector<double> run_root(const std::vector<double> &a, std::vector<double> *ieee = nullptr) {
  Dev<double> da(a), f(a.size()), q(a.size());
  root<<<(int)((a.size() + 255) / 256), 256>>>((int)a.size(), da.p, f.p, q.p);
  if (ieee) *ieee = q.get();
  return f.get();
}

int main() {
  std::mt19937_64 rng(7);
  auto mantissa = [&] { return 1.0 + (double)(rng() >> 12) * 0x1p-52; };  // [1, 2)
  auto sign = [&] { return rng() & 1 ? 1.0 : -1.0; };
  const int kPer = 256;

  // Quotients: |a| >= 2^-960 (the residual's products stay normal), |b| in [2^-1022, 2^1021), the
  // quotient normal. Both results lie within a fraction of an ulp of the exact quotient on either
  // side: they differ by at most one.
  {
    std::vector<double> a, b, want;
    for (int eb = -1022; eb < 1021; eb += 7)
      for (int eq = -1020; eq < 1022; eq += 31) {
        const int ea = eb + eq;
        if (ea < -960 || ea > 1022) continue;
        for (int k = 0; k < kPer / 8; ++k) {
          a.push_back(sign() * ldexp(mantissa(), ea));
          b.push_back(sign() * ldexp(mantissa(), eb));
        }
      }
    const std::vector<double> got = run_quotient(a, b, &want);
    double worst = 0;
    for (size_t i = 0; i < got.size(); ++i) worst = fmax(worst, ulps(got[i], want[i]));
    check("quotients over the exponents, ulp", worst <= 1, worst);
    // divisors and numerators of the solver's size, mantissas next to the powers of two
    a.clear(); b.clear();
    for (int k = 0; k < 1 << 20; ++k) {
      auto edge = [&] { return k & 1 ? mantissa() : rng() & 1 ? 1.0 + (double)(rng() % 8) * 0x1p-52 : 2.0 - (double)(1 + rng() % 8) * 0x1p-52; };
      a.push_back(sign() * ldexp(edge(), (int)(rng() % 41) - 20));
      b.push_back(ldexp(edge(), (int)(rng() % 41) - 20));
    }
    const std::vector<double> got2 = run_quotient(a, b, &want);
    worst = 0;
    for (size_t i = 0; i < got2.size(); ++i) worst = fmax(worst, ulps(got2[i], want[i]));
    check("quotients of ordinary size, ulp", worst <= 1, worst);
  }
  // Square roots of every normal number.
  {
    std::vector<double> a, want;
    for (int e = -1022; e <= 1023; ++e)
      for (int k = 0; k < kPer; ++k)
        a.push_back(ldexp(k < 8 ? 1.0 + k * 0x1p-52 : k < 16 ? 2.0 - (k - 7) * 0x1p-52 : mantissa(), e));
    const std::vector<double> got = run_root(a, &want);
    double worst = 0;
    for (size_t i = 0; i < got.size(); ++i) worst = fmax(worst, ulps(got[i], want[i]));
    check("square roots over the exponents, ulp", worst <= 1, worst);
  }
  // Outside the ranges.
  {
    const double sub = 0x1p-1030, inf = INFINITY;
    const std::vector<double> a = {1, 1, 1, inf, NAN, 1, 0, 1, inf, 1, -3};
    const std::vector<double> b = {0, sub, inf, 2, 1, NAN, 0, -sub, inf, 0x1.1p1022, 0x1.8p1023};
    const std::vector<double> got = run_quotient(a, b);
    bool ok = true;
    for (int i = 0; i < 9; ++i) ok = ok && isnan(got[i]);
    check("NaN for a divisor 0, subnormal, infinite or NaN, a numerator infinite or NaN", ok, 0);
    check("0 for a divisor above 2^1022", got[9] == 0 && got[10] == 0, got[9]);
    const std::vector<double> z = run_quotient({0.0, -0.0, 0.0}, {3.0, 3.0, -0x1p-1022});
    check("0 for a numerator 0", z[0] == 0 && z[1] == 0 && z[2] == 0, z[0]);
    // numerators below 2^-960: within 2^-36 of the quotient or 2^-1022, whichever is more
    std::vector<double> sa, sb, want;
    for (int k = 0; k < 4096; ++k) {
      sa.push_back(sign() * ldexp(mantissa(), -961 - (int)(rng() % 112)));
      sb.push_back(ldexp(mantissa(), (int)(rng() % 41) - 20));
    }
    const std::vector<double> sg = run_quotient(sa, sb, &want);
    double worst = 0;
    for (size_t i = 0; i < sg.size(); ++i) worst = fmax(worst, fabs(sg[i] - want[i]) / fmax(fabs(want[i]) * 0x1p-36, 0x1p-1022));
    check("small numerators", worst <= 1, worst);
    const std::vector<double> r = run_root({0.0, sub, -1.0, inf, NAN});
    ok = true;
    for (double x : r) ok = ok && isnan(x);
    check("NaN for the root of 0, a subnormal, a negative number, infinity or NaN", ok, 0);
  }
  // Solver. With a huge Pi, A = H = Pi and the solution is e = B / Pi, B = M0 (M0 + Pi) - M. Whatever
  // the size of the divisors (about Pi^2), a solve is handed to the general form or right (to the
  // stop test's 1e-3; the tolerance adds the Newton step after it).
  {
    std::vector<double> s, want;
    for (double Pi = 1e100; Pi < 1.3e154; Pi *= 1.05)
      for (double root : {0.3, 0.7}) {
        const double M0 = 10;
        s.insert(s.end(), {0.2, M0, M0 * (M0 + Pi) - root * Pi, Pi});
        want.push_back(root);
      }
    s.insert(s.end(), {0.2, 10, 10 * (10 + 1.3e154), 1.3e154});  // the first divisor is 2^1022.9
    want.push_back(0);
    Dev<double> ds(s), e(want.size());
    Dev<int> bad(want.size());
    solve<<<(int)((want.size() + 127) / 128), 128>>>((int)want.size(), ds.p, e.p, bad.p);
    const std::vector<double> ge = e.get();
    const std::vector<int> gb = bad.get();
    double wrong = 0;
    for (size_t i = 0; i < want.size(); ++i) wrong += !gb[i] && !(fabs(ge[i] - want[i]) <= 2e-3 * want[i]);
    check("solves with divisors of any size: wrong and not handed on", wrong == 0, wrong);
  }
  {
    std::vector<double> e;
    for (double x = 1e-7; x < 5e24; x *= 1.01) e.push_back(x);
    Dev<double> de(e), fast(e.size()), ieee(e.size());
    guess<<<(int)((e.size() + 127) / 128), 128>>>((int)e.size(), de.p, fast.p, ieee.p);
    const std::vector<double> f = fast.get(), q = ieee.get();
    double worst = 0;
    for (size_t i = 0; i < e.size(); ++i) worst = fmax(worst, ulps(f[i], q[i]));
    check("c_s^2 of the guess, ulp", worst <= 1, worst);
  }
  const cudaError_t err = cudaDeviceSynchronize();
  check(cudaGetErrorString(err), err == cudaSuccess, 0);
  printf("%d failures\n", failures);
  return failures ? 1 : 0;
}
