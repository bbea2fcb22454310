// Rounding of the FP32 SRT update over a run, on the host: a smooth flow in a
// closed box (bounce-back on every face), stepped in FP32 by the library's update
// and by the plain order of its operations with fused multiply-adds (the even half
// of the equilibrium, the odd half added, the difference, the relaxation), both
// against the library's update in FP64.  Prints the rms velocity error of both
// over the seeds, per relaxation time.
#include "lbm_d3q19.cuh"

#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

using namespace lbm;

struct Library {
  template <class V, class Emit>
  static void collide(const V (&f)[Q], const PairState<V>& ps, V ux, V uy, V uz, V w, Emit&& emit) {
    collide_srt_pairs<false, V>(f, ps, ux, uy, uz, w, emit);
  }
};
struct Plain {
  template <class V, class Emit>
  static void collide(const V (&f)[Q], const PairState<V>& ps, V ux, V uy, V uz, V w, Emit&& emit) {
    const V u2 = fma_(uz, uz, fma_(uy, uy, ux * ux)), c0 = fma_(V(-1.5), u2, V(1));
    static_for<0, Q>([&](auto qc) {
      constexpr int q = decltype(qc)::value;
      const V eu = V(cx(q)) * ux + V(cy(q)) * uy + V(cz(q)) * uz;
      const V wr = ps.rho * weight<V>(q);
      const V even = wr * fma_(V(4.5) * eu, eu, c0);
      emit(qc, fma_(fma_(V(3) * wr, eu, even) - f[q], w, f[q]));
    });
  }
};

template <class V, class Update>
struct Box {
  int n;
  V w;
  std::vector<V> f, g, u[3];
  long at(int x, int y, int z) const { return x + (long)n * (z + (long)n * y); }
  void step(bool first) {
    const long N = (long)n * n * n;
    for (int y = 0; y < n; ++y)
      for (int z = 0; z < n; ++z)
        for (int x = 0; x < n; ++x) {
          V p[Q];
          const long c = at(x, y, z);
          static_for<0, Q>([&](auto qc) {
            constexpr int q = decltype(qc)::value;
            const int xs = x - cx(q), ys = y - cy(q), zs = z - cz(q);
            const bool in = xs >= 0 && xs < n && ys >= 0 && ys < n && zs >= 0 && zs < n;
            p[q] = first ? f[q * N + c] : (in ? f[q * N + at(xs, ys, zs)] : f[opp(q) * N + c]);
          });
          PairState<V> ps;
          make_pairs<V>(p, ps);
          const V inv = vrcp(ps.rho_full);
          const V ux = ps.jx * inv, uy = ps.jy * inv, uz = ps.jz * inv;
          u[0][c] = ux;
          u[1][c] = uy;
          u[2][c] = uz;
          Update::collide(p, ps, ux, uy, uz, w,
                          [&](auto qc, V v) { g[decltype(qc)::value * N + c] = v; });
        }
    std::swap(f, g);
  }
  void run(const std::vector<float>& start, int edge, float tau, int steps) {
    n = edge;
    w = vrcp((V)tau);
    f.assign(start.begin(), start.end());
    g = f;
    for (auto& v : u) v.resize(start.size() / Q);
    for (int s = 0; s <= steps; ++s) step(s == 0);
  }
};

template <class A, class B>
double rms(const A& a, const B& b) {
  double s = 0;
  for (int i = 0; i < 3; ++i)
    for (size_t c = 0; c < a.u[i].size(); ++c) {
      const double d = (double)a.u[i][c] - b.u[i][c];
      s += d * d;
    }
  return std::sqrt(s / a.u[0].size());
}

int main() {
  constexpr int n = 24, steps = 100;
  for (float tau : {0.55f, 0.6f, 0.7f, 0.9f}) {
    double lib = 0, plain = 0;
    for (int seed = 1; seed <= 4; ++seed) {
      std::mt19937 g(seed);
      double k[4][3], ph[4][3];
      for (int i = 0; i < 4; ++i)
        for (int a = 0; a < 3; ++a) {
          k[i][a] = M_PI * (1 + (int)(g() % 3)) / (n - 1);
          ph[i][a] = 2 * M_PI * (g() / 4294967296.0);
        }
      std::vector<float> f((size_t)Q * n * n * n);
      for (int y = 0; y < n; ++y)
        for (int z = 0; z < n; ++z)
          for (int x = 0; x < n; ++x) {
            double v[4];
            for (int i = 0; i < 4; ++i)
              v[i] = (i < 3 ? 0.05 : 5e-4) * std::sin(k[i][0] * x + ph[i][0]) *
                     std::sin(k[i][1] * y + ph[i][1]) * std::sin(k[i][2] * z + ph[i][2]);
            const double u2 = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
            for (int q = 0; q < Q; ++q) {
              const double eu = cx(q) * v[0] + cy(q) * v[1] + cz(q) * v[2];
              f[q * (size_t)(n * n * n) + x + n * (z + n * y)] = (float)(
                  weight<double>(q) * (1 + v[3]) * (1 + 3 * eu + 4.5 * eu * eu - 1.5 * u2));
            }
          }
      Box<double, Library> r;
      Box<float, Library> a;
      Box<float, Plain> b;
      r.run(f, n, tau, steps);
      a.run(f, n, tau, steps);
      b.run(f, n, tau, steps);
      lib += rms(a, r) / 4;
      plain += rms(b, r) / 4;
    }
    std::printf("%g %.6e %.6e\n", tau, lib, plain);
  }
}
