// Host build of pieces of the device code whose forms were changed for speed,
// against the plain forms, bit by bit: the hill climb that tests four neighbours
// at a time (pacific_b200/csrc/gjk.cuh), and the divisions, the motion test and
// the cell index of the kicks (pacific_b200/csrc/common.cuh).  Compiled and run
// by tests/test_arith_cpu.py; prints a summary line and exits 1 on failure.
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include "../pacific_b200/csrc/gjk.cuh"

using namespace gg;

// the neighbours one by one
static int climb(const LocalBody<double>& B, V3<double> v, int cur) {
  if (!(norm2(v) > kEpsilon * kEpsilon)) return -1;
  auto at = [&](int i) { return v3<double>(B.verts[3 * i], B.verts[3 * i + 1], B.verts[3 * i + 2]); };
  int last = -1;
  double h = dot(at(cur), v);
  for (int moves = 0; moves < B.nverts; ++moves) {
    int next = -1;
    double dn = 0.;
    for (int k = B.adj_start[cur]; k < B.adj_start[cur + 1] && next < 0; ++k) {
      if (B.adj[k] == last) continue;
      const double d = dot(at(B.adj[k]), v);
      if (!(d - h < 1.e-16)) {
        next = B.adj[k];
        dn = d;
      }
    }
    if (next < 0) break;
    last = cur;
    cur = next;
    h = dn;
  }
  return cur;
}

int main() {
  std::mt19937_64 g(5);
  std::normal_distribution<double> N;
  std::uniform_real_distribution<double> U(-1., 1.);
  long failures = 0, climbs = 0;
  // a k-gon between two apexes: apexes of degree k, the others of degree 4
  for (int k = 3; k <= 13; ++k) {
    std::vector<double> verts;
    std::vector<int> start{0}, adj;
    for (int i = 0; i < k; ++i) {
      verts.insert(verts.end(), {1e-3 * std::cos(2 * kPi * i / k), 0., 1e-3 * std::sin(2 * kPi * i / k)});
      for (int o : {(i + 1) % k, k, (i + k - 1) % k, k + 1}) adj.push_back(o);
      start.push_back((int)adj.size());
    }
    verts.insert(verts.end(), {0., 8e-4, 0., 0., -8e-4, 0.});
    for (int t = 0; t < 2; ++t) {
      for (int i = 0; i < k; ++i) adj.push_back(i);
      start.push_back((int)adj.size());
    }
    LocalBody<double> B;
    B.type = 3;
    B.nverts = k + 2;
    B.verts = verts.data();
    B.adj_start = start.data();
    B.adj = adj.data();
    for (int t = 0; t < 20000; ++t) {
      V3<double> v = v3<double>(N(g), N(g), N(g));
      if (t % 5 == 1) v.y = 0.;            // ties between the apexes
      if (t % 7 == 1) v.x = v.z = 0.;      // ... and along the ring
      if (t % 11 == 1) v = sc(v, 1e-16);
      if (t % 13 == 1) v.x = NAN;
      B.cur = t % (k + 2);
      const int want = climb(B, v, B.cur);
      const V3<double> p = support_local(B, v);
      const V3<double> w = want < 0 ? v3<double>(0., 0., 0.)
                                    : v3<double>(verts[3 * want], verts[3 * want + 1], verts[3 * want + 2]);
      ++climbs;
      if (p.x != w.x || p.y != w.y || p.z != w.z || (want >= 0 && B.cur != want)) ++failures;
    }
  }
  // float division: random operands of all normal exponents whose quotient is
  // normal, and the special values
  const float special[] = {0.f, -0.f, 1.f, 6.f, INFINITY, -INFINITY, NAN, 1e-45f, 1.17549435e-38f, 3.4e38f};
  auto divide = [&](float x, float d) {
    const float a = x / d, b = Divisor<float>(d)(x);
    if (std::isnan(a) ? !std::isnan(b) : std::memcmp(&a, &b, 4)) ++failures;
  };
  for (float x : special)
    for (float d : special)
      if (std::isnan(x / d) || x / d == 0.f || std::fabs(x / d) >= 1.2e-38f) divide(x, d);
  for (long t = 0; t < 4000000; ++t) {
    const unsigned long long r = g();
    unsigned u[2] = {(unsigned)r, (unsigned)(r >> 32)};
    if (t % 3 == 0) u[0] &= ~0u << (t % 23), u[1] &= ~0u << (t / 3 % 23);  // short significands
    float f[2];
    std::memcpy(f, u, 8);
    const double q = (double)f[0] / (double)f[1];
    if (std::fabs(q) > 1.2e-38 && std::isfinite(q)) divide(f[0], f[1]);
  }
  // |t| > most, about the limit and away from it
  for (long t = 0; t < 400000; ++t) {
    const V3<double> x = sc(v3<double>(N(g), N(g), N(g)), std::pow(10., 20. * U(g)));
    double most = norm(x);
    if (t % 2) most *= 1. + 1e-13 * std::round(20. * U(g));
    if (t % 7 == 0) most = U(g);
    if (t % 31 == 0) most = 0.;
    if (longer(x, most) != (norm(x) > most)) ++failures;
  }
  // cell indices, at faces and between them
  for (long t = 0; t < 1000000; ++t) {
    const double e = std::pow(10., U(g)) * 1e-3, o = U(g);
    double x = o + e * std::round(2000. * U(g)) * (t % 4 ? 1. : 1000.);
    const int ulps = (int)(g() % 9) - 4;
    for (int u = 0; u < std::abs(ulps); ++u) x = std::nextafter(x, ulps < 0 ? -1e9 : 1e9);
    if (t % 3 == 0) x += e * U(g);
    if (cell_coord(x, o, e, 1. / e) != (int)std::floor((x - o) / e)) ++failures;
  }
  std::printf("climbs %ld failures %ld\n", climbs, failures);
  return failures ? 1 : 0;
}
