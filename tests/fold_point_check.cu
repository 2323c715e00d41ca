// Host check of fold_point (ctca_b200/csrc/fold_point.cuh): for every
// combination of periodic, face and other field boundaries, every array kind
// and grids down to two cells an axis, the value of every element equals the
// one the slab operations leave one after the other, in int64 and in FP64, and
// the shell holds every element that they change, once.  Built and run by
// tests/test_fold_point.py.
#include <cstdio>
#include <random>
#include <vector>

#include "fold_point.cuh"
#include "slab.cuh"

using namespace emsesg;

template <typename T>
static void apply(std::vector<T>& a, const FieldDesc& f, const SlabOp& o) {
  const int ax = o.axis, ea = ax == 0 ? 1 : 0, eb = ax == 2 ? 1 : 2;
  SlabArgs s;
  s.o = o;
  s.f = f;
  s.count = (int64_t)o.depth * (o.hi[ea] - o.lo[ea] + 1) * (o.hi[eb] - o.lo[eb] + 1) * o.nc;
  for (int64_t t = 0; t < s.count; t++) slab_apply(a.data(), s, t);
}

int main() {
  int bad = 0, cases = 0;
  std::mt19937_64 rng(7);
  const int dims[][3] = {{5, 6, 7}, {9, 8, 12}, {2, 3, 2}, {3, 2, 4}};
  for (const auto& n : dims)
    for (int fb = 0; fb < 27; fb++)
      for (int kind = 0; kind < 3; kind++) {
        emsesg_config c{};
        c.nx = n[0];
        c.ny = n[1];
        c.nz = n[2];
        c.nfbnd[0] = fb % 3;
        c.nfbnd[1] = fb / 3 % 3;
        c.nfbnd[2] = fb / 9;
        const int nc = kind == 0 ? 1 : 6, g = kind == 1 ? 9 : 3, lo = kind == 1 ? -4 : -1;
        const std::vector<SlabOp> ops = fold_ops(c, kind, nc);
        const FieldDesc f{nc, lo, n[0] + g, n[1] + g, n[2] + g};
        std::vector<long long> a((size_t)f.size());
        for (auto& v : a) v = (long long)(rng() % 2000001) - 1000000;
        std::vector<double> d(a.begin(), a.end());
        for (auto& v : d) v *= 0.1;
        // every element starts random, the outer guards too, which a step
        // leaves at zero
        std::vector<long long> sa = a;
        std::vector<double> sd = d;
        for (const SlabOp& o : ops) {
          apply(sa, f, o);
          apply(sd, f, o);
        }
        const FoldGeo fg = fold_geo(c, kind);
        bool same = true;
        std::vector<int> hit((size_t)(f.size() / nc), 0);
        const FoldShell s = fold_shell(f);
        for (int64_t t = 0; t < s.nzs + s.nys + s.nxs; t++) {
          int x[3];
          shell_node(s, t, x);
          hit[(size_t)(x[0] + (int64_t)f.ex * (x[1] + (int64_t)f.ey * x[2]))]++;
        }
        for (int z = 0; z < f.ez; z++)
          for (int y = 0; y < f.ey; y++)
            for (int x = 0; x < f.ex; x++) {
              const int h = hit[(size_t)(x + (int64_t)f.ex * (y + (int64_t)f.ey * z))];
              same = same && h <= 1;
              for (int q = 0; q < nc; q++) {
                const int i = x + lo, j = y + lo, k = z + lo;
                const size_t e = (size_t)f.at(q, i, j, k);
                const bool ok = fold_point(a.data(), f, fg, q, i, j, k) == sa[e] &&
                                fold_point(d.data(), f, fg, q, i, j, k) == sd[e];
                if (!ok && same) std::printf("first at c=%d (%d,%d,%d)\n", q, i, j, k);
                same = same && ok && (h == 1 || sa[e] == a[e]);
                if (fold_inner(fg, i, j, k)) same = same && sa[e] == a[e];
              }
            }
        if (!same) {
          bad++;
          std::printf("mismatch n=%dx%dx%d nfbnd=%d%d%d kind=%d\n", n[0], n[1], n[2], c.nfbnd[0], c.nfbnd[1],
                      c.nfbnd[2], kind);
        }
        cases++;
      }
  std::printf("%s cases=%d\n", bad ? "FAIL" : "ok", cases);
  return bad ? 1 : 0;
}
