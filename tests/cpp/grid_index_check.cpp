// grid_index_check.cpp -- the bucket index of gridded fields against all
// triangles, on the CPU: argv[1] a file of int64 n, n_tri, n_query, double
// xy[n][2], int32 tri[n_tri][3], double q[n_query][2].  For every query the first
// triangle that holds it must be the first of its bucket's list that does, in
// the arithmetic of the FP64 lookup and in that of the FP32 one (whose point and
// bucket are rounded), and the lists must be ascending and within range.
#include <stdarg.h>
#include <stdio.h>
#include <string.h>

#include <cmath>
#include <vector>

#include "jsh_grid_index.h"

void jsh_set_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vprintf(fmt, ap);
  va_end(ap);
}

int main(int argc, char** argv) {
  FILE* f = fopen(argv[1], "rb");
  int64_t s[3];
  if (!f || fread(s, 8, 3, f) != 3) return 2;
  const int64_t n = s[0], nt = s[1], nq = s[2];
  std::vector<double> xy(2 * n), q(2 * nq);
  std::vector<int32_t> tri(3 * nt);
  if ((int64_t)fread(xy.data(), 8, 2 * n, f) != 2 * n || (int64_t)fread(tri.data(), 4, 3 * nt, f) != 3 * nt ||
      (int64_t)fread(q.data(), 8, 2 * nq, f) != 2 * nq)
    return 2;
  fclose(f);
  // argv[2]: the lean index
  const bool lean = argc > 2;
  JshGridIndex X, full;
  if (jsh_grid_index(xy.data(), n, tri.data(), nt, false, &full)) return 3;
  if (jsh_grid_index(xy.data(), n, tri.data(), nt, lean, &X)) return 3;
  auto id = [&](int64_t b, int k) {
    if (k < 7) return X.head[8 * b + k];
    return X.head[8 * b + 7] < 0 ? -1 : X.more[X.head[8 * b + 7] + (k - 7)];
  };
  int64_t longest = 0, entries = 0;
  for (int64_t b = 0; b < (int64_t)X.nbx * X.nby; ++b) {
    int k = 0;
    for (int last = -1; id(b, k) >= 0; last = id(b, k++))
      if (id(b, k) <= last || id(b, k) >= nt) return printf("bucket %lld: not ascending\n", (long long)b), 1;
    entries += k;
    longest = std::max<int64_t>(longest, k);
  }
  auto orient = [](auto ax, auto ay, auto bx, auto by, auto cx, auto cy) { return (bx - ax) * (cy - ay) - (by - ay) * (cx - ax); };
  auto in64 = [&](int64_t t, double px, double py) {
    const double *a = &xy[2 * tri[3 * t]], *b = &xy[2 * tri[3 * t + 1]], *c = &xy[2 * tri[3 * t + 2]];
    const double area = orient(a[0], a[1], b[0], b[1], c[0], c[1]);
    if (area == 0.0) return false;
    return orient(px, py, b[0], b[1], c[0], c[1]) / area >= 0 && orient(a[0], a[1], px, py, c[0], c[1]) / area >= 0 &&
           orient(a[0], a[1], b[0], b[1], px, py) / area >= 0;
  };
  auto in32 = [&](int64_t t, float px, float py) {
    const float* r = &full.rec[12 * t];
    const float w0 = ((r[2] - px) * (r[5] - py) - (r[3] - py) * (r[4] - px)) * r[8];
    const float w1 = ((px - r[0]) * r[7] - (py - r[1]) * r[6]) * r[8];
    return w0 >= -1e-6f && w1 >= -1e-6f && 1.f - w0 - w1 >= -1e-6f;
  };
  int64_t inside = 0;
  for (int64_t k = 0; k < nq; ++k) {
    const double px = q[2 * k], py = q[2 * k + 1];
    const float fx = (float)px, fy = (float)py;
    int64_t first64 = -1, first32 = -1;
    for (int64_t t = nt; t-- > 0;) {
      if (in64(t, px, py)) first64 = t;
      if (in32(t, fx, fy)) first32 = t;
    }
    inside += first64 >= 0;
    for (int single = 0; single < 2; ++single) {
      const float inv = (float)(1.0 / X.h);
      const double bx = single ? (double)((fx - (float)X.x0) * inv) : (px - X.x0) / X.h;
      const double by = single ? (double)((fy - (float)X.y0) * inv) : (py - X.y0) / X.h;
      int64_t got = -1;
      if (bx >= 0 && by >= 0) {
        const int64_t b = (int64_t)std::min((int)by, X.nby - 1) * X.nbx + std::min((int)bx, X.nbx - 1);
        for (int c = 0; id(b, c) >= 0 && got < 0; ++c)
          if (single ? in32(id(b, c), fx, fy) : in64(id(b, c), px, py)) got = id(b, c);
      } else if (!single) {
        first64 = -1;  // outside the rectangle
      } else {
        first32 = -1;
      }
      const int64_t want = single ? first32 : first64;
      if (got != want)
        return printf("(%.17g, %.17g) %s: triangle %lld, of all %lld\n", px, py, single ? "FP32" : "FP64",
                      (long long)got, (long long)want), 1;
    }
  }
  printf("%lld buckets, %lld entries, longest %lld, %lld of %lld inside\n", (long long)X.nbx * X.nby,
         (long long)entries, (long long)longest, (long long)inside, (long long)nq);
  return 0;
}
