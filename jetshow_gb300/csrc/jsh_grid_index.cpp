// jsh_grid_index.cpp -- the bucket index and the triangle records of a
// triangulated grid (the device's lookups: jsh_fields.cuh, jsh_fields32.cuh).
//
// Square buckets, each with the triangles that it touches, in ascending order, the
// first seven inline.  The full index has about two buckets per triangle (one for
// two triangles from 2^26 buckets on) and a record per triangle; the lean one,
// where memory is short, a bucket for two triangles and no records.
//
// A mixed-precision lookup outside its hint's triangle is a chain of loads, a
// bucket and its triangles two at a time: with half a bucket per triangle,
// listed by bounding boxes, about 10 triangles a bucket, read one after another
// through a list, instead of the 3 to 4 of the full index, a 256^2 render of a
// 200 000 point grid took 25.2 + 17.3 ms (tau, IQUV kernel), now 19.8 + 15.2;
// 512^2 76 + 55, now 48 + 44.
#include "jsh_grid_index.h"

#include <string.h>

#include <algorithm>
#include <cmath>
#include <thread>
#include <vector>

#include "jsh_model.h"

namespace {

// f(k) for k in [0, n) on a thread each (on this one where none can be had).
template <typename F>
void in_parallel(int n, F f) {
  std::vector<std::thread> threads;
  threads.reserve((size_t)n);
  for (int k = 1; k < n; ++k) {
    try {
      threads.emplace_back(f, k);
    } catch (...) {  // no thread or no memory for one
      f(k);
    }
  }
  f(0);
  for (auto& t : threads) t.join();
}

struct Entry {
  uint32_t bucket, triangle;
};

}  // namespace

size_t jsh_grid_full_bytes(int64_t n_tri) {
  // heads (two buckets a triangle), records, and the longer lists: few on an
  // even grid
  return (size_t)n_tri * (2 * 8 * sizeof(int32_t) + 12 * sizeof(float));
}

int jsh_grid_index(const double* xy, int64_t n, const int32_t* tri, int64_t n_tri, bool lean, JshGridIndex* out) {
  double x0 = xy[0], x1 = xy[0], y0 = xy[1], y1 = xy[1];
  for (int64_t i = 1; i < n; ++i) {
    x0 = std::min(x0, xy[2 * i]);
    x1 = std::max(x1, xy[2 * i]);
    y0 = std::min(y0, xy[2 * i + 1]);
    y1 = std::max(y1, xy[2 * i + 1]);
  }
  if (!std::isfinite(x0) || !std::isfinite(x1) || !std::isfinite(y0) || !std::isfinite(y1)) {
    jsh_set_error("grid points must be finite");
    return JSH_ERR_INVALID;
  }
  const double ex = x1 - x0, ey = y1 - y0;
  double n_buckets = (double)n_tri / 2.0;
  if (!lean) n_buckets = std::max(n_buckets, std::min(2.0 * (double)n_tri, 67108864.0));
  double h = std::sqrt(std::max(ex * ey, 1e-300) / std::max(1.0, n_buckets));
  if (!(h > 0) || !std::isfinite(h)) h = std::max(std::max(ex, ey), 1.0);
  h = std::max(h, std::max(ex, ey) / 65536.0);  // at most 65536 buckets per side
  const int32_t nbx = std::max(1, (int32_t)std::ceil(ex / h)), nby = std::max(1, (int32_t)std::ceil(ey / h));
  const int64_t nbk = (int64_t)nbx * nby;
  // A triangle is listed in every bucket that it touches, the bucket grown so
  // that FP32 lookups near an edge still find it: by a hundredth of its side and
  // by the rounding of the coordinates, the latter by half a side at most.  A
  // grid far from the origin has sides below the rounding (z in [1e5, 1e5 + 1]
  // pc: 1e-3 pc against 0.1), where an FP32 coordinate cannot tell the buckets
  // apart and the unbounded margin listed every triangle in thousands of them.
  const double coord = std::max(std::max(std::fabs(x0), std::fabs(x1)), std::max(std::fabs(y0), std::fabs(y1)));
  const double margin = 0.01 * h + std::min(16.0 * 5.9604645e-8 * coord, 0.5 * h);
  out->x0 = x0;
  out->y0 = y0;
  out->h = h;
  out->nbx = nbx;
  out->nby = nby;
  out->rec.resize(lean ? 0 : (size_t)12 * n_tri);

  // The triangles in stretches, one a thread: each its records and its (bucket,
  // triangle) entries, once (its time: jsh_grid_upload).
  const int n_threads =
      (int)std::min<int64_t>({(int64_t)16, std::max<int64_t>(1, (int64_t)std::thread::hardware_concurrency()),
                              1 + n_tri / 8192});
  std::vector<std::vector<Entry>> entries((size_t)n_threads);
  std::vector<char> failed((size_t)n_threads, 0);
  in_parallel(n_threads, [&](int part) {
    try {
      std::vector<Entry>& E = entries[(size_t)part];
      const int64_t t0 = n_tri * part / n_threads, t1 = n_tri * (part + 1) / n_threads;
      E.reserve((size_t)(t1 - t0) * 9);
      for (int64_t t = t0; t < t1; ++t) {
        double px[3], py[3];
        for (int k = 0; k < 3; ++k) {
          px[k] = xy[2 * (int64_t)tri[3 * t + k]];
          py[k] = xy[2 * (int64_t)tri[3 * t + k] + 1];
        }
        if (!lean) {  // the FP32 operations here round as the device's would
          float* r = &out->rec[(size_t)12 * t];
          for (int k = 0; k < 3; ++k) {
            r[2 * k] = (float)px[k];
            r[2 * k + 1] = (float)py[k];
          }
          r[6] = r[4] - r[0];
          r[7] = r[5] - r[1];
          const float area32 = (r[2] - r[0]) * r[7] - (r[3] - r[1]) * r[6];
          r[8] = area32 == 0.f ? NAN : 1.f / area32;
          memcpy(r + 9, tri + 3 * t, 3 * sizeof(int32_t));
        }
        for (int k = 0; k < 3; ++k) {
          px[k] -= x0;
          py[k] -= y0;
        }
        const double bx0 = std::min(px[0], std::min(px[1], px[2])), bx1 = std::max(px[0], std::max(px[1], px[2]));
        const double by0 = std::min(py[0], std::min(py[1], py[2])), by1 = std::max(py[0], std::max(py[1], py[2]));
        const int32_t i0 = std::max(0, (int32_t)std::floor((bx0 - margin) / h)),
                      i1 = std::min(nbx - 1, (int32_t)std::floor((bx1 + margin) / h)),
                      j0 = std::max(0, (int32_t)std::floor((by0 - margin) / h)),
                      j1 = std::min(nby - 1, (int32_t)std::floor((by1 + margin) / h));
        // edge normals, outwards (none for a triangle without area: its box)
        const double area = (px[1] - px[0]) * (py[2] - py[0]) - (py[1] - py[0]) * (px[2] - px[0]);
        const double sgn = area > 0 ? 1.0 : area < 0 ? -1.0 : 0.0;
        double nx[3], ny[3], limit[3];
        for (int k = 0; k < 3; ++k) {
          const int l = (k + 1) % 3;
          nx[k] = sgn * (py[l] - py[k]);
          ny[k] = sgn * (px[k] - px[l]);
          // beyond the edge by more than half a bucket (with its margin) either way
          limit[k] = nx[k] * px[k] + ny[k] * py[k] + (0.5 * h + margin) * (std::fabs(nx[k]) + std::fabs(ny[k]));
        }
        for (int32_t j = j0; j <= j1; ++j)
          for (int32_t i = i0; i <= i1; ++i) {
            const double cx = (i + 0.5) * h, cy = (j + 0.5) * h;
            bool apart = false;
            for (int k = 0; k < 3; ++k) apart = apart || nx[k] * cx + ny[k] * cy > limit[k];
            // points beyond the last bucket's end are looked up in it
            if (!apart || i == nbx - 1 || j == nby - 1)
              E.push_back(Entry{(uint32_t)((int64_t)j * nbx + i), (uint32_t)t});
          }
      }
    } catch (const std::bad_alloc&) {
      failed[(size_t)part] = 1;
    }
  });
  for (char f : failed)
    if (f) throw std::bad_alloc();

  // The buckets in stretches, one a thread, which goes through all entries and
  // takes its own: the ids of a bucket come in ascending order.
  auto own = [&](int part, auto visit) {
    const uint32_t b0 = (uint32_t)(nbk * part / n_threads), b1 = (uint32_t)(nbk * (part + 1) / n_threads);
    for (const auto& E : entries)
      for (const Entry& e : E)
        if (e.bucket >= b0 && e.bucket < b1) visit(e);
  };
  JshRaw<uint32_t> count;
  count.resize((size_t)nbk);
  out->head.resize((size_t)nbk * 8);
  in_parallel(n_threads, [&](int part) {
    const int64_t b0 = nbk * part / n_threads, b1 = nbk * (part + 1) / n_threads;
    std::fill(&count[(size_t)b0], &count[(size_t)b0] + (b1 - b0), 0u);
    std::fill(&out->head[(size_t)b0 * 8], &out->head[(size_t)b0 * 8] + (b1 - b0) * 8, -1);
    own(part, [&](const Entry& e) { ++count[e.bucket]; });
  });
  uint64_t n_more = 0;
  for (int64_t b = 0; b < nbk; ++b) {
    const uint32_t c = count[(size_t)b];
    if (c > 7) {
      out->head[(size_t)b * 8 + 7] = (int32_t)n_more;
      n_more += c - 7 + 1;  // and a -1
    }
    if (n_more > (uint64_t)INT32_MAX) {
      jsh_set_error("grid too large");
      return JSH_ERR_INVALID;
    }
    count[(size_t)b] = 0;
  }
  out->more.resize((size_t)n_more);
  in_parallel(n_threads, [&](int part) {
    own(part, [&](const Entry& e) {
      const uint32_t c = count[e.bucket]++;
      int32_t* hd = &out->head[(size_t)e.bucket * 8];
      if (c < 7) {
        hd[c] = (int32_t)e.triangle;
      } else {
        int32_t* more = &out->more[(size_t)hd[7] + (c - 7)];
        more[0] = (int32_t)e.triangle;
        more[1] = -1;  // the next one's place, or the end
      }
    });
  });
  return JSH_OK;
}
