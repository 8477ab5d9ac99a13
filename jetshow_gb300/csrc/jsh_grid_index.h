// jsh_grid_index.h -- the bucket index and the triangle records of a
// triangulated grid, built on the host at upload.
#pragma once

#include <stddef.h>
#include <stdint.h>

#include <memory>

// An array whose elements are left as they are until they are written.
template <typename T>
struct JshRaw {
  std::unique_ptr<T[]> p;
  size_t n = 0;
  void resize(size_t m) {
    p.reset(m ? new T[m] : nullptr);
    n = m;
  }
  size_t bytes() const { return n * sizeof(T); }
  T& operator[](size_t i) { return p[i]; }
  const T& operator[](size_t i) const { return p[i]; }
};

struct JshGridIndex {
  double x0, y0, h;  // bucket (i, j) covers [x0 + i h, x0 + (i + 1) h) x ...; the last ones what lies beyond
  int32_t nbx, nby;
  // head [nbx * nby][8], more and rec [n_tri][12] (lean: none) as JshGrid::bhead, bmore and rec
  JshRaw<int32_t> head, more;
  JshRaw<float> rec;
};

// Device bytes of the arrays of a full index: about two buckets a triangle.
size_t jsh_grid_full_bytes(int64_t n_tri);

// Builds the index of triangles tri [n_tri][3] over points xy [n][2]
// (vertex ids in range).  A JSH status; throws std::bad_alloc.
int jsh_grid_index(const double* xy, int64_t n, const int32_t* tri, int64_t n_tri, bool lean, JshGridIndex* out);
