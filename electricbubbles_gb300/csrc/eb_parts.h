// A range cut into parts of about equal size, in plain C++ (host and device).
#pragma once

#ifdef __CUDACC__
#define EB_PARTS_FN __host__ __device__ __forceinline__
#else
#define EB_PARTS_FN inline
#endif

// n elements in c parts, part i from i n / c (rounded down) to (i + 1) n / c. Stepped part by
// part, so that no product i n is formed: of a leaf's points and batches of 32 it leaves 32
// bits from 262,144 points on (coincident points, a tight cluster beside an outlier).
struct EbParts {
  int q, r, c;
  int at = 0;   // start of the next part
  int acc = 0;  // the remainder of i n / c
  EB_PARTS_FN EbParts(int n, int parts) : q(n / parts), r(n % parts), c(parts) {}
  // the next part's size; `at` moves behind it
  EB_PARTS_FN int next() {
    int m = q;
    acc += r;
    if (acc >= c) {
      acc -= c;
      ++m;
    }
    at += m;
    return m;
  }
};
