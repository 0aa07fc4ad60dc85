// GPU quadtree construction for the boundary-node FMM.
//
// The reference bins the nodes into a uniform 2^l x 2^l grid at every level with a
// counting sort (ASSIGN1, cadap2.f:252-409) and loops over all 4^l boxes, empty or
// not (DOINT0DR, cadapdrop2.f:84-197). Here the nodes are sorted once by a Morton key
// at depth 20; the occupied boxes of every level are then the distinct key prefixes,
// each owning a contiguous range of the sorted nodes. Only occupied boxes exist.
// The tree is adaptive: below a uniform floor (the shallowest level of mean occupancy at
// most `leaf_target`), a box with more than `leaf_cap` points is split (DAASSI,
// dapif1.f:1165-1255, with NAPB = leaf_cap); every point's leaf level follows from the
// keys of the points leaf_cap places before and after it in sorted order. V lists follow MKINTL
// (cadap2.f:780-828: children of the parent's neighbours that are not adjacent, at most
// 27); the leaves' U and W lists follow DALI12/DALI34 (dapif2.f:3-356) for leaves of
// different levels.
#include <cooperative_groups.h>
#include <cub/cub.cuh>

#include <algorithm>
#include <cmath>

#include <atomic>
#include <mutex>

#include "eb_internal.h"

namespace {

struct __align__(16) Box4 {
  double x, y, z, w;
};
__host__ __device__ __forceinline__ Box4 mk_box4(double a, double b, double c, double d) {
  Box4 r;
  r.x = a; r.y = b; r.z = c; r.w = d;
  return r;
}

__host__ __device__ __forceinline__ unsigned long long spread2(unsigned int v) {
  unsigned long long x = v;
  x = (x | (x << 16)) & 0x0000FFFF0000FFFFull;
  x = (x | (x << 8)) & 0x00FF00FF00FF00FFull;
  x = (x | (x << 4)) & 0x0F0F0F0F0F0F0F0Full;
  x = (x | (x << 2)) & 0x3333333333333333ull;
  x = (x | (x << 1)) & 0x5555555555555555ull;
  return x;
}
__host__ __device__ __forceinline__ unsigned int compact2(unsigned long long x) {
  x &= 0x5555555555555555ull;
  x = (x | (x >> 1)) & 0x3333333333333333ull;
  x = (x | (x >> 2)) & 0x0F0F0F0F0F0F0F0Full;
  x = (x | (x >> 4)) & 0x00FF00FF00FF00FFull;
  x = (x | (x >> 8)) & 0x0000FFFF0000FFFFull;
  x = (x | (x >> 16)) & 0x00000000FFFFFFFFull;
  return (unsigned int)x;
}
__host__ __device__ __forceinline__ unsigned long long morton(unsigned int ix, unsigned int iy) {
  return spread2(ix) | (spread2(iy) << 1);
}

// The build's numbers on the device; the host reads the first part after the leaf levels
// and `last` after the counts (one copy each).
struct TreeDev {
  double sq[4];                  // as in EbTreeHost, up to hist
  int bad, lmin;
  int hist[EB_KEY_LEVELS + 1];
  int last[12];                  // leaves, groups, tiles, U and W entries, list error, chunks
  int first[EB_KEY_LEVELS + 1];  // k_gather_points' histogram
  unsigned int ticket[2];
};
static_assert(offsetof(TreeDev, last) == offsetof(EbTreeHost, last), "copied as one piece");

// True in the block of a grid that counts itself last; it then sees what the others wrote.
__device__ __forceinline__ bool last_block(unsigned int* ticket) {
  __shared__ bool s_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (s_last) __threadfence();
  return s_last;
}

// Doubles as integers in their order, so that the FP64 pipe (two lanes a cycle and SM, each
// step of a reduction 64 cycles and more) has no part in the minima and maxima.
__device__ __forceinline__ long long ordered(double x) {
  const long long b = __double_as_longlong(x);
  return b ^ ((b >> 63) & 0x7fffffffffffffffll);
}
__device__ __forceinline__ double unordered(long long b) {
  return __longlong_as_double(b ^ ((b >> 63) & 0x7fffffffffffffffll));
}
struct IBox {  // (min x, -max x, min y, -max y) as ordered integers: all four by minima
  long long v[4];
};
// The minima over the block (256 threads), in thread 0.
__device__ __forceinline__ IBox box_min(IBox b) {
  __shared__ long long s[4][8];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) b.v[q] = min(b.v[q], __shfl_xor_sync(0xffffffffu, b.v[q], o));
    if (lane == 0) s[q][w] = b.v[q];
  }
  __syncthreads();
  if (threadIdx.x == 0)
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int x = 1; x < 8; ++x) b.v[q] = min(b.v[q], s[q][x]);
  __syncthreads();
  return b;
}

// Bounding box per block; the last block forms the root square sq = (W, x0, y0, 2^20 / W):
// the box's larger side widened by 1e-9 relative, centred on the box (W = 1 for a single
// point), or the given one of a forest of independent problems in a grid of cells.
__global__ void __launch_bounds__(256) k_bbox(const double2* __restrict__ z, int n, IBox* __restrict__ part, int wall,
                                              int forest, Box4 given, TreeDev* T) {
  const long long inf = ordered(INFINITY);
  IBox b{{inf, inf, inf, inf}};
  bool nonfinite = false;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const longlong2 p = reinterpret_cast<const longlong2*>(z)[i];
    const double x = __longlong_as_double(p.x), y = __longlong_as_double(p.y);
    if ((~p.x & 0x7ff0000000000000ll) == 0 || (~p.y & 0x7ff0000000000000ll) == 0) {  // inf or NaN
      nonfinite = true;
      continue;
    }
    b.v[0] = min(b.v[0], ordered(x));
    b.v[1] = min(b.v[1], ~ordered(x));
    b.v[2] = min(b.v[2], ordered(y));
    b.v[3] = min(b.v[3], ~ordered(y));
  }
  if (nonfinite) atomicOr(&T->bad, 1);
  b = box_min(b);
  if (threadIdx.x == 0) part[blockIdx.x] = b;
  if (!last_block(&T->ticket[0])) return;
  b = IBox{{inf, inf, inf, inf}};
  for (int i = threadIdx.x; i < gridDim.x; i += blockDim.x)
#pragma unroll
    for (int q = 0; q < 4; ++q) b.v[q] = min(b.v[q], __ldcg(&part[i].v[q]));
  b = box_min(b);
  if (threadIdx.x != 0) return;
  double* sq = T->sq;
  if (forest) {
    sq[0] = given.x;
    sq[1] = given.y;
    sq[2] = given.z;
    sq[3] = __ddiv_rn((double)(1u << EB_KEY_LEVELS), given.x);
    return;
  }
  const Box4 r = mk_box4(unordered(b.v[0]), unordered(~b.v[1]), unordered(b.v[2]), unordered(~b.v[3]));
  if (wall) {
    // the square [xleft, xleft + slength] x [0, slength] of the wall-bounded CADAPDR
    // (cadapdrop.f:142-145), widened by 1e-9 so that no key needs clamping
    if (!(r.z >= 0.0)) atomicOr(&T->bad, 2);
    double w = fmax(__dadd_rn(r.y, -r.x), r.w);
    if (!(w > 0)) w = 1.0;
    w = __dmul_rn(w, 1.0 + 1e-9);
    sq[0] = w;
    sq[1] = r.x;
    sq[2] = 0.0;
    sq[3] = __ddiv_rn((double)(1u << EB_KEY_LEVELS), w);
    return;
  }
  double w = fmax(__dadd_rn(r.y, -r.x), __dadd_rn(r.w, -r.z));
  if (!(w > 0)) w = 1.0;
  w = __dmul_rn(w, 1.0 + 1e-9);
  sq[0] = w;
  sq[1] = __dadd_rn(__dmul_rn(0.5, __dadd_rn(r.x, r.y)), -__dmul_rn(0.5, w));
  sq[2] = __dadd_rn(__dmul_rn(0.5, __dadd_rn(r.z, r.w)), -__dmul_rn(0.5, w));
  sq[3] = __ddiv_rn((double)(1u << EB_KEY_LEVELS), w);
}

__global__ void k_keys(const double2* __restrict__ z, int n, const double* __restrict__ sq,
                       unsigned long long* __restrict__ keys, int* __restrict__ idx) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double x0 = sq[1], y0 = sq[2], inv_cell = sq[3];
  const double maxc = (double)((1u << EB_KEY_LEVELS) - 1);
  double fx = floor((z[i].x - x0) * inv_cell), fy = floor((z[i].y - y0) * inv_cell);
  fx = fmin(fmax(fx, 0.0), maxc);
  fy = fmin(fmax(fy, 0.0), maxc);
  keys[i] = morton((unsigned int)fx, (unsigned int)fy);
  idx[i] = i;
}

// The sort of up to SORT_MAX keys in one launch: a stable radix sort, eight bits a pass, of
// one cluster of 16 blocks whose shared memories hold all keys, each with its point's index
// below it in one word (block r the positions [r per, (r + 1) per)). Per pass a warp ranks
// its items in their order by digit (ballots), the block orders its items by digit in shared
// memory, the counts of all blocks give each digit's place, and the items go on to the block
// of their new position through distributed shared memory, neighbours of a digit side by
// side (a remote store is paid by the segments that a warp touches). For tens of thousands of
// keys a library sort's five passes are a handful of blocks each behind two launches: 95 us
// at 32,768 points. Keys and indices in two arrays and scattered straight to their
// blocks, with the keys formed on these 16 SMs as well, took 45 us, this and k_keys 31 us.
constexpr int SORT_CL = 16, SORT_BS = 1024, SORT_IPT = 4, SORT_MAX = SORT_CL * SORT_BS * SORT_IPT;
static_assert(2 * EB_KEY_LEVELS + 16 <= 64 && SORT_MAX <= 1 << 16, "key and index in one word");
struct SortSmem {
  unsigned long long item[SORT_BS * SORT_IPT];  // this block's positions
  unsigned long long loc[SORT_BS * SORT_IPT];   // its items by digit
  int wh[SORT_BS / 32][256];                    // items of a digit per warp, then before the warp
  int tot[256], lbase[256], gbase[256], sw[2][8];
};
__global__ void __cluster_dims__(SORT_CL, 1, 1) __launch_bounds__(SORT_BS)
    k_sort(const unsigned long long* __restrict__ in, int n, unsigned long long* __restrict__ keys,
           int* __restrict__ perm) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  extern __shared__ __align__(16) unsigned char sort_smem[];
  SortSmem& S = *reinterpret_cast<SortSmem*>(sort_smem);
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, r = (int)cl.block_rank();
  const int per = (n + SORT_CL - 1) / SORT_CL, p0 = r * per, nr = max(0, min(n, p0 + per) - p0);
  const int rounds = (per + SORT_BS - 1) / SORT_BS;  // of 32 items of a warp, at most SORT_IPT
  unsigned long long v[SORT_IPT];
#pragma unroll
  for (int q = 0; q < SORT_IPT; ++q) {
    const int s = (w * rounds + q) * 32 + lane;
    v[q] = q < rounds && s < nr ? in[p0 + s] << 16 | (unsigned long long)(p0 + s) : ~0ull;
  }
  for (int shift = 16; shift < 16 + 2 * EB_KEY_LEVELS; shift += 8) {
    for (int x = lane; x < 256; x += 32) S.wh[w][x] = 0;
    __syncwarp();
    int rk[SORT_IPT];
#pragma unroll
    for (int q = 0; q < SORT_IPT; ++q) {
      if (q >= rounds) break;
      const bool valid = (w * rounds + q) * 32 + lane < nr;
      const int d = (int)(v[q] >> shift) & 255;
      unsigned int m = __ballot_sync(0xffffffffu, valid);
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        const unsigned int t = __ballot_sync(0xffffffffu, (d >> b) & 1);
        m &= (d >> b) & 1 ? t : ~t;
      }
      const int old = valid ? S.wh[w][d] : 0;
      __syncwarp();
      rk[q] = old + __popc(m & ((1u << lane) - 1u));
      if (valid && (m >> lane) == 1u) S.wh[w][d] = rk[q] + 1;  // the highest lane of the digit
      __syncwarp();
    }
    __syncthreads();
    int tot = 0, incl = 0;
    if (tid < 256) {
      int c[SORT_BS / 32];
#pragma unroll
      for (int x = 0; x < SORT_BS / 32; ++x) c[x] = S.wh[x][tid];
#pragma unroll
      for (int x = 0; x < SORT_BS / 32; ++x) {
        S.wh[x][tid] = tot;
        tot += c[x];
      }
      S.tot[tid] = tot;
      incl = tot;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      if (lane == 31) S.sw[0][w] = incl;
    }
    __syncthreads();
    if (tid < 256) {
      int b = incl - tot;
      for (int x = 0; x < w; ++x) b += S.sw[0][x];
      S.lbase[tid] = b;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < SORT_IPT; ++q) {
      if (q >= rounds) break;
      const int d = (int)(v[q] >> shift) & 255;
      if ((w * rounds + q) * 32 + lane < nr) S.loc[S.lbase[d] + S.wh[w][d] + rk[q]] = v[q];
    }
    cl.sync();
    int all = 0, mine = 0;
    if (tid < 256) {
#pragma unroll
      for (int x = 0; x < SORT_CL; ++x) {
        const int t = cl.map_shared_rank(S.tot, x)[tid];
        if (x < r) mine += t;
        all += t;
      }
      incl = all;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      if (lane == 31) S.sw[1][w] = incl;
    }
    __syncthreads();
    if (tid < 256) {
      int b = incl - all + mine - S.lbase[tid];
      for (int x = 0; x < w; ++x) b += S.sw[1][x];
      S.gbase[tid] = b;  // from a place in loc to the position
    }
    __syncthreads();
    for (int s = tid; s < nr; s += SORT_BS) {
      const unsigned long long x = S.loc[s];
      const int pos = s + S.gbase[(int)(x >> shift) & 255], to = pos / per;
      cl.map_shared_rank(S.item, to)[pos - to * per] = x;
    }
    cl.sync();
#pragma unroll
    for (int q = 0; q < SORT_IPT; ++q) {
      const int s = (w * rounds + q) * 32 + lane;
      v[q] = q < rounds && s < nr ? S.item[s] : ~0ull;
    }
  }
#pragma unroll
  for (int q = 0; q < SORT_IPT; ++q) {
    const int s = (w * rounds + q) * 32 + lane;
    if (q < rounds && s < nr) {
      keys[p0 + s] = v[q] >> 16;
      perm[p0 + s] = (int)(v[q] & 0xffff);
    }
  }
}

// Sorted positions, also as float hi + lo pairs packed (hi.x, hi.y, lo.x, lo.y), and the
// histogram of the first level at which consecutive sorted keys fall in different boxes:
// the occupied boxes of level l in a uniform tree number 1 + sum_{l' <= l} first[l']. The
// last block picks the minimum leaf level from it: for one problem the shallowest level
// whose occupied boxes hold at most `target` points on average (a uniform floor, which keeps
// leaves of one level, and so no W lists, wherever the points are evenly spread), for a
// forest the level of its cells.
__global__ void __launch_bounds__(256) k_gather_points(const double2* __restrict__ z, const int* __restrict__ perm,
                                const unsigned long long* __restrict__ keys, int n, int target, int R,
                                double2* __restrict__ zs, float4* __restrict__ zhl, TreeDev* T) {
  __shared__ int sh[EB_KEY_LEVELS + 1];
  if (threadIdx.x <= EB_KEY_LEVELS) sh[threadIdx.x] = 0;
  __syncthreads();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    const double2 p = z[perm[i]];
    zs[i] = p;
    const float hx = (float)p.x, hy = (float)p.y;
    zhl[i] = make_float4(hx, hy, (float)(p.x - (double)hx), (float)(p.y - (double)hy));
    const unsigned long long x = i > 0 ? keys[i] ^ keys[i - 1] : 0ull;
    if (x != 0) atomicAdd(&sh[EB_KEY_LEVELS - (63 - __clzll((long long)x)) / 2], 1);
  }
  __syncthreads();
  if (threadIdx.x <= EB_KEY_LEVELS && sh[threadIdx.x]) atomicAdd(&T->first[threadIdx.x], sh[threadIdx.x]);
  if (!last_block(&T->ticket[1]) || threadIdx.x >= 32) return;
  const int l = threadIdx.x;
  int nb = l == 0 ? 1 : l <= EB_KEY_LEVELS ? __ldcg(&T->first[l]) : 0;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, nb, o);
    if (l >= o) nb += y;
  }
  const unsigned int ok = __ballot_sync(0xffffffffu, l <= EB_KEY_LEVELS && (double)n / nb <= (double)target);
  if (l == 0) T->lmin = R > 0 ? R : ok ? __ffs(ok) - 1 : EB_KEY_LEVELS;
}

// The points of a direct tree in their given order, with the float hi + lo copies, and a
// flag for a non-finite coordinate.
__global__ void k_direct_points(const double2* __restrict__ z, int n, int* __restrict__ perm,
                                double2* __restrict__ zs, float4* __restrict__ zhl, int* __restrict__ bad) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double2 p = z[i];
  if (!isfinite(p.x) || !isfinite(p.y)) atomicOr(bad, 1);
  perm[i] = i;
  zs[i] = p;
  float hx = (float)p.x, hy = (float)p.y;
  zhl[i] = make_float4(hx, hy, (float)(p.x - (double)hx), (float)(p.y - (double)hy));
}

// Levels shared by the keys a and b: the deepest level whose box holds both
// (EB_KEY_LEVELS when the keys are equal, -1 never: the root holds every point).
__device__ __forceinline__ int shared_levels(unsigned long long a, unsigned long long b) {
  const unsigned long long x = a ^ b;
  if (x == 0ull) return EB_KEY_LEVELS;
  const int hb = 63 - __clzll((long long)x);
  return EB_KEY_LEVELS - 1 - hb / 2;
}

// lcpw[w] = levels shared by sorted points w and w + cap (w < n - cap). The box of level
// l around a point holds more than cap points exactly when some window [w, w + cap]
// containing the point has lcpw[w] >= l (a box is a contiguous range of sorted points).
__global__ void k_lcp_window(const unsigned long long* __restrict__ keys, int n, int cap,
                             unsigned char* __restrict__ lcpw) {
  const int w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= n - cap) return;
  lcpw[w] = (unsigned char)shared_levels(keys[w], keys[w + cap]);
}

// Leaf level of every sorted point: one more than the deepest level whose box around the
// point holds more than cap points, at most EB_KEY_LEVELS (coincident points), 0 when
// n <= cap, and at least lmin (k_gather_points). Also, per block of 256 points (row l of bc,
// one entry per block), the points that start a box of level l >= 1: l is at most the
// point's leaf level and its key differs from the previous point's at level l; row 0: the
// points that start a leaf.
constexpr int TREE_BS = 256;
__global__ void __launch_bounds__(TREE_BS) k_leaf_level(const unsigned long long* __restrict__ keys, int n, int cap,
                             const unsigned char* __restrict__ lcpw, unsigned char* __restrict__ plev,
                             int* __restrict__ bc, const TreeDev* __restrict__ T) {
  const int lmin = T->lmin;
  __shared__ int sh[EB_KEY_LEVELS + 1];
  if (threadIdx.x <= EB_KEY_LEVELS) sh[threadIdx.x] = 0;
  __syncthreads();
  const int i = blockIdx.x * TREE_BS + threadIdx.x;
  if (i < n) {
    int lam = 0;
    if (n > cap) {
      const int w0 = max(0, i - cap), w1 = min(i, n - 1 - cap);
      int m = 0;
      for (int w = w0; w <= w1; ++w) m = max(m, (int)lcpw[w]);
      lam = min(EB_KEY_LEVELS, m + 1);
    }
    lam = max(lam, lmin);
    plev[i] = (unsigned char)lam;
    const int sl = i > 0 ? shared_levels(keys[i - 1], keys[i]) : -1;
    for (int l = max(1, sl + 1); l <= lam; ++l) atomicAdd(&sh[l], 1);
    if (sl < lam) atomicAdd(&sh[0], 1);
  }
  __syncthreads();
  if (threadIdx.x <= EB_KEY_LEVELS) bc[(size_t)threadIdx.x * gridDim.x + blockIdx.x] = sh[threadIdx.x];
}

// Exclusive sums of up to six arrays, a block each; the totals go to tot.
struct ScanJob {
  const int* in;
  int* out;
  int* tot;
  int n;
};
struct ScanJobs {
  ScanJob j[6];
};
constexpr int SCAN_BS = 1024, SCAN_PT = 8;
__device__ __forceinline__ void scan_array(const int* in, int* out, int n, int* tot) {
  __shared__ int sw[32], s_run;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  if (tid == 0) s_run = 0;
  for (int base = 0; base < n; base += SCAN_BS * SCAN_PT) {
    const int i0 = base + tid * SCAN_PT;
    int v[SCAN_PT], sum = 0;
#pragma unroll
    for (int q = 0; q < SCAN_PT; ++q) {
      v[q] = i0 + q < n ? in[i0 + q] : 0;
      sum += v[q];
    }
    int x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) sw[w] = x;
    __syncthreads();
    if (w == 0) {
      int y = sw[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, y, o);
        if (lane >= o) y += u;
      }
      sw[lane] = y;
    }
    __syncthreads();
    int run = s_run + (w > 0 ? sw[w - 1] : 0) + x - sum;
#pragma unroll
    for (int q = 0; q < SCAN_PT; ++q) {
      if (i0 + q < n) out[i0 + q] = run;
      run += v[q];
    }
    __syncthreads();
    if (tid == 0) s_run += sw[31];
    __syncthreads();
  }
  if (tid == 0 && tot) *tot = s_run;
}
__global__ void __launch_bounds__(SCAN_BS) k_scan(ScanJobs jobs) {
  const ScanJob j = jobs.j[blockIdx.x];
  scan_array(j.in, j.out, j.n, j.tot);
}
// The rows of k_leaf_level's counts, in place; the totals are the boxes of each level and,
// row 0, the leaves.
__global__ void __launch_bounds__(SCAN_BS) k_scan_rows(int nblk, int* bc, TreeDev* T) {
  int* row = bc + (size_t)blockIdx.x * nblk;
  scan_array(row, row, nblk, blockIdx.x == 0 ? &T->last[0] : &T->hist[blockIdx.x]);
}

struct LevOffT {
  int v[EB_KEY_LEVELS + 3];
};

// Every box, by the point that starts it: its id is the level's offset plus the heads of the
// level before the point (the block's from the scanned counts, the rest by ballots), so ids
// are in level order and in point order within a level. Box key, level, first point,
// parent and first child (the box of the next level that starts at the same point; a split
// box's points all lie in its children). Also the leaves in point order, with the flag and
// the exclusive count of leaf heads per point, and zeros for the counts of children and V
// lists.
__global__ void __launch_bounds__(TREE_BS) k_boxes(const unsigned long long* __restrict__ keys,
                            const unsigned char* __restrict__ plev, int n, int L, LevOffT lo,
                            const int* __restrict__ bc, unsigned long long* __restrict__ bkey,
                            unsigned char* __restrict__ blev, int* __restrict__ pt0, int* __restrict__ parent,
                            int* __restrict__ child0, int* __restrict__ nchild, int* __restrict__ vcount,
                            int* __restrict__ lflag, int* __restrict__ lscan, int* __restrict__ leaves) {
  constexpr int NW = TREE_BS / 32;
  __shared__ int wc[EB_KEY_LEVELS + 1][NW];  // heads per warp; row 0: leaf heads
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const int i = blockIdx.x * TREE_BS + tid;
  const bool in = i < n;
  const unsigned long long key = in ? keys[i] : 0ull;
  const int lam = in ? plev[i] : -1;
  const int sl = !in ? EB_KEY_LEVELS : i > 0 ? shared_levels(keys[i - 1], key) : -1;
  const bool head = sl < lam;  // of a leaf
  for (int l = 0; l <= L; ++l) {
    const unsigned int m = __ballot_sync(0xffffffffu, l == 0 ? head : l <= lam && l > sl);
    if (lane == 0) wc[l][w] = __popc(m);
  }
  __syncthreads();
  auto rank = [&](int l, bool f) {  // heads before this point
    const unsigned int m = __ballot_sync(0xffffffffu, f);
    int r = bc[(size_t)l * gridDim.x + blockIdx.x] + __popc(m & ((1u << lane) - 1u));
    for (int q = 0; q < w; ++q) r += wc[l][q];
    return r;
  };
  int up = 0;      // the point's box of the level above, and whether the point starts it
  bool fup = i == 0;
  if (i == 0) {
    bkey[0] = 0;
    blev[0] = 0;
    pt0[0] = 0;
    parent[0] = -1;
    child0[0] = -1;
    nchild[0] = 0;
    vcount[0] = 0;
  }
  for (int l = 1; l <= L; ++l) {
    const bool f = l <= lam && l > sl;
    const int b = lo.v[l] + rank(l, f) + (f ? 0 : -1);
    if (f) {
      bkey[b] = key >> (2 * (EB_KEY_LEVELS - l));
      blev[b] = (unsigned char)l;
      pt0[b] = i;
      parent[b] = up;
      child0[b] = -1;
      nchild[b] = 0;
      vcount[b] = 0;
      if (fup) child0[up] = b;
    }
    if (l <= lam) {
      up = b;
      fup = f;
    }
  }
  const int r = rank(0, head);
  if (in) {
    lflag[i] = head;
    lscan[i] = r;
    if (head) leaves[r] = up;
  }
}

// Point range end of every box (binary search for the first key beyond the box's prefix)
// and the children count of its parent.
__global__ void k_boxes_fin(int nbox, const unsigned long long* __restrict__ keys, int n,
                            const unsigned long long* __restrict__ bkey, const unsigned char* __restrict__ blev,
                            const int* __restrict__ pt0, const int* __restrict__ parent,
                            int* __restrict__ pt1, int* __restrict__ nchild) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= nbox) return;
  const int l = blev[b], sh = 2 * (EB_KEY_LEVELS - l);
  const unsigned long long k = bkey[b];
  int lo = pt0[b] + 1, hi = n;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if ((keys[mid] >> sh) > k) hi = mid;
    else lo = mid + 1;
  }
  pt1[b] = lo;
  if (l > 0) atomicAdd(&nchild[parent[b]], 1);
}

__device__ __forceinline__ int find_box(const unsigned long long* __restrict__ bkey, int off,
                                        int nb, unsigned long long key) {
  int lo = 0, hi = nb - 1;
  while (lo <= hi) {
    int mid = (lo + hi) >> 1;
    unsigned long long v = bkey[off + mid];
    if (v == key) return off + mid;
    if (v < key) lo = mid + 1;
    else hi = mid - 1;
  }
  return -1;
}

// V lists of every box of levels 2..L in one launch (MKINTL, cadap2.f:780-828: the
// children of the parent's neighbours that are not adjacent to the box; DALI12's list 1,
// dapif2.f:3-171). Only existing boxes are found, so the children of a neighbour that is
// a leaf are absent: its points reach the box's leaves through their U lists.
// One warp per box: the 36 candidates (the children of the 3 x 3 parents around the
// box's parent, in the fixed order qy, qx, cy, cx) are looked up by the lanes, two each,
// and the hits written in candidate order.
__global__ void k_vlist(const unsigned long long* __restrict__ bkey, LevOffT lo, int first, int nbox, int R,
                        int* __restrict__ vlist, unsigned char* __restrict__ vcode,
                        int* __restrict__ vcount) {
  const int gid = first + (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (gid >= nbox) return;  // whole warps leave together
  int lev = 0;
  while (gid >= lo.v[lev + 1]) ++lev;
  const int off = lo.v[lev], nb = lo.v[lev + 1] - off;
  const unsigned long long key = bkey[gid];
  if (lev <= R) {  // a forest's boxes of level <= R hold different problems
    if (lane == 0) vcount[gid] = 0;
    return;
  }
  const unsigned long long root = key >> (2 * (lev - R));
  const int ix = (int)compact2(key), iy = (int)compact2(key >> 1);
  const int px = ix >> 1, py = iy >> 1, half = 1 << (lev - 1), side = 1 << lev;
  int cnt = 0;
  for (int base = 0; base < 36; base += 32) {
    const int c = base + lane;
    int s = -1, code = 0;
    if (c < 36) {
      const int qy = py - 1 + c / 12, qx = px - 1 + (c / 4) % 3, cy = (c >> 1) & 1, cx = c & 1;
      const int sx = 2 * qx + cx, sy = 2 * qy + cy, dx = ix - sx, dy = iy - sy;
      const bool inside = qy >= 0 && qy < half && qx >= 0 && qx < half && sx < side && sy < side;
      const bool adjacent = dx >= -1 && dx <= 1 && dy >= -1 && dy <= 1;
      if (inside && !adjacent) {
        s = find_box(bkey, off, nb, morton((unsigned)sx, (unsigned)sy));
        if (s >= 0 && (bkey[s] >> (2 * (lev - R))) != root) s = -1;
        code = (dy + 3) * 7 + (dx + 3);
      }
    }
    const unsigned int m = __ballot_sync(0xffffffffu, s >= 0);
    if (s >= 0) {
      const int pos = cnt + __popc(m & ((1u << lane) - 1u));
      vlist[(size_t)gid * EB_VMAX + pos] = s;
      vcode[(size_t)gid * EB_VMAX + pos] = (unsigned char)code;
    }
    cnt += __popc(m);
  }
  if (lane == 0) vcount[gid] = cnt;
}

// Image lists of the wall y = 0 (the root square's bottom edge) for the boxes of levels
// 2..ld, one thread per box: the source boxes S of the box's level whose mirror image
// across the wall is not adjacent to the box T but lies among the children of the
// mirrored neighbours of T's parent, the reflected interaction list of DOINT0DR (MKINTR,
// cadap2.f:830-877; cadapdrop2.f:159-197). On level 2 every pair is listed whose images
// are not adjacent (it takes the pairs of level 1 as well, whose parents are the root);
// below, only the first two rows have such pairs: T and S in rows 0-1 and S in the
// columns of the children of T's parent's column neighbours. Mirrored, S sits at row
// -1 - iy_S, so the offset T - S' is (ix_T - ix_S, iy_T + iy_S + 1) in box units, dy in
// [1, 7]; the pairs with dy = 1 and |dx| <= 1 (both in row 0, columns adjacent) are left
// to the direct sum of level ld.
__global__ void k_imglist(const unsigned long long* __restrict__ bkey, const unsigned char* __restrict__ blev,
                          LevOffT lo, int first, int nimg, int* __restrict__ ilist,
                          unsigned char* __restrict__ icode, int* __restrict__ icount) {
  const int gid = first + blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= nimg) return;
  const int lev = blev[gid];
  const int off = lo.v[lev], nb = lo.v[lev + 1] - off;
  const unsigned long long key = bkey[gid];
  const int ix = (int)compact2(key), iy = (int)compact2(key >> 1), side = 1 << lev;
  int cnt = 0, x0, x1, y1;
  if (lev == 2) {
    x0 = 0; x1 = 3; y1 = 3;
  } else if (iy <= 1) {
    const int px = ix >> 1;
    x0 = max(2 * px - 2, 0); x1 = min(2 * px + 3, side - 1); y1 = 1;
  } else {
    icount[gid] = 0;
    return;
  }
  for (int sy = 0; sy <= y1; ++sy)
    for (int sx = x0; sx <= x1; ++sx) {
      const int dx = ix - sx, dy = iy + sy + 1;
      if (dy == 1 && dx >= -1 && dx <= 1) continue;  // adjacent images: direct sum
      const int s = find_box(bkey, off, nb, morton((unsigned)sx, (unsigned)sy));
      if (s < 0) continue;
      ilist[(size_t)gid * EB_VMAX + cnt] = s;
      icode[(size_t)gid * EB_VMAX + cnt] = (unsigned char)((dy + 3) * 7 + (dx + 3));
      ++cnt;
    }
  icount[gid] = cnt;
}

#define EB_LIST_STACK 72

// U and W lists of every leaf (DALI12 / DALI34, dapif2.f:3-356, for an adaptive tree
// without level restriction). For leaf b of level l:
//  * every existing box C of level l adjacent to b (b itself included): a leaf C goes to
//    U; below a split C, the boxes adjacent to b are followed down to leaves (U), and a
//    box that is not adjacent to b while its parent is goes to W (its multipole is
//    evaluated at b's points: M2P, DABARR's list-3 evaluation);
//  * every leaf of a coarser level m adjacent to b's ancestor of level m goes to U (the
//    dual list 4, evaluated directly: such a leaf holds at most cap points).
// Every pair of points is then covered exactly once by U, W or a V list of a common
// level. FILL = false counts, FILL = true writes at ustart / wstart, each with the leaf's (and
// box's) other work items (WorkItems).
struct WorkItems {
  const int *pt0, *pt1, *parent;
  int *gcount, *tcount, *ccount;              // per leaf (nbox + 1), per box of levels >= 2 (nb2 + 1)
  const int *gstart, *tstart, *cstart;
  int *gleaf, *gfirst;
  int4* tiles;
  int *anc, *chunk_box, *cdone;
  int nbox, cfirst, nb2, lmin, lend;
};

// Counts of thread t's work items: near-field groups of EB_GROUP targets and shared-memory
// tiles of at most EB_NTILE of leaf t (b: its box, -1 beyond the last leaf), chunks of box t.
__device__ __forceinline__ void count_items(const WorkItems& W, int t, int b, const unsigned char* blev,
                                            const int* nchild) {
  if (t <= W.nbox) {
    const int np = b >= 0 ? W.pt1[b] - W.pt0[b] : 0;
    W.gcount[t] = (np + EB_GROUP - 1) / EB_GROUP;
    W.tcount[t] = (np + EB_NTILE - 1) / EB_NTILE;
  }
  // Chunks of the boxes whose FP32 multipoles come directly from their points: every box
  // of the levels >= lmin and every leaf above them (coarser levels get theirs by M2M).
  if (W.nb2 > 0 && t <= W.nb2) {
    const int g = W.cfirst + t;
    const bool direct = t < W.nb2 && (blev[g] >= W.lmin || nchild[g] == 0);
    W.ccount[t] = direct ? (W.pt1[g] - W.pt0[g] + EB_CHUNK - 1) / EB_CHUNK : 0;
    if (t < W.nb2) W.cdone[t] = 0;
  }
}

__device__ __forceinline__ void fill_items(const WorkItems& W, int t, int b, const unsigned char* blev) {
  if (b >= 0) {
    const int a = W.pt0[b], nt = W.pt1[b] - a;
    int g0 = W.gstart[t], c = W.gcount[t];
    for (int g = 0; g < c; ++g) {
      W.gleaf[g0 + g] = t;
      W.gfirst[g0 + g] = a + g * EB_GROUP;
    }
    g0 = W.tstart[t];
    c = W.tcount[t];
    for (int g = 0; g < c; ++g)
      W.tiles[g0 + g] = make_int4(t, a + (int)((long long)g * nt / c), a + (int)((long long)(g + 1) * nt / c), 0);
    // The FP32 far field's boxes of the leaf: the leaf and its ancestors down to level
    // max(2, min(lev, lend)), -1 beyond (levels <= lend hold the L2L-accumulated locals).
    int up = b;
    const int l = blev[b], lmin = max(2, min(l, W.lend));
    for (int q = 0; q < EB_FAR_LEVELS; ++q) {
      const int lev = l - q;
      W.anc[(size_t)t * EB_FAR_LEVELS + q] = lev >= lmin ? up : -1;
      if (lev > lmin) up = W.parent[up];
    }
  }
  if (t < W.nb2)
    for (int c = 0; c < W.ccount[t]; ++c) W.chunk_box[W.cstart[t] + c] = W.cfirst + t;
}

// A warp per leaf: its neighbours on its own level (tasks 0..8) and those of its ancestors
// (eight a level, coarser levels after finer ones) go to the lanes, which look them up side
// by side; a leaf's entries stand in the tasks' order. With a thread per leaf the chains of
// binary searches, nine and more of some ten dependent loads, took 14 us to count and 16 us to
// fill at 64 x 512, now 6 and 8 us.
template <bool FILL>
__global__ void __launch_bounds__(128) k_leaf_lists(WorkItems W, int nleaf, const int* __restrict__ nleaf_d,
                             const int* __restrict__ leaves,
                             const unsigned long long* __restrict__ bkey,
                             const unsigned char* __restrict__ blev, LevOffT lo, int R,
                             const int* __restrict__ floor_d,
                             const int* __restrict__ child0, const int* __restrict__ nchild,
                             int* __restrict__ ucnt, int* __restrict__ wcnt,
                             const int* __restrict__ ustart, const int* __restrict__ wstart,
                             int* __restrict__ ulist, int* __restrict__ wlist, int* __restrict__ err) {
  const int gt = blockIdx.x * 128 + threadIdx.x, lane = threadIdx.x & 31;
  if (nleaf_d) nleaf = *nleaf_d;  // counting pass: launched for an upper bound
  // the other work items: a thread per leaf and box, the launch has 32 threads for each
  {
    const int b = gt < nleaf ? leaves[gt] : -1;
    if (FILL) fill_items(W, gt, b, blev);
    else count_items(W, gt, b, blev, nchild);
    if (!FILL && b < 0 && gt <= W.nbox) ucnt[gt] = wcnt[gt] = 0;
  }
  const int t = gt >> 5;
  if (t >= nleaf) return;
  const int b = leaves[t], l = blev[b];
  const unsigned long long kb = bkey[b];
  const int ix = (int)compact2(kb), iy = (int)compact2(kb >> 1);
  const unsigned long long root = kb >> (2 * (l - R));  // the leaf's problem (R <= l)
  // no leaf lies above the tree's floor (every box there is split)
  const int mstop = max(R, *floor_d), ntask = 9 + 8 * max(0, l - mstop);
  int nu = 0, nw = 0;  // entries of the tasks before
  int* uo = FILL ? ulist + ustart[t] : nullptr;
  int* wo = FILL ? wlist + wstart[t] : nullptr;
  for (int k0 = 0; k0 < ntask; k0 += 32) {
    const int k = k0 + lane;
    // the task's box, if it exists, belongs to the problem and (coarser levels) is a leaf
    int C = -1;
    bool split = false;
    if (k < ntask) {
      const int up = k < 9 ? 0 : 1 + (k - 9) / 8, m = l - up;
      int q = k < 9 ? k : (k - 9) % 8;
      if (k >= 9 && q >= 4) ++q;  // not the ancestor itself
      const int sx = (ix >> up) + q % 3 - 1, sy = (iy >> up) + q / 3 - 1, side = 1 << m;
      if (sx >= 0 && sy >= 0 && sx < side && sy < side) {
        C = find_box(bkey, lo.v[m], lo.v[m + 1] - lo.v[m], morton((unsigned)sx, (unsigned)sy));
        if (C >= 0 && (bkey[C] >> (2 * (m - R))) != root) C = -1;
        if (C >= 0) {
          split = nchild[C] != 0;
          if (split && k >= 9) C = -1;
        }
      }
    }
    // below a split box of the leaf's level: counted first, written with the offsets known
    auto descend = [&](int* u, int* v, int& cu, int& cw) {
      int stack[EB_LIST_STACK];
      int sp = 0;
      for (int c = 0; c < nchild[C]; ++c) stack[sp++] = child0[C] + c;
      while (sp > 0) {
        const int D = stack[--sp];
        const int f = blev[D] - l;
        const unsigned long long kd = bkey[D];
        const int jx = (int)compact2(kd), jy = (int)compact2(kd >> 1);
        const int x0 = ix << f, x1 = ((ix + 1) << f) - 1, y0 = iy << f, y1 = ((iy + 1) << f) - 1;
        const bool adj = jx >= x0 - 1 && jx <= x1 + 1 && jy >= y0 - 1 && jy <= y1 + 1;
        if (!adj) {
          if (v) v[cw] = D;
          ++cw;
        } else if (nchild[D] == 0) {
          if (u) u[cu] = D;
          ++cu;
        } else if (sp + nchild[D] <= EB_LIST_STACK) {
          for (int c = 0; c < nchild[D]; ++c) stack[sp++] = child0[D] + c;
        } else {
          atomicOr(err, 1);
        }
      }
    };
    int cu = C >= 0 && !split, cw = 0;
    if (split && C >= 0) descend(nullptr, nullptr, cu, cw);
    __syncwarp();
    int eu = cu, ew = cw;  // inclusive sums over the lanes
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int a = __shfl_up_sync(0xffffffffu, eu, o), c = __shfl_up_sync(0xffffffffu, ew, o);
      if (lane >= o) {
        eu += a;
        ew += c;
      }
    }
    if (FILL && C >= 0) {
      if (!split) {
        uo[nu + eu - cu] = C;
      } else {
        int a = 0, c = 0;
        descend(uo + nu + eu - cu, wo + nw + ew - cw, a, c);
      }
    }
    nu += __shfl_sync(0xffffffffu, eu, 31);
    nw += __shfl_sync(0xffffffffu, ew, 31);
  }
  if (!FILL && lane == 0) {
    ucnt[t] = nu;
    wcnt[t] = nw;
  }
}

// Algorithmic work of the built tree: near-field pairs (self excluded), M2P evaluations
// (W-list box, target point) and M2L pairs.
__global__ void k_pair_counts(int nleaf, const int* __restrict__ leaves, const int* __restrict__ pt0,
                              const int* __restrict__ pt1, const int* __restrict__ ustart,
                              const int* __restrict__ ulist, const int* __restrict__ wstart,
                              int vfirst, int vlast, const int* __restrict__ vcount,
                              unsigned long long* __restrict__ out) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  unsigned long long up = 0, vp = 0, wp = 0;
  if (t < nleaf) {
    const int b = leaves[t];
    const long long nt = pt1[b] - pt0[b];
    long long ns = 0;
    for (int j = ustart[t]; j < ustart[t + 1]; ++j) {
      const int s = ulist[j];
      ns += pt1[s] - pt0[s];
    }
    up = (unsigned long long)(nt * ns - nt);
    wp = (unsigned long long)(nt * (wstart[t + 1] - wstart[t]));
  }
  for (int g = vfirst + blockIdx.x * blockDim.x + threadIdx.x; g < vlast; g += gridDim.x * blockDim.x)
    vp += (unsigned long long)vcount[g];
  up = warp_sum<unsigned long long>(up);
  vp = warp_sum<unsigned long long>(vp);
  wp = warp_sum<unsigned long long>(wp);
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(&out[0], up);
    atomicAdd(&out[1], vp);
    atomicAdd(&out[2], wp);
  }
}

inline int nblk(long long n, int bs) { return (int)((n + bs - 1) / bs); }

}  // namespace

namespace {
std::atomic<unsigned long long> g_epoch{1};
thread_local bool t_capturing = false;
std::mutex g_deferred_mu;
std::vector<void*> g_deferred;
}  // namespace

unsigned long long eb_devbuf_epoch() { return g_epoch.load(); }
void eb_devbuf_set_capturing(bool on) { t_capturing = on; }
void eb_devbuf_collect() {
  std::vector<void*> v;
  {
    std::lock_guard<std::mutex> lk(g_deferred_mu);
    v.swap(g_deferred);
  }
  for (void* q : v) cudaFree(q);
  if (!v.empty()) g_epoch++;  // no cached graph may keep an address freed here
}

int DevBuf::ensure(size_t nbytes) {
  if (nbytes <= bytes && p) return EB_OK;
  if (p && t_capturing) {
    std::lock_guard<std::mutex> lk(g_deferred_mu);
    g_deferred.push_back(p);
    p = nullptr;
    bytes = 0;
    g_epoch++;
  }
  release();
  size_t want = nbytes < 256 ? 256 : nbytes;
  cudaError_t e = cudaMalloc(&p, want);
  if (e != cudaSuccess) {
    p = nullptr;
    bytes = 0;
    eb_set_last_cuda_error(e, "cudaMalloc", __FILE__, __LINE__);
    return EB_ERR_CUDA;
  }
  bytes = want;
  return EB_OK;
}

void DevBuf::release() {
  if (p) {
    cudaFree(p);
    g_epoch++;
  }
  p = nullptr;
  bytes = 0;
}

// (z - x0 - (i + 1/2) r) / r, the offset of a coordinate from the centre of its leaf in
// leaf units, with both subtractions carried exactly (two-sum, two-product), so that
// for two nodes the offsets differ by exactly (z_j - z_i)/r minus the integer index
// offset of their leaves, up to the final roundings (2^-54 of a leaf side each). The division
// is a product with rinv = 1 / r and a correction by its exact remainder, so that the quotient
// is the rounded one: the product alone would stretch the offsets, but not the index offset, by
// the rounding of rinv (up to 2^-53), and an FP64 division is some twenty instructions on
// a pipe of two lanes a cycle.
__device__ __forceinline__ double leaf_offset(double z, double x0, unsigned int i, double r, double rinv) {
  double s = __dsub_rn(z, x0);
  double bb = __dsub_rn(s, z);
  double e1 = __dadd_rn(__dsub_rn(z, __dsub_rn(s, bb)), __dsub_rn(-x0, bb));
  double ci = (double)i + 0.5;
  double c = __dmul_rn(ci, r);
  double e2 = __fma_rn(ci, r, -c);
  double u = __dsub_rn(s, c);
  double bb2 = __dsub_rn(u, s);
  double e3 = __dadd_rn(__dsub_rn(s, __dsub_rn(u, bb2)), __dsub_rn(-c, bb2));
  const double a = __dadd_rn(u, __dadd_rn(__dsub_rn(e1, e2), e3));
  const double q = __dmul_rn(a, rinv);
  return __fma_rn(__fma_rn(-q, r, a), rinv, q);
}

// Leaf-relative node coordinates as three floats hi + mid + lo (all 53 bits of the
// double offset), for the double-float near field: wa = (x.hi, y.hi, x.mid, y.mid),
// wb = (x.lo, y.lo). (hi, mid) alone is a double-float. One thread per point: with a block
// per leaf, most of its lanes idle, 1,048,576 nodes took 212 us, now 121 (112 without the
// quotients' correction).
__device__ __forceinline__ void split3(double w, float& hi, float& mid, float& lo) {
  hi = __double2float_rn(w);
  double r1 = w - (double)hi;
  mid = __double2float_rn(r1);
  lo = __double2float_rn(r1 - (double)mid);
}

__global__ void __launch_bounds__(128) k_leaf_coords(int n, const int* __restrict__ lflag,
                              const int* __restrict__ lscan, const int* __restrict__ leaves,
                              const unsigned long long* __restrict__ bkey,
                              const unsigned char* __restrict__ blev, const double2* __restrict__ zs, double x0, double y0,
                              double W, double winv, float4* __restrict__ wa, float2* __restrict__ wb) {
  const int i = blockIdx.x * 128 + threadIdx.x;
  if (i >= n) return;
  const int b = leaves[lscan[i] + lflag[i] - 1];  // leaf heads up to point i
  const unsigned long long k = bkey[b];
  const unsigned int ix = compact2(k), iy = compact2(k >> 1);
  // W / 2^level, exact, and its rounded reciprocal
  const double r = W * __hiloint2double((1023 - (int)blev[b]) << 20, 0);
  const double rinv = winv * __hiloint2double((1023 + (int)blev[b]) << 20, 0);
  const double2 z = zs[i];
  float xh, xm, xl, yh, ym, yl;
  split3(leaf_offset(z.x, x0, ix, r, rinv), xh, xm, xl);
  split3(leaf_offset(z.y, y0, iy, r, rinv), yh, ym, yl);
  wa[i] = make_float4(xh, yh, xm, ym);
  wb[i] = make_float2(xl, yl);
}

// The tree of a problem that takes the direct sums: one kernel and one readback (the
// finiteness check) instead of the build; the FMM's apply then sums all pairs.
static int direct_tree(eb_ctx* ctx, EbTree& t, const double2* z, int n, int leaf_cap) {
  cudaStream_t st = eb_stream(ctx);
  t.direct = true;
  t.n = n;
  t.cap = leaf_cap;
  t.R = 0;
  t.wall = 0;
  t.ld = 0;
  t.L = 0;
  t.nbox = 1;
  t.nleaf = 1;
  t.ngroup = 0;
  t.ntile = 0;
  t.nchunk = 0;
  t.chunk_lmin = 2;
  t.lend = 2;
  t.nu = t.nw = 0;
  t.lev_off[0] = 0;
  for (int l = 1; l < EB_KEY_LEVELS + 2; ++l) t.lev_off[l] = 1;
  t.x0 = t.y0 = 0.0;
  t.W = 1.0;
  if (!t.host) EB_CUDA_TRY(cudaMallocHost(reinterpret_cast<void**>(&t.host), sizeof(EbTreeHost)));
  EB_TRY(t.perm.ensure(sizeof(int) * (size_t)n));
  EB_TRY(t.zs.ensure(sizeof(double2) * (size_t)n));
  EB_TRY(t.zhl.ensure(sizeof(float4) * (size_t)n));
  EB_TRY(t.bbox.ensure(sizeof(int)));
  // inside an RK call (ctx->defer) the flag accumulates in ctx->d_bad, read after the call
  int* bad = ctx->defer ? ctx->d_bad.as<int>() : t.bbox.as<int>();
  if (!ctx->defer) EB_CUDA_TRY(cudaMemsetAsync(bad, 0, sizeof(int), st));
  k_direct_points<<<nblk(n, 256), 256, 0, st>>>(z, n, t.perm.as<int>(), t.zs.as<double2>(), t.zhl.as<float4>(),
                                                bad);
  eb_count_launch(ctx);
  if (!ctx->defer) {
    EB_CUDA_TRY(cudaMemcpyAsync(&t.host->bad, bad, sizeof(int), cudaMemcpyDeviceToHost, st));
    EB_CUDA_TRY(cudaStreamSynchronize(st));
    if (t.host->bad & 1) {
      eb_set_last_error_msg("non-finite node coordinate");
      return EB_ERR_NAN;
    }
  }
  t.u_pairs = (long long)n * (n - 1);
  t.v_pairs = t.w_pairs = 0;
  t.pairs_read = true;
  t.valid = true;
  return eb_check_launch(ctx, "direct tree");
}

int eb_tree_build(eb_ctx* ctx, EbTree& t, const double2* z, int n, int leaf_target, int leaf_cap,
                  const double* root_sq, int root_level, int wall) {
  cudaStream_t st = eb_stream(ctx);
  t.valid = false;
  if (n <= 0) return EB_ERR_ARG;
  if (!root_sq && !wall && ctx->nsim == 0 && ctx->opts.direct_max > 0 && n <= ctx->opts.direct_max)
    return direct_tree(ctx, t, z, n, leaf_cap < 1 ? EB_LEAF_CAP : leaf_cap);
  t.direct = false;
  if (leaf_target < 1) leaf_target = 32;
  if (leaf_cap < 1) leaf_cap = EB_LEAF_CAP;
  t.n = n;
  t.cap = leaf_cap;
  t.R = root_sq ? root_level : 0;
  t.wall = wall && !root_sq;
  t.ld = 0;
  const int BS = 256;
  if (!t.host) EB_CUDA_TRY(cudaMallocHost(reinterpret_cast<void**>(&t.host), sizeof(EbTreeHost)));
  EbTreeHost* H = t.host;
  t.pairs_read = false;
  // (the whole build is a chain of small kernels, and their number and that of the copies
  // is what it costs, about 4 us each. A solve of 64 x 512 nodes, geometry installed, spent
  // 664 us before its first Krylov vector with 80 of them under a profiler, 288 us with 25, of
  // which the build's are 14 kernels, a memset and two readbacks; without one it went from 1,897
  // to 1,664 us, and the Cauchy sum of 60,001 points from 1,060 to 870 us)
  // 1. bounding square, on the device
  const int nbb = std::min(nblk(n, BS), 1024), nb256 = nblk(n, TREE_BS);
  EB_TRY(t.partial.ensure(sizeof(IBox) * (size_t)nbb));
  EB_TRY(t.dev.ensure(sizeof(TreeDev)));
  TreeDev* T = t.dev.as<TreeDev>();
  EB_CUDA_TRY(cudaMemsetAsync(T, 0, sizeof(TreeDev), st));
  k_bbox<<<nbb, BS, 0, st>>>(z, n, t.partial.as<IBox>(), t.wall, root_sq != nullptr,
                             root_sq ? mk_box4(root_sq[0], root_sq[1], root_sq[2], 0.0) : Box4(), T);
  eb_count_launch(ctx);
  // 2. keys and sort (a non-finite coordinate gives clamped keys; reported below)
  EB_TRY(t.keys.ensure(sizeof(unsigned long long) * (size_t)n));
  EB_TRY(t.perm.ensure(sizeof(int) * (size_t)n));
  EB_TRY(t.keys_alt.ensure(sizeof(unsigned long long) * (size_t)n));
  EB_TRY(t.idx_alt.ensure(sizeof(int) * (size_t)n));
  k_keys<<<nblk(n, 128), 128, 0, st>>>(z, n, T->sq, t.keys_alt.as<unsigned long long>(), t.idx_alt.as<int>());
  eb_count_launch(ctx);
  if (n <= SORT_MAX) {
    EB_CUDA_TRY(cudaFuncSetAttribute(k_sort, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    EB_CUDA_TRY(cudaFuncSetAttribute(k_sort, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SortSmem)));
    k_sort<<<SORT_CL, SORT_BS, sizeof(SortSmem), st>>>(t.keys_alt.as<unsigned long long>(), n,
                                                       t.keys.as<unsigned long long>(), t.perm.as<int>());
  } else {
    size_t tmp_sort = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, tmp_sort, t.keys_alt.as<unsigned long long>(),
                                    t.keys.as<unsigned long long>(), t.idx_alt.as<int>(),
                                    t.perm.as<int>(), n, 0, 2 * EB_KEY_LEVELS, st);
    EB_TRY(t.cubtmp.ensure(tmp_sort));
    size_t tb = t.cubtmp.bytes;
    EB_CUDA_TRY(cub::DeviceRadixSort::SortPairs(t.cubtmp.p, tb, t.keys_alt.as<unsigned long long>(),
                                                t.keys.as<unsigned long long>(), t.idx_alt.as<int>(),
                                                t.perm.as<int>(), n, 0, 2 * EB_KEY_LEVELS, st));
  }
  eb_count_launch(ctx);
  const unsigned long long* keys = t.keys.as<unsigned long long>();
  // 3. sorted positions and the uniform floor
  EB_TRY(t.zs.ensure(sizeof(double2) * (size_t)n));
  EB_TRY(t.zhl.ensure(sizeof(float4) * (size_t)n));
  k_gather_points<<<nblk(n, 256), 256, 0, st>>>(z, t.perm.as<int>(), keys, n, leaf_target, t.R, t.zs.as<double2>(),
                                                t.zhl.as<float4>(), T);
  eb_count_launch(ctx);
  // 4. leaf level of every point, deepest level, boxes per level
  EB_TRY(t.lcpw.ensure((size_t)n));
  EB_TRY(t.plev.ensure((size_t)n));
  EB_TRY(t.bc.ensure(sizeof(int) * (EB_KEY_LEVELS + 1) * (size_t)nb256));
  if (n > leaf_cap) {
    k_lcp_window<<<nblk(n - leaf_cap, BS), BS, 0, st>>>(keys, n, leaf_cap, t.lcpw.as<unsigned char>());
    eb_count_launch(ctx);
  }
  k_leaf_level<<<nb256, TREE_BS, 0, st>>>(keys, n, leaf_cap, t.lcpw.as<unsigned char>(), t.plev.as<unsigned char>(),
                                          t.bc.as<int>(), T);
  k_scan_rows<<<EB_KEY_LEVELS + 1, SCAN_BS, 0, st>>>(nb256, t.bc.as<int>(), T);
  ctx->launches += 2;
  EB_CUDA_TRY(cudaMemcpyAsync(H->sq, T, offsetof(TreeDev, last), cudaMemcpyDeviceToHost, st));
  EB_CUDA_TRY(cudaStreamSynchronize(st));
  if (H->bad & 1) {
    eb_set_last_error_msg("non-finite node coordinate");
    return EB_ERR_NAN;
  }
  if (H->bad & 2) {
    eb_set_last_error_msg("wall-bounded flow: a node lies below the wall y = 0");
    return EB_ERR_ARG;
  }
  t.W = H->sq[0];
  t.x0 = H->sq[1];
  t.y0 = H->sq[2];
  int L = EB_KEY_LEVELS;  // the deepest leaf level: the last one with boxes
  while (L > 0 && H->hist[L] == 0) --L;
  t.L = L;
  t.lev_off[0] = 0;
  for (int l = 0; l <= L; ++l) t.lev_off[l + 1] = t.lev_off[l] + (l == 0 ? 1 : H->hist[l]);
  for (int l = L + 1; l <= EB_KEY_LEVELS; ++l) t.lev_off[l + 1] = t.lev_off[L + 1];
  t.nbox = t.lev_off[L + 1];
  t.lend = std::max(2, L - EB_FAR_LEVELS + 1);
  const size_t NB = (size_t)t.nbox;
  EB_TRY(t.bkey.ensure(sizeof(unsigned long long) * NB));
  EB_TRY(t.blev.ensure(NB));
  EB_TRY(t.pt0.ensure(sizeof(int) * NB));
  EB_TRY(t.pt1.ensure(sizeof(int) * NB));
  EB_TRY(t.parent.ensure(sizeof(int) * NB));
  EB_TRY(t.child0.ensure(sizeof(int) * NB));
  EB_TRY(t.nchild.ensure(sizeof(int) * NB));
  // 5. boxes of every level, leaves in point order
  EB_TRY(t.lflag.ensure(sizeof(int) * (size_t)n));
  EB_TRY(t.lscan.ensure(sizeof(int) * (size_t)n));
  EB_TRY(t.leaves.ensure(sizeof(int) * NB));
  EB_TRY(t.vcount.ensure(sizeof(int) * NB));
  LevOffT lo;
  for (int l = 0; l < EB_KEY_LEVELS + 3; ++l) lo.v[l] = t.lev_off[std::min(l, L + 1)];
  k_boxes<<<nb256, TREE_BS, 0, st>>>(keys, t.plev.as<unsigned char>(), n, L, lo, t.bc.as<int>(),
                                     t.bkey.as<unsigned long long>(), t.blev.as<unsigned char>(), t.pt0.as<int>(),
                                     t.parent.as<int>(), t.child0.as<int>(), t.nchild.as<int>(), t.vcount.as<int>(),
                                     t.lflag.as<int>(), t.lscan.as<int>(), t.leaves.as<int>());
  k_boxes_fin<<<nblk(t.nbox, BS), BS, 0, st>>>(t.nbox, keys, n, t.bkey.as<unsigned long long>(),
                                              t.blev.as<unsigned char>(), t.pt0.as<int>(), t.parent.as<int>(),
                                              t.pt1.as<int>(), t.nchild.as<int>());
  ctx->launches += 2;
  // 7. V lists of every box of levels >= 2
  EB_TRY(t.vlist.ensure(sizeof(int) * NB * EB_VMAX));
  EB_TRY(t.vcode.ensure(NB * EB_VMAX));
  if (L >= 2) {
    const int first = t.lev_off[2];
    k_vlist<<<nblk(32LL * (t.nbox - first), 128), 128, 0, st>>>(t.bkey.as<unsigned long long>(), lo, first, t.nbox, t.R,
                                                       t.vlist.as<int>(), t.vcode.as<unsigned char>(),
                                                       t.vcount.as<int>());
    eb_count_launch(ctx);
  }
  // 7b. image lists of the wall (levels 2..ld, ld the uniform floor)
  if (t.wall && L >= 2 && H->lmin >= 2) {
    t.ld = std::min(H->lmin, L);
    const int first = t.lev_off[2], nimg = t.lev_off[t.ld + 1];
    EB_TRY(t.ilist.ensure(sizeof(int) * (size_t)nimg * EB_VMAX));
    EB_TRY(t.icode.ensure((size_t)nimg * EB_VMAX));
    EB_TRY(t.icount.ensure(sizeof(int) * (size_t)nimg));
    EB_CUDA_TRY(cudaMemsetAsync(t.icount.p, 0, sizeof(int) * (size_t)nimg, st));
    k_imglist<<<nblk(nimg - first, 128), 128, 0, st>>>(t.bkey.as<unsigned long long>(), t.blev.as<unsigned char>(),
                                                       lo, first, nimg, t.ilist.as<int>(),
                                                       t.icode.as<unsigned char>(), t.icount.as<int>());
    eb_count_launch(ctx);
  }
  // 8. per-leaf counts, scanned so that one synchronisation sizes them all: U and W list
  // lengths, near-field groups of EB_GROUP targets, shared-memory tiles of at most
  // EB_NTILE targets, and FP32 direct-P2M chunks of at most EB_CHUNK points of every box
  // of the chunked levels (every level up to 256K points, so that no dependent M2M
  // launches remain on the critical path; above that the EB_DIRECT_LEVELS finest).
  // The leaf count is known on the device only: the counting kernel runs over nbox + 1
  // threads and leaves zeros beyond it, and the scans span nbox + 1 entries.
  const int NBi = t.nbox;
  t.nchunk = 0;
  t.chunk_lmin = n <= (1 << 18) ? 2 : std::max(2, L - EB_DIRECT_LEVELS + 1);
  const int cfirst = t.lev_off[std::min(2, L + 1)], nb2 = L >= 2 ? t.nbox - cfirst : 0;
  for (DevBuf* d : {&t.ucnt, &t.wcnt, &t.ustart, &t.wstart, &t.tcount, &t.tstart, &t.gcount, &t.gstart})
    EB_TRY(d->ensure(sizeof(int) * (NB + 1)));
  for (DevBuf* d : {&t.ccount, &t.cstart, &t.cdone}) EB_TRY(d->ensure(sizeof(int) * (size_t)(nb2 + 1)));
  WorkItems W{t.pt0.as<int>(),    t.pt1.as<int>(),    t.parent.as<int>(), t.gcount.as<int>(), t.tcount.as<int>(),
              t.ccount.as<int>(), t.gstart.as<int>(), t.tstart.as<int>(), t.cstart.as<int>(), nullptr,
              nullptr,            nullptr,            nullptr,            nullptr,            t.cdone.as<int>(),
              NBi,                cfirst,             nb2,                t.chunk_lmin,       t.lend};
  k_leaf_lists<false><<<nblk(32LL * NBi + 1, 128), 128, 0, st>>>(W, NBi, &T->last[0], t.leaves.as<int>(),
                                                       t.bkey.as<unsigned long long>(),
                                                       t.blev.as<unsigned char>(), lo, t.R, &T->lmin, t.child0.as<int>(),
                                                       t.nchild.as<int>(), t.ucnt.as<int>(), t.wcnt.as<int>(),
                                                       nullptr, nullptr, nullptr, nullptr, &T->last[5]);
  const ScanJobs jobs{{{t.gcount.as<int>(), t.gstart.as<int>(), &T->last[1], NBi + 1},
                       {t.tcount.as<int>(), t.tstart.as<int>(), &T->last[2], NBi + 1},
                       {t.ucnt.as<int>(), t.ustart.as<int>(), &T->last[3], NBi + 1},
                       {t.wcnt.as<int>(), t.wstart.as<int>(), &T->last[4], NBi + 1},
                       {t.ccount.as<int>(), t.cstart.as<int>(), &T->last[6], nb2 + 1}}};
  k_scan<<<nb2 > 0 ? 5 : 4, SCAN_BS, 0, st>>>(jobs);
  ctx->launches += 2;
  EB_CUDA_TRY(cudaMemcpyAsync(H->last, T->last, sizeof(T->last), cudaMemcpyDeviceToHost, st));
  EB_CUDA_TRY(cudaStreamSynchronize(st));
  if (H->last[5]) {
    eb_set_last_error_msg("tree build: interaction-list traversal deeper than its stack");
    return EB_ERR_WORKSPACE;
  }
  const int nl = H->last[0];
  t.nleaf = nl;
  t.ngroup = H->last[1];
  t.ntile = H->last[2];
  t.nu = H->last[3];
  t.nw = H->last[4];
  // 9. fill the lists and work items
  EB_TRY(t.ulist.ensure(sizeof(int) * (size_t)std::max<long long>(t.nu, 1)));
  EB_TRY(t.wlist.ensure(sizeof(int) * (size_t)std::max<long long>(t.nw, 1)));
  EB_TRY(t.gleaf.ensure(sizeof(int) * (size_t)t.ngroup));
  EB_TRY(t.gfirst.ensure(sizeof(int) * (size_t)t.ngroup));
  EB_TRY(t.tiles.ensure(sizeof(int4) * (size_t)t.ntile));
  EB_TRY(t.anc.ensure(sizeof(int) * (size_t)nl * EB_FAR_LEVELS));
  t.nchunk = nb2 > 0 ? H->last[6] : 0;
  EB_TRY(t.chunk_box.ensure(sizeof(int) * (size_t)std::max(t.nchunk, 1)));
  W.gleaf = t.gleaf.as<int>();
  W.gfirst = t.gfirst.as<int>();
  W.tiles = t.tiles.as<int4>();
  W.anc = t.anc.as<int>();
  W.chunk_box = t.chunk_box.as<int>();
  k_leaf_lists<true><<<nblk(std::max(32LL * nl, (long long)nb2), 128), 128, 0, st>>>(W, nl, nullptr, t.leaves.as<int>(),
                                                     t.bkey.as<unsigned long long>(),
                                                     t.blev.as<unsigned char>(), lo, t.R, &T->lmin, t.child0.as<int>(),
                                                     t.nchild.as<int>(), nullptr, nullptr, t.ustart.as<int>(),
                                                     t.wstart.as<int>(), t.ulist.as<int>(), t.wlist.as<int>(),
                                                     &T->last[5]);
  eb_count_launch(ctx);
  // 10. leaf-relative coordinates for the double-float kernels and the FP32 P2M / far field
  EB_TRY(t.wdf.ensure(sizeof(float4) * (size_t)n));
  EB_TRY(t.wdf_lo.ensure(sizeof(float2) * (size_t)n));
  k_leaf_coords<<<nblk(n, 128), 128, 0, st>>>(n, t.lflag.as<int>(), t.lscan.as<int>(), t.leaves.as<int>(),
                                   t.bkey.as<unsigned long long>(), t.blev.as<unsigned char>(), t.zs.as<double2>(),
                                   t.x0, t.y0, t.W, 1.0 / t.W, t.wdf.as<float4>(), t.wdf_lo.as<float2>());
  eb_count_launch(ctx);
  EB_TRY(eb_check_launch(ctx, "tree build"));
  t.valid = true;
  return EB_OK;
}

// Pair counts (the algorithmic work of the near field, M2P and M2L), counted on the
// device when first asked for after a build (they are statistics, not inputs of any
// apply, so the build does not spend a launch on them).
int eb_tree_pairs(eb_ctx* ctx, EbTree& t) {
  if (!t.pairs_read) {
    if (!t.valid) return EB_ERR_NOGEOM;
    cudaStream_t st = eb_stream(ctx);
    const int BS = 256, nl = t.nleaf, L = t.L;
    EB_TRY(t.pairs.ensure(3 * sizeof(unsigned long long)));
    unsigned long long* cnt = t.pairs.as<unsigned long long>();
    EB_CUDA_TRY(cudaMemsetAsync(cnt, 0, 3 * sizeof(unsigned long long), st));
    int vfirst = t.lev_off[std::min(2, L + 1)], vlast = t.nbox;
    k_pair_counts<<<std::max(nblk(nl, BS), 1), BS, 0, st>>>(nl, t.leaves.as<int>(), t.pt0.as<int>(),
                                                           t.pt1.as<int>(), t.ustart.as<int>(), t.ulist.as<int>(),
                                                           t.wstart.as<int>(), vfirst, vlast, t.vcount.as<int>(), cnt);
    eb_count_launch(ctx);
    EB_CUDA_TRY(cudaMemcpyAsync(t.host->pairs, cnt, sizeof(t.host->pairs), cudaMemcpyDeviceToHost, st));
    EB_CUDA_TRY(cudaStreamSynchronize(st));
    t.u_pairs = (long long)t.host->pairs[0];
    t.v_pairs = (long long)t.host->pairs[1];
    t.w_pairs = (long long)t.host->pairs[2];
    t.pairs_read = true;
  }
  return EB_OK;
}

EbTree::~EbTree() {
  if (host) cudaFreeHost(host);
}
