// M2L of the FP64-class operators (native FP64 and double-float) in fixed point, its
// contraction on the 5th-generation tensor cores.
//
// SLSHIFT (cadap2.f:1149-1215) and DSLNEW (dapif3.f:1200-1289) factor the M2L of an
// interaction-list entry with offset d (in box units) into two diagonal scalings around a
// fixed binomial matrix; with the powers of two shared out so that every factor is at most 1,
//   a_k = (2/d)^k M_k              (after moving psi to the target centre),
//   b_m = sum_k C(m+k-1, m) 2^-(m+k) a_k,
//   L_m += (-1)^m (2/d)^m b_m.
// GB300 issues two FP64 lanes a cycle and SM against 64 32-bit integer ones and some 4,000
// tensor multiply-adds, so nothing here is done in FP64:
//  * k_m2l_fix turns each box's multipoles into 64-bit integers, 61 bits below the largest
//    coefficient of phi and of psi, with one exponent each;
//  * the scalings are 64 x 64-bit multiplies of which the high half is kept, of operands
//    split into two signed 32-bit limbs (six 32 x 32 + 64 multiply-adds a complex part);
//  * a_k, brought to 54 bits below the entry's largest one, and the binomial matrix, 54 bits
//    below each row's largest entry, become six signed 9-bit digits each, exact in FP16; the
//    products of digits i and j go to the accumulator i + j <= 6, whose sums are integers
//    below 2^24 and so exact in FP32 (what i + j = 7 would add is below 2^-60). One tile is
//    128 rows (Re / Im of phi and psi of 32 entries, or of phi of 64) x 48 orders, 26 digit
//    pairs of three tcgen05.mma (kind::f16, M = 128, N = 48, K = 16) each, with seven
//    accumulators of 48 tensor-memory columns;
//  * the entries of a target box are added as 64-bit integers with one exponent (the same
//    result in any order) and become double or double-float once per box.
// Errors of the sums against direct sums are those of the FP64 kernel (k_m2l) or smaller (a
// single small coefficient of a high order keeps fewer bits than in FP64: all are held to the
// largest of their entry).
//
// What bounds it is the issue of the integer work before and after the products. One block
// per SM (its accumulators fill the tensor memory) of two teams of 16 warps, each with
// its own digits, runs a round of one team's integer work under the other's: the team that
// holds the tensor memory issues its products, reads the sums and passes it on.
// Measured (E = 2, p = 44; k_m2l is the FP64 CUDA-core kernel): 13,290 entries of 64 x 512
// 222 -> 71 us, 497,412 entries of 1,024 x 1,024 6.73 -> 1.44 ms (about 830 cycles an entry
// and SM); E = 1, some 73,000 entries of 60,001 scattered points 1,035 -> 201 us. In the
// double-float pipeline with the multipoles' conversion: 1,024 x 1,024 2.48 (k_m2l_df) ->
// 1.55 ms. There, E = 2 takes it always and E = 1 from 3,072 boxes on: an apply takes
// (k_m2l_df / this) 841 / 767, 409 / 383, 255 / 251, 139 / 131 and 91 / 90 us for 256 x 512,
// 64 x 1,024, 64 x 512, 16 x 512 and 1 x 2,048 nodes (E = 2), 557 / 483, 287 / 277, 187 / 188,
// 106 / 115 and 75 / 81 us for E = 1.
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <vector>

#include "eb_internal.h"

namespace {

constexpr int FX_KCH = EB_FX_K / 8;         // 16-byte chunks along K per row group
constexpr uint32_t FX_LBO = 128, FX_SBO = FX_KCH * 128;
constexpr int FX_ROWS = 128;                // rows of a tile
constexpr int FX_A = FX_ROWS * EB_FX_K * 2; // bytes of a digit of the data
constexpr int FX_B = EB_FX_K * EB_FX_K * 2; // bytes of a digit of the matrix
constexpr int FX_ND = 6;                    // digits of a number
constexpr int FX_NACC = 7;                  // accumulators (digit pairs i + j = 0 .. 6)
constexpr int FX_COLS = 512;                // tensor-memory columns (7 x 48, a power of two)
constexpr int FX_TEAM = 512;                // threads of a team
constexpr int FX_THREADS = 2 * FX_TEAM;
constexpr int FX_PITCH = FX_ROWS + 4;       // row pitch of the contributions (int64)
constexpr int FX_GROUP = 8;                 // target boxes of a work item, at most
constexpr int FX_BAD = 1 << 20;             // exponent of a box with a non-finite multipole
static_assert(EB_FX_K == 48, "the accumulators' columns and the digit layout");
static_assert(EB_FX_K * FX_PITCH * 8 <= FX_ND * FX_A, "the contributions reuse the digits' memory");

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// shared-memory matrix descriptor (K-major core matrices of 8 rows x 16 bytes, no swizzle)
__device__ __forceinline__ uint64_t fx_desc(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(FX_LBO >> 4) << 16) |
         ((uint64_t)(FX_SBO >> 4) << 32) | (1ull << 46);
}

// instruction descriptor: D f32 (bits 4-5 = 1), A and B f16 (bits 7-9, 10-12 = 0), both
// K-major, N >> 3 at bits 17-22, M >> 4 at bits 24-28
constexpr uint32_t FX_IDESC = (1u << 4) | ((uint32_t)(EB_FX_K >> 3) << 17) | ((uint32_t)(FX_ROWS >> 4) << 24);

__device__ __forceinline__ void fx_mma(uint32_t taddr, uint64_t a, uint64_t b, uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(taddr),
      "l"(a), "l"(b), "r"(FX_IDESC), "r"(acc));
}

// A 64-bit integer as two signed limbs, x = hi 2^32 + lo
struct Limb {
  int hi, lo;
};
__device__ __forceinline__ Limb limbs(long long x) {
  return Limb{(int)(x >> 32) + (int)((uint32_t)x >> 31), (int)x};
}

// a b + c of 32-bit a and b and 64-bit c in one instruction (a product of sign-extended
// truncations written in C becomes a 64-bit multiplication: three multiply-adds and shifts)
__device__ __forceinline__ long long madw(int a, int b, long long c) {
  long long d;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
  return d;
}

// (x yr + y yi) / 2^64, the lowest parts left out (an error of at most two units), for
// |x|, |y| < 2^61.5 and table entries of at most 2^62: every partial sum is below 2^63
__device__ __forceinline__ long long mul_add_hi(Limb x, int yrh, int yrl, Limb y, int yih, int yil) {
  const long long mid = madw(x.hi, yrl, madw(x.lo, yrh, madw(y.hi, yil, madw(y.lo, yih, 0x80000000ll))));
  return madw(x.hi, yrh, madw(y.hi, yih, (long long)(int)(mid >> 32)));
}

// 2^e of any e: two factors, the first clamped so that a result in range stays exact
__device__ __forceinline__ double scale2(double v, int e) {
  const int e1 = max(-1000, min(1000, e)), e2 = max(-1000, min(1000, e - e1));
  return v * __hiloint2double((1023 + e1) << 20, 0) * __hiloint2double((1023 + e2) << 20, 0);
}

// x << n, x >> n for 0 <= n < 32
__device__ __forceinline__ long long shl31(long long x, int n) {
  return (long long)(((unsigned long long)__funnelshift_l((uint32_t)x, (uint32_t)(x >> 32), n) << 32) |
                     ((uint32_t)x << n));
}
__device__ __forceinline__ long long sra31(long long x, int n) {
  return ((long long)((int)(x >> 32) >> n) << 32) | __funnelshift_r((uint32_t)x, (uint32_t)(x >> 32), n);
}

__device__ __forceinline__ int exp_above(uint32_t hiabs) {  // e with |v| < 2^e, v's high word given
  return (int)(hiabs >> 20) - 1022;
}

// Multipoles of the boxes [first, first + nb) as 64-bit integers, one warp per box:
// fx = v 2^(61 - S), 2^S above the box's largest part of phi (fs.x) and of psi (fs.y); fs.z is
// the exponent above the largest part of k phi_k, which moving psi to another centre adds.
// Double-float multipoles without FP64: the exponents are those of the high floats, and both
// floats of a part are shifted into place as integers.
__device__ __forceinline__ long long float_fix(float f, int S) {  // f 2^(61 - S), |f| < 2^S
  const uint32_t b = __float_as_uint(f);
  const int e = (int)((b >> 23) & 255u), m = (int)((b & 0x7fffffu) | (e ? 0x800000u : 0u));
  const int sh = max(e, 1) - 89 - S;
  const long long v = sh >= 0 ? (long long)m << min(sh, 40) : sh > -32 ? (long long)((m + (1 << (-sh - 1))) >> -sh) : 0;
  return (int)b < 0 ? -v : v;
}

template <int E, bool DF>
__global__ void __launch_bounds__(128) k_m2l_fix(int first, int nb, int p, const void* __restrict__ mpole,
                                                 longlong2* __restrict__ fx, int4* __restrict__ fs) {
  pdl_wait();
  const int wb = (blockIdx.x * 128 + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (wb >= nb) return;
  const size_t b = (size_t)(first + wb), n = (size_t)E * p;
  const double2* md = reinterpret_cast<const double2*>(mpole) + b * n;
  const float4* mf = reinterpret_cast<const float4*>(mpole) + b * n;
  // the largest parts' magnitude bits (double: the high words; double-float: the high floats),
  // and those of k phi_k rounded up
  uint32_t h[2] = {0u, 0u}, hk = 0u;
  for (int o = lane; o < E * p; o += 32) {
    uint32_t m;
    if (DF) {
      const float4 v = mf[o];
      m = max(__float_as_uint(v.x) & 0x7fffffffu, __float_as_uint(v.z) & 0x7fffffffu);
    } else {
      const double2 v = md[o];
      m = max((uint32_t)__double2hiint(v.x) & 0x7fffffffu, (uint32_t)__double2hiint(v.y) & 0x7fffffffu);
    }
    if (E == 1 || o < p) {
      h[0] = max(h[0], m);
      if (E == 2) {
        const float k = (float)(o + 1);
        if (DF) hk = max(hk, __float_as_uint(__fmul_ru(__uint_as_float(m), k)));
        else {  // the exponent field plus that of (top mantissa bits + 1) x k
          const float t = __fmul_ru(__uint_as_float(0x3f800000u + (((m & 0xfffffu) + 1u) << 3)), k);
          hk = max(hk, (m & 0x7ff00000u) + ((__float_as_uint(t) >> 23) - 127u) * (1u << 20));
        }
      }
    } else {
      h[1] = max(h[1], m);
    }
  }
  h[0] = __reduce_max_sync(0xffffffffu, h[0]);
  if (E == 2) {
    h[1] = __reduce_max_sync(0xffffffffu, h[1]);
    hk = __reduce_max_sync(0xffffffffu, hk);
  }
  auto above = [](uint32_t m) { return DF ? (int)(m >> 23) - 126 : exp_above(m); };
  const bool bad = max(h[0], h[1]) >= (DF ? 0x7f800000u : 0x7ff00000u);
  int S[2];
#pragma unroll
  for (int e = 0; e < E; ++e) S[e] = above(h[e]);  // down to -1022: zeros and subnormals too
  if (lane == 0) fs[b] = make_int4(bad ? FX_BAD : S[0], S[E - 1], max(above(hk), S[0]), 0);
  for (int o = lane; o < E * p; o += 32) {
    const int Se = E == 1 || o < p ? S[0] : S[E - 1];
    longlong2 r = make_longlong2(0, 0);
    if (!bad && DF) {
      const float4 v = mf[o];
      r.x = float_fix(v.x, Se) + float_fix(v.y, Se);
      r.y = float_fix(v.z, Se) + float_fix(v.w, Se);
    } else if (!bad) {
      const double2 v = md[o];
      // 2^(61 - S) as two factors (S from -1022 to 1024)
      const int e1 = (61 - Se) >> 1, e2 = 61 - Se - e1;
      const double f1 = __hiloint2double((1023 + e1) << 20, 0), f2 = __hiloint2double((1023 + e2) << 20, 0);
      r.x = __double2ll_rn(v.x * f1 * f2);
      r.y = __double2ll_rn(v.y * f1 * f2);
    }
    fx[b * n + o] = r;
  }
}

// (x c + y d) 2^-q for |x|, |y| < 2^61 and small integers (|c| + |d| < 2^10), q >= 1 such
// that the result stays below 2^62: the operands in 31-bit parts
__device__ __forceinline__ long long small_mul(long long x, int c, long long y, int d, int q) {
  const int mask = 0x7fffffff;
  const long long h = madw((int)(x >> 31), c, madw((int)(y >> 31), d, 0));
  const long long l = madw((int)x & mask, c, madw((int)y & mask, d, 0));
  return q <= 31 ? shl31(h, 31 - q) + sra31(l, q) : (h + (l >> 31)) >> min(q - 31, 63);
}

// The six digits of two neighbouring columns (k, k + 1) of a row from x0, x1 2^-r rounded
// (|x| 2^-r <= 2^53, 0 < r < 8): 256 added to every digit, so that fields of 9 bits hold
// digit + 256 >= 0; 0x6400 | f is the FP16 number 1024 + f, and minus 1280 leaves the digit.
__device__ __forceinline__ void store_digits(unsigned char* at, long long x0, long long x1, int r, long long bias) {
  const unsigned long long u = (unsigned long long)(x0 + bias), v = (unsigned long long)(x1 + bias);
  const uint32_t ul = __funnelshift_r((uint32_t)u, (uint32_t)(u >> 32), r), uh = (uint32_t)(u >> 32) >> r;
  const uint32_t vl = __funnelshift_r((uint32_t)v, (uint32_t)(v >> 32), r), vh = (uint32_t)(v >> 32) >> r;
  const uint32_t um = __funnelshift_r(ul, uh, 27), vm = __funnelshift_r(vl, vh, 27);
  auto put = [&](int i, uint32_t a, uint32_t b, uint32_t mask) {
    uint32_t pk = (__byte_perm(a, b, 0x5410) & mask) | 0x64006400u;
    asm("sub.rn.f16x2 %0, %0, %1;" : "+r"(pk) : "r"(0x65006500u));
    *reinterpret_cast<uint32_t*>(at + i * FX_A) = pk;
  };
  put(5, ul, vl, 0x01ff01ffu);
  put(4, ul >> 9, vl >> 9, 0x01ff01ffu);
  put(3, ul >> 18, vl >> 18, 0x01ff01ffu);
  put(2, um, vm, 0x01ff01ffu);
  put(1, um >> 9, vm >> 9, 0x01ff01ffu);
  put(0, um >> 18, vm >> 18, 0x03ff03ffu);  // digit 0: 0 .. 512
}

__device__ __forceinline__ uint32_t hi_abs(long long x) {
  const int h = (int)(x >> 32);
  return (uint32_t)(h < 0 ? ~h : h);
}

__device__ __forceinline__ void team_sync(int team) {
  asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "n"(FX_TEAM) : "memory");
}

template <int E, bool DF>
__global__ void __launch_bounds__(FX_THREADS, 1) k_m2l_fx(int first, int ntarget, const int* __restrict__ vlist,
                                                          const unsigned char* __restrict__ vcode,
                                                          const int* __restrict__ vcount, int p,
                                                          const uint4* __restrict__ bdig,
                                                          const int4* __restrict__ tab, const int* __restrict__ rsc,
                                                          const int* __restrict__ pdv,
                                                          const longlong2* __restrict__ fx,
                                                          const int4* __restrict__ fs, void* __restrict__ local,
                                                          int accumulate, int nsingle, int group, long long lim0,
                                                          long long lim1) {
  pdl_wait();
  constexpr int NE = FX_ROWS / (2 * E);  // entries of a round
  constexpr int NW = FX_TEAM / 32;
  // 256 in each digit, see store_digits
  constexpr long long BIAS = 256ll * (1ll + (1ll << 9) + (1ll << 18) + (1ll << 27) + (1ll << 36) + (1ll << 45));
  extern __shared__ __align__(1024) unsigned char sm[];
  __shared__ __align__(8) unsigned long long mbar[2];
  __shared__ uint32_t s_taddr;
  __shared__ int sv_src[2][NE], sv_code[2][NE], sv_pd[2][NE], sv_box[2][NE], sv_exp[2][E][NE];
  __shared__ int sv_e0[2][FX_GROUP + 1], sv_E[2][E][FX_GROUP], sv_cnt[2][FX_GROUP], s_pdv[EB_NCODE];
  // s_fail: of a team (1: no tensor memory, 2: products whose end it did not see), written by its
  // first thread before a team_sync and read by the team behind it, so that all its threads
  // leave together; s_lock: the tensor memory is taken
  __shared__ int s_fail[2], s_lock;
  const int team = threadIdx.x / FX_TEAM, tid = threadIdx.x - team * FX_TEAM, warp = tid >> 5, lane = tid & 31;
  int *s_src = sv_src[team], *s_code = sv_code[team], *s_pd = sv_pd[team], *s_box = sv_box[team];
  int *s_cnt = sv_cnt[team], *s_e0 = sv_e0[team], (*s_exp)[NE] = sv_exp[team], (*s_E)[FX_GROUP] = sv_E[team];
  unsigned char* sB = sm;                                                   // [digit][48 x 48]
  unsigned char* sA = sm + FX_ND * FX_B + (size_t)team * FX_ND * FX_A;      // [digit][128 x 48], then
  long long* sC = reinterpret_cast<long long*>(sA);                         // the contributions
  const int ldl = p + 1, ldt = p + 2;
  const int4* tabp = tab + (size_t)EB_NCODE * ldt;  // (-1)^m (2/d)^m
  for (int i = threadIdx.x; i < FX_ND * FX_B / 16; i += FX_THREADS) reinterpret_cast<uint4*>(sB)[i] = bdig[i];
  for (int i = threadIdx.x; i < EB_NCODE; i += FX_THREADS) s_pdv[i] = pdv[i];
  if (threadIdx.x == 0) {
    s_fail[0] = s_fail[1] = 0;
    s_lock = 0;
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&mbar[0])));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&mbar[1])));
    asm volatile("fence.mbarrier_init.release.cluster;");
  }
  if (threadIdx.x < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_taddr)),
                 "r"(FX_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("fence.proxy.async.shared::cta;");
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t taddr = s_taddr;
  uint32_t phase = 0;
  auto products_done = [&](uint32_t parity) {  // bounded
    uint32_t done = 0;
    for (long long it = 0; it < EB_FX_WAIT && !done; ++it)
      asm volatile(
          "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
          " selp.u32 %0, 1, 0, p;\n}\n"
          : "=r"(done)
          : "r"(smem_u32(&mbar[team])), "r"(parity)
          : "memory");
    return done != 0;
  };

  // work items: the first nsingle boxes one by one, the others in groups; teams in turn
  const int nitem = nsingle + (ntarget - nsingle + group - 1) / group, step = 2 * gridDim.x;
  auto item_box = [&](int g) { return g < nsingle ? g : min(ntarget, nsingle + (g - nsingle) * group); };
  for (int g = team * gridDim.x + blockIdx.x; g < nitem; g += step) {
    const int gb0 = item_box(g), gb1 = item_box(g + 1);
    if (tid < gb1 - gb0) s_cnt[tid] = vcount[first + gb0 + tid];
    team_sync(team);
    int b0 = gb0;
    while (b0 < gb1) {
      // a round: the next boxes of the item whose entries fit (a box has at most 27)
      int b1 = b0, ne = 0, mine = -1, mine0 = 0;
      while (b1 < gb1) {
        const int c = s_cnt[b1 - gb0];
        if (ne + c > NE) break;
        if (tid == 0) s_e0[b1 - b0] = ne;
        if (tid >= ne && tid < ne + c) {
          mine = b1;
          mine0 = ne;
        }
        ne += c;
        ++b1;
      }
      const int nbx = b1 - b0;
      if (tid == 0) s_e0[nbx] = ne;
      if (mine >= 0) {
        const size_t at = (size_t)(first + mine) * EB_VMAX + tid - mine0;
        const int code = vcode[at];
        s_src[tid] = vlist[at];
        s_code[tid] = code;
        s_pd[tid] = s_pdv[code];
        s_box[tid] = mine - b0;
      }
      team_sync(team);
      if (ne > 0) {
        // the digits of a: a warp per entry and expansion, two columns per lane (the rows of
        // entries beyond ne hold anything: a row's products stay in its row)
        for (int it = warp; it < E * ne; it += NW) {
          const int en = E == 2 ? it >> 1 : it, e = E == 2 ? it & 1 : 0;
          const int kk = 2 * lane;  // columns kk, kk + 1: orders k = kk + 1, kk + 2
          const int code = s_code[en], pd = s_pd[en], src = s_src[en];
          const longlong2* ms = fx + (size_t)src * E * p + kk;
          const int4 S = fs[src];
          const int4* tb = tab + (size_t)code * ldt + kk + 1;
          longlong2 y[2];
          int4 t[2];
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const bool in = kk + q < pd;
            y[q] = in ? ms[q + e * p] : make_longlong2(0, 0);
            t[q] = in ? tb[q] : make_int4(0, 0, 0, 0);
          }
          int ex = S.x;
          if (e) {
            // psi moved to the target centre: psi -= conj(d) (k - 1) phi of the order before
            // (none before the first), 61 bits below 2^ex: |psi'| <= |psi| + |d|_1 k |phi_k|
            const int dx = code % 7 - 3, dy = code / 7 - 3;
            ex = max(S.y, S.z + 32 - __clz(abs(dx) + abs(dy))) + 1;
            const int q_phi = ex - S.x, q_psi = min(ex - S.y, 63);
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              const longlong2 pb = kk + q >= 1 && kk + q < pd ? ms[q - 1] : make_longlong2(0, 0);
              const int dxf = dx * (kk + q), dyf = dy * (kk + q);
              y[q].x = (y[q].x >> q_psi) - small_mul(pb.x, dxf, pb.y, dyf, q_phi);
              y[q].y = (y[q].y >> q_psi) - small_mul(pb.y, dxf, pb.x, -dyf, q_phi);
            }
          }
          long long a[2][2];
          uint32_t mx = 0;
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const Limb yr = limbs(y[q].x), yi = limbs(y[q].y);
            a[0][q] = mul_add_hi(yr, t[q].x, t[q].y, yi, -t[q].z, -t[q].w);
            a[1][q] = mul_add_hi(yr, t[q].z, t[q].w, yi, t[q].x, t[q].y);
            mx = max(mx, max(hi_abs(a[0][q]), hi_abs(a[1][q])));
          }
          // |a| < 2^(64 - clz): brought below 2^53, or halved where it is far below the
          // box's scale (its last bits are those of the product then)
          const int r = max(11 - __clz(__reduce_max_sync(0xffffffffu, mx)), 1);
          // a is this integer times 2^(ex - 59) (the product kept 2^-2 of it), times 2^r
          if (lane == 0) s_exp[e][en] = S.x == FX_BAD ? FX_BAD : ex - 59 + r;
          if (kk < EB_FX_K) {
            const long long bias = (BIAS << r) + (1ll << (r - 1));
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              const int row = 2 * E * en + 2 * e + c;
              store_digits(sA + ((row >> 3) * FX_KCH + (kk >> 3)) * 128 + (row & 7) * 16 + (kk & 7) * 2, a[c][0],
                           a[c][1], r, bias);
            }
          }
        }
        // make the generic-proxy stores visible to the tensor cores' (async) proxy
        asm volatile("fence.proxy.async.shared::cta;");
        team_sync(team);
        if (tid == 0) {
          // the tensor memory (bounded; the other team gives it back after its reads). A team
          // whose products' end stays out keeps it.
          bool mine = false;
          for (long long it = 0; it < (team ? lim1 : lim0) && !mine; ++it) mine = atomicCAS(&s_lock, 0, 1) == 0;
          __threadfence_block();
          if (mine) {
            asm volatile("tcgen05.fence::after_thread_sync;");
            const uint32_t sa = smem_u32(sA), sb = smem_u32(sB);
            for (int d = 0; d < FX_NACC; ++d) {
              uint32_t acc = 0u;
              for (int i = max(0, d - (FX_ND - 1)); i <= min(d, FX_ND - 1); ++i) {
#pragma unroll
                for (int s = 0; s < EB_FX_K / 16; ++s) {
                  fx_mma(taddr + d * EB_FX_K, fx_desc(sa + i * FX_A + s * 256), fx_desc(sb + (d - i) * FX_B + s * 256),
                         acc);
                  acc = 1u;
                }
              }
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                smem_u32(&mbar[team])));
            if (!products_done(phase)) s_fail[team] = 2;
          } else {
            s_fail[team] = 1;
          }
        } else if (warp > 0 && tid - 32 < E * nbx) {
          // the common exponent of a box's entries
          const int e = (tid - 32) / nbx, bx = tid - 32 - e * nbx;
          int m = -(1 << 24);
          for (int j = s_e0[bx]; j < s_e0[bx + 1]; ++j) m = max(m, s_exp[e][j]);
          s_E[e][bx] = m;
        }
        team_sync(team);
        if (s_fail[team]) break;
        phase ^= 1u;
        asm volatile("tcgen05.fence::after_thread_sync;");
        // b_m out of the tensor memory, as integers: a warp reads the 32 rows of its quarter,
        // a part of the orders. The team then gives the tensor memory back.
        constexpr int MH = EB_FX_K / (NW / 4);
        const int row = (warp & 3) * 32 + lane, mlo = (warp >> 2) * MH;
        for (int m0 = mlo; m0 < mlo + MH; m0 += 4) {
          uint32_t v[FX_NACC][4];
#pragma unroll
          for (int d = 0; d < FX_NACC; ++d)
            asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(v[d][0]), "=r"(v[d][1]), "=r"(v[d][2]), "=r"(v[d][3])
                         : "r"(taddr + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(d * EB_FX_K + m0)));
          asm volatile("tcgen05.wait::ld.sync.aligned;");
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            int w[FX_NACC];
#pragma unroll
            for (int d = 0; d < FX_NACC; ++d) w[d] = __float2int_rn(__uint_as_float(v[d][q]));
            // sum of w_d 2^(42 - 9 d), below 2^62 (no row of the matrix sums to 8)
            const long long top = madw(w[0], 1 << 18, madw(w[1], 1 << 9, w[2]));
            const long long low = madw(w[3], 1 << 15, madw(w[4], 64, (w[5] >> 3) + (w[6] >> 12)));
            sC[(m0 + q) * FX_PITCH + row] = shl31(top, 24) + low;
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;");
        team_sync(team);
        if (tid == 0) atomicExch(&s_lock, 0);
        // contributions (-1)^m (2/d)^m b_m of the entries to their boxes, in place: a thread
        // per row and part of the orders reads both parts before either is replaced
        {
          const int en = row / (2 * E), e = E == 2 ? (row >> 1) & 1 : 0;
          const bool im = row & 1, act = en < ne;
          const int4* tb = tabp + (size_t)(act ? s_code[en] : 0) * ldt;
          const int pd = act ? s_pd[en] : -1;
          const int sh = act ? min(s_E[e][s_box[en]] - s_exp[e][en] + 2, 63) : 2;
          const long long half = 1ll << (sh - 1);
#pragma unroll 4
          for (int m = mlo; m < mlo + MH; ++m) {
            const long long own = sC[m * FX_PITCH + row], oth = __shfl_xor_sync(0xffffffffu, own, 1);
            const int4 t = m <= pd ? tb[m] : make_int4(0, 0, 0, 0);
            const long long c = mul_add_hi(limbs(own), t.x, t.y, limbs(oth), im ? t.z : -t.z, im ? t.w : -t.w);
            sC[m * FX_PITCH + row] = (c + half) >> sh;
          }
        }
        team_sync(team);
      }
      // the sums over each box's entries: one thread per part of an order
      for (int o = tid; o < nbx * EB_FX_K * 2 * E; o += FX_TEAM) {
        const int bx = o / (EB_FX_K * 2 * E), rem = o - bx * (EB_FX_K * 2 * E), m = rem / (2 * E), c = rem % (2 * E);
        if (m > p) continue;
        const int e = c >> 1, j0 = s_e0[bx], j1 = s_e0[bx + 1];
        double v = 0.0;
        if (j1 > j0) {
          long long s = 0;
          for (int j = j0; j < j1; ++j) s += sC[m * FX_PITCH + 2 * E * j + c];
          const int ex = s_E[e][bx];
          v = ex >= FX_BAD ? __longlong_as_double(0x7ff8000000000000ll) : scale2((double)s, ex - 2 - rsc[m]);
        }
        const size_t at = (((size_t)(first + b0 + bx) * E + e) * ldl + m) * 2 + (c & 1);
        if (DF) {
          float2* out = reinterpret_cast<float2*>(local) + at;
          if (accumulate) v += (double)out->x + (double)out->y;
          const float h = __double2float_rn(v);
          *out = make_float2(h, __double2float_rn(v - (double)h));
        } else {
          double* out = reinterpret_cast<double*>(local) + at;
          *out = accumulate ? *out + v : v;
        }
      }
      team_sync(team);
      b0 = b1;
    }
    if (s_fail[team]) break;  // (the whole team, or none: last written before the round's team_sync)
  }
  // no tensor memory is given up under products in flight (a second wait, bounded as the first)
  if (tid == 0 && s_fail[team] == 2) products_done(phase);
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (s_fail[0] | s_fail[1]) {
    // a wait ran out: mark this block's expansions non-finite
    for (int g = team * gridDim.x + blockIdx.x; g < nitem; g += step)
      for (int b = item_box(g); b < item_box(g + 1); ++b)
        for (int idx = tid; idx < E * ldl; idx += FX_TEAM) {
          const size_t at = (size_t)(first + b) * E * ldl + idx;
          if (DF) reinterpret_cast<float4*>(local)[at] = make_float4(__int_as_float(0x7fc00000), 0.f, 0.f, 0.f);
          else reinterpret_cast<double2*>(local)[at] = make_double2(__longlong_as_double(0x7ff8000000000000ll), 0.0);
        }
  }
  if (threadIdx.x < 32)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(FX_COLS));
}

template <int E, bool DF>
int fx_launch(eb_ctx* ctx, int first, int ntarget, int nsrc, int ncoarse, const int* vlist, const unsigned char* vcode,
              const int* vcount, EbTables& tb, EbFmmWork& w, const void* mpole, void* local, int accumulate,
              cudaStream_t st) {
  const int p = tb.p;
  EB_TRY(w.mfix.ensure((sizeof(longlong2) * E * (size_t)p + sizeof(int4)) * (size_t)(first + nsrc)));
  longlong2* fx = w.mfix.as<longlong2>();
  int4* fs = reinterpret_cast<int4*>(fx + (size_t)(first + nsrc) * E * p);
  EB_CUDA_TRY(eb_launch_next(k_m2l_fix<E, DF>, dim3((nsrc * 32 + 127) / 128), dim3(128), 0, st, first, nsrc, p, mpole, fx, fs));
  constexpr int sm = FX_ND * (2 * FX_A + FX_B) + 1024;
  EB_CUDA_TRY(cudaFuncSetAttribute(k_m2l_fx<E, DF>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm));
  // Items of about a round's entries: single boxes on the coarse levels (their lists are
  // long, and these items come first), groups on the others.
  const int group = E == 2 ? 5 : FX_GROUP;
  const int nsingle = std::min(ncoarse, ntarget);
  const int nitem = nsingle + (ntarget - nsingle + group - 1) / group;
  const int grid = std::min((nitem + 1) / 2, ctx->nsm);
  EB_CUDA_TRY(eb_launch_next(k_m2l_fx<E, DF>, dim3(grid), dim3(FX_THREADS), sm, st, first, ntarget, vlist, vcode, vcount, p, reinterpret_cast<const uint4*>(tb.fxb),
                                               tb.fxt.as<int4>(), reinterpret_cast<const int*>(tb.fxr), tb.pd.as<int>(), fx, fs, local,
                                               accumulate, nsingle, group, ctx->fx_lock_limit[0], ctx->fx_lock_limit[1]));
  ctx->launches += 2;
  return EB_OK;
}

}  // namespace

// The M2L of boxes [first, first + ntarget) from the multipoles of boxes [first,
// first + nsrc); df: double-float multipoles and locals (float4), else double2. ncoarse: how
// many of the first target boxes lie on levels of few boxes.
int eb_m2l_fx(eb_ctx* ctx, int E, bool df, int first, int ntarget, int nsrc, int ncoarse, const int* vlist,
              const unsigned char* vcode, const int* vcount, EbTables& tb, EbFmmWork& w, const void* mpole,
              void* local, int accumulate, cudaStream_t st) {
  if (ntarget <= 0) return EB_OK;
  auto go = [&](auto f) { return f(ctx, first, ntarget, nsrc, ncoarse, vlist, vcode, vcount, tb, w, mpole, local, accumulate, st); };
  if (E == 2) return df ? go(fx_launch<2, true>) : go(fx_launch<2, false>);
  return df ? go(fx_launch<1, true>) : go(fx_launch<1, false>);
}

// The fixed-point tables of an order p < 48: the digits of the binomial matrix in the tensor
// cores' operand layout, its row scalings and the powers (2/d)^j as 2^62 fractions. Constants
// of the order, formed once per process (0.6 ms).
namespace {
struct FxTables {
  std::vector<unsigned short> dig;
  std::vector<int> rsc;
  std::vector<int4> t;
};

void fx_build(int p, FxTables& T) {
  std::vector<unsigned short>& dig = T.dig;
  std::vector<int>& rsc = T.rsc;
  std::vector<int4>& t = T.t;
  dig.assign((size_t)FX_ND * FX_B / 2, 0);
  rsc.assign(EB_FX_K, 0);
  typedef unsigned __int128 u128;
  for (int m = 0; m <= p; ++m) {
    std::vector<u128> c(p);
    for (int kk = 0; kk < p; ++kk)  // C(m + kk, m), exact
      c[kk] = kk == 0 ? (u128)1 : c[kk - 1] * (u128)(m + kk) / (u128)kk;
    // C 2^-(m + k) 2^r as multiples of 2^-54, r the largest with every entry <= 1/2
    int r = 60;
    for (int kk = 0; kk < p; ++kk) {
      const int s = m + kk + 1;
      while (r > 0 && (s - r >= 1 ? c[kk] > ((u128)1 << (s - r - 1)) : true)) --r;
    }
    rsc[m] = r;
    for (int kk = 0; kk < p; ++kk) {
      const int s = m + kk + 1 - r - 54;  // the entry is c 2^-s units
      long long x;
      if (s > 0) x = (long long)((c[kk] + ((u128)1 << (s - 1))) >> s);
      else x = (long long)(c[kk] << -s);
      for (int i = FX_ND - 1; i >= 0; --i) {
        long long d = i > 0 ? ((x + 256) & 511) - 256 : x;
        x = (x - d) >> 9;
        // FP16 bits of a small integer
        unsigned short h = 0;
        if (d != 0) {
          const unsigned a = (unsigned)(d < 0 ? -d : d);
          int e = 31 - __builtin_clz(a);
          h = (unsigned short)((d < 0 ? 0x8000u : 0u) | ((unsigned)(15 + e) << 10) | ((a << (10 - e)) & 0x3ffu));
        }
        const size_t off = ((size_t)(m >> 3) * FX_KCH + (kk >> 3)) * 128 + (m & 7) * 16 + (kk & 7) * 2;
        dig[((size_t)i * FX_B + off) / 2] = h;
      }
    }
  }
  // the powers, and after them the powers times (-1)^j
  t.assign(2 * (size_t)EB_NCODE * (p + 2), make_int4(0, 0, 0, 0));
  for (int code = 0; code < EB_NCODE; ++code) {
    const int dx = code % 7 - 3, dy = code / 7 - 3;
    if (std::abs(dx) < 2 && std::abs(dy) < 2) continue;
    const long double dn = (long double)(dx * dx + dy * dy);
    const long double zr = 2.0L * dx / dn, zi = -2.0L * dy / dn;
    long double re = 1.0L, im = 0.0L;
    for (int j = 0; j < p + 2; ++j) {
      auto limb = [](long double v, int& h, int& l) {
        long long x = (long long)std::floor(v * (long double)(1ll << 62) + 0.5L);
        if ((unsigned int)x == 0x80000000u) ++x;  // a low limb that can be negated
        h = (int)((x + 0x80000000ll) >> 32);
        l = (int)(unsigned int)(unsigned long long)x;
      };
      int4& o = t[(size_t)code * (p + 2) + j];
      limb(re, o.x, o.y);
      limb(im, o.z, o.w);
      int4& n = t[(size_t)(EB_NCODE + code) * (p + 2) + j];
      limb((j & 1) ? -re : re, n.x, n.y);
      limb((j & 1) ? -im : im, n.z, n.w);
      const long double nr = re * zr - im * zi;
      im = re * zi + im * zr;
      re = nr;
    }
  }
}
}  // namespace

int eb_m2l_fx_tables(EbTables& tb) {
  if (tb.p > EB_FX_MAXP) return EB_OK;
  static std::mutex mu;
  static FxTables cache[EB_FX_MAXP + 1];
  std::lock_guard<std::mutex> lock(mu);
  FxTables& T = cache[tb.p];
  if (T.t.empty()) fx_build(tb.p, T);
  const std::vector<unsigned short>& dig = T.dig;
  const std::vector<int>& rsc = T.rsc;
  const std::vector<int4>& t = T.t;
  // one buffer and one copy: the powers, the digits, the row scalings (16-byte aligned)
  const size_t nt = t.size() * sizeof(int4), nd = dig.size() * 2, nr = rsc.size() * sizeof(int);
  std::vector<char> all(nt + nd + nr);
  memcpy(all.data(), t.data(), nt);
  memcpy(all.data() + nt, dig.data(), nd);
  memcpy(all.data() + nt + nd, rsc.data(), nr);
  EB_TRY(tb.fxt.ensure(all.size()));
  tb.fxb = tb.fxt.as<char>() + nt;
  tb.fxr = tb.fxt.as<char>() + nt + nd;
  EB_CUDA_TRY(cudaMemcpy(tb.fxt.p, all.data(), all.size(), cudaMemcpyHostToDevice));
  return EB_OK;
}

// For tests of the bounded wait: how often a team (0 or 1) of a block asks for the tensor memory
// before it gives up, in the applies from now on (graphs of solves keep theirs).
extern "C" int eb_fx_lock_limit(eb_ctx* ctx, int team, long long n) {
  if (!ctx || team < 0 || team > 1 || n < 0) return EB_ERR_ARG;
  ctx->fx_lock_limit[team] = n;
  return EB_OK;
}
