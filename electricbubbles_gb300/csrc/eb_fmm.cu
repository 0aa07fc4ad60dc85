// Complex-variable FMM for the two layer-potential sums of the hot path.
//
//  Stokes (Sherman-Lauricella), what CADAPDR / CADAPMOD compute (cadapdrop2.f,
//  cadap2.f):   GW(z) = phi(z) + s [ z conj(phi'(z)) + conj(psi(z)) ],  s = -1 / +1,
//      phi(z) = sum qa_j/(z_j - z),   psi(z) = sum qb_j/(z_j - z) + qc_j/(z_j - z)^2,
//      qc_j = -conj(z_j) qa_j   (charges of cadapdrop.f:214-222).
//  Cauchy, what DAPIF2 computes with IFLAG7 = 3 (dapif1.f:552-558):
//      F(z_i) = sum_{j != i} q_j/(z_i - z_j) = -phi(z_i).
//
// Differences from the reference's per-level uniform FMM (CADAPDR, which forms
// multipoles from the sources at every level and has no M2M/L2L):
//  * a sparse quadtree with an upward pass (P2M at leaves, M2M) and a downward pass
//    (M2L over the same interaction lists, L2L, L2P);
//  * expansions are stored scaled by the box side r (M_k / r^k, L_m r^m), so every
//    translation operator depends only on the box offset in box units;
//  * psi is kept relative to the expansion centre c: psi_c = psi + conj(c) phi', so
//    that GW = phi + s[(z - c) conj(phi') + conj(psi_c)] involves no cancellation
//    between terms of size |z|. Moving an expansion from centre c to c' adds
//    conj(c' - c) phi' to psi;
//  * M2L uses the scale / binomial / scale factorisation of SLSHIFT
//    (cadap2.f:1149-1215) with the order truncated per offset to what the offset's
//    separation ratio needs for the requested tolerance.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <functional>
#include <type_traits>
#include <utility>
#include <vector>

#include <cuda_pipeline.h>

#include "eb_df.cuh"
#include "eb_internal.h"
#include "eb_parts.h"
#include "eb_post.cuh"

namespace {

__device__ __forceinline__ unsigned int compact2d(unsigned long long x) {
  x &= 0x5555555555555555ull;
  x = (x | (x >> 1)) & 0x3333333333333333ull;
  x = (x | (x >> 2)) & 0x0F0F0F0F0F0F0F0Full;
  x = (x | (x >> 4)) & 0x00FF00FF00FF00FFull;
  x = (x | (x >> 8)) & 0x0000FFFF0000FFFFull;
  x = (x | (x >> 16)) & 0x00000000FFFFFFFFull;
  return (unsigned int)x;
}

// Morton key of the box (x, y) of a level (the even bits hold x)
__device__ __forceinline__ unsigned long long morton_key(unsigned int x, unsigned int y) {
  unsigned long long r = 0;
  for (int b = 0; b < 32; ++b)
    r |= ((unsigned long long)((x >> b) & 1u) << (2 * b)) | ((unsigned long long)((y >> b) & 1u) << (2 * b + 1));
  return r;
}

__device__ __forceinline__ double2 box_center(unsigned long long key, double x0, double y0,
                                              double r) {
  unsigned int ix = compact2d(key), iy = compact2d(key >> 1);
  return make_double2(x0 + ((double)ix + 0.5) * r, y0 + ((double)iy + 0.5) * r);
}

__device__ __forceinline__ double pow2d(int e) { return __hiloint2double((1023 + e) << 20, 0); }

__device__ __forceinline__ int quadrant(unsigned long long key) {
  return (int)(key & 3ull);  // bit 0: ix & 1, bit 1: iy & 1
}

// ---------------------------------------------------------------------------------
// Charges (sorted order). Stokes: qa, qb of cadapdrop.f:214-222, and the near-field data.
//
// The Stokes pair. With D = z_j - z_t, e = D / |D|^2 = conj(1/D) and the unit number
// f = e / conj(e) = D e, the pair's term qa/D + s (conj(qb/D) - D conj(qa/D^2)) is
//   e [qa conj(f) + s conj(qb) - s conj(qa) f],
// and qa conj(f) -+ its conjugate is twice its real (s = -1) or i times its imaginary
// part (s = +1). With f = 1 - 2 ey (dy - i dx), that is one real factor
//   v = c0 + ey (ax dx + ay dy):   s = -1: c0 = 2 qa.x - qb.x, (ax, ay) = ( 4 qa.y, -4 qa.x)
//                                  s = +1: c0 = 2 qa.y - qb.y, (ax, ay) = (-4 qa.x, -4 qa.y)
// and the term is e (v + i c1) with c1 = qb.y (s = -1) or i e (v + i c1) with
// c1 = -qb.x (s = +1; the sums over the sources are turned by i once, at their end).
// FASMVP's qb is real (conj(dz) u minus its own conjugate, over i), so c1 = 0 for its sign
// s = -1: 14 FP64 instructions a pair where the term as written takes 27. Measured on
// 1,048,576 nodes (110.6 M pairs): the double-float near field 1,425 -> 918 us, the FP32
// one 274 -> 216 us, the FP64 one below; errors against direct sums as before or smaller.
// ---------------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ void near_charge(c_t<T> a, c_t<T> b, T s, T f, c_t<T>& ca, c_t<T>& cc) {
  if (s < (T)0) {
    ca = cmk<T>((T)4 * a.y * f, (T)-4 * a.x * f);
    cc = cmk<T>(((T)2 * a.x - b.x) * f, b.y * f);
  } else {
    ca = cmk<T>((T)-4 * a.x * f, (T)-4 * a.y * f);
    cc = cmk<T>(((T)2 * a.y - b.y) * f, -b.x * f);
  }
}

// Computed in T: the FP32 operator forms its charges in FP32 (GB300's FP64 pipe is ~1/60
// of its FP32 rate). dz = null: the charges of the transposed operator's sum,
// qa = -dens, qb = conj(dens). nc: the near field's (ax, ay), (c0, c1). next: the FP64 near
// field's tile counter, set to zero.
template <typename T>
__global__ void k_charges_stokes(int n, const int* __restrict__ perm,
                                 const double2* __restrict__ dens, const double2* __restrict__ dz,
                                 const double* __restrict__ hpt, double sd,
                                 c_t<T>* __restrict__ qa, c_t<T>* __restrict__ qb,
                                 c_t<T>* __restrict__ nc, int* __restrict__ next) {
  pdl_next();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0 && next) *next = 0;
  if (i >= n) return;
  int o = perm[i];
  const double2 ud = dens[o];
  const c_t<T> u = cmk<T>((T)ud.x, (T)ud.y);
  c_t<T> a, b;
  if (dz) {
    const double2 dd = dz[o];
    const c_t<T> d = cmk<T>((T)dd.x, (T)dd.y);
    const T h = (T)hpt[o] * (T)(1.0 / (2.0 * EB_PI));
    // 1/(2 pi i) = -i/(2 pi)
    c_t<T> w = cmul<T>(u, d);
    a = cmk<T>(w.y * h, -w.x * h);
    c_t<T> v = csub<T>(cmul<T>(u, cconj<T>(d)), cmul<T>(cconj<T>(u), d));
    b = cmk<T>(v.y * h, -v.x * h);
  } else {
    a = cmk<T>(-u.x, -u.y);
    b = cconj<T>(u);
  }
  qa[i] = a;
  qb[i] = b;
  near_charge<T>(a, b, (T)sd, (T)1, nc[2 * i], nc[2 * i + 1]);
}

// The direct sums' charges of FASMVP, one block per drop, with the drop's sums za and pk
// (k_drop_reduce_stokes) from the same reads: for a few hundred nodes the sums' own launch on
// another stream and its two event waits cost as much as the sums. The direct tree's points
// are in node order, and its pairs need nc only. Measured, one drop of 256 nodes: 18.8 -> 15.3 us an apply
template <typename T>
__global__ void __launch_bounds__(256) k_charges_drop(const int* __restrict__ start, const double2* __restrict__ dens,
                                                      const double2* __restrict__ dz, const double* __restrict__ hpt,
                                                      const double2* __restrict__ pkw, double sd,
                                                      c_t<T>* __restrict__ nc, double2* __restrict__ za,
                                                      double* __restrict__ pk) {
  pdl_next();
  __shared__ double red[3][8];
  const int b = blockIdx.x, i0 = start[b], i1 = start[b + 1];
  double v[3] = {0.0, 0.0, 0.0};
  for (int i = i0 + threadIdx.x; i < i1; i += blockDim.x) {
    const double2 ud = dens[i], dd = dz[i], w = pkw[i];
    const c_t<T> u = cmk<T>((T)ud.x, (T)ud.y), d = cmk<T>((T)dd.x, (T)dd.y);
    const T h = (T)hpt[i] * (T)(1.0 / (2.0 * EB_PI));
    const c_t<T> q = cmul<T>(u, d), r = csub<T>(cmul<T>(u, cconj<T>(d)), cmul<T>(cconj<T>(u), d));
    near_charge<T>(cmk<T>(q.y * h, -q.x * h), cmk<T>(r.y * h, -r.x * h), (T)sd, (T)1, nc[2 * i], nc[2 * i + 1]);
    v[0] += ud.x;
    v[1] += ud.y;
    v[2] = fma(ud.x, w.x, fma(-ud.y, w.y, v[2]));
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    v[c] = warp_sum<double>(v[c]);
    if ((threadIdx.x & 31) == 0) red[c][threadIdx.x >> 5] = v[c];
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    const double* q = red[threadIdx.x];
    const double s = ((q[0] + q[1]) + (q[2] + q[3])) + ((q[4] + q[5]) + (q[6] + q[7]));
    const double h = 2.0 * EB_PI / (double)(i1 - i0);
    if (threadIdx.x == 0) za[b].x = h * s;
    else if (threadIdx.x == 1) za[b].y = h * s;
    else pk[b] = s;
  }
}

__device__ __forceinline__ float4 df4(double2 v) {
  float hx = __double2float_rn(v.x), hy = __double2float_rn(v.y);
  return make_float4(hx, __double2float_rn(v.x - (double)hx), hy, __double2float_rn(v.y - (double)hy));
}

// Double-float charges and near-field data, scaled by 1/r_leaf, the side of the point's
// own leaf (the near field works in leaf units): 2^lev / W.
__global__ void k_charges_stokes_df(int n, const int* __restrict__ perm, const double2* __restrict__ dens,
                                    const double2* __restrict__ dz, const double* __restrict__ hpt,
                                    double s, double winv, const unsigned char* __restrict__ plev,
                                    float4* __restrict__ qdf, float4* __restrict__ nc) {
  pdl_next();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int o = perm[i];
  const double rinv = winv * pow2d((int)plev[i]);
  double2 u = dens[o], a, b;
  if (dz) {
    double2 d = dz[o];
    double h = hpt[o] * (1.0 / (2.0 * EB_PI));
    double2 w = cmul<double>(u, d);
    a = make_double2(w.y * h, -w.x * h);
    double2 v = csub<double>(cmul<double>(u, cconj<double>(d)), cmul<double>(cconj<double>(u), d));
    b = make_double2(v.y * h, -v.x * h);
  } else {  // the transposed operator's charges
    a = make_double2(-u.x, -u.y);
    b = cconj<double>(u);
  }
  qdf[2 * i] = df4(make_double2(a.x * rinv, a.y * rinv));
  qdf[2 * i + 1] = df4(make_double2(b.x * rinv, b.y * rinv));
  double2 ca, cc;
  near_charge<double>(a, b, s, rinv, ca, cc);
  nc[2 * i] = df4(ca);
  nc[2 * i + 1] = df4(cc);
}

// Cauchy charge of node o: q[o], or u_o dz_o h_o (FASMVP_LAP, laplace.f:190-200) when
// q is null.
__device__ __forceinline__ double2 cauchy_charge(int o, const double2* q, const double* lu,
                                                 const double2* dz, const double* hpt) {
  if (q) return q[o];
  const double f = lu[o] * hpt[o];
  return make_double2(f * dz[o].x, f * dz[o].y);
}

__global__ void k_charges_cauchy_df(int n, const int* __restrict__ perm, const double2* __restrict__ q,
                                    const double* __restrict__ lu, const double2* __restrict__ dz,
                                    const double* __restrict__ hpt, double winv,
                                    const unsigned char* __restrict__ plev, float4* __restrict__ qdf) {
  pdl_next();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double rinv = winv * pow2d((int)plev[i]);
  double2 v = cauchy_charge(perm[i], q, lu, dz, hpt);
  qdf[i] = df4(make_double2(v.x * rinv, v.y * rinv));
}

template <typename T>
__global__ void k_charges_cauchy(int n, const int* __restrict__ perm,
                                 const double2* __restrict__ q, const double* __restrict__ lu,
                                 const double2* __restrict__ dz, const double* __restrict__ hpt,
                                 c_t<T>* __restrict__ qa, int* __restrict__ next) {
  pdl_next();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0 && next) *next = 0;
  if (i >= n) return;
  const int o = perm[i];
  if (q) {
    qa[i] = cmk<T>((T)q[o].x, (T)q[o].y);
  } else {
    const T f = (T)lu[o] * (T)hpt[o];
    qa[i] = cmk<T>(f * (T)dz[o].x, f * (T)dz[o].y);
  }
}

// ---------------------------------------------------------------------------------
// 1/x in FP64 for the near field: the hardware's reciprocal approximation r (about 20
// bits) and one third-order step r (1 + e + e^2) with e = 1 - x r, which cubes the
// relative error: three FP64 instructions where two Newton steps take four.
// ---------------------------------------------------------------------------------
__device__ __forceinline__ double rcp_nr(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  const double e = fma(-x, r, 1.0);
  return fma(r, fma(e, e, e), r);
}

// What a near-field pair adds (see the charges): NEAR_V the Stokes pair with c1 = 0,
// NEAR_VC with it, NEAR_Q the Cauchy pair q / (z_t - z_j), NEAR_QI only its imaginary
// part (all that FASMVP_LAP's post-processing reads).
enum { NEAR_V = 0, NEAR_VC = 1, NEAR_Q = 2, NEAR_QI = 3 };

// One pair in FP64: ca = (ax, ay), cc = (c0, c1), or ca = q.
template <int K>
__device__ __forceinline__ void near_pair64(double2 zj, double2 ca, double2 cc, double2 zi, double& gx,
                                            double& gy) {
  const double dx = zj.x - zi.x, dy = zj.y - zi.y;
  const double rr = rcp_nr(fma(dx, dx, dy * dy));
  if (K == NEAR_QI) {
    gy = fma(fma(ca.x, dy, -ca.y * dx), rr, gy);
    return;
  }
  const double ex = dx * rr, ey = dy * rr;  // conj(1/D)
  if (K == NEAR_Q) {
    gx = fma(-ca.x, ex, fma(-ca.y, ey, gx));
    gy = fma(ca.x, ey, fma(-ca.y, ex, gy));
  } else {
    const double v = fma(ey, fma(ca.x, dx, ca.y * dy), cc.x);
    gx = fma(ex, v, gx);
    gy = fma(ey, v, gy);
    if (K == NEAR_VC) {
      gx = fma(-ey, cc.y, gx);
      gy = fma(ex, cc.y, gy);
    }
  }
}

// The end of a Stokes near-field sum: s = +1 turns it by i.
template <typename T>
__device__ __forceinline__ c_t<T> near_turn(T gx, T gy, bool plus) {
  return plus ? cmk<T>(-gy, gx) : cmk<T>(gx, gy);
}

template <typename T>
__device__ __forceinline__ c_t<T> cpow_int(c_t<T> u, int n) {
  c_t<T> r = cmk<T>(1, 0), b = u;
  while (n > 0) {
    if (n & 1) r = cmul<T>(r, b);
    b = cmul<T>(b, b);
    n >>= 1;
  }
  return r;
}

// ---------------------------------------------------------------------------------
// P2M at the leaves (SLMKXP, cadap2.f:412-468, with scaled coefficients and psi
// relative to the box centre). One block per leaf (of any level): the leaf's points (32 at a time)
// write their powers w^j to shared memory, then thread j forms the power sums
//   A_j = sum a w^j,  B_j = sum b w^j,  C_j = sum conj(w) a w^j   (a = qa/r, b = qb/r)
// and M_phi[k] = -A_{k-1}, M_psi[k] = -(B_{k-1} + (k-1) C_{k-2}).
//
// FP64-bound: about 15 FP64 instructions per point and order. The powers come by doubling
// (w^j = w^(j-len) w^len, all points and orders of a step at once), and four groups of
// threads take a quarter of the points each, every thread all three sums of its order, so
// that 176 of 192 lanes are busy at p = 44. BREAL: real charges b (FASMVP's own, see the
// charges). Measured alone: 96 -> 72 us at 64 x 512, 2.25 -> 1.50 ms at 1,024 x 1,024.
// ---------------------------------------------------------------------------------
constexpr int P2M_NG = 4;  // groups of points
template <int E, bool BREAL>
__global__ void __launch_bounds__(256) k_p2m64(const int* __restrict__ leaves,
                                               const unsigned long long* __restrict__ bkey,
                                               const unsigned char* __restrict__ blev,
                                               const int* __restrict__ pt0, const int* __restrict__ pt1,
                                               const double2* __restrict__ zs,
                                               const double2* __restrict__ qa,
                                               const double2* __restrict__ qb, double x0, double y0,
                                               double W, double winv, int p, double2* __restrict__ mpole) {
  extern __shared__ double2 sm2d[];
  const int ps = p + 1;  // odd row stride: conflict-free rows
  double2* pw = sm2d;                // [32][p + 1]: w^j per point
  double2* sc = pw + 32 * ps;        // a, b, conj(w) a per point
  const int b = leaves[blockIdx.x];
  const int tid = threadIdx.x, nt = blockDim.x;
  const int lev = blev[b];
  const double rinv = winv * pow2d(lev);
  const int grp = tid / p, k = tid - grp * p;
  double2 A = make_double2(0.0, 0.0), B = A, C = A;
  const int i0 = pt0[b], i1 = pt1[b];
  pdl_wait();  // the charges
  EbParts batches(i1 - i0, (i1 - i0 + 31) / 32);  // of equal size
  while (batches.at < i1 - i0) {
    const int base = i0 + batches.at, cnt = batches.next();
    __syncthreads();
    if (tid < cnt) {
      const int i = base + tid;
      const double2 zi = zs[i];
      const double2 c = box_center(bkey[b], x0, y0, W * pow2d(-lev));
      const double2 w = make_double2((zi.x - c.x) * rinv, (zi.y - c.y) * rinv);
      const double2 ah = cscale<double>(qa[i], rinv);
      sc[tid] = ah;
      if (E == 2) {
        sc[32 + tid] = cscale<double>(qb[i], rinv);
        sc[64 + tid] = cmul<double>(cconj<double>(w), ah);
      }
      pw[tid * ps] = make_double2(1.0, 0.0);
      pw[tid * ps + 1] = w;
    }
    __syncthreads();
    for (int len = 1; len + 1 < p; len <<= 1) {
      const int span = min(len, p - 1 - len);
      for (int pr = tid; pr < cnt * span; pr += nt) {
        const int j = pr / cnt, sp = pr - j * cnt;  // lanes over the points first
        double2* row = pw + sp * ps + len + 1 + j;
        *row = cmul<double>(*(row - len), pw[sp * ps + len]);
      }
      __syncthreads();
    }
    if (grp < P2M_NG) {
      for (int s = grp; s < cnt; s += P2M_NG) {
        const double2 v = pw[s * ps + k];
        cfma<double>(A, sc[s], v);
        if (E == 2) {
          if (BREAL) crfma<double>(B, sc[32 + s].x, v);
          else cfma<double>(B, sc[32 + s], v);
          cfma<double>(C, sc[64 + s], v);
        }
      }
    }
  }
  __syncthreads();
  double2* red = sm2d;  // [E == 2 ? 3 : 1][P2M_NG][p]
  if (grp < P2M_NG) {
    red[grp * p + k] = A;
    if (E == 2) {
      red[(P2M_NG + grp) * p + k] = B;
      red[(2 * P2M_NG + grp) * p + k] = C;
    }
  }
  __syncthreads();
  auto total = [&](int which, int kk) {
    const double2* q = red + which * P2M_NG * p + kk;
    return cadd<double>(cadd<double>(q[0], q[p]), cadd<double>(q[2 * p], q[3 * p]));
  };
  for (int o = tid; o < E * p; o += nt) {
    double2 v;
    if (o < p) {
      v = total(0, o);
    } else {
      const int kk = o - p;
      v = total(1, kk);
      if (kk >= 1) crfma<double>(v, (double)kk, total(2, kk - 1));
    }
    mpole[(size_t)b * E * p + o] = make_double2(-v.x, -v.y);
  }
}

// the sum of the 4 lanes of an output (lanes 4o .. 4o+3) in a fixed order, in every lane
__device__ __forceinline__ double2 quad_sum(double2 v) {
#pragma unroll
  for (int o = 1; o <= 2; o <<= 1) {
    v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
    v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
  }
  return v;
}

// ---------------------------------------------------------------------------------
// M2M into the boxes of one level. With e the child
// centre offset in child units and a_k = e^-k M_k:  M'_n = (e/2)^n sum_{k<=n} C(n-1,k-1) a_k.
// psi is first moved to the parent centre: psi_k += conj(e) (k-1) phi_{k-1}.
//
// The four children's offsets are e_0 = (1 + i)/2 times 1, i, -1, -i (rot), so that with
// b_k = e_0^-k M_k of each child and c_k^r = sum over the children of i^(rot r) b_k,
//   M'_n = (e_0/2)^n sum_k C(n-1,k-1) c_k^((n-k) mod 4):
// one binomial sum for all children, the kernel's bulk, where a sum per child took up to
// four times the FP64 work. Four lanes per output take every 4th term each (one r per lane).
// An SM takes 16 cycles per FP64 warp instruction, so that one parent's outputs alone keep
// it busy for microseconds; on a level of few boxes they are dealt to nsplit blocks (each
// forms c anew).
// Measured (E = 2): 25.2 -> 11.9 us a level of 64 x 512 (beside the near field), 21.6 -> 8.4
// us at 4,096 nodes.
// ---------------------------------------------------------------------------------
__device__ __forceinline__ int quad_rot(int q) { return q == 3 ? 0 : q == 2 ? 1 : q == 0 ? 2 : 3; }

template <int E>
__global__ void k_m2m64(int offp, int nsplit, const unsigned long long* __restrict__ bkey,
                        const int* __restrict__ child0, const int* __restrict__ nchild, int p,
                        const double* __restrict__ binom, int ldb, const double2* __restrict__ epow2,
                        const double2* __restrict__ einv, double2* __restrict__ mpole) {
  extern __shared__ double2 sm2d[];
  double2* cr = sm2d;  // [r][E*p]
  const int P = offp + blockIdx.x / nsplit, sp = blockIdx.x % nsplit;
  const int tid = threadIdx.x, ld = p + 2, nout = E * p;
  const int c0 = child0[P], nc = nchild[P];
  pdl_wait();
  if (nc == 0) return;  // a leaf: its multipole comes from its points
  const double2* e0inv = einv + 3 * ld;
  const double2* e0pow = epow2 + 3 * ld;
  for (int o = tid; o < nout; o += blockDim.x) {
    const int e2 = o / p, kk = o - e2 * p, k = kk + 1;
    double2 c[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) c[r] = make_double2(0.0, 0.0);
    const double2 sc = e0inv[k];
    for (int ci = 0; ci < nc; ++ci) {
      const double2* mc = mpole + (size_t)(c0 + ci) * nout;
      const int q = quadrant(bkey[c0 + ci]), rot = quad_rot(q);
      double2 v = mc[o];
      if (e2 == 1 && k >= 2) {
        const double2 ec = epow2[q * ld + 1];  // e / 2
        cfma<double>(v, cscale<double>(cconj<double>(ec), 2.0 * (k - 1)), mc[kk - 1]);
      }
      const double2 b = cmul<double>(v, sc);
      c[0] = cadd<double>(c[0], b);
      if (rot == 0) {
#pragma unroll
        for (int r = 1; r < 4; ++r) c[r] = cadd<double>(c[r], b);
      } else if (rot == 2) {
        c[1] = csub<double>(c[1], b);
        c[2] = cadd<double>(c[2], b);
        c[3] = csub<double>(c[3], b);
      } else {
        const double2 ib = rot == 1 ? make_double2(-b.y, b.x) : make_double2(b.y, -b.x);
        c[1] = cadd<double>(c[1], ib);
        c[2] = csub<double>(c[2], b);
        c[3] = csub<double>(c[3], ib);
      }
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) cr[r * nout + o] = c[r];
  }
  __syncthreads();
  // a warp's 8 outputs: every nsplit-th group of 8
  const int o = ((tid >> 5) * nsplit + sp) * 8 + ((tid >> 2) & 7), part = tid & 3;
  const bool act = o < nout;
  const int oo = act ? o : 0;
  const int e = oo / p, n = oo - e * p + 1;
  double2 v = make_double2(0.0, 0.0);
  if (act) {
    const double* brow = binom + (size_t)(n - 1) * ldb;
    const double2* src = cr + ((n - 1 - part) & 3) * nout + e * p;
#pragma unroll 4
    for (int k = part; k < n; k += 4) crfma<double>(v, brow[k], src[k]);
  }
  v = quad_sum(v);
  if (act && part == 0) mpole[(size_t)P * nout + o] = cmul<double>(e0pow[n], v);
}

// ---------------------------------------------------------------------------------
// L2L from the boxes of one level to their children. With e the child offset
// in child units and a_m = (e/2)^m L_m:  L'_j += e^-j sum_{m>=j} C(m, j) a_m,
// and psi is moved to the child centre: psi'_j += conj(e) (j+1) phi'_{j+1} (of the shifted
// coefficients; shifting and moving polynomials commute).
//
// For the children e_0 i^rot (see the M2M), with a_m = (e_0/2)^m L_m and
// S_r = sum_{m = j+r mod 4} C(m, j) a_m:  L'_j = e_0^-j sum_r i^(rot r) S_r, so that the
// four lanes of an output form the S_r of all children at once and then one child each.
// On levels of few boxes the orders are dealt to nsplit blocks in ranges of about equal
// work.
// ---------------------------------------------------------------------------------
template <int E>
__global__ void k_l2l64(int offp, int nsplit, const unsigned long long* __restrict__ bkey,
                        const int* __restrict__ child0, const int* __restrict__ nchild, int p,
                        const double* __restrict__ binom, int ldb, const double2* __restrict__ epow2,
                        const double2* __restrict__ einv, double2* __restrict__ local) {
  extern __shared__ double2 sm2d[];
  double2* a = sm2d;                    // [E][p + 1]
  double2* sph = a + E * (p + 1);       // [rot][p + 1]: the children's phi', for psi
  __shared__ int s_child[4];
  const int ldl = p + 1, ld = p + 2, nout = E * ldl, tid = threadIdx.x;
  const int P = offp + blockIdx.x / nsplit, sp = blockIdx.x % nsplit;
  const int c0 = child0[P], nc = nchild[P];
  pdl_wait();
  if (nc == 0) return;
  // orders [ja, jb): the work of order j is p + 1 - j terms
  auto cut = [&](int i) { return i >= nsplit ? ldl : (int)(ldl * (1.f - sqrtf(1.f - (float)i / nsplit))); };
  const int ja = cut(sp), jb = cut(sp + 1), nj = jb - ja;
  if (tid < 4) s_child[tid] = -1;
  __syncthreads();
  if (tid < nc) s_child[quad_rot(quadrant(bkey[c0 + tid]))] = c0 + tid;
  const double2* e0inv = einv + 3 * ld;
  const double2* e0pow = epow2 + 3 * ld;
  const double2* lp = local + (size_t)P * nout;
  for (int idx = tid; idx < nout; idx += blockDim.x) {
    const int m = idx % ldl;
    if (m >= ja) a[idx] = cmul<double>(lp[idx], e0pow[m]);
  }
  __syncthreads();
  // outputs: phi of the orders [ja, min(jb + 1, p + 1)) (psi of the last one needs the next
  // phi), then psi of [ja, jb)
  const int nphi = E == 2 ? min(nj + 1, ldl - ja) : nj;
  const int o = tid >> 2, part = tid & 3;
  const bool psi = o >= nphi, act = o < nphi + (E == 2 ? nj : 0);
  const int j = !act ? p : ja + (psi ? o - nphi : o);
  const double2* ae = a + (psi && act ? ldl : 0);
  double2 s = make_double2(0.0, 0.0);
  if (act) {
#pragma unroll 4
    for (int m = j + part; m <= p; m += 4) crfma<double>(s, binom[(size_t)m * ldb + j], ae[m]);
  }
  // child `part` (rot): sum_r i^(rot r) S_r, S_r in the quad's lane r
  const int q0 = (threadIdx.x & 31) & ~3;
  double2 v = make_double2(0.0, 0.0);
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const double x = __shfl_sync(0xffffffffu, s.x, q0 + r), y = __shfl_sync(0xffffffffu, s.y, q0 + r);
    const int k = (part * r) & 3;  // times i^k
    const double tx = k & 1 ? y : x, ty = k & 1 ? x : y;
    v.x += k == 1 || k == 2 ? -tx : tx;
    v.y += k >= 2 ? -ty : ty;
  }
  v = cmul<double>(e0inv[j], v);
  if (E == 2) {
    if (act && !psi) sph[part * ldl + j] = v;
    __syncthreads();
    if (act && psi && j < p) {
      // conj(e_0 i^rot) (j + 1) phi'
      const double f = 0.5 * (j + 1);
      const double2 ec = make_double2(part == 0 || part == 3 ? f : -f, part <= 1 ? -f : f);
      cfma<double>(v, ec, sph[part * ldl + j + 1]);
    }
  }
  const int c = s_child[part];
  if (act && c >= 0 && (psi || j < jb)) {
    double2* lc = local + (size_t)c * nout + (psi ? ldl : 0) + j;
    *lc = cadd<double>(*lc, v);
  }
}

// FP32 L2L: one block per child box, one thread per output (e, j), psi moved before the
// shift: psi_m += conj(e/2) (m+1) phi_{m+1}.
template <typename T, int E>
__global__ void k_l2l(int offc, const unsigned long long* __restrict__ bkey,
                      const int* __restrict__ parent, int p, const T* __restrict__ binom,
                      int ldb, const c_t<T>* __restrict__ epow2, const c_t<T>* __restrict__ einv,
                      c_t<T>* __restrict__ local) {
  extern __shared__ unsigned char smem_raw[];
  c_t<T>* a = reinterpret_cast<c_t<T>*>(smem_raw);
  const int ldl = p + 1, ld = p + 2, nout = E * ldl, tid = threadIdx.x;
  const int c = offc + blockIdx.x;
  const int P = parent[c];
  const int q = quadrant(bkey[c]);
  c_t<T> eh = epow2[q * ld + 1];
  const c_t<T>* lp = local + (size_t)P * nout;
  pdl_wait();
  for (int idx = tid; idx < nout; idx += blockDim.x) {
    int e2 = idx / ldl, m = idx - e2 * ldl;
    c_t<T> v = lp[idx];
    if (e2 == 1 && m < p) cfma<T>(v, cscale<T>(cconj<T>(eh), (T)(m + 1)), lp[m + 1]);
    a[idx] = cmul<T>(v, epow2[q * ld + m]);
  }
  __syncthreads();
  if (tid < nout) {
    int e = tid / ldl, j = tid - e * ldl;
    const c_t<T>* ae = a + e * ldl;
    c_t<T> s0 = cmk<T>(0, 0), s1 = cmk<T>(0, 0);
    int m = j;
    for (; m + 1 <= p; m += 2) {
      crfma<T>(s0, binom[(size_t)m * ldb + j], ae[m]);
      crfma<T>(s1, binom[(size_t)(m + 1) * ldb + j], ae[m + 1]);
    }
    if (m <= p) crfma<T>(s0, binom[(size_t)m * ldb + j], ae[m]);
    c_t<T>* lc = local + (size_t)c * nout;
    c_t<T> v = lc[tid];
    cfma<T>(v, einv[q * ld + j], cadd<T>(s0, s1));
    lc[tid] = v;
  }
}

// ---------------------------------------------------------------------------------
// M2L over the interaction lists of every box of levels >= 2 (one launch for all
// levels). One block per target box; its 4 warps take every 4th entry of the V list
// and accumulate in shared memory, and the 4 partial expansions are added in a fixed
// order at the end. For offset d = (c_t - c_s)/r and a_k = M_k d^-k,
//   L_m += (-1)^m d^-m sum_{k <= pd} C(m+k-1, m) a_k,   m <= pd(d),
// after moving psi to the target centre: psi_k -= conj(d) (k-1) phi_{k-1}.
// The E (pd+1) outputs of a pair are spread over the lanes, up to 3 per lane.
// ---------------------------------------------------------------------------------
template <typename T, int NS>
__device__ __forceinline__ void m2l_slots(int ob, int lane, int nout, int ldo, int pd, int p,
                                          int ldc, const T* C2, const c_t<T>* a,
                                          const c_t<T>* dv, c_t<T>* acc, int ldl) {
  int o[NS], m[NS], e[NS];
  bool v[NS];
  c_t<T> bsum[NS];
#pragma unroll
  for (int sl = 0; sl < NS; ++sl) {
    o[sl] = ob + lane + 32 * sl;
    v[sl] = o[sl] < nout;
    e[sl] = v[sl] ? o[sl] / ldo : 0;
    m[sl] = v[sl] ? o[sl] - e[sl] * ldo : 0;
    bsum[sl] = cmk<T>(0, 0);
  }
  for (int k = 0; k < pd; ++k) {
#pragma unroll
    for (int sl = 0; sl < NS; ++sl) crfma<T>(bsum[sl], C2[k * ldc + m[sl]], a[e[sl] * p + k]);
  }
#pragma unroll
  for (int sl = 0; sl < NS; ++sl) {
    if (v[sl]) {
      c_t<T> post = dv[m[sl]];
      if (m[sl] & 1) post = cmk<T>(-post.x, -post.y);
      c_t<T>* ap = acc + e[sl] * ldl + m[sl];
      c_t<T> t = *ap;
      cfma<T>(t, post, bsum[sl]);
      *ap = t;
    }
  }
}

template <typename T, int E>
__global__ void __launch_bounds__(128) k_m2l(int first, const int* __restrict__ vlist,
                                             const unsigned char* __restrict__ vcode,
                                             const int* __restrict__ vcount, int p,
                                             const T* __restrict__ binom, int ldb,
                                             const c_t<T>* __restrict__ dinv,
                                             const int* __restrict__ pdv,
                                             const c_t<T>* __restrict__ mpole,
                                             c_t<T>* __restrict__ local, int accumulate) {
  extern __shared__ unsigned char smem_raw[];
  const int ldc = p + 1, ldl = p + 1, ldd = p + 2;
  // C2[(k-1)*(p+1) + m] = C(m+k-1, m), k = 1..p, m = 0..p
  T* C2 = reinterpret_cast<T*>(smem_raw);
  c_t<T>* sa = reinterpret_cast<c_t<T>*>(smem_raw + ((sizeof(T) * (size_t)p * ldc + 15) & ~(size_t)15));
  c_t<T>* sacc = sa + 4 * E * p;
  for (int idx = threadIdx.x; idx < p * ldc; idx += blockDim.x) {
    int k = idx / ldc + 1, m = idx % ldc;
    C2[idx] = binom[(size_t)(m + k - 1) * ldb + m];
  }
  for (int idx = threadIdx.x; idx < 4 * E * ldl; idx += blockDim.x) sacc[idx] = cmk<T>(0, 0);
  __syncthreads();
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gid = first + blockIdx.x;
  c_t<T>* a = sa + w * E * p;
  c_t<T>* acc = sacc + w * E * ldl;
  const int nv = vcount[gid];
  for (int j = w; j < nv; j += 4) {
    int s = vlist[(size_t)gid * EB_VMAX + j];
    int code = vcode[(size_t)gid * EB_VMAX + j];
    int pd = pdv[code];
    const c_t<T>* dv = dinv + (size_t)code * ldd;
    const c_t<T>* ms = mpole + (size_t)s * E * p;
    T dxr = (T)(code % 7 - 3), dyr = (T)(code / 7 - 3);
    for (int kk = lane; kk < pd; kk += 32) {
      int k = kk + 1;
      c_t<T> sc = dv[k];
      a[kk] = cmul<T>(ms[kk], sc);
      if (E == 2) {
        c_t<T> mpsi = ms[p + kk];
        if (k >= 2) cfma<T>(mpsi, cmk<T>(-dxr * (T)(k - 1), dyr * (T)(k - 1)), ms[kk - 1]);
        a[p + kk] = cmul<T>(mpsi, sc);
      }
    }
    __syncwarp();
    const int ldo = pd + 1, nout = E * ldo;
    for (int ob = 0; ob < nout; ob += 96) {
      int rem = nout - ob;
      if (rem > 64) m2l_slots<T, 3>(ob, lane, nout, ldo, pd, p, ldc, C2, a, dv, acc, ldl);
      else if (rem > 32) m2l_slots<T, 2>(ob, lane, nout, ldo, pd, p, ldc, C2, a, dv, acc, ldl);
      else m2l_slots<T, 1>(ob, lane, nout, ldo, pd, p, ldc, C2, a, dv, acc, ldl);
    }
    __syncwarp();
  }
  __syncthreads();
  const int tot = E * ldl;
  for (int idx = threadIdx.x; idx < tot; idx += blockDim.x) {
    c_t<T> v = cadd<T>(cadd<T>(sacc[idx], sacc[tot + idx]), cadd<T>(sacc[2 * tot + idx], sacc[3 * tot + idx]));
    if (accumulate) v = cadd<T>(local[(size_t)gid * tot + idx], v);
    local[(size_t)gid * tot + idx] = v;
  }
}

// Two floats in a register pair: one issue slot for two multiply-adds (the rate of the
// multiply-adds themselves is the same, 64 pairs or 128 lanes a cycle and SM)
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pk2(float x, float y) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float2 upk2(f32x2 a) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// The FP32 M2L for the default order P (20) on few boxes: a block per box, its four warps
// with a quarter of the list each. An entry's multipoles and powers d^-j come by
// asynchronous copies (all in flight at once), a_k takes the multipoles' place with a lane
// per coefficient, and then lane m <= P owns output order m of both expansions: its binomial
// column C(m+k-1, m) stays in registers (as pairs: a complex term is one packed
// multiply-add), two entries at a time, and the loop over k stops at the first multiple of 4
// past their truncation orders pd (a_k = 0 beyond an entry's own).
// The longest list decides: a warp alone issues an instruction every four cycles, and the
// 27 entries of a coarse level's box took one warp 11.5 us. At 64 x 512 (13,290 entries): 10.0 -> 8.9 us.
constexpr int M2L32_CTAS = 5;  // blocks per SM

template <int E, int P>
__global__ void __launch_bounds__(128, M2L32_CTAS) k_m2l_f32w(int first, int nt, const int* __restrict__ vlist,
                                                  const unsigned char* __restrict__ vcode,
                                                  const int* __restrict__ vcount,
                                                  const float* __restrict__ bt,
                                                  const float2* __restrict__ dinv,
                                                  const int* __restrict__ pdv,
                                                  const float2* __restrict__ mpole,
                                                  float2* __restrict__ local, int accumulate) {
  constexpr int ldl = P + 1, ldd = P + 2;
  constexpr int CM = E * P / 2, CD = ldd / 2, CPE = CM + CD;  // 16-byte pieces of an entry
  static_assert(P % 4 == 0 && P <= 31 && EB_VMAX <= 32, "whole chunks, a lane per order and entry");
  constexpr int WPB = 4, NE = (EB_VMAX + WPB - 1) / WPB;
  __shared__ float4 sa[WPB][NE * CPE];  // per entry [e][k] M_k, then a_k; d^-j
  __shared__ float2 sred[WPB][E][ldl];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m = min(lane, P);
  f32x2 c2[P];
#pragma unroll
  for (int k = 0; k < P; ++k) {
    const float c = bt[k * ldl + m];
    c2[k] = pk2(c, c);
  }
  const float sgn = (m & 1) ? -1.f : 1.f;
  float4* buf = sa[w];
  float2* buf2 = reinterpret_cast<float2*>(buf);
  for (int t = blockIdx.x; t < nt; t += gridDim.x) {
    const int gid = first + t;
    const int nv = vcount[gid];
    // this warp's entries
    const int per = (nv + WPB - 1) / WPB, e0 = min(nv, w * per), ne = min(nv, e0 + per) - e0;
    int lsrc = 0, lcode = 0, lpd = 0;
    if (lane < ne) {
      lsrc = vlist[(size_t)gid * EB_VMAX + e0 + lane];
      lcode = vcode[(size_t)gid * EB_VMAX + e0 + lane];
      lpd = pdv[lcode];
    }
    float2 acc[E];
#pragma unroll
    for (int e = 0; e < E; ++e) acc[e] = make_float2(0.f, 0.f);
    pdl_wait();  // the multipoles
    if (ne > 0) {
      for (int c0 = 0; c0 < ne * CPE; c0 += 32) {
        const int c = c0 + lane, j = min(c / CPE, ne - 1), x = c - j * CPE;
        const int src = __shfl_sync(0xffffffffu, lsrc, j), code = __shfl_sync(0xffffffffu, lcode, j);
        const float4* g = x < CM ? reinterpret_cast<const float4*>(mpole) + (size_t)src * CM + x
                                 : reinterpret_cast<const float4*>(dinv) + code * CD + (x - CM);
        if (c < ne * CPE) __pipeline_memcpy_async(buf + c, g, 16);
      }
      __pipeline_commit();
      __pipeline_wait_prior(0);
      __syncwarp();
      // a_k in place, from the last coefficient to the first: psi's shift reads phi_(k-1)
      for (int c0 = (ne * P - 1) & ~31; c0 >= 0; c0 -= 32) {
        const int c = c0 + lane, j = min(c / P, ne - 1), kk = c - j * P;
        const int code = __shfl_sync(0xffffffffu, lcode, j), pd = __shfl_sync(0xffffffffu, lpd, j);
        const bool act = c < ne * P;
        float2* mj = buf2 + j * 2 * CPE + kk;
        float2 v0 = make_float2(0.f, 0.f), v1 = v0;
        if (act && kk < pd) {
          const float2 sc = mj[E * P + 1];
          v0 = cmul<float>(mj[0], sc);
          if (E == 2) {  // psi moved to the target's centre
            float2 ps = mj[P];
            const float f = (float)kk;
            const float dxr = (float)(code % 7 - 3) * f, dyr = (float)(code / 7 - 3) * f;
            if (kk > 0) cfma<float>(ps, make_float2(-dxr, dyr), mj[-1]);
            v1 = cmul<float>(ps, sc);
          }
        }
        __syncwarp();
        if (act) {
          mj[0] = v0;
          if (E == 2) mj[P] = v1;
        }
        __syncwarp();
      }
      for (int j = 0; j < ne; j += 2) {
        const int j1 = min(j + 1, ne - 1);
        const int pd0 = __shfl_sync(0xffffffffu, lpd, j), pd1 = __shfl_sync(0xffffffffu, lpd, j1);
        const int pdm = __reduce_max_sync(0xffffffffu, max(pd0, pd1));  // (in a uniform register)
        const float4 *b0 = buf + j * CPE, *b1 = buf + j1 * CPE;
        const float2 po0 = cscale<float>(reinterpret_cast<const float2*>(b0 + CM)[m], lane <= pd0 ? sgn : 0.f);
        const float2 po1 = cscale<float>(reinterpret_cast<const float2*>(b1 + CM)[m], lane <= pd1 && j1 > j ? sgn : 0.f);
        const ulonglong2 *av = reinterpret_cast<const ulonglong2*>(b0), *bv = reinterpret_cast<const ulonglong2*>(b1);
        f32x2 b[E][2];
#pragma unroll
        for (int e = 0; e < E; ++e) b[e][0] = b[e][1] = 0;
#pragma unroll
        for (int k0 = 0; k0 < P; k0 += 4) {
          if (k0 < pdm) {
#pragma unroll
            for (int k = k0; k < k0 + 4; k += 2) {
#pragma unroll
              for (int e = 0; e < E; ++e) {
                const ulonglong2 a0 = av[(e * P + k) / 2], a1 = bv[(e * P + k) / 2];
                b[e][0] = fma2(c2[k], a0.x, b[e][0]);
                b[e][1] = fma2(c2[k], a1.x, b[e][1]);
                b[e][0] = fma2(c2[k + 1], a0.y, b[e][0]);
                b[e][1] = fma2(c2[k + 1], a1.y, b[e][1]);
              }
            }
          }
        }
#pragma unroll
        for (int e = 0; e < E; ++e) {
          cfma<float>(acc[e], po0, upk2(b[e][0]));
          cfma<float>(acc[e], po1, upk2(b[e][1]));
        }
      }
    }
    if (lane <= P) {
#pragma unroll
      for (int e = 0; e < E; ++e) sred[w][e][lane] = acc[e];
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < E * ldl; idx += 128) {
      const int e = idx / ldl, mm = idx - e * ldl;
      float2 v = sred[0][e][mm];
#pragma unroll
      for (int q = 1; q < WPB; ++q) v = cadd<float>(v, sred[q][e][mm]);
      float2* lc = local + (size_t)gid * E * ldl + idx;
      if (accumulate) v = cadd<float>(*lc, v);
      *lc = v;
    }
    __syncthreads();
  }
}

// The FP32 M2L for the default order P (20) on many boxes: a lane per list entry. A warp takes as many
// whole boxes as have 32 entries between them; the entries' multipoles come through shared
// memory (asynchronous copies, all in flight at once), each lane scales its own to a_k in
// registers and forms its 21 outputs of both expansions with the binomials C(m+k-1, m) as
// immediate operands, and the entries of a box are added through shared memory in their
// order. a_k = 0 beyond the entry's truncation order pd, outputs m > pd are left out.
// With a lane per output order every a_k is a shared-memory broadcast, and a 16-byte one
// costs four cycles of an SM however few addresses there are: two thirds of the lanes busy
// and 68 to 80 of those cycles an entry, where this way an entry takes 98 warp instructions,
// 60 of them multiply-adds. Measured (E = 2): 1,024 x 1,024 (497,412
// entries) 287 -> 113 us.
// Coarse levels' boxes, with up to 27 entries each, go one to a warp, the others nb to a
// warp. From M2L32_WIDE boxes on: an apply of 256 x 512
// (12,000 boxes) takes 125 against 134 us with a block per box, one of 64 x 1,024 (4,500)
// 66.5 against 67.3 us and one of 64 x 512 (2,244) 45.6 against 40.2 us.
constexpr int M2L32_WIDE = 8192;
template <int P>
struct M2lBinom {  // C(m+k, m) for k < P, m <= P: exact in double
  __host__ __device__ static constexpr float at(int k, int m) {
    double c = 1.0;
    for (int i = 1; i <= m; ++i) c = c * (k + i) / i;
    return (float)c;
  }
};
template <typename F, int... I>
__device__ __forceinline__ void static_for_impl(F&& f, std::integer_sequence<int, I...>) {
  (f(std::integral_constant<int, I>()), ...);
}
template <int N, typename F>
__device__ __forceinline__ void static_for(F&& f) {
  static_for_impl(f, std::make_integer_sequence<int, N>());
}

constexpr int M2L32_WARPS = 4;
template <int E, int P>
struct M2l32Smem {
  static constexpr int CM = E * P / 2;       // 16-byte pieces of a box's multipoles
  static constexpr int PITCH = CM | 1;       // rows of an odd number of pieces: no bank conflicts
  static constexpr int NOUT = E * (P + 1), CP = 33;
  static constexpr int WARP = PITCH * 32 * 2 > NOUT * CP ? PITCH * 32 * 2 : (NOUT * CP + 1) & ~1;  // float2
  float2 buf[M2L32_WARPS][WARP];             // the multipoles, then the outputs [NOUT][CP]
  float2 d[(P + 2) * EB_NCODE];              // d^-j at [j][code]
};

template <int E, int P>
__global__ void __launch_bounds__(32 * M2L32_WARPS, 4)
    k_m2l_f32p(int first, int nt, int ncoarse, int nb, const int* __restrict__ vlist,
               const unsigned char* __restrict__ vcode, const int* __restrict__ vcount,
               const float2* __restrict__ dinv, const int* __restrict__ pdv, const float2* __restrict__ mpole,
               float2* __restrict__ local, int accumulate) {
  typedef M2l32Smem<E, P> Smem;
  constexpr int ldd = P + 2, CM = Smem::CM, PITCH = Smem::PITCH, NOUT = Smem::NOUT, CP = Smem::CP;
  static_assert(EB_VMAX <= 32 && (E * P) % 2 == 0, "a box's entries fit a warp");
  extern __shared__ float4 sm4[];
  Smem& S = *reinterpret_cast<Smem*>(sm4);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = threadIdx.x; i < EB_NCODE * ldd; i += 32 * M2L32_WARPS)
    S.d[(i % ldd) * EB_NCODE + i / ldd] = dinv[i];
  __syncthreads();
  float2* buf = S.buf[w];
  const int wid = blockIdx.x * M2L32_WARPS + w;
  const int t0 = wid < ncoarse ? wid : ncoarse + (wid - ncoarse) * nb;
  const int n = wid < ncoarse ? 1 : min(nb, nt - t0);  // this warp's boxes, at most 32
  if (n <= 0) return;
  const int cnt = lane < n ? vcount[first + t0 + lane] : 0;
  int end = cnt;  // of the lane's box in the warp's entries
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, end, o);
    if (lane >= o) end += y;
  }
  for (int s = 0; s < n;) {
    const int base = __shfl_sync(0xffffffffu, end - cnt, s);
    const int e = s + __popc(__ballot_sync(0xffffffffu, lane >= s && lane < n && end - base <= 32));
    const int ne = __shfl_sync(0xffffffffu, end, e - 1) - base;
    // the lane's entry
    int bx = s, o0 = 0;
    for (int b = s; b < e; ++b) {
      const int o = __shfl_sync(0xffffffffu, end - cnt, b) - base;
      if (lane >= o) {
        bx = b;
        o0 = o;
      }
    }
    int src = 0, code = 0, pd = -1;
    if (lane < ne) {
      const size_t x = (size_t)(first + t0 + bx) * EB_VMAX + (lane - o0);
      src = vlist[x];
      code = vcode[x];
      pd = pdv[code];
    }
    pdl_wait();  // the multipoles
    for (int c0 = 0; c0 < ne * CM; c0 += 32) {
      const int c = c0 + lane, j = min(c / CM, ne - 1), x = c - j * CM;
      const int sj = __shfl_sync(0xffffffffu, src, j);
      if (c < ne * CM)
        __pipeline_memcpy_async(reinterpret_cast<float4*>(buf) + j * PITCH + x,
                                reinterpret_cast<const float4*>(mpole) + (size_t)sj * CM + x, 16);
    }
    __pipeline_commit();
    __pipeline_wait_prior(0);
    __syncwarp();
    float2 a[E][P];
    {
      const float4* row = reinterpret_cast<const float4*>(buf) + (lane < ne ? lane : 0) * PITCH;
#pragma unroll
      for (int x = 0; x < CM; ++x) {
        const float4 v = row[x];
        const int q = 2 * x;
        a[q / P][q % P] = make_float2(v.x, v.y);
        a[(q + 1) / P][(q + 1) % P] = make_float2(v.z, v.w);
      }
    }
    const float dx = (float)(code % 7 - 3), dy = (float)(code / 7 - 3);
    float2 below = make_float2(0.f, 0.f);  // phi's coefficient k - 1
#pragma unroll
    for (int k = 0; k < P; ++k) {
      float2 sc = S.d[(k + 1) * EB_NCODE + code];
      if (k >= pd) sc = make_float2(0.f, 0.f);
      const float2 ph = a[0][k];
      a[0][k] = cmul<float>(ph, sc);
      if (E == 2) {  // psi moved to the target's centre
        float2 ps = a[E - 1][k];
        if (k > 0) cfma<float>(ps, make_float2(-dx * (float)k, dy * (float)k), below);
        a[E - 1][k] = cmul<float>(ps, sc);
        below = ph;
      }
    }
    __syncwarp();  // the multipoles are consumed
    static_for<P + 1>([&](auto mc) {
      constexpr int m = decltype(mc)::value;
      float2 b[E];
#pragma unroll
      for (int x = 0; x < E; ++x) b[x] = make_float2(0.f, 0.f);
      static_for<P>([&](auto kc) {
        constexpr int k = decltype(kc)::value;
        constexpr float c = M2lBinom<P>::at(k, m);
#pragma unroll
        for (int x = 0; x < E; ++x) crfma<float>(b[x], c, a[x][k]);
      });
      float2 po = S.d[m * EB_NCODE + code];
      if (m > pd) po = make_float2(0.f, 0.f);
      if (m & 1) po = make_float2(-po.x, -po.y);
#pragma unroll
      for (int x = 0; x < E; ++x) buf[(x * (P + 1) + m) * CP + lane] = cmul<float>(po, b[x]);
    });
    __syncwarp();
    for (int i0 = 0; i0 < (e - s) * NOUT; i0 += 32) {
      const int i = i0 + lane, bi = min(i / NOUT, e - s - 1), o = i - bi * NOUT;
      const int j1 = __shfl_sync(0xffffffffu, end, s + bi) - base, j0 = j1 - __shfl_sync(0xffffffffu, cnt, s + bi);
      if (i < (e - s) * NOUT) {
        float2 v = make_float2(0.f, 0.f);
        for (int j = j0; j < j1; ++j) v = cadd<float>(v, buf[o * CP + j]);
        float2* lc = local + (size_t)(first + t0 + s + bi) * NOUT + o;
        if (accumulate) v = cadd<float>(*lc, v);
        *lc = v;
      }
    }
    __syncwarp();
    s = e;
  }
}

// ---------------------------------------------------------------------------------
// The same M2L in double-float arithmetic (FP64-class accuracy on the FP32 pipes): the
// multipoles, d^-j and binomial tables are double-float; each output's binomial sum is
// accumulated with compensation; the four warps' partial expansions are added in a
// fixed order and written as FP64.
// ---------------------------------------------------------------------------------
__device__ __forceinline__ cdf cdf_ld(const float4* p) { return cdf_from_float4(*p); }
__device__ __forceinline__ float4 cdf_f4(cdf v) { return make_float4(v.x.hi, v.x.lo, v.y.hi, v.y.lo); }

template <int NS>
__device__ __forceinline__ void m2l_slots_df(int ob, int lane, int nout, int ldo, int pd, int p, int ldc,
                                             const float2* C2, const float4* a, const float4* dv,
                                             float4* acc, int ldl) {
  int o[NS], m[NS], e[NS];
  bool v[NS];
  dfacc bx[NS], by[NS];
#pragma unroll
  for (int sl = 0; sl < NS; ++sl) {
    o[sl] = ob + lane + 32 * sl;
    v[sl] = o[sl] < nout;
    e[sl] = v[sl] ? o[sl] / ldo : 0;
    m[sl] = v[sl] ? o[sl] - e[sl] * ldo : 0;
    bx[sl] = dfacc{0.f, 0.f};
    by[sl] = dfacc{0.f, 0.f};
  }
  for (int k = 0; k < pd; ++k) {
#pragma unroll
    for (int sl = 0; sl < NS; ++sl) {
      const float2 c = C2[k * ldc + m[sl]];
      const float4 av = a[e[sl] * p + k];
      acc_prod(bx[sl], dfl{c.x, c.y}, dfl{av.x, av.y});
      acc_prod(by[sl], dfl{c.x, c.y}, dfl{av.z, av.w});
    }
  }
#pragma unroll
  for (int sl = 0; sl < NS; ++sl) {
    if (v[sl]) {
      cdf post = cdf_ld(dv + m[sl]);
      if (m[sl] & 1) post = cdf{dfl_neg(post.x), dfl_neg(post.y)};
      float4* ap = acc + e[sl] * ldl + m[sl];
      *ap = cdf_f4(cdf_add(cdf_from_float4(*ap), cdf_mul(post, cdf{acc_value(bx[sl]), acc_value(by[sl])})));
    }
  }
}

template <int E>
__global__ void __launch_bounds__(128) k_m2l_df(int first, const int* __restrict__ vlist,
                                                const unsigned char* __restrict__ vcode,
                                                const int* __restrict__ vcount, int p,
                                                const float2* __restrict__ binom, int ldb,
                                                const float4* __restrict__ dinv,
                                                const int* __restrict__ pdv,
                                                const float4* __restrict__ mpole,
                                                float4* __restrict__ local, int accumulate) {
  extern __shared__ float4 smem_f4[];
  const int ldc = p + 1, ldl = p + 1, ldd = p + 2;
  float2* C2 = reinterpret_cast<float2*>(smem_f4);
  float4* sa = smem_f4 + (p * ldc + 1) / 2;
  float4* sacc = sa + 4 * E * p;
  for (int idx = threadIdx.x; idx < p * ldc; idx += blockDim.x) {
    int k = idx / ldc + 1, m = idx % ldc;
    C2[idx] = binom[(size_t)(m + k - 1) * ldb + m];
  }
  for (int idx = threadIdx.x; idx < 4 * E * ldl; idx += blockDim.x) sacc[idx] = make_float4(0.f, 0.f, 0.f, 0.f);
  __syncthreads();
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gid = first + blockIdx.x;
  float4* a = sa + w * E * p;
  float4* acc = sacc + w * E * ldl;
  const int nv = vcount[gid];
  for (int j = w; j < nv; j += 4) {
    const int s = vlist[(size_t)gid * EB_VMAX + j];
    const int code = vcode[(size_t)gid * EB_VMAX + j];
    const int pd = pdv[code];
    const float4* dv = dinv + (size_t)code * ldd;
    const float4* ms = mpole + (size_t)s * E * p;
    const float dxr = (float)(code % 7 - 3), dyr = (float)(code / 7 - 3);
    for (int kk = lane; kk < pd; kk += 32) {
      const int k = kk + 1;
      const cdf sc = cdf_ld(dv + k);
      a[kk] = cdf_f4(cdf_mul(cdf_ld(ms + kk), sc));
      if (E == 2) {
        cdf mpsi = cdf_ld(ms + p + kk);
        if (k >= 2) {
          const cdf f = cdf{{-dxr * (float)(k - 1), 0.f}, {dyr * (float)(k - 1), 0.f}};
          mpsi = cdf_add(mpsi, cdf_mul(f, cdf_ld(ms + kk - 1)));
        }
        a[p + kk] = cdf_f4(cdf_mul(mpsi, sc));
      }
    }
    __syncwarp();
    const int ldo = pd + 1, nout = E * ldo;
    for (int ob = 0; ob < nout; ob += 96) {
      int rem = nout - ob;
      if (rem > 64) m2l_slots_df<3>(ob, lane, nout, ldo, pd, p, ldc, C2, a, dv, acc, ldl);
      else if (rem > 32) m2l_slots_df<2>(ob, lane, nout, ldo, pd, p, ldc, C2, a, dv, acc, ldl);
      else m2l_slots_df<1>(ob, lane, nout, ldo, pd, p, ldc, C2, a, dv, acc, ldl);
    }
    __syncwarp();
  }
  __syncthreads();
  const int tot = E * ldl;
  for (int idx = threadIdx.x; idx < tot; idx += blockDim.x) {
    cdf v01 = cdf_add(cdf_from_float4(sacc[idx]), cdf_from_float4(sacc[tot + idx]));
    cdf v23 = cdf_add(cdf_from_float4(sacc[2 * tot + idx]), cdf_from_float4(sacc[3 * tot + idx]));
    cdf v = cdf_add(v01, v23);
    if (accumulate) v = cdf_add(cdf_from_float4(local[(size_t)gid * tot + idx]), v);
    local[(size_t)gid * tot + idx] = cdf_f4(v);
  }
}

// ---------------------------------------------------------------------------------
// The P2M, M2M and L2L of the double-float pipeline.
// ---------------------------------------------------------------------------------
__device__ __forceinline__ cdf cdf_conj(cdf a) { return cdf{a.x, dfl_neg(a.y)}; }
__device__ __forceinline__ cdf cdf_scale(cdf a, float f) { return cdf{dfl_mul_f(a.x, f), dfl_mul_f(a.y, f)}; }

// acc += a * b (complex) with compensated real and imaginary sums
__device__ __forceinline__ void cacc_mul(dfacc& rx, dfacc& ry, cdf a, cdf b) {
  acc_prod(rx, a.x, b.x);
  acc_prod(rx, dfl_neg(a.y), b.y);
  acc_prod(ry, a.x, b.y);
  acc_prod(ry, a.y, b.x);
}

// acc += c * a (c real)
__device__ __forceinline__ void cacc_rmul(dfacc& rx, dfacc& ry, dfl c, cdf a) {
  acc_prod(rx, c, a.x);
  acc_prod(ry, c, a.y);
}

__device__ __forceinline__ cdf cacc_value(const dfacc& rx, const dfacc& ry) {
  return cdf{acc_value(rx), acc_value(ry)};
}

// P2M at the leaves from the leaf-relative offsets w (units of the leaf side) and the
// charges qa/r, qb/r: M_phi[k] = -A_{k-1}, M_psi[k] = -(B_{k-1} + (k-1) C_{k-2}).
template <int E>
__global__ void k_p2m_df(const int* __restrict__ leaves, const int* __restrict__ pt0, const int* __restrict__ pt1,
                         const float4* __restrict__ wa, const float4* __restrict__ q, int p,
                         float4* __restrict__ mpole) {
  // thread (which, k) < NA p sums one of A_k, B_k, C_k over the leaf's points
  constexpr int NA = E == 2 ? 3 : 1;
  extern __shared__ float4 sm4[];
  const int ps = p + 1;
  float4* pw = sm4;
  float4* sc = pw + 32 * ps;
  const int b = leaves[blockIdx.x], tid = threadIdx.x;
  const int which = tid / p, kq = tid - which * p;
  const bool acc_thread = which < NA;
  dfacc Rx{0.f, 0.f}, Ry{0.f, 0.f};
  const int i0 = pt0[b], i1 = pt1[b];
  pdl_wait();  // the charges
  for (int base = i0; base < i1; base += 32) {
    const int cnt = min(32, i1 - base);
    __syncthreads();
    if (tid < cnt) {
      const int i = base + tid;
      const float4 wv = wa[i];
      const cdf w = cdf{{wv.x, wv.z}, {wv.y, wv.w}};
      const cdf ah = cdf_from_float4(q[(size_t)E * i]);
      sc[tid] = cdf_f4(ah);
      if (E == 2) {
        sc[32 + tid] = q[2 * (size_t)i + 1];
        sc[64 + tid] = cdf_f4(cdf_mul(cdf_conj(w), ah));
      }
      float4* row = pw + tid * ps;
      row[0] = make_float4(1.f, 0.f, 0.f, 0.f);
      row[1] = cdf_f4(w);
    }
    __syncthreads();
    // powers w^j, j < p, by doubling: w^j = w^(j-len) w^len for len < j <= 2 len, all
    // (point, j) pairs of a step in parallel
    for (int len = 1; len + 1 < p; len <<= 1) {
      const int span = min(len, p - 1 - len);
      for (int pr = tid; pr < cnt * span; pr += blockDim.x) {
        const int sp = pr / span, jj = len + 1 + (pr - sp * span);
        float4* row = pw + sp * ps;
        row[jj] = cdf_f4(cdf_mul(cdf_from_float4(row[jj - len]), cdf_from_float4(row[len])));
      }
      __syncthreads();
    }
    if (acc_thread) {
      const float4* scw = sc + 32 * which;
      for (int s2 = 0; s2 < cnt; ++s2) cacc_mul(Rx, Ry, cdf_from_float4(scw[s2]), cdf_from_float4(pw[s2 * ps + kq]));
    }
  }
  __syncthreads();
  float4* red = pw;  // [NA][p]
  if (acc_thread) red[which * p + kq] = cdf_f4(cacc_value(Rx, Ry));
  __syncthreads();
  if (tid < p) {
    float4* mp = mpole + (size_t)b * E * p;
    const cdf A = cdf_from_float4(red[tid]);
    mp[tid] = cdf_f4(cdf{dfl_neg(A.x), dfl_neg(A.y)});
    if (E == 2) {
      cdf v = cdf_from_float4(red[p + tid]);
      if (tid >= 1) v = cdf_add(v, cdf_scale(cdf_from_float4(red[2 * p + tid - 1]), (float)tid));
      mp[p + tid] = cdf_f4(cdf{dfl_neg(v.x), dfl_neg(v.y)});
    }
  }
}

// merge the compensated complex sums of the 4 lanes of an output (lanes 4o .. 4o+3),
// in a fixed order; every lane ends with the total
__device__ __forceinline__ cdf quad_merge(dfacc rx, dfacc ry) {
  cdf v = cacc_value(rx, ry);
#pragma unroll
  for (int o = 1; o <= 2; o <<= 1) {
    cdf u{{__shfl_xor_sync(0xffffffffu, v.x.hi, o), __shfl_xor_sync(0xffffffffu, v.x.lo, o)},
          {__shfl_xor_sync(0xffffffffu, v.y.hi, o), __shfl_xor_sync(0xffffffffu, v.y.lo, o)}};
    v = (threadIdx.x & o) ? cdf_add(u, v) : cdf_add(v, u);
  }
  return v;
}

// M2M: k_m2m64's scheme (one binomial sum for all children's rotations) in double-float: 4
// lanes per output coefficient, each summing every 4th term, so that the dependent chain of
// compensated products is a sixteenth of a sum per child's. Measured (E = 2): 14.9 -> 9.4 us a level
// of 64 x 512, 79 -> 56 us at 1,024 x 1,024 (its far field beside it, with the Horner steps
// below: 22.6 -> 19.2 and 569 -> 482 us)
template <int E>
__global__ void k_m2m_df(int offp, const unsigned long long* __restrict__ bkey,
                         const int* __restrict__ child0, const int* __restrict__ nchild, int p,
                         const float2* __restrict__ binom, int ldb, const float4* __restrict__ epow2,
                         const float4* __restrict__ einv, float4* __restrict__ mpole) {
  extern __shared__ float4 sm4[];
  float4* cr = sm4;  // [r][E*p]
  const int P = offp + blockIdx.x, tid = threadIdx.x, ld = p + 2, nout = E * p;
  const int c0 = child0[P], nc = nchild[P];
  pdl_wait();
  if (nc == 0) return;  // a leaf: its multipole comes from its points
  // four lanes per coefficient: lane r forms c^r from the children's b (lane ci forms child ci's)
  const int o = tid >> 2, part = tid & 3;
  const bool act = o < nout;
  const int oo = act ? o : 0;
  const int e = oo / p, n = oo - e * p + 1;
  {
    const int q = part < nc ? quadrant(bkey[c0 + part]) : 0;
    cdf b{{0.f, 0.f}, {0.f, 0.f}};
    if (part < nc) {
      const float4* mc = mpole + (size_t)(c0 + part) * nout;
      cdf v = cdf_from_float4(mc[oo]);
      if (e == 1 && n >= 2) {
        const cdf ec = cdf_scale(cdf_from_float4(epow2[q * ld + 1]), 2.f);
        v = cdf_add(v, cdf_mul(cdf_scale(cdf_conj(ec), (float)(n - 1)), cdf_from_float4(mc[n - 2])));
      }
      b = cdf_mul(v, cdf_from_float4(einv[3 * ld + n]));
    }
    const int rot = quad_rot(q), q0 = (tid & 31) & ~3;
    cdf c{{0.f, 0.f}, {0.f, 0.f}};
#pragma unroll
    for (int ci = 0; ci < 4; ++ci) {
      const float4 f = make_float4(__shfl_sync(0xffffffffu, b.x.hi, q0 + ci), __shfl_sync(0xffffffffu, b.x.lo, q0 + ci),
                                   __shfl_sync(0xffffffffu, b.y.hi, q0 + ci), __shfl_sync(0xffffffffu, b.y.lo, q0 + ci));
      const int k = (part * __shfl_sync(0xffffffffu, rot, q0 + ci)) & 3;  // times i^k
      const cdf v = cdf_from_float4(f);
      const dfl tx = k & 1 ? v.y : v.x, ty = k & 1 ? v.x : v.y;
      c.x = dfl_add(c.x, k == 1 || k == 2 ? dfl_neg(tx) : tx);
      c.y = dfl_add(c.y, k >= 2 ? dfl_neg(ty) : ty);
    }
    if (act) cr[part * nout + o] = cdf_f4(c);
  }
  __syncthreads();
  dfacc rx{0.f, 0.f}, ry{0.f, 0.f};
  if (act) {
    const float2* brow = binom + (size_t)(n - 1) * ldb;
    const float4* src = cr + ((n - 1 - part) & 3) * nout + e * p;
#pragma unroll 4
    for (int k = part; k < n; k += 4) cacc_rmul(rx, ry, dfl{brow[k].x, brow[k].y}, cdf_from_float4(src[k]));
  }
  const cdf v = quad_merge(rx, ry);
  if (act && part == 0) mpole[(size_t)P * nout + o] = cdf_f4(cdf_mul(cdf_from_float4(epow2[3 * ld + n]), v));
}

// L2L of a level's boxes into all their children at once (see k_l2l64): the four lanes of an
// output form the sums S_r of all children, then one child each. Measured (E = 2): a level of
// 64 x 512 nodes 8.0 -> 5.8 us on average, of 1,024 x 1,024 100 -> 49 us.
template <int E>
__global__ void k_l2l_df(int offp, const unsigned long long* __restrict__ bkey,
                         const int* __restrict__ child0, const int* __restrict__ nchild, int p,
                         const float2* __restrict__ binom, int ldb, const float4* __restrict__ epow2,
                         const float4* __restrict__ einv, float4* __restrict__ local) {
  extern __shared__ float4 sm4[];
  float4* a = sm4;                  // [E][p + 1]
  float4* sph = a + E * (p + 1);    // [rot][p + 1]: the children's phi', for psi
  __shared__ int s_child[4];
  const int ldl = p + 1, ld = p + 2, nout = E * ldl, tid = threadIdx.x;
  const int P = offp + blockIdx.x;
  const int c0 = child0[P], nc = nchild[P];
  pdl_wait();
  if (nc == 0) return;
  if (tid < 4) s_child[tid] = -1;
  __syncthreads();
  if (tid < nc) s_child[quad_rot(quadrant(bkey[c0 + tid]))] = c0 + tid;
  const float4* e0pow = epow2 + 3 * ld;
  const float4* lp = local + (size_t)P * nout;
  for (int idx = tid; idx < nout; idx += blockDim.x)
    a[idx] = cdf_f4(cdf_mul(cdf_from_float4(lp[idx]), cdf_from_float4(e0pow[idx % ldl])));
  __syncthreads();
  const int o = tid >> 2, part = tid & 3;
  const bool act = o < nout, psi = act && o >= ldl;
  const int j = !act ? p : psi ? o - ldl : o;
  const float4* ae = a + (psi ? ldl : 0);
  dfacc sx{0.f, 0.f}, sy{0.f, 0.f};
  if (act) {
#pragma unroll 4
    for (int m = j + part; m <= p; m += 4) {
      const float2 bm = binom[(size_t)m * ldb + j];
      cacc_rmul(sx, sy, dfl{bm.x, bm.y}, cdf_from_float4(ae[m]));
    }
  }
  // child `part` (rot): sum_r i^(rot r) S_r, S_r in the quad's lane r
  const cdf s = cacc_value(sx, sy);
  const int q0 = (tid & 31) & ~3;
  cdf v{{0.f, 0.f}, {0.f, 0.f}};
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const cdf t{{__shfl_sync(0xffffffffu, s.x.hi, q0 + r), __shfl_sync(0xffffffffu, s.x.lo, q0 + r)},
                {__shfl_sync(0xffffffffu, s.y.hi, q0 + r), __shfl_sync(0xffffffffu, s.y.lo, q0 + r)}};
    const int k = (part * r) & 3;  // times i^k
    const dfl tx = k & 1 ? t.y : t.x, ty = k & 1 ? t.x : t.y;
    v.x = dfl_add(v.x, k == 1 || k == 2 ? dfl_neg(tx) : tx);
    v.y = dfl_add(v.y, k >= 2 ? dfl_neg(ty) : ty);
  }
  v = cdf_mul(cdf_from_float4(einv[3 * ld + j]), v);
  if (E == 2) {
    if (act && !psi) sph[part * ldl + j] = cdf_f4(v);
    __syncthreads();
    if (psi && j < p) {
      // conj(e_0 i^rot) (j + 1) phi': both parts of the conjugate are +- 1/2
      const cdf ph = cdf_from_float4(sph[part * ldl + j + 1]);
      const bool nx = part == 1 || part == 2, ny = part <= 1;  // its signs
      const dfl xx = nx ? dfl_neg(ph.x) : ph.x, xy = nx ? dfl_neg(ph.y) : ph.y;
      const dfl yx = ny ? dfl_neg(ph.x) : ph.x, yy = ny ? dfl_neg(ph.y) : ph.y;
      v = cdf_add(v, cdf_scale(cdf{dfl_sub(xx, yy), dfl_add(xy, yx)}, 0.5f * (float)(j + 1)));
    }
  }
  const int c = s_child[part];
  if (act && c >= 0) {
    float4* lc = local + (size_t)c * nout + o;
    *lc = cdf_f4(cdf_add(cdf_from_float4(*lc), v));
  }
}

// ---------------------------------------------------------------------------------
// FP32 multipoles of every box of the finest levels directly from its points, in
// parallel over those levels (no dependent M2M chain): one warp per chunk of at most
// EB_CHUNK points forms that chunk's contribution (the P2M sums of SLMKXP,
// cadap2.f:412-468, scaled by the box side and relative to the box centre), and the
// last chunk of a box to finish adds the chunks of the box in order. The offset of a point from an ancestor's centre in the
// ancestor's units is u 2^-sh + (i + 1/2) 2^-sh - (i >> sh) - 1/2 from its leaf offset
// u and leaf grid index i (sh levels between the point's leaf and the box), exact apart
// from the rounding of u.
// ---------------------------------------------------------------------------------
struct LevOff {
  int v[EB_KEY_LEVELS + 2];
  float rinv[EB_KEY_LEVELS + 2];  // 1 / (box side) per level, rounded to float on the host
};

//
// One warp per chunk, four to a block and without block-wide waits: a lane per point forms
// the powers w^k of 32 points in shared memory (rows of an odd pitch: no bank conflicts),
// then a lane per order sums the points, all three sums A, B, C from one read of a power.
// With a block per chunk, a thread per sum and order, and half of the points each, a point
// took 13 warp instructions and level, most of them addressing (E = 2, p = 20: 98 -> 72 us
// for 524,288 nodes).
constexpr int P2M_CW = 4;  // chunks of a block
__host__ __device__ constexpr int p2m_pitch(int p) { return (p < 32 ? p : 32) | 1; }
inline size_t p2m_smem(int p) { return P2M_CW * 32 * (sizeof(float2) * (p2m_pitch(p) + 1) + sizeof(float4)); }

// A part of a box's sum is written: the warp that counts the last of nc adds them in order.
__device__ __forceinline__ void p2m_finish(int lane, int nc, int nout, const float2* part, int* cdone, float2* mpole) {
  __threadfence();
  __syncwarp();
  int done = 0;
  if (lane == 0) done = atomicAdd(cdone, 1) == nc - 1;
  if (!__shfl_sync(0xffffffffu, done, 0)) return;
  __threadfence();
  for (int o = lane; o < nout; o += 32) {
    float2 acc = __ldcg(part + o);
#pragma unroll 8
    for (int q = 1; q < nc; ++q) acc = cadd<float>(acc, __ldcg(part + (size_t)q * nout + o));
    mpole[o] = acc;
  }
  if (lane == 0) *cdone = 0;
}

template <int E>
__global__ void __launch_bounds__(32 * P2M_CW) k_p2m_chunks(LevOff lo, int nchunk, int first2,
                                                    const unsigned char* __restrict__ blev,
                                                    const unsigned char* __restrict__ plev,
                                                    const int* __restrict__ chunk_box,
                                                    const int* __restrict__ cstart,
                                                    const unsigned long long* __restrict__ keys,
                                                    const int* __restrict__ pt0, const int* __restrict__ pt1,
                                                    const float4* __restrict__ wa, const float2* __restrict__ qa,
                                                    const float2* __restrict__ qb, int p,
                                                    float2* __restrict__ mpart, int* __restrict__ cdone,
                                                    float2* __restrict__ mpole) {
  // Sums per chunk: A_k = sum a w^k, B_k = sum b w^k, C_k = sum conj(w) a w^k (a, b the
  // scaled charges), multipole -A_k and -(B_k + k C_(k-1)).
  extern __shared__ float4 sm4[];
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c = blockIdx.x * P2M_CW + wid;
  if (c >= nchunk) return;
  const int pitch = p2m_pitch(p), nout = E * p;
  float4* sab = sm4 + wid * 32;  // (a, b) per point
  float2* scc = reinterpret_cast<float2*>(sm4 + P2M_CW * 32) + wid * 32 * (pitch + 1);  // conj(w) a per point
  float2* pw = scc + 32;         // [32][pitch]: w^k per point
  const int b = chunk_box[c];
  const int l = blev[b];
  const float rinv = lo.rinv[l];
  const int bb = b - first2, c0 = cstart[bb], nc = cstart[bb + 1] - c0;
  const int i0 = pt0[b] + (c - c0) * EB_CHUNK;
  const int cnt = min(pt1[b], i0 + EB_CHUNK) - i0;
  pdl_wait();  // the charges
  // a box of one chunk gets its multipole directly; otherwise the chunk's part goes to
  // mpart and the box's last chunk to finish adds the parts in chunk order
  float2* dst = nc == 1 ? mpole + (size_t)b * nout : mpart + (size_t)c * nout;
  float2 last = make_float2(0.f, 0.f);  // C of the order below this round's
  for (int k0 = 0; k0 < p; k0 += 32) {  // a lane per order
    const int kw = min(32, p - k0), k = min(lane, kw - 1);
    float2 A = make_float2(0.f, 0.f), B = A, C = A;
    for (int s0 = 0; s0 < cnt; s0 += 32) {
      const int ns = min(32, cnt - s0);
      if (s0 > 0 || k0 > 0) __syncwarp();  // the previous points are consumed
      if (lane < ns) {
        const int i = i0 + s0 + lane;
        const int lam = plev[i], sh = lam - l;
        const float f = __int_as_float((127 - sh) << 23);  // 2^-sh
        const unsigned long long kl = keys[i] >> (2 * (EB_KEY_LEVELS - lam));
        const unsigned int ix = compact2d(kl), iy = compact2d(kl >> 1);
        const float4 wv = wa[i];
        const float gx = fmaf((float)ix + 0.5f, f, -((float)(ix >> sh) + 0.5f));
        const float gy = fmaf((float)iy + 0.5f, f, -((float)(iy >> sh) + 0.5f));
        const float2 w = make_float2(fmaf(wv.x, f, gx), fmaf(wv.y, f, gy));
        const float2 ah = cscale<float>(qa[i], rinv);
        if (E == 2) {
          const float2 bh = cscale<float>(qb[i], rinv);
          sab[lane] = make_float4(ah.x, ah.y, bh.x, bh.y);
          scc[lane] = cmul<float>(cconj<float>(w), ah);
        } else {
          scc[lane] = ah;
        }
        // two chains: even and odd powers
        float2* row = pw + lane * pitch;
        const float2 w2 = cmul<float>(w, w);
        float2 ev = k0 == 0 ? make_float2(1.f, 0.f) : cpow_int<float>(w, k0), od = cmul<float>(ev, w);
        for (int j = 0; j < kw; j += 2) {
          row[j] = ev;
          if (j + 1 < kw) row[j + 1] = od;
          ev = cmul<float>(ev, w2);
          od = cmul<float>(od, w2);
        }
      }
      __syncwarp();
#pragma unroll 4
      for (int s = 0; s < ns; ++s) {
        const float2 v = pw[s * pitch + k];
        if (E == 2) {
          const float4 ab = sab[s];
          cfma<float>(A, make_float2(ab.x, ab.y), v);
          cfma<float>(B, make_float2(ab.z, ab.w), v);
          cfma<float>(C, scc[s], v);
        } else {
          cfma<float>(A, scc[s], v);
        }
      }
    }
    if (lane < kw) dst[k0 + lane] = make_float2(-A.x, -A.y);
    if (E == 2) {
      float2 cm = make_float2(__shfl_up_sync(0xffffffffu, C.x, 1), __shfl_up_sync(0xffffffffu, C.y, 1));
      if (lane == 0) cm = last;
      last = make_float2(__shfl_sync(0xffffffffu, C.x, 31), __shfl_sync(0xffffffffu, C.y, 31));
      crfma<float>(B, (float)(k0 + lane), cm);
      if (lane < kw) dst[p + k0 + lane] = make_float2(-B.x, -B.y);
    }
  }
  if (nc > 1) p2m_finish(lane, nc, nout, mpart + (size_t)c0 * nout, cdone + bb, mpole + (size_t)b * nout);
}

// The same for the default order P (20), a lane per point: its terms -a w^k and
// -(b w + k conj(w) a) w^(k-1) of every order in registers (of two points for a chunk of
// more than 32), and one sum over the lanes through shared memory at the end. A power read
// from shared memory costs its bytes for every lane that gets them (two cycles of an SM a
// warp and 8 bytes), more than the multiply-adds that it feeds; here a chunk moves 320 bytes
// a lane once. Measured (E = 2): 64 x 512 (six levels, all from the points) 16.5 -> 10.4 us
// (13.4 with k_p2m_chunks); 73 us for 524,288 nodes, as that one.
template <int E, int P>
__global__ void __launch_bounds__(32 * P2M_CW, 4) k_p2m_points(LevOff lo, int nchunk, int first2,
                                                    const unsigned char* __restrict__ blev,
                                                    const unsigned char* __restrict__ plev,
                                                    const int* __restrict__ chunk_box,
                                                    const int* __restrict__ cstart,
                                                    const unsigned long long* __restrict__ keys,
                                                    const int* __restrict__ pt0, const int* __restrict__ pt1,
                                                    const float4* __restrict__ wa, const float2* __restrict__ qa,
                                                    const float2* __restrict__ qb,
                                                    float2* __restrict__ mpart, int* __restrict__ cdone,
                                                    float2* __restrict__ mpole) {
  constexpr int NF = 2 * E * P, PITCH = 36;  // floats of a chunk; row pitch (16-byte reads without conflicts)
  __shared__ float4 sm[P2M_CW][NF * PITCH / 4];
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c = blockIdx.x * P2M_CW + wid;
  if (c >= nchunk) return;
  const int b = chunk_box[c];
  const int l = blev[b];
  const float rinv = lo.rinv[l];
  const int bb = b - first2, c0 = cstart[bb], nc = cstart[bb + 1] - c0;
  const int i0 = pt0[b] + (c - c0) * EB_CHUNK, i1 = min(pt1[b], i0 + EB_CHUNK);
  pdl_wait();  // the charges
  float2 A[P], S[E == 2 ? P : 1];
#pragma unroll
  for (int k = 0; k < P; ++k) A[k] = make_float2(0.f, 0.f);
#pragma unroll
  for (int k = 0; k < (E == 2 ? P : 1); ++k) S[k] = make_float2(0.f, 0.f);
  for (int i = i0 + lane; i < i1; i += 32) {
    const int lam = plev[i], sh = lam - l;
    const float f = __int_as_float((127 - sh) << 23);  // 2^-sh
    const unsigned long long kl = keys[i] >> (2 * (EB_KEY_LEVELS - lam));
    const unsigned int ix = compact2d(kl), iy = compact2d(kl >> 1);
    const float4 wv = wa[i];
    const float gx = fmaf((float)ix + 0.5f, f, -((float)(ix >> sh) + 0.5f));
    const float gy = fmaf((float)iy + 0.5f, f, -((float)(iy >> sh) + 0.5f));
    const float2 w = make_float2(fmaf(wv.x, f, gx), fmaf(wv.y, f, gy));
    const float2 q = cscale<float>(qa[i], -rinv);
    float2 bw = make_float2(0.f, 0.f), cq = bw, pw = make_float2(1.f, 0.f);
    A[0] = cadd<float>(A[0], q);
    if (E == 2) {
      const float2 qs = cscale<float>(qb[i], -rinv);
      S[0] = cadd<float>(S[0], qs);
      bw = cmul<float>(qs, w);
      cq = cmul<float>(cconj<float>(w), q);
    }
#pragma unroll
    for (int k = 1; k < P; ++k) {
      if (E == 2) {
        float2 t = bw;
        crfma<float>(t, (float)k, cq);
        cfma<float>(S[E == 2 ? k : 0], t, pw);
      }
      pw = cmul<float>(pw, w);
      cfma<float>(A[k], q, pw);
    }
  }
  float* row = reinterpret_cast<float*>(sm[wid]) + lane;
#pragma unroll
  for (int k = 0; k < P; ++k) {
    row[2 * k * PITCH] = A[k].x;
    row[(2 * k + 1) * PITCH] = A[k].y;
    if (E == 2) {
      row[(2 * P + 2 * k) * PITCH] = S[E == 2 ? k : 0].x;
      row[(2 * P + 2 * k + 1) * PITCH] = S[E == 2 ? k : 0].y;
    }
  }
  __syncwarp();
  // a box of one chunk gets its multipole directly; otherwise the chunk's part goes to
  // mpart and the box's last chunk to finish adds the parts in chunk order
  constexpr int nout = E * P;
  float* dst = reinterpret_cast<float*>(nc == 1 ? mpole + (size_t)b * nout : mpart + (size_t)c * nout);
#pragma unroll
  for (int o0 = 0; o0 < NF; o0 += 32) {
    const int o = o0 + lane;
    if (o < NF) {
      float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int x = 0; x < 8; ++x) {
        const float4 v = sm[wid][o * (PITCH / 4) + x];
        t.x += v.x;
        t.y += v.y;
        t.z += v.z;
        t.w += v.w;
      }
      dst[o] = (t.x + t.y) + (t.z + t.w);
    }
  }
  if (nc > 1) p2m_finish(lane, nc, nout, mpart + (size_t)c0 * nout, cdone + bb, mpole + (size_t)b * nout);
}

// M2M into the boxes of one level from their children (FP32 coarse levels): all
// children's shifted coefficients are staged in one round of loads, then each output
// sums over the children in their fixed order.
template <int E>
__global__ void k_m2m_f32(int offp, const unsigned long long* __restrict__ bkey,
                          const int* __restrict__ child0, const int* __restrict__ nchild, int p,
                          const float* __restrict__ binom, int ldb, const float2* __restrict__ epow2,
                          const float2* __restrict__ einv, float2* __restrict__ mpole) {
  extern __shared__ float2 sm2[];
  float2* a = sm2;
  const int P = offp + blockIdx.x, tid = threadIdx.x, ld = p + 2, nout = E * p;
  const int c0 = child0[P], nc = nchild[P];
  pdl_wait();
  if (nc == 0) return;  // a leaf: its multipole comes from its points
  for (int idx = tid; idx < nc * nout; idx += blockDim.x) {
    const int ci = idx / nout, o = idx - ci * nout;
    const int c = c0 + ci, q = quadrant(bkey[c]);
    const int e2 = o / p, kk = o - e2 * p, k = kk + 1;
    const float2* mc = mpole + (size_t)c * nout;
    float2 v = mc[o];
    if (e2 == 1 && k >= 2) {
      const float2 ec = cscale<float>(epow2[q * ld + 1], 2.f);
      cfma<float>(v, cscale<float>(cconj<float>(ec), (float)(k - 1)), mc[kk - 1]);
    }
    a[idx] = cmul<float>(v, einv[q * ld + k]);
  }
  __syncthreads();
  if (tid < nout) {
    const int e = tid / p, n = tid - e * p + 1;
    const float* brow = binom + (size_t)(n - 1) * ldb;
    float2 acc = make_float2(0.f, 0.f);
    for (int ci = 0; ci < nc; ++ci) {
      const int q = quadrant(bkey[c0 + ci]);
      const float2* ae = a + ci * nout + e * p;
      float2 s0 = make_float2(0.f, 0.f), s1 = s0;
      int k = 0;
      for (; k + 1 < n; k += 2) {
        crfma<float>(s0, brow[k], ae[k]);
        crfma<float>(s1, brow[k + 1], ae[k + 1]);
      }
      if (k < n) crfma<float>(s0, brow[k], ae[k]);
      cfma<float>(acc, epow2[q * ld + n], cadd<float>(s0, s1));
    }
    mpole[(size_t)P * nout + tid] = acc;
  }
}

// ---------------------------------------------------------------------------------
// Leaf evaluation: L2P plus the near field over the U list (SLSELFDR/SLDIRDR,
// cadapdrop2.f:564-620, 724-769; DABARR's pair loop, dapif3.f:460-545), self excluded.
// One warp per group of up to 8 targets of a leaf; 4 lanes per target split the
// sources (and the terms of the local expansion), and their partial sums are added
// with two shuffles in a fixed order.
// ---------------------------------------------------------------------------------
// a u + c
template <typename T>
__device__ __forceinline__ c_t<T> chorner(c_t<T> a, c_t<T> u, c_t<T> c) {
  cfma<T>(c, a, u);
  return c;
}

// Terms m0 <= m < m1 of the local expansions at u.
template <typename T, int E>
__device__ __forceinline__ void l2p_range(const c_t<T>* lb, int p, int m0, int m1, c_t<T> u, T s, T& gx,
                                          T& gy) {
  const int ldl = p + 1;
  if (m0 >= m1) return;
  c_t<T> ph = lb[m1 - 1], dph = cmk<T>(0, 0);
  c_t<T> ps = E == 2 ? lb[ldl + m1 - 1] : cmk<T>(0, 0);
  for (int m = m1 - 2; m >= m0; --m) {
    if (E == 2) dph = chorner<T>(dph, u, ph);
    ph = chorner<T>(ph, u, lb[m]);
    if (E == 2) ps = chorner<T>(ps, u, lb[ldl + m]);
  }
  if (m0 > 0) {
    c_t<T> um1 = cpow_int<T>(u, m0 - 1);  // u^(m0-1)
    // d/du (u^m0 H) = u^(m0-1) (u H' + m0 H)
    if (E == 2) dph = cmul<T>(um1, cadd<T>(cmul<T>(u, dph), cscale<T>(ph, (T)m0)));
    c_t<T> um = cmul<T>(um1, u);
    ph = cmul<T>(um, ph);
    if (E == 2) ps = cmul<T>(um, ps);
  }
  if (E == 2) {
    c_t<T> t = cmulc<T>(u, dph);
    gx += ph.x + s * (t.x + ps.x);
    gy += ph.y + s * (t.y - ps.y);
  } else {
    gx -= ph.x;
    gy -= ph.y;
  }
}

// Partial far field of lane sl of 4: a quarter of the terms.
template <typename T, int E>
__device__ __forceinline__ void l2p_part(const c_t<T>* lb, int p, int sl, c_t<T> u, T s, T& gx,
                                         T& gy) {
  const int ldl = p + 1, q = (ldl + 3) / 4;
  const int m0 = sl * q, m1 = min(ldl, m0 + q);
  l2p_range<T, E>(lb, p, m0, m1, u, s, gx, gy);
}

// M2P: the far field at u (the target's offset from the box centre in box units) of a
// box's multipole expansions M (phi at M[0, p), psi relative to the centre at M[p, 2p),
// coefficient k at index k - 1): phi = sum_k M_k u^-k, and GW += phi + s (u conj(phi_u) +
// conj(psi)) for Stokes, F -= phi for Cauchy. The evaluation of SLMVALDR
// (cadapdrop2.f:251-301) and DSLOR1 (dapif3.f:1724-1749), used for the W lists.
template <typename T, int E>
__device__ __forceinline__ void m2p_eval(const c_t<T>* M, int p, c_t<T> u, T s, T& gx, T& gy) {
  const c_t<T> v = cinv<T>(u);
  c_t<T> a = M[p - 1];
  c_t<T> da = cscale<T>(M[p - 1], (T)p);
  for (int k = p - 1; k >= 1; --k) {
    a = chorner<T>(a, v, M[k - 1]);
    if (E == 2) da = chorner<T>(da, v, cscale<T>(M[k - 1], (T)k));
  }
  const c_t<T> ph = cmul<T>(a, v);  // sum M_k v^k
  if (E == 2) {
    const c_t<T> dph = cmul<T>(da, cmul<T>(v, v));  // sum k M_k v^(k+1) = -phi_u
    c_t<T> b = M[2 * p - 1];
    for (int k = p - 1; k >= 1; --k) b = chorner<T>(b, v, M[p + k - 1]);
    const c_t<T> ps = cmul<T>(b, v);
    const c_t<T> t = cmulc<T>(u, dph);  // -u conj(phi_u)
    gx += ph.x + s * (ps.x - t.x);
    gy += ph.y - s * (ps.y + t.y);
  } else {
    gx -= ph.x;
    gy -= ph.y;
  }
}

// FP64 near field, one block per tile of up to EB_NTILE targets of one leaf. GB300 issues
// two FP64 lanes a cycle and SM, so that the kernel is bound by FP64 instructions, and a
// lane without a pair costs as much as one with: the block's threads are dealt as
// (slice, target) with as many slices of the sources as fit, 128 / T for a tile of T
// targets (87 % of the lanes busy at T = 28, where 32-target tiles with fixed slices have
// 77 % on average). Sources are staged through shared memory in slabs; a warp reads two to five
// of them at once (broadcasts). The slices are added in a fixed order; the sums go
// to nearbuf (sorted order), so that the near field runs beside the expansion passes. It
// does so with NEAR64_CTAS blocks per SM that draw tiles from a counter (zeroed by the
// charges' kernel): eight warps keep the FP64 pipe busy, while as many blocks as fit left
// the expansion passes, which share the pipe warp by warp, a seventh of it and the
// fixed-point M2L no shared memory.
// Measured: 3.25 ms for the 110.6 M pairs of 1,048,576 nodes (82 % of the FP64 issue rate
// at 14 instructions a pair), 149 us for the 4.0 M of 64 x 512; with a warp per 8 targets
// reading every source from global memory and the longer pair, near and far field
// together took 9.76 ms and 392 us (now, with the far field below, 5.7 ms and 233 us).
// HALF: a block takes half a tile. Among points spread over decades (trees with many W lists: from
// an entry per 8 leaves on) a leaf beside a dense part has thousands of sources where others have
// hundreds, and a block with a whole tile of it runs on when the others are done: 12,000 such
// points 1.4 -> 0.8 ms a Cauchy sum, with 200 and 400 a leaf 2.8 -> 1.6 and 3.3 -> 2.4 ms (2.5 and 3.1 with
// the warp per 8 targets). And with NEAR64_HALF sources a target on average (leaves of hundreds of
// points), where 126 lanes busy instead of 112 pay for staging every slab twice: 12,000 even
// points with 400 a leaf 0.94 -> 0.80 ms, 200,001 11.0 -> 9.4 (10.0 with the warp per 8 targets). On the
// other even trees half tiles take from 6 % less (64 x 1,024) to 7 % more (1,300 x 1,024).
#define NEAR64_SLAB 128
#define NEAR64_CTAS 4
#define NEAR64_HALF 1024
template <int K, bool HALF>
__global__ void __launch_bounds__(128) k_near64(int ntile, int* __restrict__ next,
                                                const int4* __restrict__ tiles, const int* __restrict__ pt0,
                                                const int* __restrict__ pt1, const int* __restrict__ ustart,
                                                const int* __restrict__ ulist, const double2* __restrict__ zs,
                                                const double2* __restrict__ q, int plus,
                                                double2* __restrict__ nearbuf) {
  constexpr bool ST = K == NEAR_V || K == NEAR_VC;
  __shared__ double2 sz[NEAR64_SLAB], sa[NEAR64_SLAB], sc[ST ? NEAR64_SLAB : 1], sred[128];
  __shared__ int sidx[NEAR64_SLAB], spre[33], sj0[32], s_tile;
  const int tid = threadIdx.x;
  for (;;) {
    if (tid == 0) s_tile = atomicAdd(next, 1);
    __syncthreads();
    const int item = s_tile;
    if (item >= (HALF ? 2 * ntile : ntile)) return;
    int4 tl = tiles[HALF ? item >> 1 : item];
    if (HALF) {
      const int mid = tl.y + ((tl.z - tl.y + 1) >> 1);
      if (item & 1) tl.y = mid;
      else tl.z = mid;
      if (tl.y == tl.z) {  // the second half of a single target
        __syncthreads();
        continue;
      }
    }
    const int T = tl.z - tl.y, nsl = 128 / T;
    const int sl = tid / T, i = tl.y + tid - sl * T;
    const double2 zi = zs[i];
    double gx = 0.0, gy = 0.0;
    const int ub = ustart[tl.x], ue = ustart[tl.x + 1];
    for (int cb = ub; cb < ue; cb += 32) {
      const int nc = min(32, ue - cb);
      if (cb > ub) __syncthreads();  // the previous boxes' slabs are consumed
      if (tid < 32) {
        int c = 0, j0 = 0;
        if (tid < nc) {
          const int sbx = ulist[cb + tid];
          j0 = pt0[sbx];
          c = pt1[sbx] - j0;
        }
        int x = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(0xffffffffu, x, o);
          if (tid >= o) x += y;
        }
        sj0[tid] = j0;
        spre[tid + 1] = x;
        if (tid == 0) spre[0] = 0;
      }
      __syncthreads();
      const int total = spre[nc];
      for (int base = 0; base < total; base += NEAR64_SLAB) {
        const int ns = min(NEAR64_SLAB, total - base);
        if (base > 0) __syncthreads();
        if (tid < ns) {
          const int gs = base + tid;
          int lo = 0, hi = nc;  // the box k with spre[k] <= gs < spre[k + 1]
          while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (spre[mid] <= gs) lo = mid;
            else hi = mid;
          }
          const int j = sj0[lo] + gs - spre[lo];
          sidx[tid] = j;
          sz[tid] = zs[j];
          if (ST) {
            sa[tid] = q[2 * (size_t)j];
            sc[tid] = q[2 * (size_t)j + 1];
          } else {
            sa[tid] = q[j];
          }
        }
        __syncthreads();
        if (sl < nsl) {
#pragma unroll 2
          for (int jj = sl; jj < ns; jj += nsl) {
            if (sidx[jj] == i) continue;
            near_pair64<K>(sz[jj], sa[jj], ST ? sc[jj] : make_double2(0.0, 0.0), zi, gx, gy);
          }
        }
      }
    }
    sred[tid] = make_double2(gx, gy);
    __syncthreads();
    if (tid < T) {
      double2 v = sred[tid];
      for (int k = 1; k < nsl; ++k) v = cadd<double>(v, sred[k * T + tid]);
      nearbuf[i] = ST ? near_turn<double>(v.x, v.y, plus) : v;
    }
  }
}

// Points from which the FP64 far field takes one lane per target: with fewer, a lane's whole
// Horner chain is longer than the FP64 pipe is busy. Measured, Horner steps
// as four FMAs and no divisions included: 83.5 -> 38.8 us at 64 x 512 and 2.48 -> 0.97 ms at
// 1,024 x 1,024 with one lane, 15.3 -> 12.3 us at 4,096 nodes with four.
constexpr int FAR64_ONE = 12288;

// FP64 far field: L2P of the leaf's local expansions and the W list, LPT lanes per target
// (LPT = 4: a warp per group of 8 targets, each lane a quarter of the terms; LPT = 1: a
// thread per target), plus the near-field sums, then the post-processing.
template <int E, int LPT>
__global__ void __launch_bounds__(128) k_far64(int n, const int* __restrict__ lflag,
                                               const int* __restrict__ lscan,
                                               const int* __restrict__ leaves, int has_far,
                                               const unsigned long long* __restrict__ bkey,
                                               const unsigned char* __restrict__ blev,
                                               const int* __restrict__ wstart, const int* __restrict__ wlist,
                                               const int* __restrict__ perm, const double2* __restrict__ zs,
                                               double x0, double y0, double W, double winv, int p, double s,
                                               const double2* __restrict__ local,
                                               const double2* __restrict__ mpole,
                                               const double2* __restrict__ nearbuf, double2* __restrict__ out,
                                               EbPost post) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = g / LPT, sl = g - i * LPT;
  const bool act = i < n;
  double gx = 0.0, gy = 0.0;
  if (act && has_far) {
    const int leaf = lscan[i] + lflag[i] - 1, b = leaves[leaf];  // leaf heads up to point i
    const double2 zi = zs[i];
    if (blev[b] >= 2) {
      const int lev = blev[b];
      const double2 c = box_center(bkey[b], x0, y0, W * pow2d(-lev));
      const double rinv = winv * pow2d(lev);
      const double2 u = make_double2((zi.x - c.x) * rinv, (zi.y - c.y) * rinv);
      const double2* lb = local + (size_t)b * E * (p + 1);
      if (LPT == 1) l2p_range<double, E>(lb, p, 0, p + 1, u, s, gx, gy);
      else l2p_part<double, E>(lb, p, sl, u, s, gx, gy);
    }
    for (int jw = wstart[leaf] + sl; jw < wstart[leaf + 1]; jw += LPT) {
      const int w = wlist[jw];
      const int lev = blev[w];
      const double2 cw = box_center(bkey[w], x0, y0, W * pow2d(-lev));
      const double rinv = winv * pow2d(lev);
      m2p_eval<double, E>(mpole + (size_t)w * E * p, p, make_double2((zi.x - cw.x) * rinv, (zi.y - cw.y) * rinv),
                          s, gx, gy);
    }
  }
  if (LPT == 4) {
    gx += __shfl_xor_sync(0xffffffffu, gx, 1);
    gy += __shfl_xor_sync(0xffffffffu, gy, 1);
    gx += __shfl_xor_sync(0xffffffffu, gx, 2);
    gy += __shfl_xor_sync(0xffffffffu, gy, 2);
  }
  if (act && sl == 0) {
    const double2 nv = nearbuf[i];
    eb_post_store(post, perm[i], make_double2(gx + nv.x, gy + nv.y), out);
  }
}

// ---------------------------------------------------------------------------------
// FP64-accurate leaf evaluation in double-float arithmetic (the sums of k_near64 and k_far64,
// about 2^-47 relative per operation, several times faster on GB300's FP32 pipes).
// Offsets are leaf-relative: for target i in leaf b and source j in neighbour b',
// (z_j - z_i)/r = w_j - (w_i - (b' - b)), exact up to the double-float rounding of w;
// the charges carry the factor 1/r. The local expansions are double-float already.
// ---------------------------------------------------------------------------------
__device__ __forceinline__ cdf cdf_pow(cdf u, int n) {
  cdf r = cdf{{1.f, 0.f}, {0.f, 0.f}}, b = u;
  while (n > 0) {
    if (n & 1) r = cdf_mul(r, b);
    b = cdf_mul(b, b);
    n >>= 1;
  }
  return r;
}

// (hi, mid, lo) - d for a small integer d, renormalised into three floats
__device__ __forceinline__ float3 tf_shift(float hi, float mid, float lo, float d) {
  dfl a = two_sum(hi, -d);
  dfl b = two_sum(mid, a.lo);
  return make_float3(a.hi, b.hi, __fadd_rn(lo, b.lo));
}

// (ah + am + al) - (b.x + b.y + b.z) as a double-float; the hi and mid differences are
// formed exactly, so the result carries the full precision of the three-float inputs.
__device__ __forceinline__ dfl tf_diff(float ah, float am, float al, float3 b) {
  dfl s = two_sum(ah, -b.x);
  dfl t = two_sum(am, -b.y);
  float u = __fadd_rn(__fadd_rn(__fsub_rn(al, b.z), s.lo), t.lo);
  dfl h = two_sum(s.hi, t.hi);
  return fast_two_sum(h.hi, __fadd_rn(h.lo, u));
}

// The near-field pair's steps without the renormalisations between them: a value's low part
// may reach a few ulps of the high one, so the products of two low parts are kept where both
// factors are of that kind (the Cauchy pair keeps normalized factors: its sums' errors were 2 %
// larger without). 1,048,576 nodes: 915 -> 825 us (Stokes).
__device__ __forceinline__ dfl dfl_mul_raw(dfl a, dfl b) {
  const float p = __fmul_rn(a.hi, b.hi);
  float e = __fmaf_rn(a.hi, b.hi, -p);
  e = __fmaf_rn(a.hi, b.lo, e);
  return dfl{p, __fmaf_rn(a.lo, b.hi, e)};
}
// a b + c d
__device__ __forceinline__ dfl dfl_dot2_raw(dfl a, dfl b, dfl c, dfl d) {
  const dfl x = dfl_mul_raw(a, b), y = dfl_mul_raw(c, d), t = two_sum(x.hi, y.hi);
  return dfl{t.hi, __fadd_rn(t.lo, __fadd_rn(x.lo, y.lo))};
}
// 1 / (x^2 + y^2): the hardware's estimate and a third-order step
__device__ __forceinline__ dfl dfl_rcp_norm(dfl x, dfl y) {
  const dfl d = dfl_dot2_raw(x, x, y, y);
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d.hi));
  const float t = __fmaf_rn(-d.lo, r, __fmaf_rn(-d.hi, r, 1.0f));
  return fast_two_sum(r, __fmul_rn(r, __fmaf_rn(t, t, t)));
}
// a + b c, and acc += b c
__device__ __forceinline__ dfl dfl_fma_raw(dfl a, dfl b, dfl c) {
  const float p = __fmul_rn(b.hi, c.hi);
  float e = __fmaf_rn(b.lo, c.lo, __fmaf_rn(b.hi, c.hi, -p));
  e = __fmaf_rn(b.hi, c.lo, e);
  e = __fmaf_rn(b.lo, c.hi, e);
  const dfl t = two_sum(p, a.hi);
  return dfl{t.hi, __fadd_rn(t.lo, __fadd_rn(e, a.lo))};
}
__device__ __forceinline__ void acc_prod_raw(dfacc& a, dfl x, dfl y) {
  const float p = __fmul_rn(x.hi, y.hi);
  float e = __fmaf_rn(x.lo, y.lo, __fmaf_rn(x.hi, y.hi, -p));
  e = __fmaf_rn(x.hi, y.lo, e);
  e = __fmaf_rn(x.lo, y.hi, e);
  acc_add(a, p);
  a.c = __fadd_rn(a.c, e);
}

// a u + c: the two products and the addend of each part summed at once
__device__ __forceinline__ dfl dfl_dot2_add(dfl a, dfl b, dfl c, dfl d, dfl s) {  // a b + c d + s
  const float p = __fmul_rn(a.hi, b.hi), q = __fmul_rn(c.hi, d.hi);
  float e = __fmaf_rn(a.hi, b.hi, -p), f = __fmaf_rn(c.hi, d.hi, -q);
  e = __fmaf_rn(a.hi, b.lo, e);
  f = __fmaf_rn(c.hi, d.lo, f);
  e = __fmaf_rn(a.lo, b.hi, e);
  f = __fmaf_rn(c.lo, d.hi, f);
  const dfl t = two_sum(p, q), u = two_sum(t.hi, s.hi);
  return fast_two_sum(u.hi, __fadd_rn(__fadd_rn(u.lo, t.lo), __fadd_rn(__fadd_rn(e, f), s.lo)));
}
__device__ __forceinline__ cdf cdf_horner(cdf a, cdf u, cdf c) {
  return cdf{dfl_dot2_add(a.x, u.x, dfl_neg(a.y), u.y, c.x), dfl_dot2_add(a.x, u.y, a.y, u.x, c.y)};
}

template <int E>
__device__ __forceinline__ void l2p_part_df(const float4* L, int p, int sl, cdf u, bool neg, dfacc& gx,
                                            dfacc& gy) {
  const int ldl = p + 1, q = (ldl + 3) / 4;
  int m0 = sl * q, m1 = min(ldl, m0 + q);
  if (m0 >= m1) return;
  cdf ph = cdf_from_float4(L[m1 - 1]), dph = cdf{{0.f, 0.f}, {0.f, 0.f}};
  for (int m = m1 - 2; m >= m0; --m) {
    if (E == 2) dph = cdf_horner(dph, u, ph);
    ph = cdf_horner(ph, u, cdf_from_float4(L[m]));
  }
  cdf ps = cdf{{0.f, 0.f}, {0.f, 0.f}};
  if (E == 2) {
    ps = cdf_from_float4(L[ldl + m1 - 1]);
    for (int m = m1 - 2; m >= m0; --m) ps = cdf_horner(ps, u, cdf_from_float4(L[ldl + m]));
  }
  if (m0 > 0) {
    cdf um1 = cdf_pow(u, m0 - 1);
    if (E == 2)
      dph = cdf_mul(um1, cdf_horner(u, dph, cdf{dfl_mul_f(ph.x, (float)m0), dfl_mul_f(ph.y, (float)m0)}));
    cdf um = cdf_mul(um1, u);
    ph = cdf_mul(um, ph);
    if (E == 2) ps = cdf_mul(um, ps);
  }
  if (E == 2) {
    // phi + s (u conj(phi') + conj(psi))
    dfl tx = dfl_add(dfl_mul(u.x, dph.x), dfl_mul(u.y, dph.y));
    dfl ty = dfl_sub(dfl_mul(u.y, dph.x), dfl_mul(u.x, dph.y));
    dfl sx = dfl_add(tx, ps.x), sy = dfl_sub(ty, ps.y);
    if (neg) {
      sx = dfl_neg(sx);
      sy = dfl_neg(sy);
    }
    acc_dfl(gx, ph.x);
    acc_dfl(gx, sx);
    acc_dfl(gy, ph.y);
    acc_dfl(gy, sy);
  } else {
    acc_dfl(gx, dfl_neg(ph.x));
    acc_dfl(gy, dfl_neg(ph.y));
  }
}

// Offset between the centres of a box of level lt (grid index it) and a box of level
// ls = lt + ds (index is), in units of the second box's side: (c_t - c_s) / r_s =
// ((2 it + 1) 2^ds - (2 is + 1)) / 2, formed in integers and exact in float for boxes
// that touch or nearly touch.
__device__ __forceinline__ float box_delta(int it, int is, int ds) {
  long long num;
  int e;
  if (ds >= 0) {
    num = ((2LL * it + 1) << ds) - (2LL * is + 1);
    e = -1;
  } else {
    num = (2LL * it + 1) - ((2LL * is + 1) << (-ds));
    e = ds - 1;
  }
  return ldexpf((float)num, e);
}

__device__ __forceinline__ float pow2f(int e) { return __int_as_float((127 + e) << 23); }

// A target's position relative to the centre of a box ds levels below (ds < 0: above)
// its leaf, in that box's units, as three floats: w 2^ds + (c_leaf - c_box) / r_box.
__device__ __forceinline__ void frame_shift(float4 wa, float2 wb, int ds, int bx, int by, int sx, int sy,
                                            float3& tx, float3& ty) {
  const float f = pow2f(ds);
  tx = tf_shift(wa.x * f, wa.z * f, wb.x * f, -box_delta(bx, sx, ds));
  ty = tf_shift(wa.y * f, wa.w * f, wb.y * f, -box_delta(by, sy, ds));
}

__device__ __forceinline__ dfl tf_to_dfl(float3 t) {
  return dfl_add(two_sum(t.x, t.y), dfl{t.z, 0.f});
}

// M2P in double-float (m2p_eval's sums): M the box's double-float multipoles, u the
// target's offset in box units.
template <int E>
__device__ __forceinline__ void m2p_df(const float4* M, int p, cdf u, bool neg, dfacc& gx, dfacc& gy) {
  const dfl rr = dfl_rcp(dfl_add(dfl_sqr(u.x), dfl_sqr(u.y)));
  const cdf v = cdf{dfl_mul(u.x, rr), dfl_neg(dfl_mul(u.y, rr))};
  cdf a = cdf_from_float4(M[p - 1]);
  cdf da = cdf_scale(a, (float)p);
  for (int k = p - 1; k >= 1; --k) {
    const cdf mk = cdf_from_float4(M[k - 1]);
    a = cdf_horner(a, v, mk);
    if (E == 2) da = cdf_horner(da, v, cdf_scale(mk, (float)k));
  }
  const cdf ph = cdf_mul(a, v);
  if (E == 2) {
    const cdf dph = cdf_mul(da, cdf_mul(v, v));  // -phi_u
    cdf b = cdf_from_float4(M[2 * p - 1]);
    for (int k = p - 1; k >= 1; --k) b = cdf_horner(b, v, cdf_from_float4(M[p + k - 1]));
    const cdf ps = cdf_mul(b, v);
    const dfl tx = dfl_add(dfl_mul(u.x, dph.x), dfl_mul(u.y, dph.y));  // -u conj(phi_u)
    const dfl ty = dfl_sub(dfl_mul(u.y, dph.x), dfl_mul(u.x, dph.y));
    dfl sx = dfl_sub(ps.x, tx), sy = dfl_neg(dfl_add(ps.y, ty));
    if (neg) {
      sx = dfl_neg(sx);
      sy = dfl_neg(sy);
    }
    acc_dfl(gx, ph.x);
    acc_dfl(gx, sx);
    acc_dfl(gy, ph.y);
    acc_dfl(gy, sy);
  } else {
    acc_dfl(gx, dfl_neg(ph.x));
    acc_dfl(gy, dfl_neg(ph.y));
  }
}

// The near field into nearbuf (sorted order): a warp per group of 8 targets of a leaf, 4
// lanes per target over the sources. K: NEAR_V, NEAR_VC or NEAR_Q; nc: (ax, ay), (c0, c1)
// per source, or q.
__device__ __forceinline__ void df_quad_sum(dfl& vx, dfl& vy, int sl) {
#pragma unroll
  for (int o = 1; o <= 2; o <<= 1) {
    dfl ox{__shfl_xor_sync(0xffffffffu, vx.hi, o), __shfl_xor_sync(0xffffffffu, vx.lo, o)};
    dfl oy{__shfl_xor_sync(0xffffffffu, vy.hi, o), __shfl_xor_sync(0xffffffffu, vy.lo, o)};
    vx = (sl & o) ? dfl_add(ox, vx) : dfl_add(vx, ox);
    vy = (sl & o) ? dfl_add(oy, vy) : dfl_add(vy, oy);
  }
}

template <int K>
__global__ void __launch_bounds__(128) k_near_df(int ngroup, const int* __restrict__ gleaf,
                                                 const int* __restrict__ gfirst, const int* __restrict__ leaves,
                                                 const unsigned long long* __restrict__ bkey,
                                                 const unsigned char* __restrict__ blev,
                                                 const int* __restrict__ pt0, const int* __restrict__ pt1,
                                                 const int* __restrict__ ustart, const int* __restrict__ ulist,
                                                 const float4* __restrict__ wa, const float2* __restrict__ wb,
                                                 const float4* __restrict__ nc, int plus,
                                                 double2* __restrict__ nearbuf) {
  const int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (g >= ngroup) return;
  const int lane = threadIdx.x & 31, tg = lane >> 2, sl = lane & 3;
  const int leaf = gleaf[g], b = leaves[leaf];
  const int i = gfirst[g] + tg;
  const bool act = i < pt1[b];
  const int ii = act ? i : gfirst[g];
  const float4 wia = wa[ii];
  const float2 wib = wb[ii];
  const int lt = blev[b];
  dfacc gx{0.f, 0.f}, gy{0.f, 0.f};
  const unsigned long long kb = bkey[b];
  const int bx = (int)compact2d(kb), by = (int)compact2d(kb >> 1);
  for (int jl = ustart[leaf]; jl < ustart[leaf + 1]; ++jl) {
    const int sb = ulist[jl];
    const unsigned long long ks = bkey[sb];
    // the target relative to the source leaf's centre, in that leaf's units (three
    // floats); the source charges carry the factor 1 / r of their own leaf
    float3 tx, ty;
    frame_shift(wia, wib, blev[sb] - lt, bx, by, (int)compact2d(ks), (int)compact2d(ks >> 1), tx, ty);
    const int j1 = pt1[sb];
    for (int j = pt0[sb] + sl; j < j1; j += 4) {
      if (j == ii) continue;
      const float4 ja = wa[j];
      const float2 jb = wb[j];
      // D / r = w_j - (w_i - offset): hi and mid parts subtracted exactly
      const dfl dx = tf_diff(ja.x, ja.z, jb.x, tx), dy = tf_diff(ja.y, ja.w, jb.y, ty);
      const dfl rr = dfl_rcp_norm(dx, dy);
      const dfl ex = K == NEAR_Q ? dfl_mul(dx, rr) : dfl_mul_raw(dx, rr);  // conj(1/D)
      const dfl ey = K == NEAR_Q ? dfl_mul(dy, rr) : dfl_mul_raw(dy, rr);
      if (K == NEAR_Q) {
        const cdf q = cdf_from_float4(nc[j]);  // q/(z_i - z_j) = -q/D
        acc_prod(gx, dfl_neg(q.x), ex);
        acc_prod(gx, dfl_neg(q.y), ey);
        acc_prod(gy, q.x, ey);
        acc_prod(gy, dfl_neg(q.y), ex);
      } else {
        const float4 a = nc[2 * (size_t)j], c = nc[2 * (size_t)j + 1];
        const dfl v = dfl_fma_raw(dfl{c.x, c.y}, ey, dfl_dot2_raw(dfl{a.x, a.y}, dx, dfl{a.z, a.w}, dy));
        acc_prod_raw(gx, ex, v);
        acc_prod_raw(gy, ey, v);
        if (K == NEAR_VC) {
          const dfl c1{c.z, c.w};
          acc_prod(gx, dfl_neg(ey), c1);
          acc_prod(gy, ex, c1);
        }
      }
    }
  }
  dfl vx = acc_value(gx), vy = acc_value(gy);
  df_quad_sum(vx, vy, sl);
  if (sl == 0 && act) {
    const double x = dfl_to_double(vx), y = dfl_to_double(vy);
    nearbuf[i] = K == NEAR_Q ? make_double2(x, y) : near_turn<double>(x, y, plus);
  }
}

// The far field (L2P and the W list) plus the near-field sums, then the post-processing.
template <int E>
__global__ void __launch_bounds__(128) k_far_df(int ngroup, const int* __restrict__ gleaf,
                                                const int* __restrict__ gfirst, const int* __restrict__ leaves,
                                                int has_far, const unsigned long long* __restrict__ bkey,
                                                const unsigned char* __restrict__ blev,
                                                const int* __restrict__ pt1,
                                                const int* __restrict__ wstart, const int* __restrict__ wlist,
                                                const float4* __restrict__ mpole, const int* __restrict__ perm,
                                                const float4* __restrict__ wa, const float2* __restrict__ wb,
                                                int p, double s, const float4* __restrict__ local,
                                                double2* __restrict__ out, EbPost post,
                                                const double2* __restrict__ nearbuf) {
  const int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (g >= ngroup) return;
  const int lane = threadIdx.x & 31, tg = lane >> 2, sl = lane & 3;
  const int leaf = gleaf[g], b = leaves[leaf];
  const int i = gfirst[g] + tg;
  const bool act = i < pt1[b];
  const int ii = act ? i : gfirst[g];
  const float4 wia = wa[ii];
  const float2 wib = wb[ii];
  const cdf wi = cdf{{wia.x, wia.z}, {wia.y, wia.w}};
  const bool neg = s < 0.0;
  const int lt = blev[b];
  dfacc gx{0.f, 0.f}, gy{0.f, 0.f};
  if (has_far && lt >= 2) l2p_part_df<E>(local + (size_t)b * E * (p + 1), p, sl, wi, neg, gx, gy);
  if (has_far) {
    const unsigned long long kb = bkey[b];
    const int bx = (int)compact2d(kb), by = (int)compact2d(kb >> 1);
    // W list: the lanes of a target take every 4th box
    for (int jw = wstart[leaf] + sl; jw < wstart[leaf + 1]; jw += 4) {
      const int w = wlist[jw];
      const unsigned long long kw = bkey[w];
      float3 tx, ty;
      frame_shift(wia, wib, blev[w] - lt, bx, by, (int)compact2d(kw), (int)compact2d(kw >> 1), tx, ty);
      m2p_df<E>(mpole + (size_t)w * E * p, p, cdf{tf_to_dfl(tx), tf_to_dfl(ty)}, neg, gx, gy);
    }
  }
  dfl vx = acc_value(gx), vy = acc_value(gy);
  df_quad_sum(vx, vy, sl);
  if (sl == 0 && act) {
    const double2 nv = nearbuf[i];
    eb_post_store(post, perm[i], make_double2(dfl_to_double(vx) + nv.x, dfl_to_double(vy) + nv.y), out);
  }
}

// FP32 far field, one block per tile of the near field: the local expansions of the
// leaf and of its nearest ancestors (at most EB_FAR_LEVELS boxes, the coarsest holding
// the L2L-accumulated expansion of the levels above) are staged in shared memory, and
// each expansion is evaluated directly about its own centre at every target (the sum
// equals L2P of the L2L-accumulated leaf expansion). Each half-warp takes one level, and
// every EB_FAR_LEVELS-th box of the leaf's W list, whose multipoles are evaluated at the
// targets (M2P). Adds the near-field sums of k_near32 and applies the post-processing.
//
// Its Horner steps bound it (12 multiply-adds an order, level and target of E = 2). A lane
// holds two targets of the tile and takes them through packed multiply-adds, with each
// coefficient staged twice (x, x, y, y): 8 instructions an order for 32 targets of two
// levels, where a lane per target and warps that took every fourth of six levels had 28.
// Measured (E = 2): 1,048,576 nodes 227 -> 183 us, 64 x 512 10.8 -> 9.1 us.
constexpr int FAR_THREADS = 16 * EB_FAR_LEVELS;

__device__ __forceinline__ void chorner2(f32x2& ax, f32x2& ay, f32x2 ux, f32x2 uy, f32x2 nuy, f32x2 cx, f32x2 cy) {
  const f32x2 x = fma2(ax, ux, fma2(ay, nuy, cx));
  ay = fma2(ax, uy, fma2(ay, ux, cy));
  ax = x;
}

template <int E>
__global__ void __launch_bounds__(FAR_THREADS) k_far32(const int4* __restrict__ tiles, const int* __restrict__ leaves,
                                               const unsigned long long* __restrict__ bkey,
                                               const unsigned char* __restrict__ blev,
                                               const int* __restrict__ anc, const int* __restrict__ wstart,
                                               const int* __restrict__ wlist,
                                               const int* __restrict__ perm,
                                               const float4* __restrict__ wa, int p, float s,
                                               const float2* __restrict__ local,
                                               const float2* __restrict__ mpole,
                                               double2* __restrict__ out, EbPost post,
                                               const double2* __restrict__ nearbuf) {
  constexpr int T = EB_NTILE, NS = EB_FAR_LEVELS;
  static_assert(T == 32, "two targets per lane of a half-warp");
  extern __shared__ float4 sloc[];  // [nf][p + 1][E]: a coefficient as (x, x, y, y)
  __shared__ float2 sred[NS][T];
  const int4 tl = tiles[blockIdx.x];
  const int leaf = tl.x, b = leaves[leaf];
  const int tid = threadIdx.x, tt = tid & 15, sl = tid >> 4;
  const int i0 = tl.y + tt, i1 = i0 + 16;
  const bool two = tl.z - tl.y > 16;  // the tile's second half holds targets
  const int ldl = p + 1, nco = E * ldl;
  const int box = anc[(size_t)leaf * EB_FAR_LEVELS + sl];  // this half-warp's
  if (box >= 0) {
    const float2* lc = local + (size_t)box * nco;
    for (int m = tt; m < ldl; m += 16)
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const float2 v = lc[e * ldl + m];
        sloc[sl * nco + m * E + e] = make_float4(v.x, v.x, v.y, v.y);
      }
  }
  const unsigned long long kb = bkey[b];
  const unsigned int ix = compact2d(kb), iy = compact2d(kb >> 1);
  const float4 w0 = wa[i0 < tl.z ? i0 : tl.y], w1 = wa[i1 < tl.z ? i1 : tl.y];
  float2 f0 = make_float2(0.f, 0.f), f1 = f0;
  __syncwarp();
  // With u the leaf-scaled offset, the offset scaled to the ancestor sl levels up is
  //   u 2^-sl + (i + 1/2) 2^-sl - (i >> sl) - 1/2   (i the leaf's grid index),
  // whose constant part is exact in FP32 (i < 2^20).
  if (box >= 0) {
    const float f = __int_as_float((127 - sl) << 23);  // 2^-sl
    const float gx = fmaf((float)ix + 0.5f, f, -((float)(ix >> sl) + 0.5f));
    const float gy = fmaf((float)iy + 0.5f, f, -((float)(iy >> sl) + 0.5f));
    const f32x2 ff = pk2(f, f), gx2 = pk2(gx, gx), gy2 = pk2(gy, gy);
    const f32x2 ux = fma2(pk2(w0.x, w1.x), ff, gx2), uy = fma2(pk2(w0.y, w1.y), ff, gy2);
    const f32x2 nuy = mul2(uy, pk2(-1.f, -1.f));
    const ulonglong2* lb = reinterpret_cast<const ulonglong2*>(sloc + sl * nco);
    ulonglong2 c = lb[p * E];
    f32x2 phx = c.x, phy = c.y, dx = 0, dy = 0, psx = 0, psy = 0;
    if (E == 2) {
      c = lb[p * E + 1];
      psx = c.x;
      psy = c.y;
    }
#pragma unroll 4
    for (int m = p - 1; m >= 0; --m) {
      if (E == 2) chorner2(dx, dy, ux, uy, nuy, phx, phy);
      c = lb[m * E];
      chorner2(phx, phy, ux, uy, nuy, c.x, c.y);
      if (E == 2) {
        c = lb[m * E + 1];
        chorner2(psx, psy, ux, uy, nuy, c.x, c.y);
      }
    }
    f32x2 gx_, gy_;
    if (E == 2) {  // phi + s (u conj(phi') + conj(psi))
      const f32x2 ss = pk2(s, s), ns = pk2(-s, -s);
      gx_ = fma2(ss, fma2(ux, dx, fma2(uy, dy, psx)), phx);
      gy_ = fma2(ns, fma2(ux, dy, fma2(nuy, dx, psy)), phy);
    } else {
      gx_ = mul2(phx, pk2(-1.f, -1.f));
      gy_ = mul2(phy, pk2(-1.f, -1.f));
    }
    const float2 vx = upk2(gx_), vy = upk2(gy_);
    f0 = make_float2(vx.x, vy.x);
    f1 = make_float2(vx.y, vy.y);
  }
  // W list (boxes below the leaf's level): the target's offset in the box's units is
  // u 2^ds + (c_leaf - c_box) / r_box, the high part of u first, so that the cancelling
  // terms meet exactly, then the middle part
  const int lt = blev[b];
  for (int jw = wstart[leaf] + sl; jw < wstart[leaf + 1]; jw += NS) {
    const int w = wlist[jw];
    const unsigned long long kw = bkey[w];
    const int ds = blev[w] - lt;
    const float f = pow2f(ds);
    const float dx = box_delta((int)ix, (int)compact2d(kw), ds), dy = box_delta((int)iy, (int)compact2d(kw >> 1), ds);
    const float2* mw = mpole + (size_t)w * E * p;
    const float2 u0 = make_float2(fmaf(w0.z, f, fmaf(w0.x, f, dx)), fmaf(w0.w, f, fmaf(w0.y, f, dy)));
    m2p_eval<float, E>(mw, p, u0, s, f0.x, f0.y);
    if (two) {
      const float2 u1 = make_float2(fmaf(w1.z, f, fmaf(w1.x, f, dx)), fmaf(w1.w, f, fmaf(w1.y, f, dy)));
      m2p_eval<float, E>(mw, p, u1, s, f1.x, f1.y);
    }
  }
  sred[sl][tt] = f0;
  sred[sl][tt + 16] = f1;
  __syncthreads();
  const int i = tl.y + tid;
  if (tid < T && i < tl.z) {
    float2 v = sred[0][tid];
#pragma unroll
    for (int q = 1; q < NS; ++q) {
      v.x += sred[q][tid].x;
      v.y += sred[q][tid].y;
    }
    const double2 nv = nearbuf[i];
    eb_post_store_f32(post, perm[i], make_float2(v.x + (float)nv.x, v.y + (float)nv.y), out);
  }
}

// FP32 near field, one block per tile of up to EB_NTILE (32) targets of one leaf: the
// sources of the leaf's U list (32 boxes at a time) are staged through shared memory in
// slabs of NEAR_SLAB, source q of a slab beside source q + half the slab. Each thread holds
// two targets of the tile (lanes l and l + 16 of the tile; one, if the tile has no more than
// 16) and each half-warp takes one of 4 slices of the source pairs, so every staged pair is
// read once per two targets (a broadcast within the half-warp). The slices are added in
// a fixed order. The self pair needs no test: its offset is exactly zero, and with the
// squared distance offset by 1e-36 its terms are exact zeros. Plain FP32 sums: the error
// of the FP32 terms themselves (~1e-6 of the largest) dominates the summation error, so
// compensated sums buy nothing. Writes the near-field sums in sorted order. Positions are
// absolute (float hi + lo), so sources of any level are alike.
// The issue of the pairs bounds it: two sources go through packed arithmetic at once, 17
// instructions with the two reciprocals, where single ones with a division took 30 each.
// A tile takes two warps: with four, the waits of its start and end weighed twice as much.
// Measured (Stokes): the 57.1 M pairs of 524,288 nodes 112 -> 72 us, 95 us with four warps.
#define NEAR_SLAB 256
#define NEAR32_THREADS 64

// 1 / x to an ulp for normal x (the squared distance is at least 1e-36)
__device__ __forceinline__ float rcp32(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

template <int K>
__device__ __forceinline__ void near_pair(const float4 hlj, const float4 c, const float4 hl, float& gx, float& gy) {
  const float dx = (hlj.x - hl.x) + (hlj.z - hl.z);
  const float dy = (hlj.y - hl.y) + (hlj.w - hl.w);
  const float rr = rcp32(fmaf(dx, dx, fmaf(dy, dy, 1e-36f)));
  const float ex = dx * rr, ey = dy * rr;  // conj(1/D), D = z_s - z_t
  if (K == NEAR_Q) {  // c = (q, -, -)
    gx = fmaf(-c.x, ex, fmaf(-c.y, ey, gx));
    gy = fmaf(c.x, ey, fmaf(-c.y, ex, gy));
  } else {  // c = (ax, ay, c0, c1)
    const float v = fmaf(ey, fmaf(c.x, dx, c.y * dy), c.z);
    gx = fmaf(ex, v, gx);
    gy = fmaf(ey, v, gy);
    if (K == NEAR_VC) {
      gx = fmaf(-ey, c.w, gx);
      gy = fmaf(ex, c.w, gy);
    }
  }
}

// A target against the sources of a slab pair by pair: its negated position, and the two
// sources' sums side by side.
struct NearT {
  f32x2 hx, hy, lx, ly, gx, gy;
};
__device__ __forceinline__ NearT near_target(float4 h) {
  return NearT{pk2(-h.x, -h.x), pk2(-h.y, -h.y), pk2(-h.z, -h.z), pk2(-h.w, -h.w), 0, 0};
}

// The pair of near_pair for two sources: H = (x, x', y, y') of the high parts, L of the low
// ones, C = (ax, ax', ay, ay') or (q, q'), D = (c0, c0', c1, c1').
template <int K>
__device__ __forceinline__ void near_pair2(ulonglong2 H, ulonglong2 L, ulonglong2 C, ulonglong2 D, NearT& t) {
  const f32x2 dx = add2(add2(H.x, t.hx), add2(L.x, t.lx));
  const f32x2 dy = add2(add2(H.y, t.hy), add2(L.y, t.ly));
  const float2 dd = upk2(fma2(dx, dx, fma2(dy, dy, pk2(1e-36f, 1e-36f))));
  const f32x2 rr = pk2(rcp32(dd.x), rcp32(dd.y));
  const f32x2 ex = mul2(dx, rr), ey = mul2(dy, rr);
  if (K == NEAR_Q) {
    const f32x2 neg = pk2(-1.f, -1.f), nex = mul2(ex, neg);
    t.gx = fma2(C.x, nex, fma2(mul2(C.y, neg), ey, t.gx));
    t.gy = fma2(C.x, ey, fma2(C.y, nex, t.gy));
  } else {
    const f32x2 v = fma2(ey, fma2(C.x, dx, mul2(C.y, dy)), D.x);
    t.gx = fma2(ex, v, t.gx);
    t.gy = fma2(ey, v, t.gy);
    if (K == NEAR_VC) {
      t.gx = fma2(mul2(ey, pk2(-1.f, -1.f)), D.y, t.gx);
      t.gy = fma2(ex, D.y, t.gy);
    }
  }
}

template <int K>
__global__ void __launch_bounds__(NEAR32_THREADS, 16) k_near32(const int4* __restrict__ tiles, const int* __restrict__ pt0,
                                                   const int* __restrict__ pt1,
                                                   const int* __restrict__ ustart, const int* __restrict__ ulist,
                                                   const float4* __restrict__ zhl,
                                                   const float2* __restrict__ qn, int plus,
                                                   double2* __restrict__ nearbuf) {
  constexpr bool ST = K != NEAR_Q;
  static_assert(EB_NTILE == 32, "two targets per thread over 16 lanes");
  constexpr int NS = NEAR32_THREADS / 16, NP = NEAR_SLAB / 2;
  __shared__ float4 sh[NP], slo[NP], sc[NP];
  __shared__ float4 sd[K == NEAR_VC ? NP : 1];
  __shared__ float2 sd0[K == NEAR_V ? NP : 1];
  __shared__ int spre[33], sj0[32];
  __shared__ float2 sred[NS][EB_NTILE];
  const int4 tl = tiles[blockIdx.x];
  const int leaf = tl.x;
  const int tid = threadIdx.x;
  const int sl = tid >> 4;    // source slice
  const int t0 = tid & 15;    // targets t0 and t0 + 16 of the tile
  const int i0 = tl.y + t0, i1 = i0 + 16;
  const bool two = tl.z - tl.y > 16;
  NearT a0 = near_target(zhl[i0 < tl.z ? i0 : tl.y]), a1 = near_target(zhl[i1 < tl.z ? i1 : tl.y]);
  const int ub = ustart[leaf], ue = ustart[leaf + 1];
  for (int cb = ub; cb < ue; cb += 32) {
    const int nc = min(32, ue - cb);
    if (cb > ub) __syncthreads();  // the previous boxes' slabs are consumed
    if (tid < 32) {
      int c = 0, j0 = 0;
      if (tid < nc) {
        const int sbx = ulist[cb + tid];
        j0 = pt0[sbx];
        c = pt1[sbx] - j0;
      }
      int x = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (tid >= o) x += y;
      }
      sj0[tid] = j0;
      spre[tid + 1] = x;
      if (tid == 0) spre[0] = 0;
    }
    __syncthreads();
    const int total = spre[nc];
    for (int base = 0; base < total; base += NEAR_SLAB) {
      const int ns = min(NEAR_SLAB, total - base), np = (ns + 1) >> 1;
      if (base > 0) __syncthreads();
      for (int s2 = tid; s2 < np; s2 += NEAR32_THREADS) {
        auto find = [&](int gs) {
          int lo = 0, hi = nc;  // the box k with spre[k] <= gs < spre[k + 1]
          while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (spre[mid] <= gs) lo = mid;
            else hi = mid;
          }
          return sj0[lo] + gs - spre[lo];
        };
        const bool odd = s2 + np >= ns;  // no second source: the first with charges of zero
        const int j = find(base + s2), k = odd ? j : find(base + np + s2);
        const float4 zj = zhl[j], zk = zhl[k];
        sh[s2] = make_float4(zj.x, zk.x, zj.y, zk.y);
        slo[s2] = make_float4(zj.z, zk.z, zj.w, zk.w);
        if (ST) {
          const float4 cj = reinterpret_cast<const float4*>(qn)[j];
          float4 ck = reinterpret_cast<const float4*>(qn)[k];
          if (odd) ck = make_float4(0.f, 0.f, 0.f, 0.f);
          sc[s2] = make_float4(cj.x, ck.x, cj.y, ck.y);
          if (K == NEAR_VC) sd[s2] = make_float4(cj.z, ck.z, cj.w, ck.w);
          else sd0[s2] = make_float2(cj.z, ck.z);
        } else {
          const float2 cj = qn[j];
          float2 ck = qn[k];
          if (odd) ck = make_float2(0.f, 0.f);
          sc[s2] = make_float4(cj.x, ck.x, cj.y, ck.y);
        }
      }
      __syncthreads();
      auto run = [&](auto both) {
#pragma unroll 2
        for (int q = sl; q < np; q += NS) {
          const ulonglong2 H = reinterpret_cast<const ulonglong2*>(sh)[q];
          const ulonglong2 L = reinterpret_cast<const ulonglong2*>(slo)[q];
          const ulonglong2 C = reinterpret_cast<const ulonglong2*>(sc)[q];
          ulonglong2 D = make_ulonglong2(0, 0);
          if (K == NEAR_VC) D = reinterpret_cast<const ulonglong2*>(sd)[q];
          if (K == NEAR_V) D.x = reinterpret_cast<const f32x2*>(sd0)[q];
          near_pair2<K>(H, L, C, D, a0);
          if (both.value) near_pair2<K>(H, L, C, D, a1);
        }
      };
      if (two) run(std::true_type());
      else run(std::false_type());
    }
  }
  auto sum2 = [](f32x2 v) {
    const float2 f = upk2(v);
    return f.x + f.y;
  };
  sred[sl][t0] = make_float2(sum2(a0.gx), sum2(a0.gy));
  sred[sl][t0 + 16] = make_float2(sum2(a1.gx), sum2(a1.gy));
  __syncthreads();
  if (tid < EB_NTILE && tl.y + tid < tl.z) {
    float2 v = sred[0][tid];
#pragma unroll
    for (int q = 1; q < NS; ++q) {
      v.x += sred[q][tid].x;
      v.y += sred[q][tid].y;
    }
    if (ST) v = near_turn<float>(v.x, v.y, plus);
    nearbuf[tl.y + tid] = make_double2((double)v.x, (double)v.y);
  }
}

// ---------------------------------------------------------------------------------
// Direct sums for small point sets (at most eb_opts.direct_max points, one problem, free
// space). Every pair by the near-field formula of the leaf kernels, with the FMM's charges
// (sorted order) and its fused post-processing; one block of 128 threads per target, the
// threads over the sources, their partial sums added in a fixed order (direct_block_sum). On a few hundred points the
// FMM's chain of about a dozen dependent launches, each on a handful of SMs, costs far
// more than all N^2 pairs: an FP64 pair is 14 FP64 instructions, so 1,024 points take
// 25 us of the GPU's FP64 rate. The sums are exact up to rounding (no truncation).
// ---------------------------------------------------------------------------------
// The sum of a block's partial sums, in thread 0 (warp butterflies, then the warps in
// order through shared memory).
template <typename T>
__device__ __forceinline__ void direct_block_sum(T& gx, T& gy) {
  __shared__ T sx[4], sy[4];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    gx += __shfl_xor_sync(0xffffffffu, gx, o);
    gy += __shfl_xor_sync(0xffffffffu, gy, o);
  }
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    sx[w] = gx;
    sy[w] = gy;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    gx = sx[0] + sx[1] + sx[2] + sx[3];
    gy = sy[0] + sy[1] + sy[2] + sy[3];
  }
}

// Where the charges come from: the arrays of the charges' kernels, or from the density in place:
// FASMVP's (with the drops' sums za and pk of k_charges_drop, formed by every block), or
// FASMVP_LAP's. A launch costs as much as the charges of a few hundred points formed by
// every block: an apply takes (own launch / in place) 13.8 / 12.7 us at 256 points, 16.4 / 14.4 at
// 384, 20.5 / 22.6 at 512 (FASMVP), 13.8 / 12.2 at 512 and 14.4 / 16.4 at 640 (FASMVP_LAP).
enum { SRC_Q = 0, SRC_STOKES = 1, SRC_LAPLACE = 2 };
constexpr int DIRECT_STOKES = 400, DIRECT_LAPLACE = 512;  // points, at most

template <int K, int SRC>
__global__ void __launch_bounds__(128) k_direct64(int n, const double2* __restrict__ zs,
                                                  const double2* __restrict__ q, const int* __restrict__ perm,
                                                  int plus, double2* __restrict__ out, EbPost post) {
  pdl_wait();
  constexpr bool ST = K == NEAR_V || K == NEAR_VC;
  static_assert(SRC != SRC_STOKES || K == NEAR_V, "FASMVP's charges with its sign");
  const int i = blockIdx.x;  // one block of 128 threads per target, the threads over the sources
  const double2 zi = zs[i];
  double gx = 0.0, gy = 0.0;
  // SRC_STOKES: the sums of dens and of the singular terms over the target's drop [a0, a1),
  // and of the latter over the drop of pinf [b0, b1)
  double v[4] = {0.0, 0.0, 0.0, 0.0};
  int a0 = 0, a1 = 0, b0 = 0, b1 = 0;
  if (SRC == SRC_STOKES) {
    const int d = post.drop_of[i], d0 = post.pinf_drop ? post.pinf_drop[d] : 0;
    a0 = post.start[d];
    a1 = post.start[d + 1];
    b0 = post.start[d0];
    b1 = post.start[d0 + 1];
  }
  for (int j = threadIdx.x; j < n; j += 128) {
    double2 ca, cc = make_double2(0.0, 0.0);
    if (SRC == SRC_Q) {
      ca = ST ? q[2 * j] : q[j];
      if (ST) cc = q[2 * j + 1];
    } else if (SRC == SRC_LAPLACE) {
      ca = cscale<double>(post.dz[j], post.u[j] * post.hpt[j]);
    } else {
      // (near_charge's values for s = -1: with h = 4 hpt / (2 pi), -h dens dz and the real
      // h Re(dens) Im(dz))
      const double2 u = post.dens[j], d = post.dz[j], kw = post.pkw[j];
      const double h = post.hpt[j] * (2.0 / EB_PI);
      const double2 hd = make_double2(h * d.x, h * d.y);
      ca = make_double2(fma(u.y, hd.y, -(u.x * hd.x)), fma(-u.y, hd.x, -(u.x * hd.y)));
      cc.x = u.x * hd.y;
      const double t = fma(u.x, kw.x, -(u.y * kw.y));
      if (j >= a0 && j < a1) {
        v[0] += u.x;
        v[1] += u.y;
        v[2] += t;
      }
      if (j >= b0 && j < b1) v[3] += t;
    }
    if (j != i) near_pair64<K>(zs[j], ca, cc, zi, gx, gy);
  }
  if (SRC == SRC_STOKES) {
    // all six sums through shared memory: 16 threads each, eight values a thread
    __shared__ double part[6][128], tot[6];
    part[0][threadIdx.x] = gx;
    part[1][threadIdx.x] = gy;
#pragma unroll
    for (int c = 0; c < 4; ++c) part[2 + c][threadIdx.x] = v[c];
    __syncthreads();
    if (threadIdx.x < 96) {
      const double* r = part[threadIdx.x >> 4] + (threadIdx.x & 15);
      double s = ((r[0] + r[16]) + (r[32] + r[48])) + ((r[64] + r[80]) + (r[96] + r[112]));
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if ((threadIdx.x & 15) == 0) tot[threadIdx.x >> 4] = s;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      const double h = 2.0 * EB_PI / (double)(a1 - a0);
      eb_post_stokes(post, i, near_turn<double>(tot[0], tot[1], plus), make_double2(h * tot[2], h * tot[3]), tot[4],
                     tot[5]);
    }
    return;
  }
  direct_block_sum<double>(gx, gy);
  if (threadIdx.x == 0) {
    const double2 w = ST ? near_turn<double>(gx, gy, plus) : make_double2(gx, gy);
    eb_post_store(post, perm[i], w, out);
  }
}

// The FP32 operator's direct sums: positions as float hi + lo, the pair of k_near32.
template <int K>
__global__ void __launch_bounds__(128) k_direct32(int n, const float4* __restrict__ zhl,
                                                  const float2* __restrict__ nc, const int* __restrict__ perm,
                                                  int plus, double2* __restrict__ out, EbPost post) {
  pdl_wait();
  constexpr bool ST = K != NEAR_Q;
  const int i = blockIdx.x;
  const float4 hi = zhl[i];
  float gx = 0.f, gy = 0.f;
  for (int j = threadIdx.x; j < n; j += 128) {
    if (j == i) continue;
    const float4 c = ST ? reinterpret_cast<const float4*>(nc)[j] : make_float4(nc[j].x, nc[j].y, 0.f, 0.f);
    near_pair<K>(zhl[j], c, hi, gx, gy);
  }
  direct_block_sum<float>(gx, gy);
  if (threadIdx.x == 0) {
    const float2 v = ST ? near_turn<float>(gx, gy, plus) : make_float2(gx, gy);
    eb_post_store_f32(post, perm[i], v, out);
  }
}

// ---------------------------------------------------------------------------------
// Wall-bounded flow (IFLAG2 = 1 of CADAPDR / CADAPMOD): the images of the sources across
// the wall y = 0, the bottom edge of the root square.
// ---------------------------------------------------------------------------------
// MPREFLECT (cadap2.f:1468-1507) for scaled coefficients with psi relative to the
// centre: a box of centre c, side r and height yh = Im(c) / r = iy + 1/2 has the
// mirrored expansions about conj(c)
//   Mphi'[k] = conj(-Mpsi[k] + (k+1) Mphi[k] + 2 i yh k Mphi[k-1]),
//   Mpsi'[k] = -conj(Mphi[k]) + (k+1) Mphi'[k] - 2 i yh k Mphi'[k-1]
// (the reference's formulas with its absolute psi, psi = psi_c - conj(c) phi', and the
// factor r^(k+1) of each coefficient taken out). One thread per (box, k).
// Mphi'[k] from Mphi[k], Mpsi[k] and Mphi[k-1]:
template <typename T>
__device__ __forceinline__ c_t<T> reflect_phi(c_t<T> phk, c_t<T> psk, c_t<T> phk1, int k, T yh) {
  c_t<T> v = csub<T>(cscale<T>(phk, (T)(k + 1)), psk);
  const T f = (T)2 * yh * (T)k;  // + 2 i yh k Mphi[k-1]
  v.x -= f * phk1.y;
  v.y += f * phk1.x;
  return cconj<T>(v);
}

// Mphi'[k] and Mpsi'[k] from the orders k, k-1 and k-2 (zeros below order 0)
template <typename T>
__device__ __forceinline__ void reflect_pair(c_t<T> phk, c_t<T> psk, c_t<T> phk1, c_t<T> psk1, c_t<T> phk2,
                                             int k, T yh, c_t<T>& a, c_t<T>& b) {
  a = reflect_phi<T>(phk, psk, phk1, k, yh);
  b = csub<T>(cscale<T>(a, (T)(k + 1)), cconj<T>(phk));
  if (k >= 1) {
    const c_t<T> a1 = reflect_phi<T>(phk1, psk1, phk2, k - 1, yh);
    const T f = (T)2 * yh * (T)k;  // - 2 i yh k Mphi'[k-1]
    b.x += f * a1.y;
    b.y -= f * a1.x;
  }
}

template <typename T>
__global__ void k_reflect(int first, int nb, const unsigned long long* __restrict__ bkey, int p,
                          const c_t<T>* __restrict__ mpole, c_t<T>* __restrict__ mimg) {
  const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (idx >= (long long)nb * p) return;
  const int b = first + (int)(idx / p), k = (int)(idx % p);
  const T yh = (T)compact2d(bkey[b] >> 1) + (T)0.5;
  const c_t<T>* m = mpole + (size_t)b * 2 * p;
  const c_t<T> z = cmk<T>(0, 0);
  c_t<T> a, c;
  reflect_pair<T>(m[k], m[p + k], k >= 1 ? m[k - 1] : z, k >= 1 ? m[p + k - 1] : z, k >= 2 ? m[k - 2] : z, k, yh,
                  a, c);
  mimg[(size_t)b * 2 * p + k] = a;
  mimg[(size_t)b * 2 * p + p + k] = c;
}

// The same for double-float multipoles, the mirror formed in FP64
__global__ void k_reflect_df(int first, int nb, const unsigned long long* __restrict__ bkey, int p,
                             const float4* __restrict__ mpole, float4* __restrict__ mimg) {
  const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (idx >= (long long)nb * p) return;
  const int b = first + (int)(idx / p), k = (int)(idx % p);
  const double yh = (double)compact2d(bkey[b] >> 1) + 0.5;
  const float4* m = mpole + (size_t)b * 2 * p;
  auto ld = [&](int i, int lo) {
    if (i < lo) return make_double2(0.0, 0.0);
    const float4 v = m[i];
    return make_double2((double)v.x + (double)v.y, (double)v.z + (double)v.w);
  };
  double2 a, c;
  reflect_pair<double>(ld(k, 0), ld(p + k, 0), ld(k - 1, 0), ld(p + k - 1, p), ld(k - 2, 0), k, yh, a, c);
  mimg[(size_t)b * 2 * p + k] = df4(a);
  mimg[(size_t)b * 2 * p + p + k] = df4(c);
}

// The reflected near field: for every box T of level ld in the first row (on the wall),
// the images of the points of the first-row boxes next to T and of T's own at T's points
// (DONN0DR's IFLAG2 loop with MKNBRRFL, cadapdrop2.f:690-721, and the pair terms of
// SLDREFDR / SLDREF, cadapdrop2.f:857-934 and cadap2.f:1509-1586), in FP64 whatever the
// operator's arithmetic, added to the operator's output. With qc = -conj(z) qa,
//   gamma1 = conj(qa) - conj(qb), gamma2 = 2 i y_j conj(qa), delta1 = -conj(qb),
//   t = 1 / (conj(z_j) - z):  Phi = gamma1 t + gamma2 t^2, and
//   z conj(Phi') + conj(Psi) = (z - z_j) conj(gamma1 t^2 + 2 gamma2 t^3)
//                              + 2 conj(gamma2 t^2) + conj(delta1 t),
// which has no terms of size |z|. One block per box of level ld (blocks off the wall
// return at once); sources staged through shared memory. Added to the near-field sums
// (sorted order).
#define IMG_TILE 128
__global__ void __launch_bounds__(IMG_TILE) k_img_near(int off, int nb, int lev,
                                                       const unsigned long long* __restrict__ bkey,
                                                       const int* __restrict__ pt0, const int* __restrict__ pt1,
                                                       const double2* __restrict__ zs, const int* __restrict__ perm,
                                                       const double2* __restrict__ dens,
                                                       const double2* __restrict__ dz,
                                                       const double* __restrict__ hpt, double s,
                                                       double2* __restrict__ nearbuf) {
  __shared__ double2 sz[IMG_TILE], sg1[IMG_TILE], sg2[IMG_TILE], sd1[IMG_TILE];
  const int b = off + blockIdx.x;
  const unsigned long long key = bkey[b];
  if (compact2d(key >> 1) != 0) return;
  const int ix = (int)compact2d(key), side = 1 << lev;
  int src[3], nsrc = 0;
  for (int dx = -1; dx <= 1; ++dx) {
    const int sx = ix + dx;
    if (sx < 0 || sx >= side) continue;
    const unsigned long long kk = morton_key((unsigned)sx, 0u);
    int lo = 0, hi = nb - 1, f = -1;
    while (lo <= hi) {
      const int mid = (lo + hi) >> 1;
      const unsigned long long v = bkey[off + mid];
      if (v == kk) {
        f = off + mid;
        break;
      }
      if (v < kk) lo = mid + 1;
      else hi = mid - 1;
    }
    if (f >= 0) src[nsrc++] = f;
  }
  const double c2pi = 1.0 / (2.0 * EB_PI);
  for (int tb = pt0[b]; tb < pt1[b]; tb += IMG_TILE) {
    const int i = tb + threadIdx.x;
    const bool act = i < pt1[b];
    const double2 zt = zs[act ? i : pt0[b]];
    double2 acc = make_double2(0.0, 0.0);
    for (int q = 0; q < nsrc; ++q) {
      for (int jb = pt0[src[q]]; jb < pt1[src[q]]; jb += IMG_TILE) {
        const int cnt = min(IMG_TILE, pt1[src[q]] - jb);
        __syncthreads();
        if (threadIdx.x < cnt) {
          const int j = jb + threadIdx.x, o = perm[j];
          const double2 u = dens[o], d = dz[o];
          const double h = hpt[o] * c2pi;
          const double2 w = cmul<double>(u, d);
          const double2 qa = make_double2(w.y * h, -w.x * h);  // u dz h / (2 pi i)
          const double2 v = csub<double>(cmul<double>(u, cconj<double>(d)), cmul<double>(cconj<double>(u), d));
          const double2 qb = make_double2(v.y * h, -v.x * h);
          const double2 zj = zs[j];
          sz[threadIdx.x] = zj;
          sg1[threadIdx.x] = make_double2(qa.x - qb.x, qb.y - qa.y);            // conj(qa) - conj(qb)
          sg2[threadIdx.x] = make_double2(2.0 * zj.y * qa.y, 2.0 * zj.y * qa.x);  // 2 i y conj(qa)
          sd1[threadIdx.x] = make_double2(-qb.x, qb.y);                         // -conj(qb)
        }
        __syncthreads();
        if (act) {
          for (int jj = 0; jj < cnt; ++jj) {
            const double2 zj = sz[jj], g1 = sg1[jj], g2 = sg2[jj], d1 = sd1[jj];
            const double2 ze = make_double2(zj.x - zt.x, -zj.y - zt.y);  // conj(z_j) - z
            const double rd = 1.0 / (ze.x * ze.x + ze.y * ze.y);
            const double2 t1 = make_double2(ze.x * rd, -ze.y * rd);
            const double2 t2 = cmul<double>(t1, t1);
            const double2 dd = make_double2(zt.x - zj.x, zt.y - zj.y);
            const double2 g2t2 = cmul<double>(g2, t2);
            const double2 phi = cadd<double>(cmul<double>(g1, t1), g2t2);
            const double2 dphi = cadd<double>(cmul<double>(g1, t2), cscale<double>(cmul<double>(g2t2, t1), 2.0));
            const double2 r = cadd<double>(cmul<double>(dd, cconj<double>(dphi)),
                                           cadd<double>(cscale<double>(cconj<double>(g2t2), 2.0),
                                                        cconj<double>(cmul<double>(d1, t1))));
            acc.x += phi.x + s * r.x;
            acc.y += phi.y + s * r.y;
          }
        }
      }
    }
    if (act) nearbuf[i] = make_double2(nearbuf[i].x + acc.x, nearbuf[i].y + acc.y);
  }
}

inline int nblk(long long n, int bs) { return (int)((n + bs - 1) / bs); }
inline int round32(int n) { return (n + 31) & ~31; }
template <typename T>
int tables_build(EbTables& tb, int p, double tol) {
  tb.p = p;
  std::vector<char> blob;
  std::vector<std::pair<EbTab*, size_t>> at;
  auto put = [&](EbTab& tab, const auto& v) {
    const size_t o = (blob.size() + 255) & ~(size_t)255, nb = sizeof(v[0]) * v.size();
    blob.resize(o + nb);
    memcpy(blob.data() + o, v.data(), nb);
    at.emplace_back(&tab, o);
  };
  const int ldb = 2 * p + 2, ld = p + 2;
  std::vector<T> binom((size_t)ldb * ldb, (T)0);
  std::vector<double> bd((size_t)ldb * ldb, 0.0);
  for (int i = 0; i < ldb; ++i) {
    bd[(size_t)i * ldb] = 1.0;
    for (int j = 1; j <= i; ++j) bd[(size_t)i * ldb + j] = bd[(size_t)(i - 1) * ldb + j - 1] + (j <= i - 1 ? bd[(size_t)(i - 1) * ldb + j] : 0.0);
  }
  for (size_t i = 0; i < bd.size(); ++i) binom[i] = (T)bd[i];
  std::vector<c_t<T>> dinv((size_t)EB_NCODE * ld), epow2((size_t)4 * ld), einv((size_t)4 * ld);
  std::vector<int> pd(EB_NCODE, 0);
  const double rad = std::sqrt(0.5);
  for (int code = 0; code < EB_NCODE; ++code) {
    int dx = code % 7 - 3, dy = code / 7 - 3;
    bool valid = std::abs(dx) >= 2 || std::abs(dy) >= 2;
    double re = 1.0, im = 0.0;  // d^-j
    double dn = (double)dx * dx + (double)dy * dy;
    double ivr = valid ? dx / dn : 0.0, ivi = valid ? -dy / dn : 0.0;
    for (int j = 0; j < ld; ++j) {
      dinv[(size_t)code * ld + j] = cmk<T>((T)(valid ? re : 0.0), (T)(valid ? im : 0.0));
      double nr = re * ivr - im * ivi, ni = re * ivi + im * ivr;
      re = nr;
      im = ni;
    }
    if (valid) {
      double rho = rad / (std::sqrt(dn) - rad);
      int need = (int)std::ceil(std::log(tol) / std::log(rho));
      pd[code] = std::max(2, std::min(p, need));
    }
  }
  for (int q = 0; q < 4; ++q) {
    double er = (q & 1) - 0.5, ei = ((q >> 1) & 1) - 0.5;
    double pr = 1.0, pi = 0.0, vr = 1.0, vi = 0.0;
    double hr = 0.5 * er, hi = 0.5 * ei;
    double en = er * er + ei * ei, ir = er / en, ii = -ei / en;
    for (int j = 0; j < ld; ++j) {
      epow2[(size_t)q * ld + j] = cmk<T>((T)pr, (T)pi);
      einv[(size_t)q * ld + j] = cmk<T>((T)vr, (T)vi);
      double nr = pr * hr - pi * hi, ni = pr * hi + pi * hr;
      pr = nr; pi = ni;
      nr = vr * ir - vi * ii; ni = vr * ii + vi * ir;
      vr = nr; vi = ni;
    }
  }
  put(tb.binom, binom);
  put(tb.dinv, dinv);
  put(tb.pd, pd);
  put(tb.epow, epow2);
  put(tb.einv, einv);
  if (sizeof(T) == 4) {  // M2L's binomials with the output order innermost
    std::vector<T> bt((size_t)p * (p + 1));
    for (int k = 0; k < p; ++k)
      for (int m = 0; m <= p; ++m) bt[(size_t)k * (p + 1) + m] = binom[(size_t)(m + k) * ldb + m];
    put(tb.binom_t, bt);
  }
  if (sizeof(T) == 8) {
    auto split = [](double v, float& h, float& l) {
      h = (float)v;
      l = (float)(v - (double)h);
    };
    std::vector<float2> bdf(bd.size());
    for (size_t i = 0; i < bd.size(); ++i) split(bd[i], bdf[i].x, bdf[i].y);
    auto to_df = [&](const std::vector<c_t<T>>& v) {
      std::vector<float4> o(v.size());
      for (size_t i = 0; i < v.size(); ++i) {
        split((double)v[i].x, o[i].x, o[i].y);
        split((double)v[i].y, o[i].z, o[i].w);
      }
      return o;
    };
    std::vector<float4> ddf = to_df(dinv), edf = to_df(epow2), idf = to_df(einv);
    put(tb.binom_df, bdf);
    put(tb.dinv_df, ddf);
    put(tb.epow_df, edf);
    put(tb.einv_df, idf);
  }
  EB_TRY(tb.all.ensure(blob.size()));
  EB_CUDA_TRY(cudaMemcpy(tb.all.p, blob.data(), blob.size(), cudaMemcpyHostToDevice));
  for (auto& a : at) a.first->p = static_cast<const char*>(tb.all.p) + a.second;
  return EB_OK;
}

struct ProfScope {
  eb_ctx* ctx;
  int cls;
  cudaStream_t st;
  cudaEvent_t e0, e1;
  ProfScope(eb_ctx* c, int k, cudaStream_t s) : ctx(c), cls(k), st(s) {
    e0 = k == 2 ? ctx->ev_near0 : ctx->ev0;
    e1 = k == 2 ? ctx->ev_near1 : ctx->ev1;
    if (ctx->profiling) cudaEventRecord(e0, st);
  }
  void done() {
    if (!ctx->profiling) return;
    cudaEventRecord(e1, st);
    cudaEventSynchronize(e1);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    ctx->prof_launch[cls]++;
    ctx->prof_ms[cls] += ms;
  }
};

// Blocks per box of the FP64 M2M / L2L of a level of nb boxes.
int level_split(const eb_ctx* ctx, int nb) { return nb <= ctx->nsm ? 4 : nb <= 3 * ctx->nsm ? 2 : 1; }

// M2M into the boxes of level l, L2L out of them.
template <int E>
int launch_m2m64(eb_ctx* ctx, EbTree& t, EbTables& tb, int l, double2* mpole, cudaStream_t st) {
  const int p = tb.p, nb = t.lev_off[l + 1] - t.lev_off[l], ns = level_split(ctx, nb);
  const int groups = ((E * p + 7) / 8 + ns - 1) / ns;
  EB_CUDA_TRY(eb_launch_next(k_m2m64<E>, dim3(nb * ns), dim3(32 * groups), sizeof(double2) * 4 * E * p, st, t.lev_off[l], ns, t.bkey.as<unsigned long long>(), t.child0.as<int>(), t.nchild.as<int>(), p,
      tb.binom.as<double>(), 2 * p + 2, tb.epow.as<double2>(), tb.einv.as<double2>(), mpole));
  return EB_OK;
}
template <int E>
int launch_l2l64(eb_ctx* ctx, EbTree& t, EbTables& tb, int l, double2* local, cudaStream_t st) {
  const int p = tb.p, nb = t.lev_off[l + 1] - t.lev_off[l], ns = level_split(ctx, nb);
  // the widest range of orders is the last one
  const int ldl = p + 1, nj = ldl - (ns == 1 ? 0 : (int)(ldl * (1.f - std::sqrt(1.f / ns)))) + 1;
  EB_CUDA_TRY(eb_launch_next(k_l2l64<E>, dim3(nb * ns), dim3(round32(4 * (E * nj + E - 1))), sizeof(double2) * (E + 4) * (p + 1), st, t.lev_off[l], ns, t.bkey.as<unsigned long long>(), t.child0.as<int>(), t.nchild.as<int>(), p,
      tb.binom.as<double>(), 2 * p + 2, tb.epow.as<double2>(), tb.einv.as<double2>(), local));
  return EB_OK;
}

// Boxes and order from which the double-float pipeline takes the fixed-point M2L (the boxes'
// figures, at the default order, in eb_m2l_fx.cu). Its time hardly depends on the order, that of
// k_m2l_df goes with its square: an apply takes (k_m2l_df / fixed) at orders 12, 30, 36 and 44
// 115 / 171, 168 / 196, 203 / 204 and 224 / 214 us for 64 x 512 nodes, 2.14 / 2.91, 3.35 / 3.51, 4.20 /
// 3.75 and 4.87 / 4.13 ms for 1,024 x 1,024 (E = 2); 1.70 / 2.00, 2.22 / 2.27, 2.85 / 2.48 and 3.22 / 2.64
// ms for the latter with E = 1.
template <int E>
constexpr int FX_DF = E == 2 ? 0 : 3072;
constexpr int FX_DF_P = 36;

// Boxes of the levels 2, 3, .. of at most 384 boxes: their V lists are the long ones.
int coarse_boxes(const EbTree& t) {
  int l = 2;
  while (l <= t.L && t.lev_off[l + 1] - t.lev_off[l] <= 384) ++l;
  return t.lev_off[l] - t.lev_off[2];
}

// Upward pass, M2L and downward pass, shared by both kernels. Leaves the local
// expansions of every box in w.local.
// Expansions of the double-float pipeline (FP64-class accuracy on the FP32 pipes):
// P2M, M2M per level, M2L, L2L per level; multipoles and locals stay double-float.
template <int E>
int fmm_expansions_df(eb_ctx* ctx, EbTree& t, EbTables& tb, EbFmmWork& w) {
  cudaStream_t st = eb_stream(ctx);
  const int p = tb.p, L = t.L;
  const int ldb = 2 * p + 2;
  EB_TRY(w.mpole_df.ensure(sizeof(float4) * (size_t)t.nbox * E * p));
  EB_TRY(w.local_df.ensure(sizeof(float4) * (size_t)t.nbox * E * (p + 1)));
  float4* mp = w.mpole_df.as<float4>();
  float4* lo = w.local_df.as<float4>();
  {
    size_t sm = sizeof(float4) * (32 * (size_t)(p + 1) + 96);
    if (sm > 48 * 1024) EB_CUDA_TRY(cudaFuncSetAttribute(k_p2m_df<E>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    EB_CUDA_TRY(eb_launch_next(k_p2m_df<E>, dim3(t.nleaf), dim3(std::max(128, round32((E == 2 ? 3 : 1) * p))), sm, st, t.leaves.as<int>(), t.pt0.as<int>(), t.pt1.as<int>(), t.wdf.as<float4>(),
                                          E == 2 ? w.qdf.as<float4>() : w.ncdf.as<float4>(), p, mp));
    eb_count_launch(ctx);
  }
  for (int l = L - 1; l >= 2; --l) {
    int nb = t.lev_off[l + 1] - t.lev_off[l];
    EB_CUDA_TRY(eb_launch_next(k_m2m_df<E>, dim3(nb), dim3(round32(4 * E * p)), sizeof(float4) * 4 * E * p, st, t.lev_off[l], t.bkey.as<unsigned long long>(), t.child0.as<int>(), t.nchild.as<int>(), p,
        tb.binom_df.as<float2>(), ldb, tb.epow_df.as<float4>(), tb.einv_df.as<float4>(), mp));
    eb_count_launch(ctx);
  }
  {
    int first = t.lev_off[2], nt = t.nbox - first;
    size_t sm = sizeof(float4) * ((size_t)(p * (p + 1) + 1) / 2 + 4 * E * (size_t)(2 * p + 1));
    if (sm > 48 * 1024)
      EB_CUDA_TRY(cudaFuncSetAttribute(k_m2l_df<E>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    ProfScope ps(ctx, 1, st);
    const bool fixed = p >= FX_DF_P && p <= EB_FX_MAXP && nt >= FX_DF<E>;
    const int ncoarse = coarse_boxes(t);
    if (nt > 0 && fixed) {
      EB_TRY(eb_m2l_fx(ctx, E, true, first, nt, nt, ncoarse, t.vlist.as<int>(), t.vcode.as<unsigned char>(), t.vcount.as<int>(),
                       tb, w, mp, lo, 0, st));
    } else if (nt > 0) {
      k_m2l_df<E><<<nt, 128, sm, st>>>(first, t.vlist.as<int>(), t.vcode.as<unsigned char>(), t.vcount.as<int>(),
                                       p, tb.binom_df.as<float2>(), ldb, tb.dinv_df.as<float4>(), tb.pd.as<int>(),
                                       mp, lo, 0);
      eb_count_launch(ctx);
    }
    if (E == 2 && t.wall && t.ld >= 2) {  // the wall's reflected boxes
      const int nimg = t.lev_off[t.ld + 1], nbi = nimg - first;
      EB_TRY(w.mimg.ensure(sizeof(float4) * (size_t)nimg * E * p));
      k_reflect_df<<<nblk((long long)nbi * p, 128), 128, 0, st>>>(first, nbi, t.bkey.as<unsigned long long>(), p,
                                                                 mp, w.mimg.as<float4>());
      eb_count_launch(ctx);
      if (fixed) {
        EB_TRY(eb_m2l_fx(ctx, E, true, first, nbi, nbi, ncoarse, t.ilist.as<int>(), t.icode.as<unsigned char>(),
                         t.icount.as<int>(), tb, w, w.mimg.p, lo, 1, st));
      } else {
        k_m2l_df<E><<<nbi, 128, sm, st>>>(first, t.ilist.as<int>(), t.icode.as<unsigned char>(), t.icount.as<int>(),
                                          p, tb.binom_df.as<float2>(), ldb, tb.dinv_df.as<float4>(), tb.pd.as<int>(),
                                          w.mimg.as<float4>(), lo, 1);
        eb_count_launch(ctx);
      }
    }
    ps.done();
  }
  for (int l = 2; l < L; ++l) {
    const int nb = t.lev_off[l + 1] - t.lev_off[l];
    EB_CUDA_TRY(eb_launch_next(k_l2l_df<E>, dim3(nb), dim3(round32(4 * E * (p + 1))),
                               sizeof(float4) * (E + (E == 2 ? 4 : 0)) * (p + 1), st, t.lev_off[l],
                               t.bkey.as<unsigned long long>(), t.child0.as<int>(), t.nchild.as<int>(), p,
                               tb.binom_df.as<float2>(), ldb, tb.epow_df.as<float4>(), tb.einv_df.as<float4>(), lo));
    eb_count_launch(ctx);
  }
  return EB_OK;
}

// breal: the charges b are real (see the charges).
template <typename T, int E>
int fmm_expansions(eb_ctx* ctx, EbTree& t, EbTables& tb, EbFmmWork& w, bool breal,
                   const std::function<int()>& after_p2m) {
  cudaStream_t st = eb_stream(ctx);
  const int p = tb.p, L = t.L;
  const int ldb = 2 * p + 2;
  EB_TRY(w.mpole.ensure(sizeof(c_t<T>) * (size_t)t.nbox * E * p));
  EB_TRY(w.local.ensure(sizeof(c_t<T>) * (size_t)t.nbox * E * (p + 1)));
  // Upward pass. FP32: direct P2M (in chunks) for every box of the EB_DIRECT_LEVELS
  // finest levels in one launch, then M2M per coarser level. FP64: P2M and one M2M
  // launch per level.
  if (sizeof(T) == 4) {
    const int lmin = t.chunk_lmin;
    const int first2 = t.lev_off[2], nout = E * p;
    EB_TRY(w.mpart.ensure(sizeof(float2) * (size_t)t.nchunk * nout));
    LevOff lo;
    for (int l = 0; l < EB_KEY_LEVELS + 2; ++l) {
      lo.v[l] = t.lev_off[l];
      lo.rinv[l] = (float)((double)(1u << std::min(l, 30)) / t.W);
    }
    auto p2m = [&](auto kern, size_t sm, auto... order) {
      return eb_launch_next(
          kern, dim3(nblk(t.nchunk, P2M_CW)), dim3(32 * P2M_CW), sm, st, lo, t.nchunk, first2, t.blev.as<unsigned char>(), t.plev.as<unsigned char>(), t.chunk_box.as<int>(),
          t.cstart.as<int>(), t.keys.as<unsigned long long>(), t.pt0.as<int>(), t.pt1.as<int>(), t.wdf.as<float4>(),
          reinterpret_cast<const float2*>(w.qa.p), reinterpret_cast<const float2*>(w.qb.p), order...,
          w.mpart.as<float2>(), t.cdone.as<int>(), reinterpret_cast<float2*>(w.mpole.p));
    };
    if (p == 20) EB_CUDA_TRY(p2m(k_p2m_points<E, 20>, 0));
    else EB_CUDA_TRY(p2m(k_p2m_chunks<E>, p2m_smem(p), p));
    eb_count_launch(ctx);
    for (int l = lmin - 1; l >= 2; --l) {
      int nb = t.lev_off[l + 1] - t.lev_off[l];
      size_t sm2 = sizeof(float2) * 4 * (size_t)nout;
      EB_CUDA_TRY(eb_launch_next(k_m2m_f32<E>, dim3(nb), dim3(std::max(128, round32(nout))), sm2, st, t.lev_off[l], t.bkey.as<unsigned long long>(), t.child0.as<int>(), t.nchild.as<int>(), p,
          reinterpret_cast<const float*>(tb.binom.p), ldb, reinterpret_cast<const float2*>(tb.epow.p),
          reinterpret_cast<const float2*>(tb.einv.p), reinterpret_cast<float2*>(w.mpole.p)));
      eb_count_launch(ctx);
    }
  } else {
    const size_t sm = sizeof(double2) * std::max(32 * (size_t)(p + 1) + 96, (size_t)(E == 2 ? 3 : 1) * P2M_NG * p);
    auto go = [&](auto kern) -> int {
      if (sm > 48 * 1024)
        EB_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
      EB_CUDA_TRY(eb_launch_next(kern, dim3(t.nleaf), dim3(round32(P2M_NG * p)), sm, st, t.leaves.as<int>(), t.bkey.as<unsigned long long>(),
                                                     t.blev.as<unsigned char>(), t.pt0.as<int>(), t.pt1.as<int>(),
                                                     t.zs.as<double2>(), w.qa.as<double2>(), w.qb.as<double2>(), t.x0,
                                                     t.y0, t.W, 1.0 / t.W, p, w.mpole.as<double2>()));
      return EB_OK;
    };
    if (E == 2 && breal) EB_TRY(go(k_p2m64<E, true>));
    else EB_TRY(go(k_p2m64<E, false>));
    eb_count_launch(ctx);
    if (after_p2m) EB_TRY(after_p2m());
    for (int l = L - 1; l >= 2; --l) {
      EB_TRY(launch_m2m64<E>(ctx, t, tb, l, w.mpole.as<double2>(), st));
      eb_count_launch(ctx);
    }
  }
  {
    int first = t.lev_off[2], nt = t.nbox - first;
    size_t c2 = (sizeof(T) * (size_t)p * (p + 1) + 15) & ~(size_t)15;
    size_t sm = c2 + sizeof(c_t<T>) * 4 * E * (size_t)(2 * p + 1);
    if (sm > 48 * 1024)
      EB_CUDA_TRY(cudaFuncSetAttribute(k_m2l<T, E>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    ProfScope ps(ctx, 1, st);
    const bool fixed = sizeof(T) == 8 && p <= EB_FX_MAXP;
    const int ncoarse = coarse_boxes(t);
    auto m2l32 = [&](int n, DevBuf& list, DevBuf& code, DevBuf& count, DevBuf& mp, int accumulate) -> int {
      const float2* dinv = reinterpret_cast<const float2*>(tb.dinv.p);
      const float2* m = reinterpret_cast<const float2*>(mp.p);
      float2* out = reinterpret_cast<float2*>(w.local.p);
      if (n < M2L32_WIDE) {
        EB_CUDA_TRY(eb_launch_next(k_m2l_f32w<E, 20>, dim3(std::min(n, M2L32_CTAS * ctx->nsm)), dim3(128), 0, st, first, n, list.as<int>(), code.as<unsigned char>(), count.as<int>(), tb.binom_t.as<float>(), dinv,
            tb.pd.as<int>(), m, out, accumulate));
        return EB_OK;
      }
      // boxes per warp: 6 have the 32 entries of a round on average, 16 in several rounds
      // leave fewer lanes without one where there are warps enough (256 x 512: 125.0 against
      // 143.0 us an apply; 1,024 x 1,024: 745 against 722 us)
      const int nc = std::min(ncoarse, n), nb = n >= 256 * ctx->nsm ? 16 : 6;
      constexpr size_t sm = sizeof(M2l32Smem<E, 20>);
      EB_CUDA_TRY(cudaFuncSetAttribute(k_m2l_f32p<E, 20>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
      EB_CUDA_TRY(eb_launch_next(k_m2l_f32p<E, 20>, dim3(nblk(nc + nblk(n - nc, nb), M2L32_WARPS)), dim3(32 * M2L32_WARPS), sm, st, first, n, nc, nb, list.as<int>(), code.as<unsigned char>(), count.as<int>(), dinv, tb.pd.as<int>(), m, out,
          accumulate));
      return EB_OK;
    };
    if (nt > 0 && sizeof(T) == 4 && p == 20 && ctx->opts.m2l_tc > 0) {
      EB_TRY(eb_m2l_tc(ctx, E, first, nt, t.vlist.as<int>(), t.vcode.as<unsigned char>(), t.vcount.as<int>(),
                       reinterpret_cast<const float*>(tb.binom.p), ldb, reinterpret_cast<const float2*>(tb.dinv.p),
                       tb.pd.as<int>(), reinterpret_cast<const float2*>(w.mpole.p),
                       reinterpret_cast<float2*>(w.local.p), st));
    } else if (nt > 0 && sizeof(T) == 4 && p == 20) {
      EB_TRY(m2l32(nt, t.vlist, t.vcode, t.vcount, w.mpole, 0));
      eb_count_launch(ctx);
    } else if (nt > 0 && fixed) {
      EB_TRY(eb_m2l_fx(ctx, E, false, first, nt, nt, ncoarse, t.vlist.as<int>(), t.vcode.as<unsigned char>(),
                       t.vcount.as<int>(), tb, w, w.mpole.p, w.local.p, 0, st));
    } else if (nt > 0) {
      k_m2l<T, E><<<nt, 128, sm, st>>>(first, t.vlist.as<int>(), t.vcode.as<unsigned char>(),
                                       t.vcount.as<int>(), p, tb.binom.as<T>(), ldb,
                                       tb.dinv.as<c_t<T>>(), tb.pd.as<int>(), w.mpole.as<c_t<T>>(),
                                       w.local.as<c_t<T>>(), 0);
      eb_count_launch(ctx);
    }
    if (E == 2 && t.wall && t.ld >= 2) {  // the wall's reflected boxes
      const int nimg = t.lev_off[t.ld + 1], nbi = nimg - first;
      EB_TRY(w.mimg.ensure(sizeof(c_t<T>) * (size_t)nimg * E * p));
      k_reflect<T><<<nblk((long long)nbi * p, 128), 128, 0, st>>>(first, nbi, t.bkey.as<unsigned long long>(), p,
                                                                 w.mpole.as<c_t<T>>(), w.mimg.as<c_t<T>>());
      if (sizeof(T) == 4 && p == 20)
        EB_TRY(m2l32(nbi, t.ilist, t.icode, t.icount, w.mimg, 1));
      else if (fixed)
        EB_TRY(eb_m2l_fx(ctx, E, false, first, nbi, nbi, ncoarse, t.ilist.as<int>(), t.icode.as<unsigned char>(),
                         t.icount.as<int>(), tb, w, w.mimg.p, w.local.p, 1, st));
      else
        k_m2l<T, E><<<nbi, 128, sm, st>>>(first, t.ilist.as<int>(), t.icode.as<unsigned char>(), t.icount.as<int>(),
                                          p, tb.binom.as<T>(), ldb, tb.dinv.as<c_t<T>>(), tb.pd.as<int>(),
                                          w.mimg.as<c_t<T>>(), w.local.as<c_t<T>>(), 1);
      ctx->launches += fixed ? 1 : 2;
    }
    ps.done();
  }
  // Downward pass. FP64: L2L level by level. FP32: L2L only into the level lend, the
  // coarsest of the EB_FAR_LEVELS finest levels; the far-field kernel evaluates the M2L
  // expansions of the levels below it directly (cheap FP32 work instead of a dependent
  // chain of shifts).
  {
    const int lend = sizeof(T) == 8 ? L : t.lend;
    for (int l = 3; l <= lend; ++l) {
      int nb = t.lev_off[l + 1] - t.lev_off[l];
      if (sizeof(T) == 8)
        EB_TRY(launch_l2l64<E>(ctx, t, tb, l - 1, w.local.as<double2>(), st));
      else
        EB_CUDA_TRY(eb_launch_next(k_l2l<float, E>, dim3(nb), dim3(round32(E * (p + 1))), sizeof(float2) * E * (p + 1), st, t.lev_off[l], t.bkey.as<unsigned long long>(), t.parent.as<int>(), p, tb.binom.as<float>(), ldb,
            tb.epow.as<float2>(), tb.einv.as<float2>(), w.local.as<float2>()));
      eb_count_launch(ctx);
    }
  }
  return EB_OK;
}

// What the near-field pair needs (see the charges): FASMVP's charges with its sign have
// c1 = 0, and FASMVP_LAP's post-processing (kind 2) reads the imaginary part only.
template <int E>
int near_kind(int sign, const double2* dz, const EbPost& post) {
  if (E == 1) return post.kind == 2 ? NEAR_QI : NEAR_Q;
  return dz && sign < 0 ? NEAR_V : NEAR_VC;
}

// The direct path of a small problem: the FMM's charges, k_direct64 / k_direct32, and
// the post-processing. FP64-class requests (native or double-float) run in native FP64.
template <int E>
int direct_run(eb_ctx* ctx, EbTree& t, bool f32, int sign, const double2* dens, const double2* dz,
               const double* hpt, const double2* q_in, double2* out, const EbPost* postp, cudaEvent_t join) {
  EbPost post{};
  if (postp) post = *postp;
  cudaStream_t st = eb_stream(ctx);
  const int n = t.n;
  EbFmmWork& w = f32 ? ctx->work32 : ctx->work64;
  const size_t cs = f32 ? sizeof(float2) : sizeof(double2);
  EB_TRY(w.qa.ensure(cs * (size_t)n));
  if (E == 2) {
    EB_TRY(w.qb.ensure(cs * (size_t)n));
    EB_TRY(w.nc.ensure(cs * 2 * (size_t)n));
  }
  const int g = n;  // one block of 128 threads per target
  const int kind = near_kind<E>(sign, dz, post);
  const bool plus = sign > 0;
  // right behind the charges, unless another stream's sums have to be waited for too
  cudaError_t ce = cudaSuccess;
  auto go = [&](auto kern, auto... a) {
    if (join) kern<<<g, 128, 0, st>>>(a...);
    else ce = eb_launch_next(kern, dim3(g), dim3(128), 0, st, a...);
  };
  if (f32) {
    const float4* zh = t.zhl.as<float4>();
    const float2* q = E == 2 ? w.nc.as<float2>() : w.qa.as<float2>();
    if (E == 2 && post.start)
      k_charges_drop<float><<<post.k, 256, 0, st>>>(post.start, dens, dz, hpt, post.pkw, (double)sign,
                                                    w.nc.as<float2>(), const_cast<double2*>(post.za),
                                                    const_cast<double*>(post.pk));
    else if (E == 2)
      k_charges_stokes<float><<<nblk(n, 256), 256, 0, st>>>(n, t.perm.as<int>(), dens, dz, hpt, (double)sign,
                                                            w.qa.as<float2>(), w.qb.as<float2>(),
                                                            w.nc.as<float2>(), nullptr);
    else
      k_charges_cauchy<float><<<nblk(n, 256), 256, 0, st>>>(n, t.perm.as<int>(), q_in, post.u, post.dz, post.hpt,
                                                            w.qa.as<float2>(), nullptr);
    if (join) EB_CUDA_TRY(cudaStreamWaitEvent(st, join, 0));
    if (E == 1) go(k_direct32<NEAR_Q>, n, zh, q, t.perm.as<int>(), 0, out, post);
    else if (kind == NEAR_V) go(k_direct32<NEAR_V>, n, zh, q, t.perm.as<int>(), plus, out, post);
    else go(k_direct32<NEAR_VC>, n, zh, q, t.perm.as<int>(), plus, out, post);
  } else {
    const double2* zz = t.zs.as<double2>();
    const double2* q = E == 2 ? w.nc.as<double2>() : w.qa.as<double2>();
    // in place, unless a result overwrites what another block still reads (y = x)
    auto apart = [n](const void* a, size_t abytes, const void* b, size_t bbytes) {
      const uintptr_t x = reinterpret_cast<uintptr_t>(a), y = reinterpret_cast<uintptr_t>(b);
      return x + (size_t)n * abytes <= y || y + (size_t)n * bbytes <= x;
    };
    const void* res = post.kind == 0 ? static_cast<const void*>(out) : post.y;
    const bool own = E == 2 ? post.start && n <= DIRECT_STOKES && apart(dens, 16, res, 16)
                            : (q_in ? apart(q_in, 16, res, post.kind == 2 ? 8 : 16)
                                    : n <= DIRECT_LAPLACE && apart(post.u, 8, res, post.kind == 2 ? 8 : 16));
    if (own) {
      // no charges' kernel (the points of a direct tree are in their given order)
      if (q_in) q = q_in;
      if (E == 2) {
        post.dz = dz;
        post.hpt = hpt;
      }
      ctx->launches -= 1;
    } else if (E == 2 && post.start) {
      k_charges_drop<double><<<post.k, 256, 0, st>>>(post.start, dens, dz, hpt, post.pkw, (double)sign,
                                                     w.nc.as<double2>(), const_cast<double2*>(post.za),
                                                     const_cast<double*>(post.pk));
    } else if (E == 2) {
      k_charges_stokes<double><<<nblk(n, 256), 256, 0, st>>>(n, t.perm.as<int>(), dens, dz, hpt, (double)sign,
                                                             w.qa.as<double2>(), w.qb.as<double2>(),
                                                             w.nc.as<double2>(), nullptr);
    } else {
      k_charges_cauchy<double><<<nblk(n, 256), 256, 0, st>>>(n, t.perm.as<int>(), q_in, post.u, post.dz, post.hpt,
                                                             w.qa.as<double2>(), nullptr);
    }
    if (join) EB_CUDA_TRY(cudaStreamWaitEvent(st, join, 0));
    auto run = [&](auto kern) {
      if (own || join) kern<<<g, 128, 0, st>>>(n, zz, q, t.perm.as<int>(), plus, out, post);
      else ce = eb_launch_next(kern, dim3(g), dim3(128), 0, st, n, zz, q, t.perm.as<int>(), (int)plus, out, post);
    };
    if (E == 2) {
      if (own) run(k_direct64<NEAR_V, SRC_STOKES>);
      else if (kind == NEAR_V) run(k_direct64<NEAR_V, SRC_Q>);
      else run(k_direct64<NEAR_VC, SRC_Q>);
    } else {
      const bool lap = own && !q_in;
      if (kind == NEAR_QI) lap ? run(k_direct64<NEAR_QI, SRC_LAPLACE>) : run(k_direct64<NEAR_QI, SRC_Q>);
      else lap ? run(k_direct64<NEAR_Q, SRC_LAPLACE>) : run(k_direct64<NEAR_Q, SRC_Q>);
    }
  }
  EB_CUDA_TRY(ce);
  ctx->launches += 2;
  return eb_check_launch(ctx, "direct sum");
}

template <typename T, int E>
int fmm_run(eb_ctx* ctx, EbTree& t, int sign, const double2* dens, const double2* dz,
            const double* hpt, const double2* q, double2* out, const EbPost* postp,
            cudaEvent_t join, bool df_req) {
  // a direct tree (eb_tree_build: at most eb_opts.direct_max points, one problem -- a
  // batch's forest keeps its simulations apart through the tree -- and no wall)
  if (t.direct) return direct_run<E>(ctx, t, sizeof(T) == 4, sign, dens, dz, hpt, q, out, postp, join);
  EbPost post{};
  if (postp) post = *postp;
  cudaStream_t st = eb_stream(ctx);
  const bool f64 = sizeof(T) == 8;
  EbTables& tb = f64 ? ctx->tab64 : ctx->tab32;
  EbFmmWork& w = f64 ? ctx->work64 : ctx->work32;
  const int n = t.n;
  const bool df = f64 && df_req;
  if (df) {
    EB_TRY(w.ncdf.ensure(sizeof(float4) * E * (size_t)n));
    if (E == 2) EB_TRY(w.qdf.ensure(sizeof(float4) * 2 * (size_t)n));
  } else {
    EB_TRY(w.qa.ensure(sizeof(c_t<T>) * (size_t)n));
    if (E == 2) {
      EB_TRY(w.qb.ensure(sizeof(c_t<T>) * (size_t)n));
      EB_TRY(w.nc.ensure(sizeof(c_t<T>) * 2 * (size_t)n));
    }
  }
  int* next = nullptr;
  if (f64 && !df) {
    EB_TRY(w.next.ensure(sizeof(int)));
    next = w.next.as<int>();
  }
  if (df && E == 2) {
    k_charges_stokes_df<<<nblk(n, 256), 256, 0, st>>>(n, t.perm.as<int>(), dens, dz, hpt, (double)sign,
                                                      1.0 / t.W, t.plev.as<unsigned char>(), w.qdf.as<float4>(),
                                                      w.ncdf.as<float4>());
  } else if (df) {
    k_charges_cauchy_df<<<nblk(n, 256), 256, 0, st>>>(n, t.perm.as<int>(), q, post.u, post.dz, post.hpt,
                                                      1.0 / t.W, t.plev.as<unsigned char>(), w.ncdf.as<float4>());
  } else if (E == 2) {
    k_charges_stokes<T><<<nblk(n, 256), 256, 0, st>>>(n, t.perm.as<int>(), dens, dz, hpt, (double)sign,
                                                      w.qa.as<c_t<T>>(), w.qb.as<c_t<T>>(), w.nc.as<c_t<T>>(),
                                                      next);
  } else {
    k_charges_cauchy<T><<<nblk(n, 256), 256, 0, st>>>(n, t.perm.as<int>(), q, post.u, post.dz, post.hpt,
                                                      w.qa.as<c_t<T>>(), next);
  }
  eb_count_launch(ctx);
  const int has_far = t.L >= 2;
  int blocks = nblk((long long)t.ngroup * 32, 128);
  const int kind = near_kind<E>(sign, dz, post);
  const int plus = sign > 0;
  EB_TRY(w.nearbuf.ensure(sizeof(double2) * (size_t)n));
  double2* nb = w.nearbuf.as<double2>();
  auto near = [&](cudaStream_t ns) {
    if (df) {
      auto go = [&](auto kern) {
        kern<<<blocks, 128, 0, ns>>>(t.ngroup, t.gleaf.as<int>(), t.gfirst.as<int>(), t.leaves.as<int>(),
                                     t.bkey.as<unsigned long long>(), t.blev.as<unsigned char>(), t.pt0.as<int>(),
                                     t.pt1.as<int>(), t.ustart.as<int>(), t.ulist.as<int>(), t.wdf.as<float4>(),
                                     t.wdf_lo.as<float2>(), w.ncdf.as<float4>(), plus, nb);
      };
      if (E == 1) go(k_near_df<NEAR_Q>);
      else if (kind == NEAR_V) go(k_near_df<NEAR_V>);
      else go(k_near_df<NEAR_VC>);
    } else if (f64) {
      const double2* nq = E == 2 ? w.nc.as<double2>() : w.qa.as<double2>();
      // many W lists, or many sources a target on average: see the kernel
      const bool half = t.nw >= (t.nleaf + 7) / 8 || (double)t.nu / t.nleaf * t.n / t.nleaf >= NEAR64_HALF;
      auto go = [&](auto whole, auto halves) {
        (half ? halves : whole)<<<std::min(half ? 2 * t.ntile : t.ntile, NEAR64_CTAS * ctx->nsm), 128, 0, ns>>>(
            t.ntile, next, t.tiles.as<int4>(), t.pt0.as<int>(), t.pt1.as<int>(), t.ustart.as<int>(),
            t.ulist.as<int>(), t.zs.as<double2>(), nq, plus, nb);
      };
      if (kind == NEAR_Q) go(k_near64<NEAR_Q, false>, k_near64<NEAR_Q, true>);
      else if (kind == NEAR_QI) go(k_near64<NEAR_QI, false>, k_near64<NEAR_QI, true>);
      else if (kind == NEAR_V) go(k_near64<NEAR_V, false>, k_near64<NEAR_V, true>);
      else go(k_near64<NEAR_VC, false>, k_near64<NEAR_VC, true>);
    } else {
      const float2* nq = E == 2 ? w.nc.as<float2>() : w.qa.as<float2>();
      auto go = [&](auto kern) {
        kern<<<t.ntile, NEAR32_THREADS, 0, ns>>>(t.tiles.as<int4>(), t.pt0.as<int>(), t.pt1.as<int>(),
                                      t.ustart.as<int>(), t.ulist.as<int>(), t.zhl.as<float4>(), nq, plus, nb);
      };
      if (E == 1) go(k_near32<NEAR_Q>);
      else if (kind == NEAR_V) go(k_near32<NEAR_V>);
      else go(k_near32<NEAR_VC>);
    }
    eb_count_launch(ctx);
    if (E == 2 && t.wall && dz) {  // the wall's reflected near field joins the near-field sums
      const int ld = t.ld, nbl = t.lev_off[ld + 1] - t.lev_off[ld];
      k_img_near<<<nbl, IMG_TILE, 0, ns>>>(t.lev_off[ld], nbl, ld, t.bkey.as<unsigned long long>(), t.pt0.as<int>(),
                                           t.pt1.as<int>(), t.zs.as<double2>(), t.perm.as<int>(), dens, dz, hpt,
                                           (double)sign, nb);
      eb_count_launch(ctx);
    }
  };
  // The near field runs on the side stream while the expansion passes run on the main
  // stream, and the far-field kernel adds both. Measured up to
  // 2^20 nodes it pays at every size (the expansion passes' coarse levels stay
  // latency-bound): against a limit of 2^18, the 285,440-node batch's RK2 step 35.1 →
  // 33.6 ms and the 1,048,576-node refined solve 45.7 → 44.3 ms. Above that, and under the
  // per-kernel profiling timer, it precedes the far field on the main stream.
  const bool split = has_far && !ctx->profiling && n <= (1 << 20);
  auto fork_near = [&]() -> int {
    EB_CUDA_TRY(cudaEventRecord(ctx->ev_c, st));
    EB_CUDA_TRY(cudaStreamWaitEvent(ctx->side_stream, ctx->ev_c, 0));
    near(ctx->side_stream);
    EB_CUDA_TRY(cudaEventRecord(ctx->ev_p2p, ctx->side_stream));
    return EB_OK;
  };
  // FP64 on few tiles (the near field is the shorter side then): forked once the P2M, which
  // the FP64 pipe bounds as well, has run. 4,096 nodes over a wall 3.68 -> 3.56 ms a solve,
  // 14,401 nodes 233 -> 227 us an apply; 64 x 512 the other way, 6.72 -> 7.82 ms a solve.
  const bool late = f64 && !df && t.ntile <= 8 * ctx->nsm;
  if (split && !late) EB_TRY(fork_near());
  if (has_far && df) EB_TRY(fmm_expansions_df<E>(ctx, t, tb, w));
  else if (has_far) EB_TRY((fmm_expansions<T, E>(ctx, t, tb, w, dz != nullptr,
                                                 split && late ? std::function<int()>(fork_near) : nullptr)));
  if (!has_far) {
    EB_TRY(w.local.ensure(sizeof(c_t<T>) * (size_t)(E * (tb.p + 1))));
    EB_TRY(w.local_df.ensure(sizeof(float4) * (size_t)(E * (tb.p + 1))));
  }
  const int far_lev = has_far ? std::min(t.L - 1, EB_FAR_LEVELS) : 0;  // far boxes per leaf, at most
  const size_t far_sm = sizeof(float4) * (size_t)far_lev * E * (tb.p + 1);
  if (split) EB_CUDA_TRY(cudaStreamWaitEvent(st, ctx->ev_p2p, 0));
  if (join) EB_CUDA_TRY(cudaStreamWaitEvent(st, join, 0));
  if (!split && !f64) {
    ProfScope pn(ctx, 2, st);
    near(st);
    pn.done();
  }
  ProfScope ps(ctx, 0, st);
  if (!split && f64) near(st);
  if (df) {
    k_far_df<E><<<blocks, 128, 0, st>>>(
        t.ngroup, t.gleaf.as<int>(), t.gfirst.as<int>(), t.leaves.as<int>(), has_far, t.bkey.as<unsigned long long>(),
        t.blev.as<unsigned char>(), t.pt1.as<int>(), t.wstart.as<int>(), t.wlist.as<int>(), w.mpole_df.as<float4>(),
        t.perm.as<int>(), t.wdf.as<float4>(), t.wdf_lo.as<float2>(), tb.p, (double)sign, w.local_df.as<float4>(),
        out, post, nb);
  } else if (f64) {
    const int lpt = n >= FAR64_ONE ? 1 : 4;
    auto go = [&](auto kern) {
      kern<<<nblk((long long)n * lpt, 128), 128, 0, st>>>(
          n, t.lflag.as<int>(), t.lscan.as<int>(), t.leaves.as<int>(), has_far, t.bkey.as<unsigned long long>(),
          t.blev.as<unsigned char>(), t.wstart.as<int>(), t.wlist.as<int>(), t.perm.as<int>(), t.zs.as<double2>(),
          t.x0, t.y0, t.W, 1.0 / t.W, tb.p, (double)sign, w.local.as<double2>(), w.mpole.as<double2>(), nb, out, post);
    };
    if (lpt == 1) go(k_far64<E, 1>);
    else go(k_far64<E, 4>);
  } else {
    k_far32<E><<<t.ntile, FAR_THREADS, far_sm, st>>>(t.tiles.as<int4>(), t.leaves.as<int>(),
                                             t.bkey.as<unsigned long long>(), t.blev.as<unsigned char>(),
                                             t.anc.as<int>(), t.wstart.as<int>(), t.wlist.as<int>(), t.perm.as<int>(),
                                             t.wdf.as<float4>(), tb.p, (float)sign, w.local.as<float2>(),
                                             w.mpole.as<float2>(), out, post, nb);
  }
  eb_count_launch(ctx);
  ps.done();
  ctx->last_p = tb.p;
  return eb_check_launch(ctx, "fmm apply");
}

}  // namespace

int eb_tables_init(eb_ctx* ctx) {
  int p64 = ctx->opts.p64, p32 = ctx->opts.p32;
  if (p64 < 2 || p64 > EB_MAX_P || p32 < 2 || p32 > EB_MAX_P) {
    eb_set_last_error_msg("expansion order outside [2, 60]");
    return EB_ERR_TOL;
  }
  EB_TRY(tables_build<double>(ctx->tab64, p64, ctx->opts.tol64));
  EB_TRY(eb_m2l_fx_tables(ctx->tab64));
  EB_TRY(tables_build<float>(ctx->tab32, p32, ctx->opts.tol32));
  return EB_OK;
}

int eb_fmm_apply(eb_ctx* ctx, EbTree& t, int kernel, int sign, int precision,
                 const double2* dens, const double2* dz, const double* hpt, double2* out,
                 const EbPost* post, cudaEvent_t join) {
  if (!t.valid) return EB_ERR_NOGEOM;
  if (kernel != 0) return EB_ERR_ARG;
  const bool df = precision == EB_PREC_DF || ctx->opts.df64 > 0;
  if (precision == EB_FP32) return eb_fp32_apply(ctx, t, sign, dens, dz, hpt, out, post, join);
  if (precision != EB_PREC_INNER) return fmm_run<double, 2>(ctx, t, sign, dens, dz, hpt, nullptr, out, post, join, df);
  return fmm_run<float, 2>(ctx, t, sign, dens, dz, hpt, nullptr, out, post, join, false);
}

int eb_fmm_apply_cauchy(eb_ctx* ctx, EbTree& t, int precision, const double2* q, double2* out,
                        const EbPost* post) {
  if (!t.valid) return EB_ERR_NOGEOM;
  const bool df = precision == EB_PREC_DF || ctx->opts.df64 > 0;
  if (precision == EB_FP32) return eb_fp32_apply_cauchy(ctx, t, q, out, post);
  if (precision != EB_PREC_INNER) return fmm_run<double, 1>(ctx, t, 0, nullptr, nullptr, nullptr, q, out, post, nullptr, df);
  return fmm_run<float, 1>(ctx, t, 0, nullptr, nullptr, nullptr, q, out, post, nullptr, false);
}
