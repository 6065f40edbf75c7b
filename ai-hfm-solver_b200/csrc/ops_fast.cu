// Register-queue plane-marching stencil kernels.  Layout and semantics are those of
// ops_generic.cu; these kernels differ only in how they move data:
//   * a thread owns V consecutive x (V = 4 where rows and pointers allow it: one 16-byte
//     float32 / 8-byte 16-bit load; else 2 or 1, for the ragged grids) of a row and marches
//     along z through a chunk of planes, so z neighbours, the z-face coefficient and 27-point
//     partial sums stay in registers;
//   * x neighbours come from the adjacent lanes by warp shuffle (lanes hold consecutive
//     vectors of the flattened (row, x-vector) index); only lanes 0 / 31 load them;
//   * y neighbours are vector loads served mostly by L1 (the rows belong to the same block).
// Modes: SMOOTH (weighted Jacobi), RESID (A phi - b, optional norm partials), RESTRICT
// (residuals of 2 rows x 2 planes x 2 columns averaged into the coarse grid; a lane pair
// holds the two rows).
#include <map>
#include <mutex>

#include "hfm_internal.cuh"

namespace hfm {

namespace {

constexpr int kFastThreads = 256;

enum { M_SMOOTH = FAST_SMOOTH, M_RESID = FAST_RESID, M_RESTRICT = FAST_RESTRICT };
enum { C_NONE = 0, C_COARSE = 1, C_SAME = 2 };

template <int V> struct FV {
  float v[V];
};

// V consecutive values (V sizeof(T)-byte access).
template <class T, int V> __device__ __forceinline__ FV<V> ldv(const T *p) {
  FV<V> r;
  if constexpr (V == 1) {
    r.v[0] = St<T>::ld(p);
  } else if constexpr (sizeof(T) == 4) {
    if constexpr (V == 4) {
      const float4 a = __ldg(reinterpret_cast<const float4 *>(p));
      r.v[0] = a.x; r.v[1] = a.y; r.v[2] = a.z; r.v[3] = a.w;
    } else {
      const float2 a = __ldg(reinterpret_cast<const float2 *>(p));
      r.v[0] = a.x; r.v[1] = a.y;
    }
  } else {
    unsigned u[V / 2];
    if constexpr (V == 4) {
      const uint2 q = __ldg(reinterpret_cast<const uint2 *>(p));
      u[0] = q.x;
      u[1] = q.y;
    } else {
      u[0] = __ldg(reinterpret_cast<const unsigned *>(p));
    }
#pragma unroll
    for (int k = 0; k < V / 2; ++k) {
      const T *h = reinterpret_cast<const T *>(&u[k]);
      r.v[2 * k] = St<T>::to(h[0]);
      r.v[2 * k + 1] = St<T>::to(h[1]);
    }
  }
  return r;
}

template <class T, int V> __device__ __forceinline__ void stv(T *p, const FV<V> &v) {
  if constexpr (V == 1) {
    *p = St<T>::from(v.v[0]);
  } else if constexpr (sizeof(T) == 4) {
    if constexpr (V == 4) *reinterpret_cast<float4 *>(p) = make_float4(v.v[0], v.v[1], v.v[2], v.v[3]);
    else *reinterpret_cast<float2 *>(p) = make_float2(v.v[0], v.v[1]);
  } else {
    alignas(8) T h[V];
#pragma unroll
    for (int k = 0; k < V; ++k) h[k] = St<T>::from(v.v[k]);
    if constexpr (V == 4) *reinterpret_cast<uint2 *>(p) = *reinterpret_cast<const uint2 *>(h);
    else *reinterpret_cast<unsigned *>(p) = *reinterpret_cast<const unsigned *>(h);
  }
}
// The sweep's quotient: the ragged grids (V < 4) keep the IEEE division of the generic kernels.
template <int V> __device__ __forceinline__ float quotient(float n, float d) {
  return V < 4 ? n / d : __fdividef(n, d);
}
template <int V> __device__ __forceinline__ FV<V> filled(float x) {
  FV<V> r;
#pragma unroll
  for (int e = 0; e < V; ++e) r.v[e] = x;
  return r;
}

template <class T> struct FastArgs {
  DevOp op;
  const T *base;      // phi (nullable = zero)
  const T *corr;      // correction (nullable)
  const T *rhs;       // b / f (nullable = zero)
  T *out;             // smoothed phi / residual (nullable in RESTRICT mode)
  T *coarse;          // RESTRICT output
  double *partials;   // [inst][blocks] squared-residual partial sums (nullable)
  const int *active;
  int64_t stride, corr_stride, coarse_stride;
  int Z, Y, X;
  float omega, corr_sign;
  int zero_xend;      // input: phi' = 0 on x = X-1 (NS correction before the sweep)
  int zero_xend_out;  // output: residual = 0 on x = X-1 (NS residual)
  int top_copy;
  int dot_phi;        // partials of res * phi instead of res^2 (RESID)
  int dot_rhs;        // partials of out * rhs (SMOOTH)
  ZPlan zp;           // planes of a block (last: its table would lie between the scalars)
};

template <class T, int CORR>
__device__ __forceinline__ float phi_scalar(const FastArgs<T> &a, int64_t ib, int64_t ic, int z,
                                            int y, int x) {
  float v = a.base ? St<T>::ld(a.base + ib + ((int64_t)z * a.Y + y) * a.X + x) : 0.f;
  if (CORR == C_COARSE)
    v += a.corr_sign *
         St<T>::ld(a.corr + ic + ((int64_t)(z >> 1) * (a.Y >> 1) + (y >> 1)) * (a.X >> 1) + (x >> 1));
  else if (CORR == C_SAME)
    v += a.corr_sign * St<T>::ld(a.corr + ic + ((int64_t)z * a.Y + y) * a.X + x);
  if (a.zero_xend && x == a.X - 1) v = 0.f;
  return v;
}

// Load phi' (V-vector) at (z, y, x0); zero outside the grid.
template <class T, int CORR, int V>
__device__ __forceinline__ FV<V> phi_vec(const FastArgs<T> &a, int64_t ib, int64_t ic, int z, int y,
                                         int x0, bool inb) {
  FV<V> v = filled<V>(0.f);
  if (!inb) return v;
  if (a.base) v = ldv<T, V>(a.base + ib + ((int64_t)z * a.Y + y) * a.X + x0);
  if (CORR == C_COARSE) {
    const T *p = a.corr + ic + ((int64_t)(z >> 1) * (a.Y >> 1) + (y >> 1)) * (a.X >> 1) + (x0 >> 1);
    constexpr int H = V > 1 ? V / 2 : 1;
    const FV<H> c = ldv<T, H>(p);
#pragma unroll
    for (int e = 0; e < V; ++e) v.v[e] += a.corr_sign * c.v[e >> 1];
  } else if (CORR == C_SAME) {
    const FV<V> c = ldv<T, V>(a.corr + ic + ((int64_t)z * a.Y + y) * a.X + x0);
#pragma unroll
    for (int e = 0; e < V; ++e) v.v[e] += a.corr_sign * c.v[e];
  }
  if (a.zero_xend && x0 + V == a.X) v.v[V - 1] = 0.f;
  return v;
}

// Neighbours across the vector boundary by shuffle (all lanes must call).  LS: lanes between a
// row's vectors (2 in the restriction, where a lane pair holds a pair of rows).
template <class T, int CORR, int V, int LS>
__device__ __forceinline__ void halo_x(const FastArgs<T> &a, int64_t ib, int64_t ic, int z, int y,
                                       int x0, bool inb, const FV<V> &c, float &l, float &r) {
  const int lane = threadIdx.x & 31;
  float sl = __shfl_up_sync(0xffffffffu, c.v[V - 1], LS);
  float sr = __shfl_down_sync(0xffffffffu, c.v[0], LS);
  l = 0.f;
  r = 0.f;
  if (inb) {
    if (x0 > 0) l = lane >= LS ? sl : phi_scalar<T, CORR>(a, ib, ic, z, y, x0 - 1);
    if (x0 + V < a.X) r = lane < 32 - LS ? sr : phi_scalar<T, CORR>(a, ib, ic, z, y, x0 + V);
  }
}

template <class T, int V, int LS>
__device__ __forceinline__ void coef_halo_x(const T *s, int64_t base_off, int x0, int X, bool inb,
                                            const FV<V> &c, float &l, float &r) {
  const int lane = threadIdx.x & 31;
  float sl = __shfl_up_sync(0xffffffffu, c.v[V - 1], LS);
  float sr = __shfl_down_sync(0xffffffffu, c.v[0], LS);
  l = c.v[0];  // wall: ghost sigma = interior sigma
  r = c.v[V - 1];
  if (inb) {
    if (x0 > 0) l = lane >= LS ? sl : St<T>::ld(s + base_off - 1);
    if (x0 + V < X) r = lane < 32 - LS ? sr : St<T>::ld(s + base_off + V);
  }
}

// The (y, x0) of a thread: consecutive lanes hold consecutive vectors of a row; in RESTRICT a
// lane pair holds the two rows of a coarse row at one x0, so that neither a second row per
// thread (123 registers, half the warps) nor shared memory is needed to average them: one
// 32^3 SIGMA7 instance, float32, 7.6 -> 4.1 us.
constexpr int lane_step(int mode) { return mode == M_RESTRICT ? 2 : 1; }
template <int MODE, int V>
__device__ __forceinline__ bool thread_row(int X, int Y, int &y, int &x0) {
  constexpr int LS = lane_step(MODE);
  const int nvx = X / V;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool valid = i < Y * nvx;  // RESTRICT: Y is even
  const int j = valid ? i / LS : 0;
  const int g = j / nvx;
  y = g * LS + (valid ? i % LS : 0);
  x0 = (j - g * nvx) * V;
  return valid;
}

// RESTRICT: a lane pair holds the two rows of its coarse cells; they gain plane z of the
// residuals (x pairs within the vector, y pairs across the two lanes), and an odd plane
// completes and stores them.
template <class T, int V>
__device__ __forceinline__ void coarse_cells(const FastArgs<T> &a, int64_t inst, int z, int y, int x0,
                                             bool valid, const FV<V> &res, float (&cpart)[2]) {
  if constexpr (V > 1) {
#pragma unroll
    for (int k = 0; k < V / 2; ++k) {
      const float pk = res.v[2 * k] + res.v[2 * k + 1];
      cpart[k] += 0.125f * (pk + __shfl_xor_sync(0xffffffffu, pk, 1));
    }
    if (!(z & 1)) return;
    if (valid && !(y & 1)) {
      const int Yc = a.Y >> 1, Xc = a.X >> 1;
      T *cp = a.coarse + inst * a.coarse_stride + ((int64_t)(z >> 1) * Yc + (y >> 1)) * Xc + (x0 >> 1);
      if (sizeof(T) == 4 && V == 4) {
        *reinterpret_cast<float2 *>(cp) = make_float2(cpart[0], cpart[1]);
      } else {
        cp[0] = St<T>::from(cpart[0]);
        if (V == 4) cp[1] = St<T>::from(cpart[1]);
      }
    }
    cpart[0] = cpart[1] = 0.f;
  }
}

// ---------------------------------------------------------------------------------------
// 7-point forms (CONST7, SIGMA7, FACE7).
// ---------------------------------------------------------------------------------------
template <int KIND, class T, int MODE, int CORR, bool SUMS, int V>
__global__ void __launch_bounds__(kFastThreads, MODE == M_RESTRICT ? 2 : 4)
    k_fast7(const __grid_constant__ FastArgs<T> a) {
  using F4 = FV<V>;  // a thread's cells of a row
  constexpr int LS = lane_step(MODE);
  constexpr int NP = MODE == M_RESTRICT ? 2 : 1;  // planes whose loads are in flight together
  int64_t inst;
  int z0, z1;
  if (!block_planes(a.zp, a.active, a.Z, inst, z0, z1)) return;
  const int X = a.X, Y = a.Y, Z = a.Z;
  int y, x0;
  const bool valid = thread_row<MODE, V>(X, Y, y, x0);
  const int64_t ib = inst * a.stride, ic = inst * a.corr_stride;
  const int64_t plane = (int64_t)Y * X;

  // coefficient setup
  float kx = 0.f, ky = 0.f, kz = 0.f, dconst = 0.f, cx = 0.f, cy = 0.f, cz = 0.f;
  const T *sx = nullptr, *sy = nullptr, *sz = nullptr;
  if (KIND == HFM_OP_CONST7) {
    kz = a.op.k[0];
    ky = a.op.k[1];
    kx = a.op.k[2];
    dconst = 2.f * (kx + ky + kz);
  } else {
    const float s = a.op.scale;
    cz = a.op.c[0] * s;
    cy = a.op.c[1] * s;
    cx = a.op.c[2] * s;
    if (KIND == HFM_OP_FACE7) {  // instance strides follow from the extents
      sx = (const T *)a.op.coef[0] + inst * face7_nx(Z, Y, X);
      sy = (const T *)a.op.coef[1] + inst * face7_ny(Z, Y, X);
      sz = (const T *)a.op.coef[2] + inst * face7_nz(Z, Y, X);
    } else {
      sx = (const T *)a.op.coef[0] + inst * a.op.coef_stride;
      sy = (const T *)a.op.coef[1] + inst * a.op.coef_stride;
      sz = (const T *)a.op.coef[2] + inst * a.op.coef_stride;
    }
  }

  // offsets of (z, y, x0) that advance by a plane, so that a load costs one addition, not the
  // 64-bit products of its coordinates
  const T *phi = a.base + ib, *cor = a.corr + ic, *rhs = a.rhs + ib;  // read only where not null
  int64_t o = (int64_t)z0 * plane + (int64_t)y * X + x0;
  int64_t ox = ((int64_t)z0 * Y + y) * (X + 8) + x0, oy = ((int64_t)z0 * (Y + 1) + y) * X + x0;  // FACE7
  const int Xc = X >> 1;
  const int64_t plane_c = (int64_t)(Y >> 1) * Xc;
  // phi' of row y + dy of plane zz, at offset oo
  auto phi_at = [&](int64_t oo, int zz, int dy, bool in) {
    F4 v = filled<V>(0.f);
    if (!in) return v;
    if (a.base) v = ldv<T, V>(phi + oo);
    if (CORR == C_COARSE) {
      constexpr int H = V > 1 ? V / 2 : 1;
      const FV<H> c = ldv<T, H>(cor + (zz >> 1) * plane_c + ((y + dy) >> 1) * Xc + (x0 >> 1));
#pragma unroll
      for (int e = 0; e < V; ++e) v.v[e] += a.corr_sign * c.v[e >> 1];
    } else if (CORR == C_SAME) {
      const FV<V> c = ldv<T, V>(cor + oo);
#pragma unroll
      for (int e = 0; e < V; ++e) v.v[e] += a.corr_sign * c.v[e];
    }
    if (a.zero_xend && x0 + V == X) v.v[V - 1] = 0.f;
    return v;
  };

  // z queue: phi' at z-1, z, z+1; for SIGMA7 also sigma_z at z, and the z- face
  F4 pm, pc, szc, azlo;
  pm = phi_at(o - plane, z0 - 1, 0, valid && z0 > 0);
  pc = phi_at(o, z0, 0, valid);
  if (KIND == HFM_OP_SIGMA7) {
    szc = valid ? ldv<T, V>(sz + o) : filled<V>(1.f);
    if (z0 > 0 && valid) {
      F4 sm = ldv<T, V>(sz + o - plane);
#pragma unroll
      for (int e = 0; e < V; ++e) azlo.v[e] = cz * 0.5f * (szc.v[e] + sm.v[e]);
    } else {
#pragma unroll
      for (int e = 0; e < V; ++e) azlo.v[e] = cz * szc.v[e];
    }
  } else if (KIND == HFM_OP_FACE7) {
    // the z face below plane z0 (wall faces included in the array), times the scale
    const float s = a.op.scale;
    const F4 fz = valid ? ldv<T, V>(sz + o) : filled<V>(0.f);
#pragma unroll
    for (int e = 0; e < V; ++e) azlo.v[e] = s * fz.v[e];
  }
  double acc = 0.0;
  int seg_end = min(z0 + a.zp.seg, z1);
  float cpart[2] = {0.f, 0.f};  // RESTRICT: the two coarse cells of this vector, summed over planes

  for (int zb = z0; zb < z1; zb += NP) {
    // what plane z reads besides the queue; RESTRICT (whole plane pairs) loads two planes'
    // before it uses either, and the y neighbour the lane pair holds comes by shuffle
    F4 pp[NP], pyo[NP], f[NP], c0[NP], c1[NP], c2[NP], c3[NP], c4[NP];
    F4 pym, pyp;
    float fx4[NP], pl, pr;
    const int64_t ob = o;
#pragma unroll
    for (int n = 0; n < NP; ++n) {
      const int z = zb + n;
      pp[n] = phi_at(o + plane, z + 1, 0, valid && z + 1 < Z);
      if (MODE == M_RESTRICT) {
        const int dy = (y & 1) ? 1 : -1;
        pyo[n] = phi_at(o + dy * X, z, dy, valid && y + dy >= 0 && y + dy < Y);
      } else {
        halo_x<T, CORR, V, LS>(a, ib, ic, z, y, x0, valid, pc, pl, pr);
        pym = phi_at(o - X, z, -1, valid && y > 0);
        pyp = phi_at(o + X, z, 1, valid && y + 1 < Y);
      }
      if (KIND == HFM_OP_FACE7) {
        // stored faces (scale applied later): the x faces of the V cells and the one right of
        // the last, the y faces below and above, the z face above (the one below is carried)
        c0[n] = c1[n] = c2[n] = c3[n] = filled<V>(0.f);
        fx4[n] = 0.f;
        if (valid) {
          c0[n] = ldv<T, V>(sx + ox);
          fx4[n] = St<T>::ld(sx + ox + V);
          c1[n] = ldv<T, V>(sy + oy);
          c2[n] = ldv<T, V>(sy + oy + X);
          c3[n] = ldv<T, V>(sz + o + plane);
        }
        ox += (int64_t)Y * (X + 8);
        oy += plane + X;
      } else if (KIND == HFM_OP_SIGMA7) {
        c0[n] = valid ? ldv<T, V>(sx + o) : filled<V>(1.f);
        c1[n] = valid ? ldv<T, V>(sy + o) : filled<V>(1.f);
        c2[n] = (valid && y > 0) ? ldv<T, V>(sy + o - X) : c1[n];
        c3[n] = (valid && y + 1 < Y) ? ldv<T, V>(sy + o + X) : c1[n];
        if (z + 1 < Z && valid) c4[n] = ldv<T, V>(sz + o + plane);
        else c4[n] = n ? c4[0] : szc;
      }
      if (MODE == M_RESTRICT) f[n] = a.rhs && valid ? ldv<T, V>(rhs + o) : filled<V>(0.f);
      o += plane;
    }
#pragma unroll
    for (int n = 0; n < NP; ++n) {
      const int z = zb + n;
      const int64_t off = ob + n * plane;
      if (MODE == M_RESTRICT) {
        halo_x<T, CORR, V, LS>(a, ib, ic, z, y, x0, valid, pc, pl, pr);
#pragma unroll
        for (int e = 0; e < V; ++e) {
          const float sh = __shfl_xor_sync(0xffffffffu, pc.v[e], 1);
          pym.v[e] = (y & 1) ? sh : pyo[n].v[e];
          pyp.v[e] = (y & 1) ? pyo[n].v[e] : sh;
        }
      }
      F4 Ax, dg, res;
      if (KIND == HFM_OP_CONST7) {
#pragma unroll
        for (int e = 0; e < V; ++e) {
          float xm = e == 0 ? pl : pc.v[e - 1];
          float xp = e == V - 1 ? pr : pc.v[e + 1];
          Ax.v[e] = dconst * pc.v[e] - kz * (pm.v[e] + pp[n].v[e]) - ky * (pym.v[e] + pyp.v[e]) -
                    kx * (xm + xp);
          dg.v[e] = dconst;
        }
      } else if (KIND == HFM_OP_FACE7) {
        const float s = a.op.scale;
        F4 azhi;
#pragma unroll
        for (int e = 0; e < V; ++e) {
          const float axm = s * c0[n].v[e], axp = s * (e == V - 1 ? fx4[n] : c0[n].v[e + 1]);
          const float aym = s * c1[n].v[e], ayp = s * c2[n].v[e];
          azhi.v[e] = s * c3[n].v[e];
          const float xm = e == 0 ? pl : pc.v[e - 1];
          const float xp = e == V - 1 ? pr : pc.v[e + 1];
          const float p = pc.v[e];
          Ax.v[e] = axm * (p - xm) + axp * (p - xp) + aym * (p - pym.v[e]) + ayp * (p - pyp.v[e]) +
                    azlo.v[e] * (p - pm.v[e]) + azhi.v[e] * (p - pp[n].v[e]);
          dg.v[e] = ((axm + axp) + (aym + ayp)) + (azlo.v[e] + azhi.v[e]);
        }
        azlo = azhi;
      } else {
        float sxl, sxr;
        coef_halo_x<T, V, LS>(sx, off, x0, X, valid, c0[n], sxl, sxr);
        F4 azhi;
#pragma unroll
        for (int e = 0; e < V; ++e) {
          const float sxe = c0[n].v[e];
          const float sxm = e == 0 ? sxl : c0[n].v[e - 1];
          const float sxp = e == V - 1 ? sxr : c0[n].v[e + 1];
          // wall faces use the interior sigma (sxl / sxr already do at x = 0 / X-1)
          const float axm = cx * 0.5f * (sxe + sxm);
          const float axp = cx * 0.5f * (sxe + sxp);
          const float aym = cy * 0.5f * (c1[n].v[e] + c2[n].v[e]);
          const float ayp = cy * 0.5f * (c1[n].v[e] + c3[n].v[e]);
          azhi.v[e] = cz * 0.5f * (szc.v[e] + c4[n].v[e]);
          const float xm = e == 0 ? pl : pc.v[e - 1];
          const float xp = e == V - 1 ? pr : pc.v[e + 1];
          const float p = pc.v[e];
          Ax.v[e] = axm * (p - xm) + axp * (p - xp) + aym * (p - pym.v[e]) + ayp * (p - pyp.v[e]) +
                    azlo.v[e] * (p - pm.v[e]) + azhi.v[e] * (p - pp[n].v[e]);
          dg.v[e] = axm + axp + aym + ayp + azlo.v[e] + azhi.v[e];
        }
        azlo = azhi;
        szc = c4[n];
      }
      if (MODE != M_RESTRICT) f[n] = a.rhs && valid ? ldv<T, V>(rhs + off) : filled<V>(0.f);
      if (MODE == M_SMOOTH) {
#pragma unroll
        for (int e = 0; e < V; ++e) res.v[e] = pc.v[e] + a.omega * quotient<V>(f[n].v[e] - Ax.v[e], dg.v[e]);
        if (SUMS && valid) {
#pragma unroll
          for (int e = 0; e < V; ++e) acc += (double)res.v[e] * f[n].v[e];
        }
      } else {
#pragma unroll
        for (int e = 0; e < V; ++e) res.v[e] = Ax.v[e] - f[n].v[e];
        if (a.zero_xend_out && x0 + V == X) res.v[V - 1] = 0.f;
        if (SUMS && valid) {
#pragma unroll
          for (int e = 0; e < V; ++e) acc += (double)res.v[e] * (a.dot_phi ? pc.v[e] : res.v[e]);
        }
      }
      if (valid && a.out) {
        if (MODE == M_SMOOTH && a.top_copy && z == 1) stv<T, V>(a.out + ib + y * X + x0, res);
        if (!(MODE == M_SMOOTH && a.top_copy && z == 0 && Z > 1)) stv<T, V>(a.out + ib + off, res);
      }
      pm = pc;
      pc = pp[n];
      if (MODE == M_RESTRICT) coarse_cells<T, V>(a, inst, z, y, x0, valid, res, cpart);
      if (SUMS && z + 1 == seg_end) seg_end = segment_sum<kFastThreads / 32>(a.zp, a.partials, inst, Z, seg_end, z0, z1, acc);
    }
  }
}

// ---------------------------------------------------------------------------------------
// 7-point forms on rows of an odd number of cells (or off every vector boundary): one column
// of cells per thread.  Nine 4-byte loads per cell are then the least the pass can do, so it is
// bound by their latency unless they are issued early: the loads of plane z + 1 go out before
// plane z is computed, and the index arithmetic is kept to 32-bit byte offsets from the
// instance's pointers (64-bit element offsets made 257 instructions per cell, these 173).
// 4 x 75 x 90 x 101, SIGMA7: a sweep 19.3 us, 3.4 TB/s (k_fast7 with one cell per thread, loads
// and use in one plane, 40 us; one thread per cell with 64-bit divisions 53 us).  The arithmetic
// is k_fast7's.
// ---------------------------------------------------------------------------------------
template <int KIND, class T, int MODE, int CORR, bool SUMS>
__global__ void __launch_bounds__(kFastThreads, 3) k_column7(const __grid_constant__ FastArgs<T> a) {
  int64_t inst;
  int z0, z1;
  if (!block_planes(a.zp, a.active, a.Z, inst, z0, z1)) return;
  constexpr bool SIG = KIND == HFM_OP_SIGMA7;
  constexpr unsigned ES = sizeof(T);
  const int X = a.X, Y = a.Y, Z = a.Z;
  const int lane = threadIdx.x & 31;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool valid = i < X * Y;
  const int y = valid ? i / X : 0, x = valid ? i - y * X : 0;
  const T *phi = a.base + inst * a.stride;  // not read when base is null
  const T *cor = a.corr + inst * a.corr_stride;
  const T *rhs = a.rhs + inst * a.stride;
  T *out = a.out + inst * a.stride;
  const T *sx = nullptr, *sy = nullptr, *sz = nullptr;
  float cx = 0.f, cy = 0.f, cz = 0.f, kx = 0.f, ky = 0.f, kz = 0.f;
  if (SIG) {
    sx = (const T *)a.op.coef[0] + inst * a.op.coef_stride;
    sy = (const T *)a.op.coef[1] + inst * a.op.coef_stride;
    sz = (const T *)a.op.coef[2] + inst * a.op.coef_stride;
    cz = a.op.c[0] * a.op.scale;
    cy = a.op.c[1] * a.op.scale;
    cx = a.op.c[2] * a.op.scale;
  } else {
    kz = a.op.k[0];
    ky = a.op.k[1];
    kx = a.op.k[2];
  }
  // value at a byte offset from an instance pointer (uniform base, 32-bit offset)
  auto ld = [](const T *base, unsigned off) {
    return St<T>::ld(reinterpret_cast<const T *>(reinterpret_cast<const char *>(base) + off));
  };
  // phi' at byte offset o, cell (zz, yy, xx); `p`: the cell is in the grid and not zeroed by the
  // x-end rule
  const bool has = a.base != nullptr;
  auto at = [&](bool p, int zz, int yy, int xx, unsigned o) -> float {
    float v = 0.f;
    if (has && p) v = ld(phi, o);
    if (CORR == C_COARSE && p)
      v += a.corr_sign * ld(cor, ES * (unsigned)(((zz >> 1) * (Y >> 1) + (yy >> 1)) * (X >> 1) + (xx >> 1)));
    if (CORR == C_SAME && p) v += a.corr_sign * ld(cor, o);
    return v;
  };
  // lanes 0 and 31 load the row neighbour the shuffles cannot give
  const int dx = lane == 0 ? -1 : 1;
  const bool edge = valid && ((lane == 0 && x > 0) || (lane == 31 && x + 1 < X));
  const bool live = valid && !(a.zero_xend && x == X - 1);
  const bool live_lo = live && y > 0, live_hi = live && y + 1 < Y;
  const bool live_e = edge && !(a.zero_xend && x + dx == X - 1);
  const bool f_in = a.rhs && valid;
  const unsigned row = ES * (unsigned)X, plane = row * (unsigned)Y;
  const unsigned ylo = valid && y > 0 ? row : 0u, yhi = valid && y + 1 < Y ? row : 0u;  // wall: own sigma
  const unsigned xe = edge ? (unsigned)((int)ES * dx) : 0u;
  struct Plane {
    float pp, ym, yp, pe, f;           // phi' above, before / after in y, at the edge; rhs
    float sxc, sxe, syc, sym, syp, szp;
  };
  auto load = [&](int z, unsigned o, Plane &q) {
    q.pp = at(live && z + 1 < Z, z + 1, y, x, o + plane);
    q.ym = at(live_lo, z, y - 1, x, o - row);
    q.yp = at(live_hi, z, y + 1, x, o + row);
    q.pe = at(live_e, z, y, x + dx, o + (unsigned)((int)ES * dx));
    q.f = f_in ? ld(rhs, o) : 0.f;
    if (SIG) {
      q.sxc = ld(sx, o);
      q.sxe = edge ? ld(sx, o + xe) : q.sxc;
      q.syc = ld(sy, o);
      q.sym = ld(sy, o - ylo);
      q.syp = ld(sy, o + yhi);
      q.szp = ld(sz, z + 1 < Z ? o + plane : o);
    }
  };
  // threads past the plane read cell (z, 0, 0)'s conductivities and store nothing
  unsigned o = ES * (unsigned)(z0 * X * Y + (valid ? i : 0));
  float pm = at(live && z0 > 0, z0 - 1, y, x, o - plane);
  float pc = at(live, z0, y, x, o);
  Plane nx;
  load(z0, o, nx);
  float szc = 1.f, azlo = 0.f;
  if (SIG) {
    szc = ld(sz, o);
    azlo = z0 > 0 ? cz * 0.5f * (szc + ld(sz, o - plane)) : cz * szc;
  }
  int seg_end = min(z0 + a.zp.seg, z1);
  double acc = 0.0;
  for (int z = z0; z < z1; ++z) {
    const Plane q = nx;
    const unsigned here = o;
    o += plane;
    if (z + 1 < z1) load(z + 1, o, nx);
    float l = __shfl_up_sync(0xffffffffu, pc, 1), r = __shfl_down_sync(0xffffffffu, pc, 1);
    l = lane == 0 ? q.pe : l;
    r = lane == 31 ? q.pe : r;
    if (x == 0) l = 0.f;
    if (x + 1 == X) r = 0.f;
    float Ax, dg;
    if (SIG) {
      float sl = __shfl_up_sync(0xffffffffu, q.sxc, 1), sr = __shfl_down_sync(0xffffffffu, q.sxc, 1);
      sl = lane == 0 ? q.sxe : sl;
      sr = lane == 31 ? q.sxe : sr;
      if (x == 0) sl = q.sxc;  // wall: ghost sigma = interior sigma
      if (x + 1 == X) sr = q.sxc;
      const float axm = cx * 0.5f * (q.sxc + sl), axp = cx * 0.5f * (q.sxc + sr);
      const float aym = cy * 0.5f * (q.syc + q.sym), ayp = cy * 0.5f * (q.syc + q.syp);
      const float azhi = cz * 0.5f * (szc + q.szp);
      Ax = axm * (pc - l) + axp * (pc - r) + aym * (pc - q.ym) + ayp * (pc - q.yp) + azlo * (pc - pm) +
           azhi * (pc - q.pp);
      dg = axm + axp + aym + ayp + azlo + azhi;
      azlo = azhi;
      szc = q.szp;
    } else {
      dg = 2.f * (kx + ky + kz);
      Ax = dg * pc - kz * (pm + q.pp) - ky * (q.ym + q.yp) - kx * (l + r);
    }
    float v;
    if (MODE == M_SMOOTH) {
      v = pc + a.omega * quotient<1>(q.f - Ax, dg);
    } else {
      v = Ax - q.f;
      if (a.zero_xend_out && x == X - 1) v = 0.f;
    }
    if (SUMS && valid) acc += (double)v * (MODE == M_SMOOTH ? q.f : a.dot_phi ? pc : v);
    if (valid) {
      T *dst = reinterpret_cast<T *>(reinterpret_cast<char *>(out) + here);
      if (MODE == M_SMOOTH && a.top_copy && Z > 1) {
        if (z > 0) *dst = St<T>::from(v);
        if (z == 1) out[i] = St<T>::from(v);
      } else {
        *dst = St<T>::from(v);
      }
    }
    pm = pc;
    pc = q.pp;
    if (SUMS && z + 1 == seg_end) seg_end = segment_sum<kFastThreads / 32>(a.zp, a.partials, inst, Z, seg_end, z0, z1, acc);
  }
}

// ---------------------------------------------------------------------------------------
// 27-point form (K27): per-plane partial sums into three pending outputs.  On one instance of
// 16 x 32 x 32 the residual + restriction takes 5.2 us, bound by its chain of dependent loads
// (7.8 us with two rows per thread; a thread per coarse cell with 216 bounds-checked loads took
// 21 us, and 82 us on 64 x 128 x 128, where the plane-marching TMA kernel takes 8 us).
// SKIP: as skips_zero_weights() says.
// ---------------------------------------------------------------------------------------
template <class T, int MODE, int CORR, bool SUMS, int V, bool SKIP>
__global__ void __launch_bounds__(kFastThreads)
    k_fast27(const __grid_constant__ FastArgs<T> a) {
  using F4 = FV<V>;  // a thread's cells of a row
  int64_t inst;
  int z0, z1;
  if (!block_planes(a.zp, a.active, a.Z, inst, z0, z1)) return;
  const int X = a.X, Y = a.Y, Z = a.Z;
  int y, x0;
  const bool valid = thread_row<MODE, V>(X, Y, y, x0);
  const int64_t ib = inst * a.stride, ic = inst * a.corr_stride;
  const int64_t plane = (int64_t)Y * X;
  const float *K = a.op.k;

  // s_a of plane p = sum_{b,c} K[a][b][c] phi'(p, y+b-1, x+c-1)
  auto plane_sums = [&](int p, F4 &s0, F4 &s1, F4 &s2, F4 &centre) {
    F4 rows[3];
    float ls[3], rs[3];
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      const int yy = y + b - 1;
      const bool in = valid && p >= 0 && p < Z && yy >= 0 && yy < Y;
      rows[b] = phi_vec<T, CORR, V>(a, ib, ic, p, yy, x0, in);
      halo_x<T, CORR, V, lane_step(MODE)>(a, ib, ic, p, yy, x0, in, rows[b], ls[b], rs[b]);
    }
    centre = rows[1];
#pragma unroll
    for (int e = 0; e < V; ++e) {
      float t0 = 0.f, t1 = 0.f, t2 = 0.f;
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        const float xm = e == 0 ? ls[b] : rows[b].v[e - 1];
        const float xc = rows[b].v[e];
        const float xp = e == V - 1 ? rs[b] : rows[b].v[e + 1];
        auto wx = [&](int j, float x) { return K[j] * (SKIP && K[j] == 0.f ? 0.f : x); };
        t0 += wx(3 * b, xm) + wx(3 * b + 1, xc) + wx(3 * b + 2, xp);
        t1 += wx(9 + 3 * b, xm) + wx(9 + 3 * b + 1, xc) + wx(9 + 3 * b + 2, xp);
        t2 += wx(18 + 3 * b, xm) + wx(18 + 3 * b + 1, xc) + wx(18 + 3 * b + 2, xp);
      }
      s0.v[e] = t0;
      s1.v[e] = t1;
      s2.v[e] = t2;
    }
  };

  // pending: out(z) = s0(z-1) + s1(z) + s2(z+1)
  F4 acc_cur, acc_next, cen_cur, cen_next;
  {
    F4 d0, d1, d2, dc, s1;
    plane_sums(z0 - 1, d0, d1, d2, dc);
    plane_sums(z0, acc_next, s1, d2, cen_cur);
#pragma unroll
    for (int e = 0; e < V; ++e) acc_cur.v[e] = d0.v[e] + s1.v[e];
  }
  const float diag = K[13];
  double acc2 = 0.0;
  int seg_end = min(z0 + a.zp.seg, z1);
  float cpart[2] = {0.f, 0.f};  // RESTRICT: the two coarse cells of this vector, summed over planes
  for (int z = z0; z < z1; ++z) {
    const int64_t off = (int64_t)z * plane + (int64_t)y * X + x0;
    F4 f = filled<V>(0.f);
    if (a.rhs && valid) f = ldv<T, V>(a.rhs + ib + off);
    F4 n0, n1, n2, res;
    plane_sums(z + 1, n0, n1, n2, cen_next);
    F4 Ax;
#pragma unroll
    for (int e = 0; e < V; ++e) Ax.v[e] = acc_cur.v[e] + n2.v[e];
    if (MODE == M_SMOOTH) {
#pragma unroll
      for (int e = 0; e < V; ++e) res.v[e] = cen_cur.v[e] + a.omega * quotient<V>(f.v[e] - Ax.v[e], diag);
      if (SUMS && valid) {
#pragma unroll
        for (int e = 0; e < V; ++e) acc2 += (double)res.v[e] * f.v[e];
      }
    } else {
#pragma unroll
      for (int e = 0; e < V; ++e) res.v[e] = Ax.v[e] - f.v[e];
      if (a.zero_xend_out && x0 + V == X) res.v[V - 1] = 0.f;
      if (valid) {
#pragma unroll
        for (int e = 0; e < V; ++e) acc2 += (double)res.v[e] * (a.dot_phi ? cen_cur.v[e] : res.v[e]);
      }
    }
    if (valid && a.out) {
      if (MODE == M_SMOOTH && a.top_copy && z == 1) stv<T, V>(a.out + ib + y * X + x0, res);
      if (!(MODE == M_SMOOTH && a.top_copy && z == 0 && Z > 1)) stv<T, V>(a.out + ib + off, res);
    }
#pragma unroll
    for (int e = 0; e < V; ++e) {
      acc_cur.v[e] = acc_next.v[e] + n1.v[e];
      acc_next.v[e] = n0.v[e];
    }
    cen_cur = cen_next;
    if (MODE == M_RESTRICT) coarse_cells<T, V>(a, inst, z, y, x0, valid, res, cpart);
    if (SUMS && z + 1 == seg_end) seg_end = segment_sum<kFastThreads / 32>(a.zp, a.partials, inst, Z, seg_end, z0, z1, acc2);
  }
}

// Resident blocks per SM of a kernel (its registers decide: 2-3 blocks of 256 threads),
// looked up once per kernel.
int resident_blocks(const void *kernel) {
  static std::mutex mu;
  static std::map<const void *, int> cache;
  std::lock_guard<std::mutex> lk(mu);
  auto it = cache.find(kernel);
  if (it != cache.end()) return it->second;
  int nb = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel, kFastThreads, 0) != cudaSuccess || nb < 1)
    nb = 2;
  cache[kernel] = nb;
  return nb;
}

// Grid shape: (plane tiles, z chunks, instances); z chunks sized so that the launch fills the
// GPU's resident blocks once (a second, partly filled wave doubled the time of the small
// levels: 64 instances of 32^3 made 512 blocks against 444 resident).  Where chunks of 4 planes
// leave resident blocks idle, a plane more per block is a step more in a chain of dependent
// loads and nothing else runs meanwhile, so the chunks go down to one plane (two for the
// restriction): one instance, float32 SIGMA7, 32^3 .. 8^3, a sweep takes 6.7 us with 4-plane
// chunks and 3.2 us with one-plane chunks.  Chunks of fewer than 4 planes are taken only while
// the whole launch is resident, which also bounds the partial sums per instance.
template <class T>
dim3 fast_grid(FastArgs<T> &a, int B, int V, bool even_chunks, bool sums, int per_sm, int *nblk_out) {
  const int64_t vecs = (int64_t)a.Y * (a.X / V);
  const int tiles = (int)((vecs + kFastThreads - 1) / kFastThreads);
  const int64_t target = (int64_t)sm_count() * per_sm;
  // sums per plane on the small grids, where a block that must march 4 is a chain 4 long
  // (32^3: 8.1 us with a few of 64 instances active, 5.0 per plane), else per 4 planes
  const int seg = tiles * a.Z <= 64 ? 1 : 4;
  const int Z = a.Z, step = std::max(sums && a.active && B > 1 ? seg : 1, even_chunks ? 2 : 1);
  fill_zplan(a.zp, Z, B, a.active != nullptr, seg, [&](int n, int64_t limit) {
    const int64_t chunks = std::min(std::max<int64_t>(1, target / ((int64_t)tiles * n)), limit);
    int zc = (int)((Z + chunks - 1) / chunks);
    if (zc < 4 && (int64_t)tiles * n * ((Z + zc - 1) / zc) > target) zc = 4;
    zc = (zc + step - 1) / step * step;
    return zc > Z ? Z : zc;
  });
  if (nblk_out) *nblk_out = tiles * ((Z + a.zp.seg - 1) / a.zp.seg);
  return dim3(tiles, (Z + a.zp.chunk - 1) / a.zp.chunk, B);
}

}  // namespace

bool fast_eligible(int kind, Grid3 g, bool restrict_mode) {
  if (kind != HFM_OP_CONST7 && kind != HFM_OP_SIGMA7 && kind != HFM_OP_K27 && kind != HFM_OP_FACE7)
    return false;
  if ((g.X & 3) || g.X < 4) return false;
  if (restrict_mode) {
    if ((g.Y & 1) || (g.Z & 1)) return false;
  }
  return true;
}

// Cells per thread of the register-queue kernels for a grid and its pointers, 0: the generic
// kernels.  V = 4 needs rows of a multiple of 4 and pointers aligned to 4 elements; the other
// grids of the 7- and 27-point forms take V = 2 (even rows, pointers aligned to 2 elements) or
// V = 1 from 8 columns up: 4 x 75 x 90 x 101, a SIGMA7 sweep 53 -> 20 us.  Narrower rows, of
// a few hundred cells at most where they occur, stay with one thread per cell.  A correction
// from the coarse grid of a fine grid with odd extents does too, at every width: its last cells
// have no coarse cell, and these kernels do not test for that.
template <class T>
int fast_width(int kind, const DevOp &op, const PhiSrc<T> &phi, const T *rhs, const T *out,
               const T *coarse, int64_t stride, Grid3 g, bool restrict_mode) {
  const int64_t es = (int64_t)sizeof(T);
  if ((restrict_mode || (phi.corr && phi.corr_coarse)) && ((g.Z | g.Y | g.X) & 1)) return 0;
  if (fast_eligible(kind, g, restrict_mode) && vec_aligned<T>(kind, op, phi, rhs, out, coarse, stride, 4 * es))
    return 4;
  if ((kind != HFM_OP_CONST7 && kind != HFM_OP_SIGMA7 && kind != HFM_OP_K27) || g.X < 8) return 0;
  if (!(g.X & 1) && vec_aligned<T>(kind, op, phi, rhs, out, coarse, stride, 2 * es)) return 2;
  // k_column7 keeps 32-bit byte offsets within an instance
  return restrict_mode || g.n() * es >= ((int64_t)1 << 32) || g.n() >= ((int64_t)1 << 31) ? 0 : 1;
}

template <class T, int V, int KIND>
int fast_go(int mode, int corr, FastArgs<T> &a, int B, int *nblk_out, cudaStream_t s) {
  const bool sums = a.partials && (mode != M_SMOOTH || a.dot_rhs);
#define HFM_FAST_GO(KER)                                                                       \
  do {                                                                                         \
    const dim3 grid = fast_grid<T>(a, B, V, mode == M_RESTRICT, sums,                          \
                                   resident_blocks((const void *)KER), nblk_out);              \
    KER<<<grid, kFastThreads, 0, s>>>(a);                                                      \
  } while (0)
#define HFM_FAST_S(M, C, S)                                                                    \
  do {                                                                                         \
    if constexpr (KIND == HFM_OP_K27) {                                                        \
      if constexpr (!S && (V < 4 || M == M_RESTRICT)) {                                        \
        if (skips_zero_weights(KIND, a.op, a.active)) {                                        \
          HFM_FAST_GO((k_fast27<T, M, C, S, V, true>));                                        \
          break;                                                                               \
        }                                                                                      \
      }                                                                                        \
      HFM_FAST_GO((k_fast27<T, M, C, S, V, false>));                                           \
    } else if constexpr (V == 1) HFM_FAST_GO((k_column7<KIND, T, M, C, S>));                     \
    else HFM_FAST_GO((k_fast7<KIND, T, M, C, S, V>));                                          \
  } while (0)
#define HFM_FAST_K(M, C)                                                                       \
  do {                                                                                         \
    if (sums) HFM_FAST_S(M, C, true);                                                          \
    else HFM_FAST_S(M, C, false);                                                              \
  } while (0)
  if (mode == M_SMOOTH) {
    if (corr == C_NONE) HFM_FAST_K(M_SMOOTH, C_NONE);
    else if (corr == C_COARSE) HFM_FAST_K(M_SMOOTH, C_COARSE);
    else HFM_FAST_K(M_SMOOTH, C_SAME);
  } else {
    if (corr != C_NONE) return fail(HFM_ERR_UNSUPPORTED, "fast path: corrected residual");
    if (mode == M_RESID) {
      HFM_FAST_K(M_RESID, C_NONE);
    } else if constexpr (V > 1) {
      HFM_FAST_K(M_RESTRICT, C_NONE);
    } else {
      return fail(HFM_ERR_UNSUPPORTED, "fast path: restriction of odd rows");
    }
  }
#undef HFM_FAST_K
#undef HFM_FAST_S
#undef HFM_FAST_GO
  HFM_CHECK_LAUNCH("fast stencil kernel");
  return HFM_OK;
}

template <class T>
int fast_launch(int kind, int mode, int V, const DevOp &op, const PhiSrc<T> &phi, const T *rhs,
                T *out, T *coarse, int64_t stride, int64_t coarse_stride, int B, Grid3 g,
                float omega, unsigned flags, const int *active, double *partials,
                int *nblk_out, cudaStream_t s) {
  FastArgs<T> a;
  a.op = op;
  a.base = phi.base;
  a.corr = phi.corr;
  a.rhs = rhs;
  a.out = out;
  a.coarse = coarse;
  a.partials = partials;
  a.active = active;
  a.stride = stride;
  a.corr_stride = phi.corr_stride;
  a.coarse_stride = coarse_stride;
  a.Z = g.Z;
  a.Y = g.Y;
  a.X = g.X;
  a.omega = omega;
  a.corr_sign = phi.corr_sign;
  a.zero_xend = phi.zero_xend ? 1 : 0;
  a.zero_xend_out = (mode != M_SMOOTH && (flags & HFM_FLAG_ZERO_XEND)) ? 1 : 0;
  a.top_copy = (mode == M_SMOOTH && (flags & HFM_FLAG_TOP_COPY)) ? 1 : 0;
  a.dot_phi = (mode == M_RESID && (flags & HFM_INT_DOT_PHI)) ? 1 : 0;
  a.dot_rhs = (mode == M_SMOOTH && (flags & HFM_INT_DOT_RHS) && partials) ? 1 : 0;
  if (phi.base && phi.base_stride != stride) return fail(HFM_ERR_BAD_ARG, "fast path: stride mismatch");
  const int corr = phi.corr ? (phi.corr_coarse ? C_COARSE : C_SAME) : C_NONE;
#define HFM_FAST_V(KIND)                                                          \
  (V == 4 ? fast_go<T, 4, KIND>(mode, corr, a, B, nblk_out, s)                    \
   : V == 2 ? fast_go<T, 2, KIND>(mode, corr, a, B, nblk_out, s)                  \
            : fast_go<T, 1, KIND>(mode, corr, a, B, nblk_out, s))
  if (kind == HFM_OP_FACE7) return fast_go<T, 4, HFM_OP_FACE7>(mode, corr, a, B, nblk_out, s);
  if (kind == HFM_OP_K27) return HFM_FAST_V(HFM_OP_K27);
  if (kind == HFM_OP_CONST7) return HFM_FAST_V(HFM_OP_CONST7);
  return HFM_FAST_V(HFM_OP_SIGMA7);
#undef HFM_FAST_V
}

#define HFM_FAST_INST(T)                                                                       \
  template int fast_width<T>(int, const DevOp &, const PhiSrc<T> &, const T *, const T *,      \
                             const T *, int64_t, Grid3, bool);                                 \
  template int fast_launch<T>(int, int, int, const DevOp &, const PhiSrc<T> &, const T *, T *, \
                              T *, int64_t, int64_t, int, Grid3, float, unsigned, const int *, \
                              double *, int *, cudaStream_t);
HFM_FAST_INST(float)
HFM_FAST_INST(__nv_bfloat16)
HFM_FAST_INST(__half)

}  // namespace hfm
