// Operators of the NS time stepper: fused two-stage momentum
// update, pressure-gradient correction, divergence right-hand side with the source boundary
// rule, sigma-mask immersed body, and the velocity / pressure boundary rules.
//
// Every 3x3x3 kernel (diffusion w1, smoothed central differences w2-w4, divergence w6-w8) is
// passed by value as 27 weights (dz, dy, dx) and applied as a cross-correlation with zero
// padding, exactly like the reference's frozen Conv3D layers (naiver_stokes_3D.py:166-236).
#include <cstring>
#include <initializer_list>

#include "hfm_internal.cuh"

namespace hfm {
namespace {

struct K4 {
  float k[4][27];  // diffusion, x, y, z kernels
};
__device__ __forceinline__ float at(const float *f, int z, int y, int x, int Z, int Y, int X) {
  if (z < 0 || z >= Z || y < 0 || y >= Y || x < 0 || x >= X) return 0.f;
  return __ldg(f + ((int64_t)z * Y + y) * X + x);
}

// Stencils over rows of four cells.  A thread owns four consecutive x of one row, lanes own
// consecutive quads; each of the nine rows of the 3x3x3 neighbourhood is read once (one
// 16-byte load, the two edge values from the neighbouring lanes) and serves every kernel and
// all four cells, and the products run two cells per instruction on the packed float32 pipe
// (fma.rn.f32x2, each weight stored twice).  Taps are summed in the order (dz, dy, dx) with
// one fused multiply-add each, zero weights included.  Bound by the packed FMA issue and the
// L1 loads, about equally: at 64 x 128 x 128 k_momentum takes 22 us, k_divergence 13 us and
// k_pgrad 11 us; one cell per thread with a bounds check per tap took 68, 73 and 31 us.  Rows
// that are no multiple of four cells take the same quads with scalar loads (27, 22 and 14 us
// at 64 x 128 x 130).
constexpr int kRowThreads = 128;

struct W4 {
  float2 k[27][4];  // tap -> (w, w) of the diffusion, x, y, z kernels
};
struct W3 {
  float2 k[27][3];
};

template <class W, int N> W pack_weights(const float *const (&w)[N]) {
  W p;
  for (int j = 0; j < 27; ++j)
    for (int q = 0; q < N; ++q) p.k[j][q] = make_float2(w[q][j], w[q][j]);
  return p;
}

struct Quad {
  int z, y, x0;
  bool valid;
};
__device__ __forceinline__ Quad my_quad(int64_t nq, int Y, int nvx) {
  const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  Quad c;
  c.valid = q < nq;
  const int64_t t = c.valid ? q / nvx : 0;
  c.x0 = c.valid ? (int)(q - t * nvx) * 4 : 0;
  c.y = (int)(t % Y);
  c.z = (int)(t / Y);
  return c;
}

// A row of one field around a thread's quad, loaded (the loads of several rows are issued
// before the first is used) and then completed to the values x0 - 1 .. x0 + 4, zero outside
// the grid.  VEC: X a multiple of 4 and f 16-byte aligned - one 16-byte load, the two edge
// values from the neighbouring lanes (lanes 0 and 31 load theirs); every lane of the warp
// calls both.
template <bool VEC> struct Row {
  float m[VEC ? 5 : 6];  // VEC: the quad and the edge that lanes 0 / 31 load
  bool in;
  __device__ __forceinline__ void load(const float *f, int z, int y, const Quad &c, int Z, int Y, int X) {
    in = c.valid && z >= 0 && z < Z && y >= 0 && y < Y;
    const float *r = f + ((int64_t)z * Y + y) * X + c.x0;
    if (VEC) {
      float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
      if (in) q = __ldg(reinterpret_cast<const float4 *>(r));
      m[0] = q.x; m[1] = q.y; m[2] = q.z; m[3] = q.w;
      const int lane = threadIdx.x & 31;
      m[4] = 0.f;
      if (in && lane == 0 && c.x0 > 0) m[4] = __ldg(r - 1);
      if (in && lane == 31 && c.x0 + 4 < X) m[4] = __ldg(r + 4);
    } else {
#pragma unroll
      for (int e = 0; e < 6; ++e) {
        const int x = c.x0 + e - 1;
        m[e % (VEC ? 5 : 6)] = in && x >= 0 && x < X ? __ldg(r + e - 1) : 0.f;
      }
    }
  }
  __device__ __forceinline__ void values(const Quad &c, int X, float (&v)[6]) const {
    if (VEC) {
      const int lane = threadIdx.x & 31;
      const float l = __shfl_up_sync(0xffffffffu, m[3], 1), h = __shfl_down_sync(0xffffffffu, m[0], 1);
      v[0] = in && c.x0 > 0 ? (lane == 0 ? m[4] : l) : 0.f;
      v[5] = in && c.x0 + 4 < X ? (lane == 31 ? m[4] : h) : 0.f;
#pragma unroll
      for (int e = 0; e < 4; ++e) v[e + 1] = m[e];
    } else {
#pragma unroll
      for (int e = 0; e < 6; ++e) v[e] = m[e % (VEC ? 5 : 6)];
    }
  }
};

template <bool VEC>
__device__ __forceinline__ void ldq(const float *p, const Quad &c, int X, float (&v)[4]) {
  if (VEC) {
    const float4 m = *reinterpret_cast<const float4 *>(p);
    v[0] = m.x; v[1] = m.y; v[2] = m.z; v[3] = m.w;
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] = c.x0 + e < X ? p[e] : 0.f;
  }
}
template <bool VEC>
__device__ __forceinline__ void stq(float *p, const Quad &c, int X, const float (&v)[4]) {
  if (VEC) {
    *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (c.x0 + e < X) p[e] = v[e];
  }
}

// out_f = base_f + coef * (Dif(a_f) - a_u Dx(a_f) - a_v Dy(a_f) - a_w Dz(a_f)), f in {u, v, w}
// (naiver_stokes_3D.py:580-622: stage 1 with a = base = u^n, coef 1/2; stage 2 with a = b,
// base = u^n, coef 1).  With ex / ey / ez (and a zero diffusion kernel) the diffusion term is
// the given field instead: the Petrov-Galerkin form of INHALE_demo.ipynb cell 24.
struct MomArgs {
  const float *a[3], *b[3], *e[3];
  float *o[3];
  int Z, Y, X, nvx;
  float coef;
  W4 K;
};
template <bool VEC>
__global__ void __launch_bounds__(kRowThreads) k_momentum(const __grid_constant__ MomArgs m) {
  const int Z = m.Z, Y = m.Y, X = m.X;
  const Quad c = my_quad((int64_t)Z * Y * m.nvx, Y, m.nvx);
  float2 d[3][4][2];
#pragma unroll
  for (int f = 0; f < 3; ++f)
#pragma unroll
    for (int q = 0; q < 4; ++q) d[f][q][0] = d[f][q][1] = make_float2(0.f, 0.f);
  float cen[3][4];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    Row<VEC> rows[3][3];  // a plane's nine rows in flight together
#pragma unroll
    for (int b = 0; b < 3; ++b)
#pragma unroll
      for (int f = 0; f < 3; ++f) rows[b][f].load(m.a[f], c.z + a - 1, c.y + b - 1, c, Z, Y, X);
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      float v[3][6];
#pragma unroll
      for (int f = 0; f < 3; ++f) {
        rows[b][f].values(c, X, v[f]);
        if (a == 1 && b == 1) {
#pragma unroll
          for (int e = 0; e < 4; ++e) cen[f][e] = v[f][e + 1];
        }
      }
#pragma unroll
      for (int t = 0; t < 3; ++t)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float2 w = m.K.k[9 * a + 3 * b + t][q];
#pragma unroll
          for (int f = 0; f < 3; ++f) {
            d[f][q][0] = __ffma2_rn(w, make_float2(v[f][t], v[f][t + 1]), d[f][q][0]);
            d[f][q][1] = __ffma2_rn(w, make_float2(v[f][t + 2], v[f][t + 3]), d[f][q][1]);
          }
        }
    }
  }
  if (!c.valid) return;
  const int64_t i = ((int64_t)c.z * Y + c.y) * X + c.x0;
#pragma unroll
  for (int f = 0; f < 3; ++f) {
    float base[4], ext[4], out[4];
    ldq<VEC>(m.b[f] + i, c, X, base);
    if (m.e[f]) ldq<VEC>(m.e[f] + i, c, X, ext);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      auto D = [&](int q) { return e & 1 ? d[f][q][e >> 1].y : d[f][q][e >> 1].x; };
      const float d0 = m.e[f] ? ext[e] : D(0);
      const float acc = ((d0 - cen[0][e] * D(1)) - cen[1][e] * D(2)) - cen[2][e] * D(3);
      out[e] = m.coef * acc + base[e];
    }
    stq<VEC>(m.o[f] + i, c, X, out);
  }
}

// Petrov-Galerkin dissipation (INHALE_demo.ipynb cell 20), on the velocities damped by the
// immersed body, u_d = u / (1 + dt sigma).  Pass 1, per component f:
//   k_f = min(2 |(|u_d| + |v_d| + |w_d|) / 3 * Dif(f_d)| /
//             (eps + (|Dx f_d| + |Dy f_d| + |Dz f_d|) / 3), 0.5) / (1 + dt sigma)
__device__ __forceinline__ float damped(const float *f, const float *sg, float dt, int z, int y,
                                        int x, int Z, int Y, int X) {
  if (z < 0 || z >= Z || y < 0 || y >= Y || x < 0 || x >= X) return 0.f;
  const int64_t i = ((int64_t)z * Y + y) * X + x;
  return __ldg(f + i) / (1.f + dt * __ldg(sg + i));
}

__global__ void __launch_bounds__(256)
    k_pg_coef(const float *__restrict__ u, const float *__restrict__ v, const float *__restrict__ w,
              const float *__restrict__ sg, float *__restrict__ ku, float *__restrict__ kv,
              float *__restrict__ kw, int Z, int Y, int X, K4 K, float dt, float eps) {
  const int64_t n = (int64_t)Z * Y * X;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int x = (int)(i % X);
    const int64_t t = i / X;
    const int y = (int)(t % Y), z = (int)(t / Y);
    const float den = 1.f + dt * __ldg(sg + i);
    const float speed = (fabsf(__ldg(u + i) / den) + fabsf(__ldg(v + i) / den)) + fabsf(__ldg(w + i) / den);
    const float *fs[3] = {u, v, w};
    float *ks[3] = {ku, kv, kw};
#pragma unroll
    for (int f = 0; f < 3; ++f) {
      float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b)
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const int j = 9 * a + 3 * b + c;
            const float val = damped(fs[f], sg, dt, z + a - 1, y + b - 1, x + c - 1, Z, Y, X);
#pragma unroll
            for (int q = 0; q < 4; ++q) d[q] += K.k[q][j] * val;
          }
      const float num = 2.f * fabsf(speed / 3.f * d[0]);
      const float k = num / (eps + ((fabsf(d[1]) + fabsf(d[2])) + fabsf(d[3])) / 3.f);
      ks[f][i] = fminf(k, 0.5f) / den;
    }
  }
}

// Pass 2: out_f = 1.5 (k_f Dif(f_d) + Dif(f_d k_f) - f_d Dif(k_f)).
__global__ void __launch_bounds__(256)
    k_pg_flux(const float *__restrict__ u, const float *__restrict__ v, const float *__restrict__ w,
              const float *__restrict__ sg, const float *__restrict__ ku,
              const float *__restrict__ kv, const float *__restrict__ kw, float *__restrict__ ox,
              float *__restrict__ oy, float *__restrict__ oz, int Z, int Y, int X, K4 K,
              float dt) {
  const int64_t n = (int64_t)Z * Y * X;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int x = (int)(i % X);
    const int64_t t = i / X;
    const int y = (int)(t % Y), z = (int)(t / Y);
    const float *fs[3] = {u, v, w};
    const float *ks[3] = {ku, kv, kw};
    float *os[3] = {ox, oy, oz};
#pragma unroll
    for (int f = 0; f < 3; ++f) {
      float df = 0.f, dfk = 0.f, dk = 0.f;
#pragma unroll
      for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b)
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const float wgt = K.k[0][9 * a + 3 * b + c];
            const int zz = z + a - 1, yy = y + b - 1, xx = x + c - 1;
            const float fv = damped(fs[f], sg, dt, zz, yy, xx, Z, Y, X);
            const float kv_ = at(ks[f], zz, yy, xx, Z, Y, X);
            df += wgt * fv;
            dfk += wgt * (fv * kv_);
            dk += wgt * kv_;
          }
      const float fc = __ldg(fs[f] + i) / (1.f + dt * __ldg(sg + i));
      os[f][i] = 1.5f * ((__ldg(ks[f] + i) * df + dfk) - fc * dk);
    }
  }
}

// u -= conv(p, Kx), v -= conv(p, Ky), w -= conv(p, Kz)  (naiver_stokes_3D.py:631-633)
struct GradArgs {
  const float *p;
  float *o[3];
  int Z, Y, X, nvx;
  W3 K;
};
template <bool VEC>
__global__ void __launch_bounds__(kRowThreads) k_pgrad(const __grid_constant__ GradArgs m) {
  const int Z = m.Z, Y = m.Y, X = m.X;
  const Quad c = my_quad((int64_t)Z * Y * m.nvx, Y, m.nvx);
  float2 d[3][2];
#pragma unroll
  for (int q = 0; q < 3; ++q) d[q][0] = d[q][1] = make_float2(0.f, 0.f);
  Row<VEC> rows[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) rows[k].load(m.p, c.z + k / 3 - 1, c.y + k % 3 - 1, c, Z, Y, X);
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      float v[6];
      rows[3 * a + b].values(c, X, v);
#pragma unroll
      for (int t = 0; t < 3; ++t)
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          const float2 w = m.K.k[9 * a + 3 * b + t][q];
          d[q][0] = __ffma2_rn(w, make_float2(v[t], v[t + 1]), d[q][0]);
          d[q][1] = __ffma2_rn(w, make_float2(v[t + 2], v[t + 3]), d[q][1]);
        }
    }
  if (!c.valid) return;
  const int64_t i = ((int64_t)c.z * Y + c.y) * X + c.x0;
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    float o[4];
    ldq<VEC>(m.o[q] + i, c, X, o);
    o[0] -= d[q][0].x; o[1] -= d[q][0].y; o[2] -= d[q][1].x; o[3] -= d[q][1].y;
    stq<VEC>(m.o[q] + i, c, X, o);
  }
}

// b = -(Su(u) + Sv(v) + Sw(w)); with bc_source the plane x = 0 takes the value of x = 1
// (boundary_condition_source, naiver_stokes_3D.py:467-473), computed in place.
struct DivArgs {
  const float *a[3];
  float *b;
  int Z, Y, X, nvx, bc_source;
  W3 K;
};
template <bool VEC>
__global__ void __launch_bounds__(kRowThreads) k_divergence(const __grid_constant__ DivArgs m) {
  const int Z = m.Z, Y = m.Y, X = m.X;
  const Quad c = my_quad((int64_t)Z * Y * m.nvx, Y, m.nvx);
  float2 d[3][2];
#pragma unroll
  for (int q = 0; q < 3; ++q) d[q][0] = d[q][1] = make_float2(0.f, 0.f);
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    Row<VEC> rows[3][3];
#pragma unroll
    for (int b = 0; b < 3; ++b)
#pragma unroll
      for (int q = 0; q < 3; ++q) rows[b][q].load(m.a[q], c.z + a - 1, c.y + b - 1, c, Z, Y, X);
#pragma unroll
    for (int b = 0; b < 3; ++b)
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        float v[6];
        rows[b][q].values(c, X, v);
#pragma unroll
        for (int t = 0; t < 3; ++t) {
          const float2 w = m.K.k[9 * a + 3 * b + t][q];
          d[q][0] = __ffma2_rn(w, make_float2(v[t], v[t + 1]), d[q][0]);
          d[q][1] = __ffma2_rn(w, make_float2(v[t + 2], v[t + 3]), d[q][1]);
        }
      }
  }
  if (!c.valid) return;
  float o[4];
  o[0] = -((d[0][0].x + d[1][0].x) + d[2][0].x);
  o[1] = -((d[0][0].y + d[1][0].y) + d[2][0].y);
  o[2] = -((d[0][1].x + d[1][1].x) + d[2][1].x);
  o[3] = -((d[0][1].y + d[1][1].y) + d[2][1].y);
  if (m.bc_source && c.x0 == 0 && X > 1) o[0] = o[1];
  stq<VEC>(m.b + ((int64_t)c.z * Y + c.y) * X + c.x0, c, X, o);
}

// One thread per quad of a row; the 16-byte form where rows and pointers allow it.
bool rows_vec(int X, std::initializer_list<const void *> ptrs) {
  if (X & 3) return false;
  for (const void *p : ptrs)
    if ((uintptr_t)p & 15) return false;
  return true;
}
int64_t row_blocks(int Z, int Y, int nvx) { return ((int64_t)Z * Y * nvx + kRowThreads - 1) / kRowThreads; }

int launch_momentum(MomArgs &m, cudaStream_t s) {
  m.nvx = (m.X + 3) / 4;
  const int64_t nb = row_blocks(m.Z, m.Y, m.nvx);
  const bool vec = rows_vec(m.X, {m.a[0], m.a[1], m.a[2], m.b[0], m.b[1], m.b[2], m.e[0], m.e[1], m.e[2],
                                  m.o[0], m.o[1], m.o[2]});
  if (vec) k_momentum<true><<<nb, kRowThreads, 0, s>>>(m);
  else k_momentum<false><<<nb, kRowThreads, 0, s>>>(m);
  HFM_CHECK_LAUNCH("k_momentum");
  return HFM_OK;
}

__global__ void k_ibm(float *__restrict__ u, float *__restrict__ v, float *__restrict__ w,
                      const float *__restrict__ sigma, int64_t n, float dt) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const float d = 1.f + dt * __ldg(sigma + i);
    u[i] = u[i] / d;
    v[i] = v[i] / d;
    w[i] = w[i] / d;
  }
}

// Boundary shell enumeration: planes z = 0, Z-1 (2XY cells), then y = 0, Y-1 for interior z
// (2(Z-2)X), then x = 0, X-1 for interior z, y (2(Z-2)(Y-2)).
__device__ __forceinline__ void shell_cell(int64_t k, int Z, int Y, int X, int &z, int &y, int &x) {
  const int64_t A = 2LL * Y * X, Bn = 2LL * (Z - 2) * X;
  if (k < A) {
    z = k < (int64_t)Y * X ? 0 : Z - 1;
    const int64_t r = k % ((int64_t)Y * X);
    y = (int)(r / X);
    x = (int)(r % X);
  } else if (k < A + Bn) {
    const int64_t r = k - A;
    const int64_t half = (int64_t)(Z - 2) * X;
    y = r < half ? 0 : Y - 1;
    const int64_t q = r % half;
    z = 1 + (int)(q / X);
    x = (int)(q % X);
  } else {
    const int64_t r = k - A - Bn;
    const int64_t half = (int64_t)(Z - 2) * (Y - 2);
    x = r < half ? 0 : X - 1;
    const int64_t q = r % half;
    z = 1 + (int)(q / (Y - 2));
    y = 1 + (int)(q % (Y - 2));
  }
}

// Final boundary values of boundary_condition_velocity / _pressure (later assignments win:
// z planes over y planes over x planes; copies read the input arrays), gathered into scratch
// before any is written.
__global__ void k_bc_gather(const float *__restrict__ u, const float *__restrict__ v,
                            const float *__restrict__ w, float *__restrict__ scratch, int64_t S,
                            int Z, int Y, int X, float ub, int pressure) {
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < S;
       k += (int64_t)gridDim.x * blockDim.x) {
    int z, y, x;
    shell_cell(k, Z, Y, X, z, y, x);
    auto I = [&](int zz, int yy, int xx) { return ((int64_t)zz * Y + yy) * X + xx; };
    if (pressure) {
      float p;
      if (z == Z - 1) p = u[I(Z - 2, y, x)];
      else if (z == 0) p = u[I(1, y, x)];
      else if (y == Y - 1) p = u[I(z, Y - 2, x)];
      else if (y == 0) p = u[I(z, 1, x)];
      else if (x == 0) p = u[I(z, y, 1)];
      else p = 0.f;  // x = X-1 (outflow)
      scratch[k] = p;
    } else {
      float fu, fv;
      if (z == Z - 1) {
        fu = u[I(Z - 2, y, x)];
        fv = v[I(Z - 2, y, x)];
      } else if (z == 0) {
        fu = fv = 0.f;
      } else if (y == Y - 1) {
        fu = u[I(z, Y - 2, x)];
        fv = 0.f;
      } else if (y == 0) {
        fu = u[I(z, 1, x)];
        fv = 0.f;
      } else {  // x = 0 (inflow) or x = X-1
        fu = ub;
        fv = 0.f;
      }
      scratch[k] = fu;
      scratch[S + k] = fv;
      scratch[2 * S + k] = 0.f;  // w = 0 on every boundary plane
    }
  }
}

__global__ void k_bc_scatter(float *__restrict__ u, float *__restrict__ v, float *__restrict__ w,
                             const float *__restrict__ scratch, int64_t S, int Z, int Y, int X,
                             int pressure) {
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < S;
       k += (int64_t)gridDim.x * blockDim.x) {
    int z, y, x;
    shell_cell(k, Z, Y, X, z, y, x);
    const int64_t i = ((int64_t)z * Y + y) * X + x;
    u[i] = scratch[k];
    if (!pressure) {
      v[i] = scratch[S + k];
      w[i] = scratch[2 * S + k];
    }
  }
}

int grid_for(int64_t n) {
  int64_t b = (n + 255) / 256;
  const int64_t cap = (int64_t)sm_count() * 8;
  return (int)(b < 1 ? 1 : (b > cap ? cap : b));
}

int64_t shell_size(int Z, int Y, int X) {
  return 2LL * Y * X + 2LL * (Z - 2) * X + 2LL * (Z - 2) * (Y - 2);
}

int check_ns(int Z, int Y, int X) {
  if (Z < 3 || Y < 3 || X < 3) return fail(HFM_ERR_BAD_ARG, "NS operators need extents >= 3");
  return HFM_OK;
}

}  // namespace
}  // namespace hfm

using namespace hfm;

extern "C" {

size_t hfm_ns_bc_scratch_bytes(int Z, int Y, int X) {
  if (Z < 3 || Y < 3 || X < 3) return 0;
  return (size_t)shell_size(Z, Y, X) * 3 * sizeof(float);
}

int hfm_ns_bc_velocity(float *u, float *v, float *w, int Z, int Y, int X, float ub,
                       void *scratch, hfm_stream_t stream) {
  int st;
  if ((st = check_ns(Z, Y, X))) return st;
  if (!u || !v || !w || !scratch) return fail(HFM_ERR_BAD_ARG, "hfm_ns_bc_velocity: NULL");
  const int64_t S = shell_size(Z, Y, X);
  cudaStream_t s = (cudaStream_t)stream;
  k_bc_gather<<<grid_for(S), 256, 0, s>>>(u, v, w, (float *)scratch, S, Z, Y, X, ub, 0);
  HFM_CHECK_LAUNCH("k_bc_gather");
  k_bc_scatter<<<grid_for(S), 256, 0, s>>>(u, v, w, (const float *)scratch, S, Z, Y, X, 0);
  HFM_CHECK_LAUNCH("k_bc_scatter");
  return HFM_OK;
}

int hfm_ns_bc_pressure(float *p, int Z, int Y, int X, void *scratch, hfm_stream_t stream) {
  int st;
  if ((st = check_ns(Z, Y, X))) return st;
  if (!p || !scratch) return fail(HFM_ERR_BAD_ARG, "hfm_ns_bc_pressure: NULL");
  const int64_t S = shell_size(Z, Y, X);
  cudaStream_t s = (cudaStream_t)stream;
  k_bc_gather<<<grid_for(S), 256, 0, s>>>(p, p, p, (float *)scratch, S, Z, Y, X, 0.f, 1);
  HFM_CHECK_LAUNCH("k_bc_gather");
  k_bc_scatter<<<grid_for(S), 256, 0, s>>>(p, p, p, (const float *)scratch, S, Z, Y, X, 1);
  HFM_CHECK_LAUNCH("k_bc_scatter");
  return HFM_OK;
}

int hfm_ns_momentum(const float *adv_u, const float *adv_v, const float *adv_w,
                    const float *base_u, const float *base_v, const float *base_w, float *out_u,
                    float *out_v, float *out_w, int Z, int Y, int X, const float *w_dif,
                    const float *w_dx, const float *w_dy, const float *w_dz, float coef,
                    hfm_stream_t stream) {
  int st;
  if ((st = check_ns(Z, Y, X))) return st;
  if (!adv_u || !adv_v || !adv_w || !base_u || !base_v || !base_w || !out_u || !out_v || !out_w ||
      !w_dif || !w_dx || !w_dy || !w_dz)
    return fail(HFM_ERR_BAD_ARG, "hfm_ns_momentum: NULL");
  if (out_u == adv_u || out_v == adv_v || out_w == adv_w || out_u == adv_v || out_u == adv_w ||
      out_v == adv_u || out_v == adv_w || out_w == adv_u || out_w == adv_v)
    return fail(HFM_ERR_BAD_ARG, "hfm_ns_momentum: outputs must not alias the advected fields");
  const float *const w4[4] = {w_dif, w_dx, w_dy, w_dz};
  MomArgs m{{adv_u, adv_v, adv_w}, {base_u, base_v, base_w}, {nullptr, nullptr, nullptr},
            {out_u, out_v, out_w}, Z, Y, X, 0, coef, pack_weights<W4>(w4)};
  return launch_momentum(m, (cudaStream_t)stream);
}

int hfm_ns_momentum_pg(const float *adv_u, const float *adv_v, const float *adv_w,
                       const float *base_u, const float *base_v, const float *base_w,
                       float *out_u, float *out_v, float *out_w, const float *k_x,
                       const float *k_y, const float *k_z, int Z, int Y, int X, const float *w_dx,
                       const float *w_dy, const float *w_dz, float coef, hfm_stream_t stream) {
  int st;
  if ((st = check_ns(Z, Y, X))) return st;
  if (!adv_u || !adv_v || !adv_w || !base_u || !base_v || !base_w || !out_u || !out_v || !out_w ||
      !k_x || !k_y || !k_z || !w_dx || !w_dy || !w_dz)
    return fail(HFM_ERR_BAD_ARG, "hfm_ns_momentum_pg: NULL");
  if (out_u == adv_u || out_v == adv_v || out_w == adv_w || out_u == adv_v || out_u == adv_w ||
      out_v == adv_u || out_v == adv_w || out_w == adv_u || out_w == adv_v)
    return fail(HFM_ERR_BAD_ARG, "hfm_ns_momentum_pg: outputs must not alias the advected fields");
  static const float none[27] = {0.f};
  const float *const w4[4] = {none, w_dx, w_dy, w_dz};
  MomArgs m{{adv_u, adv_v, adv_w}, {base_u, base_v, base_w}, {k_x, k_y, k_z},
            {out_u, out_v, out_w}, Z, Y, X, 0, coef, pack_weights<W4>(w4)};
  return launch_momentum(m, (cudaStream_t)stream);
}

size_t hfm_ns_pg_scratch_bytes(int Z, int Y, int X) {
  if (Z <= 0 || Y <= 0 || X <= 0) return 0;
  return (size_t)3 * Z * Y * X * sizeof(float);
}

int hfm_ns_pg_dissipation(const float *u, const float *v, const float *w, const float *sigma,
                          float *k_x, float *k_y, float *k_z, int Z, int Y, int X,
                          const float *w_dif, const float *w_dx, const float *w_dy,
                          const float *w_dz, float dt, float eps_k, void *scratch,
                          hfm_stream_t stream) {
  int st;
  if ((st = check_ns(Z, Y, X))) return st;
  if (!u || !v || !w || !sigma || !k_x || !k_y || !k_z || !w_dif || !w_dx || !w_dy || !w_dz || !scratch)
    return fail(HFM_ERR_BAD_ARG, "hfm_ns_pg_dissipation: NULL");
  K4 K;
  memcpy(K.k[0], w_dif, 27 * 4);
  memcpy(K.k[1], w_dx, 27 * 4);
  memcpy(K.k[2], w_dy, 27 * 4);
  memcpy(K.k[3], w_dz, 27 * 4);
  const int64_t n = (int64_t)Z * Y * X;
  float *ku = (float *)scratch, *kv = ku + n, *kw = kv + n;
  k_pg_coef<<<grid_for(n), 256, 0, (cudaStream_t)stream>>>(u, v, w, sigma, ku, kv, kw, Z, Y, X, K,
                                                            dt, eps_k);
  HFM_CHECK_LAUNCH("k_pg_coef");
  k_pg_flux<<<grid_for(n), 256, 0, (cudaStream_t)stream>>>(u, v, w, sigma, ku, kv, kw, k_x, k_y, k_z,
                                                            Z, Y, X, K, dt);
  HFM_CHECK_LAUNCH("k_pg_flux");
  return HFM_OK;
}

int hfm_ns_pressure_gradient(const float *p, float *u, float *v, float *w, int Z, int Y, int X,
                             const float *w_px, const float *w_py, const float *w_pz,
                             hfm_stream_t stream) {
  if (!p || !u || !v || !w || !w_px || !w_py || !w_pz || Z < 1 || Y < 1 || X < 1)
    return fail(HFM_ERR_BAD_ARG, "hfm_ns_pressure_gradient: bad argument");
  const float *const w3[3] = {w_px, w_py, w_pz};
  const GradArgs m{p, {u, v, w}, Z, Y, X, (X + 3) / 4, pack_weights<W3>(w3)};
  const int64_t nb = row_blocks(Z, Y, m.nvx);
  if (rows_vec(X, {p, u, v, w})) k_pgrad<true><<<nb, kRowThreads, 0, (cudaStream_t)stream>>>(m);
  else k_pgrad<false><<<nb, kRowThreads, 0, (cudaStream_t)stream>>>(m);
  HFM_CHECK_LAUNCH("k_pgrad");
  return HFM_OK;
}

int hfm_ns_divergence(const float *u, const float *v, const float *w, float *b, int Z, int Y,
                      int X, const float *w_su, const float *w_sv, const float *w_sw,
                      int bc_source, hfm_stream_t stream) {
  if (!u || !v || !w || !b || !w_su || !w_sv || !w_sw || Z < 1 || Y < 1 || X < 1)
    return fail(HFM_ERR_BAD_ARG, "hfm_ns_divergence: bad argument");
  const float *const w3[3] = {w_su, w_sv, w_sw};
  const DivArgs m{{u, v, w}, b, Z, Y, X, (X + 3) / 4, bc_source, pack_weights<W3>(w3)};
  const int64_t nb = row_blocks(Z, Y, m.nvx);
  if (rows_vec(X, {u, v, w, b})) k_divergence<true><<<nb, kRowThreads, 0, (cudaStream_t)stream>>>(m);
  else k_divergence<false><<<nb, kRowThreads, 0, (cudaStream_t)stream>>>(m);
  HFM_CHECK_LAUNCH("k_divergence");
  return HFM_OK;
}

int hfm_ns_immersed_body(float *u, float *v, float *w, const float *sigma, int Z, int Y, int X,
                         float dt, hfm_stream_t stream) {
  if (!u || !v || !w || !sigma || Z < 1 || Y < 1 || X < 1)
    return fail(HFM_ERR_BAD_ARG, "hfm_ns_immersed_body: bad argument");
  const int64_t n = (int64_t)Z * Y * X;
  k_ibm<<<grid_for(n), 256, 0, (cudaStream_t)stream>>>(u, v, w, sigma, n, dt);
  HFM_CHECK_LAUNCH("k_ibm");
  return HFM_OK;
}

}  // extern "C"
