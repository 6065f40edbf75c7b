// The coarse end of a V-cycle in one kernel: one thread block per instance runs the V-cycle
// of every level from l0 (at most 4096 cells) down to the coarsest and back, with all fields
// of those levels in shared memory.
//
// On the deep levels the stencil kernels are a few microseconds of work behind a launch and a
// dependency each (the 16^3, 8^3, 4^3 levels of 64 instances make ~15 launches per cycle);
// this kernel replaces them with one launch whose sweeps are separated by __syncthreads().
// The sequence is the one the multi-kernel V-cycle runs (nu_pre sweeps from zero, residual +
// 2x2x2 averaging restriction, recursion, coarsest level `coarse_sweeps` sweeps from zero with
// coarse_omega, nearest prolongation + correction fused with the first post-sweep, the
// remaining post-sweeps); iterates stay in float32 between sweeps (the multi-kernel path
// rounds them to the storage type).  Operators as the other kernels evaluate them, ghost
// phi = 0: SIGMA7 face coefficients c_d (s_i + s_j) / 2 (wall face c_d s_i); CONST7 the
// anisotropic 7-point stencil with diagonal 2 (kz + ky + kx); K27 any 3x3x3 kernel, diagonal
// its centre weight.
#include <algorithm>

#include "hfm_internal.cuh"

namespace hfm {

namespace {

constexpr int kSubThreads = 512;

// Shared-memory layout of one level (floats): phi and tmp with a one-cell ghost layer on every
// side, kept zero ((Z+2)(Y+2)(X+2) each), so a stencil reads its neighbours without bounds
// checks; rhs (Z Y X); for SIGMA7 the level's face coefficients Fx [Z][Y][X+1], Fy
// [Z][Y+1][X], Fz [Z+1][Y][X] (c_d (s_i + s_j) / 2, wall faces c_d s_i) and the diagonal
// (Z Y X), formed once per launch from the conductivities in global memory.
__host__ __device__ __forceinline__ int sub_padded(int Z, int Y, int X) { return (Z + 2) * (Y + 2) * (X + 2); }
__host__ __device__ __forceinline__ int sub_faces(int Z, int Y, int X) {
  return Z * Y * (X + 1) + Z * (Y + 1) * X + (Z + 1) * Y * X;
}

// Index of cell (z, y, x) (each may be -1 .. extent) in a padded field.
__device__ __forceinline__ int pix(int z, int y, int x, int Y, int X) {
  return ((z + 1) * (Y + 2) + (y + 1)) * (X + 2) + (x + 1);
}

// A phi at cell (z, y, x), whose padded index is ip, with its diagonal.  ph is a padded field
// (ghosts zero); the face coefficients (SIGMA7) and diagonals come from the level's shared
// arrays.  The products and sums are those the conductivity form evaluates.
template <int KIND, class T>
__device__ __forceinline__ float sub_apply(const SubLevel<T> &L, const float *ph, const float *Fc,
                                           int z, int y, int x, int ip, int i, float *diag) {
  const int X = L.X, Y = L.Y, Z = L.Z;
  const int PX = X + 2, PXY = (X + 2) * (Y + 2);
  if (KIND == HFM_OP_K27) {
    float acc = 0.f;
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = 0; b < 3; ++b)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const float wgt = L.k[9 * a + 3 * b + c];
          if (wgt != 0.f) acc += wgt * ph[ip + (a - 1) * PXY + (b - 1) * PX + (c - 1)];
        }
    *diag = L.k[13];
    return acc;
  }
  if (KIND == HFM_OP_CONST7) {
    const float kz = L.k[0], ky = L.k[1], kx = L.k[2], d = 2.f * (kz + ky + kx);
    *diag = d;
    return d * ph[ip] - kz * (ph[ip - PXY] + ph[ip + PXY]) - ky * (ph[ip - PX] + ph[ip + PX]) -
           kx * (ph[ip - 1] + ph[ip + 1]);
  }
  const float *fx = Fc, *fy = fx + Z * Y * (X + 1), *fz = fy + Z * (Y + 1) * X, *dg = fz + (Z + 1) * Y * X;
  const int ixf = (z * Y + y) * (X + 1) + x, iyf = (z * (Y + 1) + y) * X + x;
  const float axm = fx[ixf], axp = fx[ixf + 1];
  const float aym = fy[iyf], ayp = fy[iyf + X];
  const float azm = fz[i], azp = fz[i + X * Y];
  const float pc = ph[ip];
  *diag = dg[i];
  return axm * (pc - ph[ip - 1]) + axp * (pc - ph[ip + 1]) + aym * (pc - ph[ip - PX]) +
         ayp * (pc - ph[ip + PX]) + azm * (pc - ph[ip - PXY]) + azp * (pc - ph[ip + PXY]);
}

// Coordinates of the cells a thread visits in a block-strided loop over a Z x Y x X grid: the
// first from one division, the next ones by adding the stride's own coordinates with carries
// (dx < X, dy < Y, so at most one carry each) instead of dividing per cell.
struct Walk {
  int z, y, x, dz, dy, dx;
  __device__ Walk(int i, int stride, int Y, int X) {
    x = i % X;
    const int t = i / X;
    y = t % Y;
    z = t / Y;
    dx = stride % X;
    const int u = stride / X;
    dy = u % Y;
    dz = u / Y;
  }
  __device__ void step(int Y, int X) {
    x += dx;
    int cy = 0;
    if (x >= X) {
      x -= X;
      cy = 1;
    }
    y += dy + cy;
    int cz = 0;
    if (y >= Y) {
      y -= Y;
      cz = 1;
    }
    z += dz + cz;
  }
};

// out = in + om (f - A in) / diag over the level's cells (in may be null: a zero iterate;
// in and out are padded fields, only out's interior is written)
template <int KIND, class T>
__device__ void sub_sweep(const SubLevel<T> &L, const float *in, const float *Fc, const float *f,
                          float *out, float om, const float *zero_pad) {
  // a zero iterate: A in = 0 and the diagonal from zero_pad's call (a zero-filled field)
  const float *ph = in ? in : zero_pad;
  Walk w(threadIdx.x, blockDim.x, L.Y, L.X);
  for (int i = threadIdx.x; i < L.n; i += blockDim.x, w.step(L.Y, L.X)) {
    const int ip = pix(w.z, w.y, w.x, L.Y, L.X);
    float dg;
    float ax = sub_apply<KIND, T>(L, ph, Fc, w.z, w.y, w.x, ip, i, &dg);
    if (!in) ax = 0.f;
    const float pc = in ? in[ip] : 0.f;
    out[ip] = pc + om * __fdividef(f[i] - ax, dg);
  }
  __syncthreads();
}

// phi -= P(coarse) on the level's interior (nearest prolongation; phi identically zero when
// `zero`: phi = -P(coarse)).  Both fields padded.
template <class T>
__device__ void sub_correct(const SubLevel<T> &L, float *ph, const SubLevel<T> &Lc,
                            const float *coarse, bool zero) {
  Walk w(threadIdx.x, blockDim.x, L.Y, L.X);
  for (int i = threadIdx.x; i < L.n; i += blockDim.x, w.step(L.Y, L.X)) {
    const int ip = pix(w.z, w.y, w.x, L.Y, L.X);
    const float c = coarse[pix(w.z >> 1, w.y >> 1, w.x >> 1, Lc.Y, Lc.X)];
    ph[ip] = zero ? -c : ph[ip] - c;
  }
  __syncthreads();
}

// fc = R(A phi - f): 0.125 times the sum over each coarse cell's eight fine residuals (ph
// padded, or null for a zero iterate)
template <int KIND, class T>
__device__ void sub_resid_restrict(const SubLevel<T> &L, const float *ph, const float *Fc,
                                   const float *f, const SubLevel<T> &Lc, float *fc) {
  Walk w(threadIdx.x, blockDim.x, Lc.Y, Lc.X);
  for (int j = threadIdx.x; j < Lc.n; j += blockDim.x, w.step(Lc.Y, Lc.X)) {
    const int xc = w.x, yc = w.y, zc = w.z;
    float sum = 0.f;
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int b = 0; b < 2; ++b)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int z = 2 * zc + a, y = 2 * yc + b, x = 2 * xc + c;
          const int i = (z * L.Y + y) * L.X + x;
          float dg;
          const float ax = ph ? sub_apply<KIND, T>(L, ph, Fc, z, y, x, pix(z, y, x, L.Y, L.X), i, &dg) : 0.f;
          sum += ax - f[i];
        }
    fc[j] = 0.125f * sum;
  }
  __syncthreads();
}

// A 16-bit or float32 value read through L2 (ld.global.cg): data another block of the same
// launch may have written (the persistent kernel's restricted residual).
template <class T> __device__ __forceinline__ T ld_l2(const T *p);
template <> __device__ __forceinline__ float ld_l2<float>(const float *p) { return __ldcg(p); }
template <> __device__ __forceinline__ __nv_bfloat16 ld_l2<__nv_bfloat16>(const __nv_bfloat16 *p) {
  return __ushort_as_bfloat16(__ldcg(reinterpret_cast<const unsigned short *>(p)));
}
template <> __device__ __forceinline__ __half ld_l2<__half>(const __half *p) {
  return __ushort_as_half(__ldcg(reinterpret_cast<const unsigned short *>(p)));
}

// The face coefficients and diagonals of a SIGMA7 level of instance `inst` into its shared
// arrays, from the conductivities in global memory, as the conductivity form forms them.
template <class T>
__device__ void sub_faces_init(const SubLevel<T> &L, int64_t inst, float *Fc) {
  const int X = L.X, Y = L.Y, Z = L.Z;
  const int64_t g = inst * (int64_t)L.n;
  const T *sx = L.sx + g, *sy = L.sy + g, *sz = L.sz + g;
  float *fx = Fc, *fy = fx + Z * Y * (X + 1), *fz = fy + Z * (Y + 1) * X;
  const int nx = Z * Y * (X + 1), ny = Z * (Y + 1) * X, nz = (Z + 1) * Y * X;
  for (int k = threadIdx.x; k < nx; k += blockDim.x) {
    const int i = k % (X + 1), row = k / (X + 1);
    const float a = i > 0 ? St<T>::to(sx[row * X + i - 1]) : 0.f, b = i < X ? St<T>::to(sx[row * X + i]) : 0.f;
    fx[k] = L.cx * (i == 0 ? b : (i == X ? a : 0.5f * (b + a)));
  }
  for (int k = threadIdx.x; k < ny; k += blockDim.x) {
    const int x = k % X, t = k / X, j = t % (Y + 1), z = t / (Y + 1);
    const int c0 = (z * Y + j) * X + x;
    const float a = j > 0 ? St<T>::to(sy[c0 - X]) : 0.f, b = j < Y ? St<T>::to(sy[c0]) : 0.f;
    fy[k] = L.cy * (j == 0 ? b : (j == Y ? a : 0.5f * (b + a)));
  }
  for (int k = threadIdx.x; k < nz; k += blockDim.x) {
    const int yx = k % (Y * X), kz = k / (Y * X);
    const float a = kz > 0 ? St<T>::to(sz[(kz - 1) * Y * X + yx]) : 0.f, b = kz < Z ? St<T>::to(sz[kz * Y * X + yx]) : 0.f;
    fz[k] = L.cz * (kz == 0 ? b : (kz == Z ? a : 0.5f * (b + a)));
  }
  __syncthreads();
  float *dg = fz + nz;
  Walk w(threadIdx.x, blockDim.x, Y, X);
  for (int i = threadIdx.x; i < L.n; i += blockDim.x, w.step(Y, X)) {
    const int ixf = (w.z * Y + w.y) * (X + 1) + w.x, iyf = (w.z * (Y + 1) + w.y) * X + w.x;
    dg[i] = fx[ixf] + fx[ixf + 1] + fy[iyf] + fy[iyf + X] + fz[i] + fz[i + X * Y];
  }
}

// The coarse-end V-cycle of one instance with the block's shared memory `sub_smem`, for the
// persistent kernel below: other blocks of the same launch wrote the right-hand side, so it is
// read through L2.
template <int KIND, class T>
__device__ void subcycle_body(const SubArgs<T> &a, int64_t inst, unsigned char *sub_smem) {
  float *F = reinterpret_cast<float *>(sub_smem);
  const int nl = a.nlev;
  // zero every padded field (ghosts stay zero: sweeps write interiors only), faces, rhs
  for (int l = 0; l < nl; ++l) {
    const SubLevel<T> &L = a.lv[l];
    const int np = 2 * sub_padded(L.Z, L.Y, L.X);
    for (int i = threadIdx.x; i < np; i += blockDim.x) F[L.o_phi + i] = 0.f;
    if (KIND == HFM_OP_SIGMA7) sub_faces_init<T>(L, inst, F + L.o_face);
  }
  for (int i = threadIdx.x; i < a.lv[0].n; i += blockDim.x) {
    F[a.lv[0].o_rhs + i] = St<T>::to(ld_l2<T>(a.rhs + inst * (int64_t)a.lv[0].n + i));
  }
  __syncthreads();

  int cur[kMaxSubLevels];    // 0: iterate in phi, 1: in tmp
  bool zero[kMaxSubLevels];  // iterate still identically zero (nu_pre == 0)
  // down: pre-smoothing from zero, residual, restriction
  for (int l = 0; l < nl - 1; ++l) {
    const SubLevel<T> &L = a.lv[l];
    float *buf[2] = {F + L.o_phi, F + L.o_tmp};
    const float *f = F + L.o_rhs, *Fc = F + L.o_face;
    int c = 0;
    for (int k = 0; k < a.nu_pre; ++k) {
      sub_sweep<KIND, T>(L, k == 0 ? nullptr : buf[c], Fc, f, buf[c ^ 1], a.omega, buf[c]);
      c ^= 1;
    }
    cur[l] = c;
    zero[l] = a.nu_pre == 0;
    sub_resid_restrict<KIND, T>(L, zero[l] ? nullptr : buf[c], Fc, f, a.lv[l + 1], F + a.lv[l + 1].o_rhs);
  }
  // coarsest: coarse_sweeps sweeps from zero; a level of at most 64 cells (4^3, 3^3) on one
  // warp, two cells a lane with their indices computed once, __syncwarp() between the
  // sweeps instead of a block barrier (the per-cell arithmetic is sub_sweep's)
  {
    const SubLevel<T> &L = a.lv[nl - 1];
    float *buf[2] = {F + L.o_phi, F + L.o_tmp};
    const float *Fc = F + L.o_face;
    int c = 0;
    if (L.n <= 64 && a.coarse_sweeps > 0) {
      if (threadIdx.x < 32) {
        const float *f = F + L.o_rhs;
        int zz[2], yy[2], xx[2], ipp[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int i = threadIdx.x + 32 * q;
          xx[q] = i % L.X;
          const int t = i / L.X;
          yy[q] = t % L.Y;
          zz[q] = t / L.Y;
          ipp[q] = pix(zz[q], yy[q], xx[q], L.Y, L.X);
        }
        for (int k = 0; k < a.coarse_sweeps; ++k) {
          const float *in = k == 0 ? nullptr : buf[c];
          float *out = buf[c ^ 1];
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int i = threadIdx.x + 32 * q;
            if (i < L.n) {
              float dg;
              const float ax = sub_apply<KIND, T>(L, in ? in : buf[c], Fc, zz[q], yy[q], xx[q], ipp[q], i, &dg);
              const float axv = in ? ax : 0.f;
              const float pc = in ? in[ipp[q]] : 0.f;
              out[ipp[q]] = pc + a.coarse_omega * __fdividef(f[i] - axv, dg);
            }
          }
          __syncwarp();
          c ^= 1;
        }
      } else {
        c = a.coarse_sweeps & 1;
      }
      __syncthreads();
    } else {
      for (int k = 0; k < a.coarse_sweeps; ++k) {
        sub_sweep<KIND, T>(L, k == 0 ? nullptr : buf[c], Fc, F + L.o_rhs, buf[c ^ 1], a.coarse_omega, buf[c]);
        c ^= 1;
      }
    }
    cur[nl - 1] = c;
  }
  // up: prolongation + correction (in place), then the post-sweeps
  const int post = a.nu_post > 0 ? a.nu_post : 1;
  for (int l = nl - 2; l >= 0; --l) {
    const SubLevel<T> &L = a.lv[l];
    const SubLevel<T> &Lc = a.lv[l + 1];
    float *buf[2] = {F + L.o_phi, F + L.o_tmp};
    const float *coarse = F + (cur[l + 1] ? Lc.o_tmp : Lc.o_phi);
    const float *Fc = F + L.o_face;
    int c = cur[l];
    sub_correct<T>(L, buf[c], Lc, coarse, zero[l]);
    for (int k = 0; k < post; ++k) {
      const float om = a.nu_post == 0 ? 0.f : a.omega;
      sub_sweep<KIND, T>(L, buf[c], Fc, F + L.o_rhs, buf[c ^ 1], om, buf[c]);
      c ^= 1;
    }
    cur[l] = c;
  }
  const SubLevel<T> &L0 = a.lv[0];
  const float *res = F + (cur[0] ? L0.o_tmp : L0.o_phi);
  Walk w(threadIdx.x, blockDim.x, L0.Y, L0.X);
  for (int i = threadIdx.x; i < L0.n; i += blockDim.x, w.step(L0.Y, L0.X))
    a.out[inst * (int64_t)L0.n + i] = St<T>::from(res[pix(w.z, w.y, w.x, L0.Y, L0.X)]);
}

// ------------------------------------------------------------------ the program kernel
// One block of 512 threads per instance interprets a list of steps (V or F cycles from a zero
// or a given iterate, or the reference's sawtooth leg) over the levels from l0 down.  It is
// bound by the chain of barrier-separated passes on one SM - each pass by its shared-memory
// wavefronts - so each pass reads as little as it can:
//   * level l0 (TOP: rows of a multiple of 4 cells) belongs to the threads in pairs of quads,
//     4 cells of x in two planes: a thread keeps its right-hand side, face coefficients,
//     1 / diagonal and iterate in registers for the whole launch, x neighbours come by
//     shuffle, and a sweep reads six 16-byte rows of fields without x padding, free of bank
//     conflicts;
//   * the next level (MID, not the coarsest) has a pair of cells in z per thread, their
//     coefficients in registers; the levels below run from shared memory;
//   * the coarsest level's sweeps keep the pairs' coefficients in registers too and synchronise
//     only the warps that hold cells;
//   * the face coefficients of all shared-memory levels are formed cell by cell in one pass
//     whose global loads are all in flight together.
// One instance of 16^3 .. 4^3 (SIGMA7 float32, V(2,2), 32 coarsest sweeps): 14.3 us a launch,
// against 47 us for the eleven launches it replaces and 24 us with 1024 threads, one quad per
// thread and the levels below walked cell by cell with integer divisions.  8 x 16 x 16 and
// 4 x 8 x 8 of the 27-point operator, the F-cycle's F and V visits in one launch: 20 us
// (35 us before, 160 us launch by launch).  In a served bf16 stream, beside other kernels: 22 us
// (34 us before).  Left over: 3.7 us of set-up (global loads), 0.11 us per coarsest sweep, 0.6 us
// per sweep of 16^3.
constexpr int kProgThreads = 512;

// Cell i of a level: padded index and coordinates, from a table formed once per launch.  It takes 8
// bytes a cell, or, where these would not fit (NARROW), 4: 16 bits of padded index (at most 36882,
// 1 x 1 x 4096) below the coordinates, whose bits add up to 15 at most (a level has 4096 cells at
// most).  (With narrow tables the compiler keeps fewer of the 27-point weights in registers where
// level l0 is in quads: 16 x 32 x 32 takes 24 us, not 20.)
struct Cell {
  int ip, z, y, x;
};
template <bool NARROW, class T> __device__ __forceinline__ Cell cell_of(const SubLevel<T> &L, const float *F, int i) {
  if constexpr (!NARROW) {
    const uint2 u = reinterpret_cast<const uint2 *>(F + L.o_idx)[i];
    return Cell{(int)(u.x & 0xffffu), (int)(u.x >> 16), (int)(u.y >> 16), (int)(u.y & 0xffffu)};
  } else {
    const unsigned u = reinterpret_cast<const unsigned *>(F + L.o_idx)[i], c = u >> 16;
    return Cell{(int)(u & 0xffffu), (int)(c >> (L.bx + L.by)), (int)((c >> L.bx) & ((1u << L.by) - 1u)),
                (int)(c & ((1u << L.bx) - 1u))};
  }
}
template <bool NARROW, class T>
__device__ __forceinline__ void set_cell(const SubLevel<T> &L, float *F, int i, int z, int y, int x) {
  const unsigned ip = (unsigned)pix(z, y, x, L.Y, L.X);
  if constexpr (!NARROW)
    reinterpret_cast<uint2 *>(F + L.o_idx)[i] = make_uint2(ip | ((unsigned)z << 16), ((unsigned)y << 16) | (unsigned)x);
  else
    reinterpret_cast<unsigned *>(F + L.o_idx)[i] =
        ip | ((unsigned)x << 16) | ((unsigned)y << (16 + L.bx)) | ((unsigned)z << (16 + L.bx + L.by));
}

// A thread-strided pass over the cells of level L.
#define HFM_FOR_CELLS(L, F)                                                              \
  for (int i = threadIdx.x; i < (L).n; i += kProgThreads) {                              \
    const Cell q = cell_of<NARROW>(L, F, i);

// Cell i of level L: its table entry and, for SIGMA7, its face coefficients (the low ones,
// and the high ones at the walls) and 1 / diagonal.  The global loads and the shared-memory
// stores are apart, so that the loads can be in flight while the block clears its fields.
template <int KIND, class T, bool NARROW> struct CellInit {
  int x, y, z, t, i;
  float vx, vy, vz, xl, xh, yl, yh, zl, zh;
  __device__ __forceinline__ void load(const SubLevel<T> &L, int64_t inst, int cell) {
    const int X = L.X, Y = L.Y, P = X * Y;
    i = cell;
    x = i % X;
    t = i / X;
    y = t % Y;
    z = t / Y;
    if (KIND == HFM_OP_SIGMA7) {
      const int64_t g = inst * (int64_t)L.n + i;
      const T *sx = L.sx + g, *sy = L.sy + g, *sz = L.sz + g;
      // at a wall the neighbour's conductivity is the cell's own: (s + s) / 2 = s
      vx = St<T>::ld(sx);
      vy = St<T>::ld(sy);
      vz = St<T>::ld(sz);
      xl = St<T>::ld(sx - (x > 0 ? 1 : 0));
      xh = St<T>::ld(sx + (x + 1 < X ? 1 : 0));
      yl = St<T>::ld(sy - (y > 0 ? X : 0));
      yh = St<T>::ld(sy + (y + 1 < Y ? X : 0));
      zl = St<T>::ld(sz - (z > 0 ? P : 0));
      zh = St<T>::ld(sz + (z + 1 < L.Z ? P : 0));
    }
  }
  __device__ __forceinline__ void store(const SubLevel<T> &L, float *F) const {
    const int X = L.X, Y = L.Y, Z = L.Z, P = X * Y;
    set_cell<NARROW>(L, F, i, z, y, x);
    if (KIND == HFM_OP_SIGMA7) {
      const float axm = L.cx * (0.5f * (vx + xl)), axp = L.cx * (0.5f * (vx + xh));
      const float aym = L.cy * (0.5f * (vy + yl)), ayp = L.cy * (0.5f * (vy + yh));
      const float azm = L.cz * (0.5f * (vz + zl)), azp = L.cz * (0.5f * (vz + zh));
      float *fx = F + L.o_face, *fy = fx + Z * Y * (X + 1), *fz = fy + Z * (Y + 1) * X;
      const int ixf = i + t, iyf = i + z * X;
      fx[ixf] = axm;
      if (x + 1 == X) fx[ixf + 1] = axp;
      fy[iyf] = aym;
      if (y + 1 == Y) fy[iyf + X] = ayp;
      fz[i] = azm;
      if (z + 1 == Z) fz[i + P] = azp;
      (fz + (Z + 1) * P)[i] = __fdividef(1.f, axm + axp + aym + ayp + azm + azp);
    }
  }
};

// Two cells, (z, y, x) and (z + 1, y, x) with z even, and their coefficients in registers (MID
// and the coarsest level): a neighbour row read from shared memory serves both.
__host__ __device__ __forceinline__ int cell_pairs(int Z, int Y, int X) { return ((Z + 1) >> 1) * Y * X; }
template <int KIND> struct CellPair {
  static constexpr bool SIG = KIND == HFM_OP_SIGMA7;
  float w[KIND == HFM_OP_K27 ? 27 : 3];              // K27 weights / CONST7 kz, ky, kx
  float xy[2][SIG ? 4 : 1], zf[SIG ? 3 : 1], rd[2];  // SIGMA7 faces; 1 / diagonal
  float v[2];                                        // the iterate
  int ip, i;  // padded and unpadded index of the first cell
  bool valid, two;
  template <class T> __device__ __forceinline__ void load(const SubLevel<T> &L, const float *F, int t) {
    const int X = L.X, Y = L.Y, Z = L.Z;
    valid = t < cell_pairs(Z, Y, X);
    if (!valid) t = 0;
    const int x = t % X, r = t / X, y = r % Y, z = 2 * (r / Y), P = X * Y;
    two = valid && z + 1 < Z;
    i = (z * Y + y) * X + x;
    ip = pix(z, y, x, Y, X);
    v[0] = v[1] = 0.f;
    if constexpr (KIND == HFM_OP_K27) {
#pragma unroll
      for (int j = 0; j < 27; ++j) w[j] = L.k[j];
      rd[0] = rd[1] = __fdividef(1.f, L.k[13]);
    } else if constexpr (KIND == HFM_OP_CONST7) {
#pragma unroll
      for (int j = 0; j < 3; ++j) w[j] = L.k[j];
      rd[0] = rd[1] = __fdividef(1.f, 2.f * (L.k[0] + L.k[1] + L.k[2]));
    } else {
      const float *fx = F + L.o_face, *fy = fx + Z * Y * (X + 1), *fz = fy + Z * (Y + 1) * X;
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        const int zg = g == 0 || two ? z + g : z, ig = i + (zg - z) * P;
        const int ixf = ig + zg * Y + y, iyf = ig + zg * X;
        xy[g][0] = fx[ixf];
        xy[g][1] = fx[ixf + 1];
        xy[g][2] = fy[iyf];
        xy[g][3] = fy[iyf + X];
        rd[g] = (fz + (Z + 1) * P)[ig];
      }
      zf[0] = fz[i];
      zf[1] = fz[i + P];
      zf[2] = fz[i + (two ? 2 * P : P)];
    }
  }
  template <class T> __device__ __forceinline__ void rhs(const SubLevel<T> &L, const float *f, float (&r)[2]) const {
    r[0] = f[i];
    r[1] = f[i + (two ? L.X * L.Y : 0)];
  }
  template <class T> __device__ __forceinline__ void store(const SubLevel<T> &L, float *ph, const float (&u)[2]) const {
    if (valid) ph[ip] = u[0];
    if (two) ph[ip + (L.X + 2) * (L.Y + 2)] = u[1];
  }
  // s += the neighbours times their coefficients (K27: minus the weights); SIGMA7 / CONST7 with
  // `diff`: s += the sum of coefficient (neighbour - own)
  template <class T>
  __device__ __forceinline__ void around(const SubLevel<T> &L, const float *ph, float (&s)[2], bool diff) const {
    const float *p = ph + ip;
    const int PX = L.X + 2, PXY = PX * (L.Y + 2);
    if constexpr (KIND == HFM_OP_K27) {
      float t[2][3] = {{s[0], 0.f, 0.f}, {s[1], 0.f, 0.f}};
      const int top = two ? 2 * PXY : PXY;  // plane z + 2
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 9; ++b) {
          const float n = p[(a == 3 ? top : (a - 1) * PXY) + (b / 3 - 1) * PX + (b % 3 - 1)];
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            const int k = a - g;
            if (k < 0 || k > 2 || (k == 1 && b == 4)) continue;
            t[g][b / 3] -= w[9 * k + b] * n;
          }
        }
      s[0] = (t[0][0] + t[0][1]) + t[0][2];
      s[1] = (t[1][0] + t[1][1]) + t[1][2];
    } else {
      const float zm = p[-PXY], zp = p[two ? 2 * PXY : PXY];
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        const float *q = p + g * PXY;
        const float o = diff ? v[g] : 0.f, zl = g == 0 ? zm : v[0], zh = g == 0 ? v[1] : zp;
        float a, b;
        if constexpr (SIG) {
          a = xy[g][0] * (q[-1] - o) + xy[g][1] * (q[1] - o);
          b = xy[g][2] * (q[-PX] - o) + xy[g][3] * (q[PX] - o);
          s[g] = (s[g] + a) + (b + (zf[g] * (zl - o) + zf[g + 1] * (zh - o)));
        } else {
          a = w[2] * ((q[-1] - o) + (q[1] - o));
          b = w[1] * ((q[-PX] - o) + (q[PX] - o));
          s[g] = (s[g] + a) + (b + w[0] * ((zl - o) + (zh - o)));
        }
      }
    }
  }
  // v + om (f - A phi) / D, as (1 - om) v + (om / D) (f + neighbours)
  template <class T>
  __device__ __forceinline__ void sweep(const SubLevel<T> &L, const float *ph, const float (&f)[2], float om) {
    float s[2] = {f[0], f[1]};
    around(L, ph, s, false);
    v[0] = (1.f - om) * v[0] + (om * rd[0]) * s[0];
    v[1] = two ? (1.f - om) * v[1] + (om * rd[1]) * s[1] : 0.f;
  }
  __device__ __forceinline__ void sweep0(const float (&f)[2], float om) {
    v[0] = (om * rd[0]) * f[0];
    v[1] = two ? (om * rd[1]) * f[1] : 0.f;
  }
  // A phi - f, the 7-point forms difference by difference
  template <class T>
  __device__ __forceinline__ void residual(const SubLevel<T> &L, const float *ph, const float (&f)[2], float (&r)[2]) const {
    float s[2] = {0.f, 0.f};
    if constexpr (KIND == HFM_OP_K27) {
      s[0] = -(w[13] * v[0]);
      s[1] = -(w[13] * v[1]);
    }
    around(L, ph, s, true);
    r[0] = -s[0] - f[0];
    r[1] = -s[1] - f[1];
  }
};

// One sweep of a level's iterate `in` (null: zero) into `out`.
template <int KIND, bool NARROW, class T>
__device__ void prog_sweep(const SubLevel<T> &L, float *F, const float *in, float *out, float om) {
  const float *f = F + L.o_rhs, *Fc = F + L.o_face;
  const float *rd = Fc + sub_faces(L.Z, L.Y, L.X);
  const float rc = KIND == HFM_OP_SIGMA7 ? 0.f
                   : __fdividef(1.f, KIND == HFM_OP_K27 ? L.k[13] : 2.f * (L.k[0] + L.k[1] + L.k[2]));
  HFM_FOR_CELLS(L, F)
    const float r = KIND == HFM_OP_SIGMA7 ? rd[i] : rc;
    if (in) {
      float dg;
      const float ax = sub_apply<KIND, T>(L, in, Fc, q.z, q.y, q.x, q.ip, i, &dg);
      out[q.ip] = in[q.ip] + om * ((f[i] - ax) * r);
    } else {
      out[q.ip] = om * (f[i] * r);
    }
  }
  __syncthreads();
}

// The second phase of a restriction: each coarse cell's eight fine residuals (padded field,
// ordered z, y, x), averaged into the coarse level's right-hand side.
template <bool NARROW, class T>
__device__ void prog_sum8(const SubLevel<T> &L, float *F, const float *res, const SubLevel<T> &Lc) {
  __syncthreads();
  const int PX = L.X + 2, PXY = PX * (L.Y + 2);
  HFM_FOR_CELLS(Lc, F)
    const float *r = res + pix(2 * q.z, 2 * q.y, 2 * q.x, L.Y, L.X);
    float sum = 0.f;
#pragma unroll
    for (int c = 0; c < 8; ++c) sum += r[(c >> 2) * PXY + ((c >> 1) & 1) * PX + (c & 1)];
    F[Lc.o_rhs + i] = 0.125f * sum;
  }
  __syncthreads();
}

// Next level's right-hand side = R(A phi - f) (phi null: zero): every fine residual by its own
// thread into `res`, then the sums.
template <int KIND, bool NARROW, class T>
__device__ void prog_restrict(const SubLevel<T> &L, float *F, const float *ph, float *res,
                              const SubLevel<T> &Lc) {
  const float *f = F + L.o_rhs, *Fc = F + L.o_face;
  HFM_FOR_CELLS(L, F)
    float dg;
    const float ax = ph ? sub_apply<KIND, T>(L, ph, Fc, q.z, q.y, q.x, q.ip, i, &dg) : 0.f;
    res[q.ip] = ax - f[i];
  }
  prog_sum8<NARROW, T>(L, F, res, Lc);
}

// Next level's right-hand side = R f
template <bool NARROW, class T>
__device__ void prog_restrict_rhs(const SubLevel<T> &L, float *F, const SubLevel<T> &Lc) {
  const float *f = F + L.o_rhs;
  HFM_FOR_CELLS(Lc, F)
    const float *r = f + (2 * q.z * L.Y + 2 * q.y) * L.X + 2 * q.x;
    float sum = 0.f;
#pragma unroll
    for (int c = 0; c < 8; ++c) sum += 0.125f * r[((c >> 2) * L.Y + ((c >> 1) & 1)) * L.X + (c & 1)];
    F[Lc.o_rhs + i] = sum;
  }
  __syncthreads();
}

// phi = [phi] + sign * P(coarse) on the level's interior (both padded)
template <bool NARROW, class T>
__device__ void prog_correct(const SubLevel<T> &L, float *F, float *ph, const SubLevel<T> &Lc,
                             const float *coarse, float sign, bool zero) {
  HFM_FOR_CELLS(L, F)
    const float c = sign * coarse[pix(q.z >> 1, q.y >> 1, q.x >> 1, Lc.Y, Lc.X)];
    ph[q.ip] = zero ? c : ph[q.ip] + c;
  }
  __syncthreads();
}

// The coarsest level's sweeps of a 7-point operator, one cell per thread (a warp's chain of
// dependent instructions sets the time of these sweeps: 218 cycles for 64 cells on two warps,
// 456 in pairs on one warp).  Unrolled by two, so that each field's addresses are formed once.
template <int KIND, bool NARROW, class T>
__device__ __forceinline__ void coarse_cells7(const SubLevel<T> &L, float *F, float om, int sweeps, int nthr) {
  const int X = L.X, Y = L.Y, Z = L.Z, PX = X + 2, PXY = PX * (Y + 2), P = X * Y;
  const bool in = (int)threadIdx.x < L.n;
  const int i = in ? threadIdx.x : L.n - 1;
  const Cell q = cell_of<NARROW>(L, F, i);
  float c[6], od;
  if (KIND == HFM_OP_CONST7) {
    c[0] = c[1] = L.k[2];
    c[2] = c[3] = L.k[1];
    c[4] = c[5] = L.k[0];
    od = om * __fdividef(1.f, 2.f * (L.k[0] + L.k[1] + L.k[2]));
  } else {
    const float *fx = F + L.o_face, *fy = fx + Z * Y * (X + 1), *fz = fy + Z * (Y + 1) * X;
    const int ixf = i + q.z * Y + q.y, iyf = i + q.z * X;
    c[0] = fx[ixf];
    c[1] = fx[ixf + 1];
    c[2] = fy[iyf];
    c[3] = fy[iyf + X];
    c[4] = fz[i];
    c[5] = fz[i + P];
    od = om * (fz + (Z + 1) * P)[i];
  }
  const float f = F[L.o_rhs + i], keep = 1.f - om;
  float *p0 = F + L.o_phi + q.ip, *p1 = F + L.o_tmp + q.ip;
  float v = od * f;
  auto sweep = [&](const float *p, float *out) {
    if (nthr == 32) __syncwarp();
    else asm volatile("bar.sync 1, %0;" ::"r"(nthr) : "memory");
    const float a = f + c[0] * p[-1] + c[1] * p[1], b = c[2] * p[-PX] + c[3] * p[PX];
    v = keep * v + od * ((a + b) + (c[4] * p[-PXY] + c[5] * p[PXY]));
    if (in) *out = v;
  };
  if (in) *p1 = v;
  for (int k = 1; k < sweeps; k += 2) {
    sweep(p1, p0);
    if (k + 1 < sweeps) sweep(p0, p1);
  }
}

// `sweeps` sweeps from zero on the coarsest level; returns the buffer holding the result.
// Where the block has a thread for each cell (K27: for each pair of cells, whose 27 neighbours
// mostly coincide), coefficients stay in registers and a barrier among the warps that hold
// cells (a warp barrier when one does) parts the sweeps.
template <int KIND, bool NARROW, bool TOP, class T>
__device__ int prog_coarse(const SubLevel<T> &L, float *F, float om, int sweeps) {
  const int np = KIND == HFM_OP_K27 ? cell_pairs(L.Z, L.Y, L.X) : L.n;
  if (np > kProgThreads) {
    for (int k = 0; k < sweeps; ++k)
      prog_sweep<KIND, NARROW, T>(L, F, k == 0 ? nullptr : F + (k & 1 ? L.o_tmp : L.o_phi), F + (k & 1 ? L.o_phi : L.o_tmp), om);
    return sweeps & 1;
  }
  const int nthr = (np + 31) & ~31;
  if ((int)threadIdx.x < nthr) {
    if constexpr (KIND != HFM_OP_K27) {
      coarse_cells7<KIND, NARROW, T>(L, F, om, sweeps, nthr);
    } else {
      CellPair<KIND> c;
      c.load(L, F, threadIdx.x);
      if (!TOP) {  // left alone the compiler reads the weights anew in every sweep (6 x 10 x 14: 33.0, not 36.9 us)
#pragma unroll
        for (int j = 0; j < 27; ++j) asm volatile("" : "+f"(c.w[j]));
      }
      float f[2];
      c.rhs(L, F + L.o_rhs, f);
      c.sweep0(f, om);
      c.store(L, F + L.o_tmp, c.v);
      for (int k = 1; k < sweeps; ++k) {
        if (nthr == 32) __syncwarp();
        else asm volatile("bar.sync 1, %0;" ::"r"(nthr) : "memory");
        c.sweep(L, F + (k & 1 ? L.o_tmp : L.o_phi), f, om);
        c.store(L, F + (k & 1 ? L.o_phi : L.o_tmp), c.v);
      }
    }
  }
  __syncthreads();
  return sweeps & 1;
}

// Four consecutive values of T as float and back (16 or 8 bytes).
template <class T> __device__ __forceinline__ void ldq4(const T *p, float (&v)[4]) {
  if constexpr (sizeof(T) == 4) {
    const float4 m = *reinterpret_cast<const float4 *>(p);
    v[0] = m.x; v[1] = m.y; v[2] = m.z; v[3] = m.w;
  } else {
    const uint2 u = *reinterpret_cast<const uint2 *>(p);
    const T *h = reinterpret_cast<const T *>(&u);
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] = St<T>::to(h[e]);
  }
}
template <class T> __device__ __forceinline__ void stq4(T *p, const float (&v)[4]) {
  if constexpr (sizeof(T) == 4) {
    *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
  } else {
    T h[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) h[e] = St<T>::from(v[e]);
    *reinterpret_cast<uint2 *>(p) = *reinterpret_cast<const uint2 *>(h);
  }
}

// A thread's pair of quads of level l0: cells x0 .. x0 + 3 of row y in planes z and z + 1 (z
// even; the second one outside the grid when Z is odd and z the last plane).  Fields are
// [Z + 2][Y + 2][X], the ghost rows and planes zero; `ip` is the first quad's first cell.
// A sweep is evaluated as p = (1 - om) p + (om / D) (f + S) with S the neighbours times their
// coefficients (8 operations a cell; forming f - A p difference by difference takes 15, and
// a sweep was bound by the issue of those); the residuals that are restricted keep the
// differences.
template <int KIND> struct TopPair {
  static constexpr bool SIG = KIND == HFM_OP_SIGMA7;
  int ip, ic;       // the first cell in the fields, its parent in the next level's padded field
  bool valid, two;  // holds cells; in both planes
  bool first, last;  // the quad starts / ends its row
  float f[2][4], p[2][4];
  // SIGMA7: x faces of each quad, y faces below / above, z faces below, between and above,
  // omega / diagonal
  float ax[2][SIG ? 5 : 1], ay[2][2][SIG ? 4 : 1], az[3][SIG ? 4 : 1], od[2][SIG ? 4 : 1];

  // neighbours across the ends of a quad's row values v (r: the row in the field)
  template <class T>
  __device__ __forceinline__ void ends(const SubLevel<T> &L, const float *r, const float (&v)[4], float &l, float &h) const {
    l = __shfl_up_sync(0xffffffffu, v[3], 1);
    h = __shfl_down_sync(0xffffffffu, v[0], 1);
    if (128 % L.X) {  // rows continue in the next warp
      const int lane = threadIdx.x & 31;
      if (lane == 0 && !first) l = r[-1];
      if (lane == 31 && !last) h = r[4];
    }
    l = first ? 0.f : l;
    h = last ? 0.f : h;
  }
  struct Around {  // the rows around the pair
    float zm[4], zp[4], ym[2][4], yp[2][4], l[2], h[2];
  };
  template <class T> __device__ __forceinline__ void gather(const SubLevel<T> &L, const float *ph, Around &n) const {
    const float *c = ph + ip;
    const int X = L.X, PZ = (L.Y + 2) * X;
    ldq4<float>(c - PZ, n.zm);
    ldq4<float>(two ? c + 2 * PZ : c + PZ, n.zp);
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      ldq4<float>(c + g * PZ - X, n.ym[g]);
      ldq4<float>(c + g * PZ + X, n.yp[g]);
      ends(L, c + g * PZ, p[g], n.l[g], n.h[g]);
    }
  }
  // K27: s -= the 26 neighbours times their weights
  template <class T>
  __device__ __forceinline__ void around27(const SubLevel<T> &L, const float *ph, float (&s)[2][4]) const {
    const float *c = ph + ip;
    const int X = L.X, PZ = (L.Y + 2) * X;
#pragma unroll
    for (int a = 0; a < 4; ++a)  // planes z - 1 .. z + 2
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        // past the ghost plane (second quad outside): its sums are never used
        const float *r = c + ((a == 3 && !two ? 2 : a) - 1) * PZ + (b - 1) * X;
        float m[4], l, h;
        ldq4<float>(r, m);
        ends(L, r, m, l, h);
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          const int k = a - g;  // plane k of quad g's stencil
          if (k < 0 || k > 2) continue;
          const float k0 = L.k[9 * k + 3 * b], k1 = L.k[9 * k + 3 * b + 1], k2 = L.k[9 * k + 3 * b + 2];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            s[g][e] -= k0 * (e == 0 ? l : m[e - 1]);
            if (k != 1 || b != 1) s[g][e] -= k1 * m[e];
            s[g][e] -= k2 * (e == 3 ? h : m[e + 1]);
          }
        }
      }
  }
  template <class T>
  __device__ __forceinline__ void sweep(const SubLevel<T> &L, const float *ph, float om) {
    float s[2][4];
#pragma unroll
    for (int g = 0; g < 2; ++g)
#pragma unroll
      for (int e = 0; e < 4; ++e) s[g][e] = f[g][e];
    if constexpr (KIND == HFM_OP_K27) {
      around27(L, ph, s);
    } else {
      Around n;
      gather(L, ph, n);
#pragma unroll
      for (int g = 0; g < 2; ++g)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float xm = e == 0 ? n.l[g] : p[g][e - 1], xp = e == 3 ? n.h[g] : p[g][e + 1];
          const float zl = g == 0 ? n.zm[e] : p[0][e], zh = g == 0 ? p[1][e] : n.zp[e];
          if constexpr (KIND == HFM_OP_CONST7) {
            const float kz = L.k[0], ky = L.k[1], kx = L.k[2];
            s[g][e] += kz * (zl + zh);
            s[g][e] += ky * (n.ym[g][e] + n.yp[g][e]);
            s[g][e] += kx * (xm + xp);
          } else {
            s[g][e] += az[g][e] * zl;
            s[g][e] += az[g + 1][e] * zh;
            s[g][e] += ay[g][0][e] * n.ym[g][e];
            s[g][e] += ay[g][1][e] * n.yp[g][e];
            s[g][e] += ax[g][e] * xm;
            s[g][e] += ax[g][e + 1] * xp;
          }
        }
    }
    const float keep = 1.f - om;
#pragma unroll
    for (int g = 0; g < 2; ++g)
#pragma unroll
      for (int e = 0; e < 4; ++e) p[g][e] = keep * p[g][e] + odiag(L, g, e, om) * s[g][e];
  }
  template <class T> __device__ __forceinline__ float odiag(const SubLevel<T> &L, int g, int e, float om) const {
    if constexpr (SIG) return od[g][e];
    return om * __fdividef(1.f, KIND == HFM_OP_K27 ? L.k[13] : 2.f * (L.k[0] + L.k[1] + L.k[2]));
  }
  // r = A phi - f
  template <class T>
  __device__ __forceinline__ void residual(const SubLevel<T> &L, const float *ph, float (&r)[2][4]) const {
    if constexpr (KIND == HFM_OP_K27) {
#pragma unroll
      for (int g = 0; g < 2; ++g)
#pragma unroll
        for (int e = 0; e < 4; ++e) r[g][e] = -(L.k[13] * p[g][e]);
      around27(L, ph, r);
#pragma unroll
      for (int g = 0; g < 2; ++g)
#pragma unroll
        for (int e = 0; e < 4; ++e) r[g][e] = -r[g][e] - f[g][e];
    } else {
      Around n;
      gather(L, ph, n);
#pragma unroll
      for (int g = 0; g < 2; ++g)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float xm = e == 0 ? n.l[g] : p[g][e - 1], xp = e == 3 ? n.h[g] : p[g][e + 1];
          const float zl = g == 0 ? n.zm[e] : p[0][e], zh = g == 0 ? p[1][e] : n.zp[e], q = p[g][e];
          if constexpr (KIND == HFM_OP_CONST7) {
            const float kz = L.k[0], ky = L.k[1], kx = L.k[2], d = 2.f * (kz + ky + kx);
            r[g][e] = d * q - kz * (zl + zh) - ky * (n.ym[g][e] + n.yp[g][e]) - kx * (xm + xp) - f[g][e];
          } else {
            r[g][e] = ax[g][e] * (q - xm) + ax[g][e + 1] * (q - xp) + ay[g][0][e] * (q - n.ym[g][e]) +
                      ay[g][1][e] * (q - n.yp[g][e]) + az[g][e] * (q - zl) + az[g + 1][e] * (q - zh) - f[g][e];
          }
        }
    }
  }
  // x pairs of both planes' values: what the restriction adds up of this pair
  __device__ __forceinline__ void pairs(const float (&r)[2][4], float *out) const {
    if (two)
      *reinterpret_cast<float2 *>(out + 2 * threadIdx.x) =
          make_float2((r[0][0] + r[0][1]) + (r[1][0] + r[1][1]), (r[0][2] + r[0][3]) + (r[1][2] + r[1][3]));
  }
  template <class T> __device__ __forceinline__ void store(const SubLevel<T> &L, float *ph) const {
    if (valid) *reinterpret_cast<float4 *>(ph + ip) = make_float4(p[0][0], p[0][1], p[0][2], p[0][3]);
    if (two) *reinterpret_cast<float4 *>(ph + ip + (L.Y + 2) * L.X) = make_float4(p[1][0], p[1][1], p[1][2], p[1][3]);
  }
  // Index in an unpadded field of the level (plane z + 1: X Y further); 0 without cells.
  template <class T> static __device__ __forceinline__ int place(const SubLevel<T> &L, int &x0, int &y, int &z) {
    const int nvx = L.X >> 2, np = ((L.Z + 1) >> 1) * L.Y * nvx;
    const int q = (int)threadIdx.x < np ? threadIdx.x : 0, t = q / nvx;
    x0 = 4 * (q - t * nvx);
    y = t % L.Y;
    z = 2 * (t / L.Y);
    return (z * L.Y + y) * L.X + x0;
  }
  // Threads of warps without cells stay out (the shuffles need whole warps of the others).
  template <class T> static __device__ __forceinline__ bool working(const SubLevel<T> &L) {
    return (int)(threadIdx.x & ~31u) < ((L.Z + 1) >> 1) * L.Y * (L.X >> 2);
  }
  template <class T> __device__ __forceinline__ void load(const SubLevel<T> &L, const T *src, float (&v)[2][4]) const {
    int x0, y, z;
    const int i = place(L, x0, y, z);
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      if (g == 0 ? valid : two) {
        ldq4<T>(src + i + g * L.X * L.Y, v[g]);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) v[g][e] = 0.f;
      }
    }
  }
  template <class T>
  __device__ __forceinline__ void init(const SubLevel<T> &L, const SubLevel<T> &Lc, int64_t inst, const T *rhs, float om) {
    const int X = L.X, Y = L.Y, Z = L.Z, P = X * Y;
    int x0, y, z;
    const int i = place(L, x0, y, z);
    valid = (int)threadIdx.x < ((Z + 1) >> 1) * Y * (X >> 2);
    two = valid && z + 1 < Z;
    first = x0 == 0;
    last = x0 + 4 == X;
    ip = ((z + 1) * (Y + 2) + (y + 1)) * X + x0;
    ic = pix(z >> 1, y >> 1, x0 >> 1, Lc.Y, Lc.X);
    const int64_t i0 = inst * (int64_t)L.n + i;
    load<T>(L, rhs + inst * (int64_t)L.n, f);
#pragma unroll
    for (int g = 0; g < 2; ++g)
#pragma unroll
      for (int e = 0; e < 4; ++e) p[g][e] = 0.f;
    if constexpr (SIG) {
      float c[4], lo[4], hi[4];
      const T *sz = L.sz + i0;
      ldq4<T>(sz, c);
      ldq4<T>(z > 0 ? sz - P : sz, lo);
      ldq4<T>(z + 1 < Z ? sz + P : sz, hi);
#pragma unroll
      for (int e = 0; e < 4; ++e) {  // at a wall the cell's own conductivity: (s + s) / 2 = s
        az[0][e] = L.cz * (0.5f * (c[e] + lo[e]));
        az[1][e] = L.cz * (0.5f * (c[e] + hi[e]));
      }
      ldq4<T>(z + 2 < Z ? sz + 2 * P : (z + 1 < Z ? sz + P : sz), c);
#pragma unroll
      for (int e = 0; e < 4; ++e) az[2][e] = L.cz * (0.5f * (hi[e] + c[e]));
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        const int64_t k = i0 + (z + g < Z ? g * P : 0);
        const T *sx = L.sx + k, *sy = L.sy + k;
        ldq4<T>(sx, c);
        ax[g][0] = L.cx * (0.5f * (c[0] + St<T>::to(sx[first ? 0 : -1])));
        ax[g][4] = L.cx * (0.5f * (c[3] + St<T>::to(sx[last ? 3 : 4])));
#pragma unroll
        for (int e = 1; e < 4; ++e) ax[g][e] = L.cx * (0.5f * (c[e] + c[e - 1]));
        ldq4<T>(sy, c);
        ldq4<T>(y > 0 ? sy - X : sy, lo);
        ldq4<T>(y + 1 < Y ? sy + X : sy, hi);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          ay[g][0][e] = L.cy * (0.5f * (c[e] + lo[e]));
          ay[g][1][e] = L.cy * (0.5f * (c[e] + hi[e]));
          od[g][e] = om * __fdividef(1.f, ax[g][e] + ax[g][e + 1] + ay[g][0][e] + ay[g][1][e] + az[g][e] + az[g + 1][e]);
        }
      }
    }
  }
};

template <int KIND, class T, bool TOP, bool NARROW>
__global__ void __launch_bounds__(kProgThreads) k_subprog(const __grid_constant__ SubProgram<T> P) {
  const SubArgs<T> &a = P.a;
  const int64_t inst = blockIdx.x;
  if (a.active && !a.active[inst]) return;
  extern __shared__ __align__(16) unsigned char sub_smem[];
  float *F = reinterpret_cast<float *>(sub_smem);
  const int nl = a.nlev;
  const SubLevel<T> &L0 = a.lv[0];
  // the cells of the shared-memory levels as one list, the coarsest first: a thread's first
  // cell is loaded, then its quads; meanwhile the block clears its shared memory (the ghosts
  // of the fields stay zero)
  constexpr int LB = TOP ? 1 : 0;
  CellInit<KIND, T, NARROW> ci;
  int l = nl - 1, first = 0;
  int k = threadIdx.x;
  auto find = [&]() {
    while (l >= LB && k >= first + a.lv[l].n) first += a.lv[l--].n;
    return l >= LB;
  };
  bool more = find();
  if (more) ci.load(a.lv[l], inst, k - first);
  for (int i = threadIdx.x; i < P.clear; i += kProgThreads) reinterpret_cast<float4 *>(F)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  TopPair<KIND> tp;
  if (TOP) tp.template init<T>(L0, a.lv[1], inst, a.rhs, a.omega);
  __syncthreads();
  while (more) {
    ci.store(a.lv[l], F);
    k += kProgThreads;
    more = find();
    if (more) ci.load(a.lv[l], inst, k - first);
  }
  if (!TOP)
    for (int i = threadIdx.x; i < L0.n; i += kProgThreads) F[L0.o_rhs + i] = St<T>::to(a.rhs[inst * (int64_t)L0.n + i]);
  __syncthreads();
  const SubLevel<T> &L1 = a.lv[1];
  const bool mid = nl > 2 && cell_pairs(L1.Z, L1.Y, L1.X) <= kProgThreads;  // level 1 in registers
  CellPair<KIND> mc;
  if (mid) mc.load(L1, F, threadIdx.x);
  if (P.phi0) {  // the given iterate of l0, in its first field
    const T *src = P.phi0 + inst * (int64_t)L0.n;
    if (TOP) {
      tp.template load<T>(L0, src, tp.p);
      tp.store(L0, F + L0.o_phi);
    } else {
      HFM_FOR_CELLS(L0, F)
        F[L0.o_phi + q.ip] = St<T>::to(src[i]);
      }
    }
    __syncthreads();
  }
  unsigned cur = 0;  // bit l: level l's iterate is in tmp
  for (int s = 0; s < P.nsteps; ++s) {
    const int op = P.op[s], cnt = P.cnt[s];
    l = P.lev[s];
    const SubLevel<T> &L = a.lv[l];
    const SubLevel<T> &Lc = a.lv[l + 1 < nl ? l + 1 : l];
    const int c = (cur >> l) & 1;
    float *ph = F + (c ? L.o_tmp : L.o_phi);    // the iterate
    float *other = F + (c ? L.o_phi : L.o_tmp);
    float *coarse = F + (((cur >> (l + 1)) & 1) ? Lc.o_tmp : Lc.o_phi);
    if (op == SO_COARSE) {
      const int r = prog_coarse<KIND, NARROW, TOP, T>(L, F, a.coarse_omega, cnt);
      cur = (cur & ~(1u << l)) | ((unsigned)r << l);
    } else if (op == SO_SWEEP0 || op == SO_SWEEP) {
      for (int n = 0; n < cnt; ++n) {
        const bool zero = op == SO_SWEEP0 && n == 0;
        if (TOP && l == 0) {
          if (tp.working(L0)) {
            if (zero) {
#pragma unroll
              for (int g = 0; g < 2; ++g)
#pragma unroll
                for (int e = 0; e < 4; ++e) tp.p[g][e] = tp.odiag(L0, g, e, a.omega) * tp.f[g][e];
            } else {
              tp.sweep(L0, ph, a.omega);
            }
            if (!tp.two) {  // the second quad is outside the grid
#pragma unroll
              for (int e = 0; e < 4; ++e) tp.p[1][e] = 0.f;
            }
            tp.store(L0, other);
          }
          __syncthreads();
        } else if (mid && l == 1) {
          if (mc.valid) {
            float f[2];
            mc.rhs(L1, F + L1.o_rhs, f);
            if (zero) mc.sweep0(f, a.omega);
            else mc.sweep(L1, ph, f, a.omega);
            mc.store(L1, other, mc.v);
          }
          __syncthreads();
        } else {
          prog_sweep<KIND, NARROW, T>(L, F, zero ? nullptr : ph, other, a.omega);
        }
        float *t = ph;
        ph = other;
        other = t;
      }
      if (cnt & 1) cur ^= 1u << l;
    } else if (op == SO_RESTRICT || op == SO_RESTRICT0) {
      const bool zero = op == SO_RESTRICT0;
      if (TOP && l == 0) {
        float *pairs = F + P.o_top;
        if (tp.working(L0)) {
          float r[2][4];
          if (zero) {
#pragma unroll
            for (int g = 0; g < 2; ++g)
#pragma unroll
              for (int e = 0; e < 4; ++e) r[g][e] = -tp.f[g][e];
          } else {
            tp.residual(L0, ph, r);
          }
          tp.pairs(r, pairs);
        }
        __syncthreads();
        const int Xh = L.X >> 1;
        HFM_FOR_CELLS(Lc, F)
          const float *r = pairs + (q.z * L.Y + 2 * q.y) * Xh + q.x;
          F[Lc.o_rhs + i] = 0.125f * (r[0] + r[Xh]);
        }
        __syncthreads();
      } else if (mid && l == 1) {
        if (mc.valid) {
          float f[2], r[2];
          mc.rhs(L1, F + L1.o_rhs, f);
          if (zero) {
            r[0] = -f[0];
            r[1] = -f[1];
          } else {
            mc.residual(L1, ph, f, r);
          }
          mc.store(L1, other, r);
        }
        prog_sum8<NARROW, T>(L1, F, other, Lc);
      } else {
        prog_restrict<KIND, NARROW, T>(L, F, zero ? nullptr : ph, other, Lc);
      }
    } else if (op == SO_RESTRICT_RHS) {
      if (TOP && l == 0) {
        float *pairs = F + P.o_top;
        tp.pairs(tp.f, pairs);
        __syncthreads();
        const int Xh = L.X >> 1;
        HFM_FOR_CELLS(Lc, F)
          const float *r = pairs + (q.z * L.Y + 2 * q.y) * Xh + q.x;
          F[Lc.o_rhs + i] = 0.125f * (r[0] + r[Xh]);
        }
        __syncthreads();
      } else {
        prog_restrict_rhs<NARROW, T>(L, F, Lc);
      }
    } else {  // SO_CORRECT0, SO_CORRECT, SO_PROLONG
      const float sign = op == SO_PROLONG ? 1.f : -1.f;
      const bool zero = op != SO_CORRECT;
      if (TOP && l == 0) {
        if (tp.valid) {
          const float c0 = sign * coarse[tp.ic], c1 = sign * coarse[tp.ic + 1];
#pragma unroll
          for (int g = 0; g < 2; ++g)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float d = e < 2 ? c0 : c1;
              tp.p[g][e] = (g == 0 || tp.two) ? (zero ? d : tp.p[g][e] + d) : 0.f;
            }
          tp.store(L0, ph);
        }
        __syncthreads();
      } else if (mid && l == 1) {
        if (mc.valid) {
          const Cell q = cell_of<NARROW>(L1, F, mc.i);
          const float d = sign * coarse[pix(q.z >> 1, q.y >> 1, q.x >> 1, Lc.Y, Lc.X)];
          mc.v[0] = zero ? d : mc.v[0] + d;
          mc.v[1] = !mc.two ? 0.f : zero ? d : mc.v[1] + d;
          mc.store(L1, ph, mc.v);
        }
        __syncthreads();
      } else {
        prog_correct<NARROW, T>(L, F, ph, Lc, coarse, sign, zero);
      }
    }
  }
  T *out = a.out + inst * (int64_t)L0.n;
  if (TOP) {
    int x0, y, z;
    const int i = tp.place(L0, x0, y, z);
    if (tp.valid) stq4<T>(out + i, tp.p[0]);
    if (tp.two) stq4<T>(out + i + L0.X * L0.Y, tp.p[1]);
  } else {
    const float *res = F + ((cur & 1) ? L0.o_tmp : L0.o_phi);
    HFM_FOR_CELLS(L0, F)
      out[i] = St<T>::from(res[q.ip]);
    }
  }
  for (l = 1; l < nl; ++l) {
    const SubLevel<T> &L = a.lv[l];
    const float *res = F + (((cur >> l) & 1) ? L.o_tmp : L.o_phi);
    HFM_FOR_CELLS(L, F)
      P.g_rhs[l][inst * (int64_t)L.n + i] = St<T>::from(F[L.o_rhs + i]);
      P.g_phi[l][inst * (int64_t)L.n + i] = St<T>::from(res[q.ip]);
    }
  }
}

}  // namespace

size_t subcycle_smem_bytes(const Grid3 *g, int nlev, bool sigma) {
  size_t f = 0;
  for (int l = 0; l < nlev; ++l) {
    const int Z = g[l].Z, Y = g[l].Y, X = g[l].X, n = Z * Y * X;
    f += (size_t)2 * sub_padded(Z, Y, X) + n;
    if (sigma) f += (size_t)sub_faces(Z, Y, X) + n;
  }
  return ((f * 4 + 15) / 16) * 16;
}

// Shared-memory layout of the coarse-end cycle, level after level: phi and tmp (padded), rhs,
// and for SIGMA7 the face arrays and the diagonal.  Returns the bytes, 0 if they exceed the
// limit.
template <class T> size_t layout_sub(int kind, SubArgs<T> &a) {
  Grid3 g[kMaxSubLevels];
  int off = 0;
  for (int l = 0; l < a.nlev; ++l) {
    SubLevel<T> &L = a.lv[l];
    g[l] = Grid3{L.Z, L.Y, L.X};
    const int np = sub_padded(L.Z, L.Y, L.X);
    L.o_phi = off;
    L.o_tmp = off + np;
    L.o_rhs = off + 2 * np;
    L.o_face = L.o_rhs + L.n;
    off = L.o_face + (kind == HFM_OP_SIGMA7 ? sub_faces(L.Z, L.Y, L.X) + L.n : 0);
  }
  const size_t smem = subcycle_smem_bytes(g, a.nlev, kind == HFM_OP_SIGMA7);
  return smem > kSubcycleMaxSmem ? 0 : smem;
}

// ------------------------------------------------------------------ persistent small end
// Level l1 of a V-cycle and the coarse end below it in one launch.  A block takes work items
// in order from a global ticket: (step, instance, z tile) for the sweeps and the residual +
// restriction of level l1, (SUB, instance) for the coarse end, which runs in the block's
// shared memory exactly as in k_subprog.  Items are numbered step by step, so an item
// only waits for items with smaller numbers - items other running blocks have already taken
// - and the waits always end; each is still bounded (the wait budget), and one that runs out
// is counted in the device's wait-failure counters (the handle then ends its slots with
// HFM_ERR_TIMEOUT) and the item is skipped.  Iterates, the restricted residual and the
// correction written in this launch are read through L2; conductivities, 1 / diag and f are
// read-only here.

// Iterate source of a sweep of the persistent kernel: phi' = (src or 0) - P(wc), or the
// fused first sweep's phi1 = omega f / diag.
template <class T> struct SmallPhi {
  const T *base, *corr, *f, *invd;
  int64_t stride, cstride;
  int Yc, Xc;
  float omega;
  int pre2;
  __device__ __forceinline__ float operator()(int64_t inst, int z, int y, int x, int Y, int X) const {
    const int64_t i = inst * stride + ((int64_t)z * Y + y) * X + x;
    if (pre2) return omega * St<T>::ld(f + i) * St<T>::ld(invd + i);
    float v = base ? St<T>::to(ld_l2<T>(base + i)) : 0.f;
    if (corr) v -= St<T>::to(ld_l2<T>(corr + inst * cstride + ((int64_t)(z >> 1) * Yc + (y >> 1)) * Xc + (x >> 1)));
    return v;
  }
};

template <int KIND, class T>
__device__ void small_sweep(const SmallArgs<T> &a, int sidx, int64_t inst, int tile) {
  const int X = a.X, Y = a.Y, Z = a.Z;
  const int z0 = tile * a.zc, z1 = min(Z, z0 + a.zc);
  SmallPhi<T> ph;
  ph.base = a.src[sidx] >= 0 ? a.buf[a.src[sidx]] : nullptr;
  ph.corr = a.corr[sidx] ? a.sub.out : nullptr;
  ph.f = a.f;
  ph.invd = a.invd;
  ph.stride = a.n;
  ph.cstride = a.sub.lv[0].n;
  ph.Yc = a.sub.lv[0].Y;
  ph.Xc = a.sub.lv[0].X;
  ph.omega = a.om[sidx];
  ph.pre2 = a.kind[sidx] == SK_PRE2;
  T *out = a.buf[a.dst[sidx]] + inst * a.n;
  const float om = a.om[sidx];
  double acc = 0.0;
  const int64_t cells = (int64_t)(z1 - z0) * Y * X;
  for (int64_t k = threadIdx.x; k < cells; k += blockDim.x) {
    const int x = (int)(k % X);
    const int64_t t = k / X;
    const int y = (int)(t % Y), z = z0 + (int)(t / Y);
    float dg;
    const float ax = op_apply_at<KIND, T>(a.op, ph, inst, z, y, x, Z, Y, X, &dg);
    const int64_t i = ((int64_t)z * Y + y) * X + x;
    const float fv = St<T>::ld(a.f + inst * a.n + i);
    const float pc = ph(inst, z, y, x, Y, X);
    const float v = pc + om * __fdividef(fv - ax, dg);
    out[i] = St<T>::from(v);
    if (a.dot[sidx]) acc += (double)v * fv;
  }
  if (a.dot[sidx] && a.partials) {
    __shared__ double sh[32];
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
      double tot = 0.0;
      for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tot += sh[w];
      a.partials[inst * a.tiles + tile] = tot;
    }
  }
}

// r_c = R(A phi - f) for the coarse planes of z tile `tile` (zc even).
template <int KIND, class T>
__device__ void small_restrict(const SmallArgs<T> &a, int sidx, int64_t inst, int tile) {
  const int X = a.X, Y = a.Y, Z = a.Z;
  const SubLevel<T> &C = a.sub.lv[0];
  SmallPhi<T> ph;
  ph.base = a.src[sidx] >= 0 ? a.buf[a.src[sidx]] : nullptr;
  ph.corr = nullptr;
  ph.f = a.f;
  ph.invd = a.invd;
  ph.stride = a.n;
  ph.pre2 = 0;
  T *fc = const_cast<T *>(a.sub.rhs) + inst * (int64_t)C.n;
  const int c0 = tile * a.zc / 2, c1 = min(C.Z, (tile * a.zc + a.zc) / 2);
  const int64_t cells = (int64_t)(c1 - c0) * C.Y * C.X;
  for (int64_t k = threadIdx.x; k < cells; k += blockDim.x) {
    const int xc = (int)(k % C.X);
    const int64_t t = k / C.X;
    const int yc = (int)(t % C.Y), zcc = c0 + (int)(t / C.Y);
    float sum = 0.f;
#pragma unroll
    for (int aa = 0; aa < 2; ++aa)
#pragma unroll
      for (int bb = 0; bb < 2; ++bb)
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) {
          const int z = 2 * zcc + aa, y = 2 * yc + bb, x = 2 * xc + cc;
          float dg;
          const float ax = op_apply_at<KIND, T>(a.op, ph, inst, z, y, x, Z, Y, X, &dg);
          sum += 0.125f * (ax - St<T>::ld(a.f + inst * a.n + ((int64_t)z * Y + y) * X + x));
        }
    fc[((int64_t)zcc * C.Y + yc) * C.X + xc] = St<T>::from(sum);
  }
}

__device__ __forceinline__ int ld_acquire(const int *p) {
  int v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

template <int KIND, class T>
__global__ void __launch_bounds__(kSubThreads) k_small(const __grid_constant__ SmallArgs<T> a) {
  extern __shared__ __align__(16) unsigned char sub_smem[];
  __shared__ int item_sh, ok_sh;
  const int total = a.base[a.nsteps];
  for (;;) {
    if (threadIdx.x == 0) item_sh = atomicAdd(a.ticket, 1);
    __syncthreads();
    const int item = item_sh;
    if (item >= total) break;
    int s = 0;
    while (item >= a.base[s + 1]) ++s;
    const int cnt = a.kind[s] == SK_SUB ? 1 : a.tiles;
    const int local = item - a.base[s];
    const int64_t inst = local / cnt;
    const int tile = local % cnt;
    if (a.active && !a.active[inst]) {
      __syncthreads();  // item_sh is rewritten by the next take
      continue;
    }
    if (threadIdx.x == 0) {
      int ok = 1;
      if (a.need[s] > 0) {
        ok = 0;
        for (int i = 0; i < a.wait_budget; ++i)
          if (ld_acquire(a.done + inst) >= a.need[s]) {
            ok = 1;
            break;
          }
        if (!ok) atomicAdd(a.wait_fail, 1);
      }
      ok_sh = ok;
    }
    __syncthreads();
    if (ok_sh) {
      if (a.kind[s] == SK_SUB) subcycle_body<KIND, T>(a.sub, inst, sub_smem);
      else if (a.kind[s] == SK_RESTRICT) small_restrict<KIND, T>(a, s, inst, tile);
      else small_sweep<KIND, T>(a, s, inst, tile);
    }
    // publish: every thread's writes, then the instance's count
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) atomicAdd(a.done + inst, 1);
  }
}

template <int KIND, class T>
int go_small(const SmallArgs<T> &a, size_t smem, cudaStream_t s) {
  const void *fn = (const void *)k_small<KIND, T>;
  int st = set_max_dynamic_smem(fn, (int)kSubcycleMaxSmem, "cudaFuncSetAttribute(k_small)");
  if (st) return st;
  int per_sm = 0;
  HFM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kSubThreads, smem));
  if (per_sm < 1) per_sm = 1;
  const int total = a.base[a.nsteps];
  const int blocks = std::min(total, per_sm * sm_count());
  k_small<KIND, T><<<blocks, kSubThreads, smem, s>>>(a);
  HFM_CHECK_LAUNCH("k_small");
  return HFM_OK;
}

template <class T>
int launch_small(int kind, SmallArgs<T> a, int B, cudaStream_t s) {
  const size_t smem = layout_sub<T>(kind, a.sub);
  if (!smem) return fail(HFM_ERR_BAD_ARG, "small-level kernel: coarse levels exceed shared memory");
  (void)B;
  switch (kind) {
    case HFM_OP_SIGMA7: return go_small<HFM_OP_SIGMA7, T>(a, smem, s);
    case HFM_OP_CONST7: return go_small<HFM_OP_CONST7, T>(a, smem, s);
    case HFM_OP_K27: return go_small<HFM_OP_K27, T>(a, smem, s);
    default: return fail(HFM_ERR_UNSUPPORTED, "small-level kernel: operator kind");
  }
}

template int launch_small<float>(int, SmallArgs<float>, int, cudaStream_t);
template int launch_small<__nv_bfloat16>(int, SmallArgs<__nv_bfloat16>, int, cudaStream_t);
template int launch_small<__half>(int, SmallArgs<__half>, int, cudaStream_t);

template <int KIND, class T, bool TOP, bool NARROW>
int go_subprog(const SubProgram<T> &p, int B, size_t smem, cudaStream_t s) {
  int st = set_max_dynamic_smem((const void *)k_subprog<KIND, T, TOP, NARROW>, (int)kProgramMaxSmem,
                                "cudaFuncSetAttribute(k_subprog)");
  if (st) return st;
  k_subprog<KIND, T, TOP, NARROW><<<B, kProgThreads, smem, s>>>(p);
  HFM_CHECK_LAUNCH("k_subprog");
  return HFM_OK;
}

// The quad form of level l0: whole quads per row, at most one pair of quads per thread, and two
// rows and planes for its restriction to pair.
template <class T> bool program_top(const SubProgram<T> &p) {
  const SubLevel<T> &L = p.a.lv[0];
  return (L.X & 3) == 0 && L.Y > 1 && L.Z > 1 && ((L.Z + 1) >> 1) * L.Y * (L.X >> 2) <= kProgThreads;
}

// Shared-memory layout of a program: per level the fields, right-hand side and faces as
// layout_sub places them, then the cell table; the quad form of level l0 keeps two fields
// without x ghosts and the pair sums only.  Returns the bytes.
template <class T> size_t layout_program(int kind, SubProgram<T> &p, bool narrow) {
  const bool top = program_top(p);
  int64_t off = 0;
  for (int l = 0; l < p.a.nlev; ++l) {
    SubLevel<T> &q = p.a.lv[l];
    const int np = sub_padded(q.Z, q.Y, q.X);
    auto bits = [](int e) {
      int b = 0;
      while ((1 << b) < e) ++b;
      return b;
    };
    q.bx = bits(q.X);
    q.by = bits(q.Y);
    q.o_phi = (int)off;
    if (top && l == 0) {
      const int nt = (q.Z + 2) * (q.Y + 2) * q.X;
      q.o_tmp = nt;
      q.o_rhs = q.o_face = q.o_idx = p.o_top = 2 * nt;
      off = 2 * nt + ((q.Z + 1) >> 1) * q.Y * (q.X >> 1);
      continue;
    }
    q.o_tmp = (int)off + np;
    q.o_rhs = (int)off + 2 * np;
    q.o_face = q.o_rhs + q.n;
    off = q.o_face + (kind == HFM_OP_SIGMA7 ? sub_faces(q.Z, q.Y, q.X) + q.n : 0);
    off = (off + 1) & ~1;
    q.o_idx = (int)off;
    off = (off + (narrow ? 1 : 2) * q.n + 3) & ~3;
  }
  off = (off + 3) & ~3;
  p.clear = (int)(off / 4);
  return (size_t)off * 4;
}

// Lays the program out, with narrow cell tables where the wide ones do not fit.  Level l0 in
// quads always leaves room for wide ones.
template <class T> size_t place_program(int kind, SubProgram<T> &p, bool &narrow) {
  size_t smem = layout_program<T>(kind, p, narrow = false);
  if (smem > kProgramMaxSmem && !program_top(p)) smem = layout_program<T>(kind, p, narrow = true);
  return smem;
}

template <class T> bool subprogram_fits(int kind, SubProgram<T> &p) {
  bool narrow;
  return place_program<T>(kind, p, narrow) <= kProgramMaxSmem;
}

template <class T>
int launch_subprogram(int kind, SubProgram<T> &p, int B, cudaStream_t s) {
  bool narrow;
  const size_t smem = place_program<T>(kind, p, narrow);
  if (smem > kProgramMaxSmem) return fail(HFM_ERR_BAD_ARG, "subcycle: levels exceed shared memory");
  const bool top = program_top(p);
#define HFM_SUBPROG(KIND)                                                   \
  return top      ? go_subprog<KIND, T, true, false>(p, B, smem, s)         \
         : narrow ? go_subprog<KIND, T, false, true>(p, B, smem, s)         \
                  : go_subprog<KIND, T, false, false>(p, B, smem, s)
  switch (kind) {
    case HFM_OP_SIGMA7: HFM_SUBPROG(HFM_OP_SIGMA7);
    case HFM_OP_CONST7: HFM_SUBPROG(HFM_OP_CONST7);
    case HFM_OP_K27: HFM_SUBPROG(HFM_OP_K27);
    default: return fail(HFM_ERR_UNSUPPORTED, "subcycle: operator kind");
  }
#undef HFM_SUBPROG
}

template bool subprogram_fits<float>(int, SubProgram<float> &);
template bool subprogram_fits<__nv_bfloat16>(int, SubProgram<__nv_bfloat16> &);
template bool subprogram_fits<__half>(int, SubProgram<__half> &);
template int launch_subprogram<float>(int, SubProgram<float> &, int, cudaStream_t);
template int launch_subprogram<__nv_bfloat16>(int, SubProgram<__nv_bfloat16> &, int, cudaStream_t);
template int launch_subprogram<__half>(int, SubProgram<__half> &, int, cudaStream_t);

}  // namespace hfm
