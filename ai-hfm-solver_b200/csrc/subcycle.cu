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

// The coarse-end V-cycle of one instance with the block's shared memory `sub_smem`.  COH:
// the right-hand side was written by other blocks of the same launch (read through L2).
template <int KIND, class T, bool COH>
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
    const T *src = a.rhs + inst * (int64_t)a.lv[0].n + i;
    F[a.lv[0].o_rhs + i] = St<T>::to(COH ? ld_l2<T>(src) : *src);
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
// One block of 1024 threads per instance interprets a list of steps (V or F cycles from a
// zero or a given iterate, or the reference's sawtooth leg) over the levels from l0 down.  It
// is bound by the chain of barrier-separated passes on one SM, so each pass is made short:
//   * level l0 (TOP: rows of a multiple of 4 cells) belongs to the threads quad by quad: a
//     thread keeps its quad's right-hand side, face coefficients, 1 / diagonal and iterate in
//     registers for the whole launch, x neighbours come by shuffle, and a sweep reads four
//     16-byte rows (y and z neighbours) of unpadded-in-x fields, free of bank conflicts;
//   * the levels below run one cell per thread from shared memory; the restricted residual
//     forms every fine residual in its own thread and then sums eight;
//   * the coarsest level's sweeps keep each cell's coefficients in registers and synchronise
//     only the warps that hold cells.
// One instance of 16^3 .. 4^3 (SIGMA7 float32, V(2,2), 32 coarsest sweeps): 24 us a launch
// against 47 us for the eleven launches it replaces; in a served bf16 stream, beside other
// kernels, 34 us against 55 us for 512 threads with all fields and faces in padded shared
// arrays.  8 x 16 x 16 and 4 x 8 x 8 of the 27-point operator, the F-cycle's F and V visits
// in one launch: 35 us against 160 us launch by launch.
constexpr int kProgThreads = 1024;

// fc = R(A phi - f), in two phases: every fine residual by its own thread into `res` (padded,
// interior), then the eight of each coarse cell in the order z, y, x.
template <int KIND, class T>
__device__ void prog_restrict(const SubLevel<T> &L, const float *ph, const float *Fc, const float *f,
                              float *res, const SubLevel<T> &Lc, float *fc) {
  Walk w(threadIdx.x, blockDim.x, L.Y, L.X);
  for (int i = threadIdx.x; i < L.n; i += blockDim.x, w.step(L.Y, L.X)) {
    const int ip = pix(w.z, w.y, w.x, L.Y, L.X);
    float dg;
    const float ax = ph ? sub_apply<KIND, T>(L, ph, Fc, w.z, w.y, w.x, ip, i, &dg) : 0.f;
    res[ip] = ax - f[i];
  }
  __syncthreads();
  const int PX = L.X + 2, PXY = PX * (L.Y + 2);
  Walk v(threadIdx.x, blockDim.x, Lc.Y, Lc.X);
  for (int j = threadIdx.x; j < Lc.n; j += blockDim.x, v.step(Lc.Y, Lc.X)) {
    const float *q = res + pix(2 * v.z, 2 * v.y, 2 * v.x, L.Y, L.X);
    float sum = 0.f;
#pragma unroll
    for (int c = 0; c < 8; ++c) sum += q[(c >> 2) * PXY + ((c >> 1) & 1) * PX + (c & 1)];
    fc[j] = 0.125f * sum;
  }
  __syncthreads();
}

// fc = R f (f unpadded)
template <class T>
__device__ void prog_restrict_rhs(const SubLevel<T> &L, const float *f, const SubLevel<T> &Lc, float *fc) {
  Walk v(threadIdx.x, blockDim.x, Lc.Y, Lc.X);
  for (int j = threadIdx.x; j < Lc.n; j += blockDim.x, v.step(Lc.Y, Lc.X)) {
    const float *q = f + (2 * v.z * L.Y + 2 * v.y) * L.X + 2 * v.x;
    float sum = 0.f;
#pragma unroll
    for (int c = 0; c < 8; ++c) sum += 0.125f * q[((c >> 2) * L.Y + ((c >> 1) & 1)) * L.X + (c & 1)];
    fc[j] = sum;
  }
  __syncthreads();
}

// phi = [phi] + sign * P(coarse) on the level's interior (both padded)
template <class T>
__device__ void prog_correct(const SubLevel<T> &L, float *ph, const SubLevel<T> &Lc, const float *coarse,
                             float sign, bool zero) {
  Walk w(threadIdx.x, blockDim.x, L.Y, L.X);
  for (int i = threadIdx.x; i < L.n; i += blockDim.x, w.step(L.Y, L.X)) {
    const int ip = pix(w.z, w.y, w.x, L.Y, L.X);
    const float c = sign * coarse[pix(w.z >> 1, w.y >> 1, w.x >> 1, Lc.Y, Lc.X)];
    ph[ip] = zero ? c : ph[ip] + c;
  }
  __syncthreads();
}

// `sweeps` sweeps from zero on the coarsest level; returns the buffer holding the result.
// Up to 1024 cells: one per thread, its coefficients in registers, a barrier among the warps
// that hold cells (a warp barrier when one does).
template <int KIND, class T>
__device__ int prog_coarse(const SubLevel<T> &L, float *F, float om, int sweeps) {
  float *buf[2] = {F + L.o_phi, F + L.o_tmp};
  const float *f = F + L.o_rhs, *Fc = F + L.o_face;
  const int n = L.n;
  if (n > (int)blockDim.x) {
    for (int k = 0; k < sweeps; ++k)
      sub_sweep<KIND, T>(L, k == 0 ? nullptr : buf[k & 1], Fc, f, buf[(k & 1) ^ 1], om, buf[k & 1]);
    return sweeps & 1;
  }
  const int nthr = (n + 31) & ~31;
  if ((int)threadIdx.x < nthr) {
    const int X = L.X, Y = L.Y, Z = L.Z, PX = X + 2, PXY = PX * (Y + 2);
    const int i = min((int)threadIdx.x, n - 1);
    const bool in = (int)threadIdx.x < n;
    const int x = i % X, t = i / X, y = t % Y, z = t / Y;
    const int ip = pix(z, y, x, Y, X);
    constexpr int NK = KIND == HFM_OP_K27 ? 27 : 6;
    float c[NK], rd;
    if (KIND == HFM_OP_K27) {
#pragma unroll
      for (int j = 0; j < NK; ++j) c[j] = L.k[j];
      rd = __fdividef(1.f, L.k[13]);
    } else if (KIND == HFM_OP_CONST7) {
      c[0] = c[1] = L.k[2];
      c[2] = c[3] = L.k[1];
      c[4] = c[5] = L.k[0];
      rd = __fdividef(1.f, 2.f * (L.k[0] + L.k[1] + L.k[2]));
    } else {
      const float *fx = Fc, *fy = fx + Z * Y * (X + 1), *fz = fy + Z * (Y + 1) * X, *dg = fz + (Z + 1) * Y * X;
      const int ixf = (z * Y + y) * (X + 1) + x, iyf = (z * (Y + 1) + y) * X + x;
      c[0] = fx[ixf];
      c[1] = fx[ixf + 1];
      c[2] = fy[iyf];
      c[3] = fy[iyf + X];
      c[4] = fz[i];
      c[5] = fz[i + X * Y];
      rd = __fdividef(1.f, dg[i]);
    }
    const float fv = f[i];
    float v = om * (fv * rd);
    if (in) buf[1][ip] = v;
    for (int k = 1; k < sweeps; ++k) {
      if (nthr == 32) __syncwarp();
      else asm volatile("bar.sync 1, %0;" ::"r"(nthr) : "memory");
      const float *p = buf[k & 1] + ip;
      float ax;
      if (KIND == HFM_OP_K27) {
        ax = 0.f;
#pragma unroll
        for (int j = 0; j < 27; ++j)
          if (c[j] != 0.f) ax += c[j] * p[(j / 9 - 1) * PXY + ((j / 3) % 3 - 1) * PX + (j % 3 - 1)];
      } else if (KIND == HFM_OP_CONST7) {
        ax = 2.f * (c[4] + c[2] + c[0]) * v - c[4] * (p[-PXY] + p[PXY]) - c[2] * (p[-PX] + p[PX]) -
             c[0] * (p[-1] + p[1]);
      } else {
        ax = c[0] * (v - p[-1]) + c[1] * (v - p[1]) + c[2] * (v - p[-PX]) + c[3] * (v - p[PX]) +
             c[4] * (v - p[-PXY]) + c[5] * (v - p[PXY]);
      }
      v += om * ((fv - ax) * rd);
      if (in) buf[(k & 1) ^ 1][ip] = v;
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

// A thread's quad of level l0 (quad form).  Fields are [Z + 2][Y + 2][X], the ghost rows and
// planes zero; `ip` is the quad's first cell in them.
template <int KIND> struct TopQuad {
  int x0, y, z, ip, X, Y, PZ;
  bool valid, work;  // holds cells; its warp does (the shuffles need whole warps)
  float f[4], p[4];
  // SIGMA7: x faces of the four cells, y and z faces below and above, 1 / diagonal
  float ax[KIND == HFM_OP_SIGMA7 ? 5 : 1], ay[2][KIND == HFM_OP_SIGMA7 ? 4 : 1],
      az[2][KIND == HFM_OP_SIGMA7 ? 4 : 1], rd[KIND == HFM_OP_SIGMA7 ? 4 : 1];

  // neighbours across the quad's ends of row values v (row base pointer r, in the grid)
  __device__ __forceinline__ void ends(const float *r, const float (&v)[4], float &l, float &h) const {
    l = __shfl_up_sync(0xffffffffu, v[3], 1);
    h = __shfl_down_sync(0xffffffffu, v[0], 1);
    const int lane = threadIdx.x & 31;
    if (lane == 0 && x0 > 0) l = r[-1];
    if (lane == 31 && x0 + 4 < X) h = r[4];
    if (x0 == 0) l = 0.f;
    if (x0 + 4 == X) h = 0.f;
  }
  template <class T>
  __device__ __forceinline__ void apply(const SubLevel<T> &L, const float *ph, float (&A)[4]) const {
    const float *c = ph + ip;
    if (KIND == HFM_OP_K27) {
#pragma unroll
      for (int e = 0; e < 4; ++e) A[e] = 0.f;
#pragma unroll
      for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) {
          const float *r = c + (a - 1) * PZ + (b - 1) * X;
          float m[4], l, h;
          if (a == 1 && b == 1) {
#pragma unroll
            for (int e = 0; e < 4; ++e) m[e] = p[e];
          } else {
            ldq4<float>(r, m);
          }
          ends(r, m, l, h);
          const float k0 = L.k[9 * a + 3 * b], k1 = L.k[9 * a + 3 * b + 1], k2 = L.k[9 * a + 3 * b + 2];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            A[e] += k0 * (e == 0 ? l : m[e - 1]);
            A[e] += k1 * m[e];
            A[e] += k2 * (e == 3 ? h : m[e + 1]);
          }
        }
      return;
    }
    float l, h, ym[4], yp[4], zm[4], zp[4];
    ldq4<float>(c - X, ym);
    ldq4<float>(c + X, yp);
    ldq4<float>(c - PZ, zm);
    ldq4<float>(c + PZ, zp);
    ends(c, p, l, h);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float xm = e == 0 ? l : p[e - 1], xp = e == 3 ? h : p[e + 1];
      if (KIND == HFM_OP_CONST7) {
        const float kz = L.k[0], ky = L.k[1], kx = L.k[2], d = 2.f * (kz + ky + kx);
        A[e] = d * p[e] - kz * (zm[e] + zp[e]) - ky * (ym[e] + yp[e]) - kx * (xm + xp);
      } else {
        A[e] = ax[e] * (p[e] - xm) + ax[e + 1] * (p[e] - xp) + ay[0][e] * (p[e] - ym[e]) +
               ay[1][e] * (p[e] - yp[e]) + az[0][e] * (p[e] - zm[e]) + az[1][e] * (p[e] - zp[e]);
      }
    }
  }
  template <class T> __device__ __forceinline__ float rdiag(const SubLevel<T> &L, int e) const {
    if (KIND == HFM_OP_SIGMA7) return rd[e];
    return __fdividef(1.f, KIND == HFM_OP_K27 ? L.k[13] : 2.f * (L.k[0] + L.k[1] + L.k[2]));
  }
  __device__ __forceinline__ void store(float *ph) const {
    if (valid) *reinterpret_cast<float4 *>(ph + ip) = make_float4(p[0], p[1], p[2], p[3]);
  }
  template <class T> __device__ void init(const SubLevel<T> &L, int64_t inst, const T *rhs) {
    X = L.X;
    Y = L.Y;
    PZ = (Y + 2) * X;
    const int nvx = X >> 2, nq = L.n >> 2, q = threadIdx.x;
    valid = q < nq;
    work = (q & ~31) < nq;
    const int qq = valid ? q : 0;
    const int t = qq / nvx;
    x0 = 4 * (qq - t * nvx);
    y = t % Y;
    z = t / Y;
    ip = (z + 1) * PZ + (y + 1) * X + x0;
    if (!valid) x0 = 0;
    const int64_t i = inst * (int64_t)L.n + 4 * qq;
    ldq4<T>(rhs + i, f);
#pragma unroll
    for (int e = 0; e < 4; ++e) p[e] = 0.f;
    if (KIND == HFM_OP_SIGMA7) {
      const T *sx = L.sx + i, *sy = L.sy + i, *sz = L.sz + i;
      const int P = X * Y;
      float c[4], lo[4], hi[4];
      ldq4<T>(sx, c);
      ax[0] = L.cx * (x0 > 0 ? 0.5f * (c[0] + St<T>::to(sx[-1])) : c[0]);
      ax[4] = L.cx * (x0 + 4 < X ? 0.5f * (c[3] + St<T>::to(sx[4])) : c[3]);
#pragma unroll
      for (int e = 1; e < 4; ++e) ax[e] = L.cx * (0.5f * (c[e] + c[e - 1]));
      ldq4<T>(sy, c);
      ldq4<T>(y > 0 ? sy - X : sy, lo);
      ldq4<T>(y + 1 < Y ? sy + X : sy, hi);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        ay[0][e] = L.cy * (0.5f * (c[e] + lo[e]));  // at a wall (s + s) / 2 = s
        ay[1][e] = L.cy * (0.5f * (c[e] + hi[e]));
      }
      ldq4<T>(sz, c);
      ldq4<T>(z > 0 ? sz - P : sz, lo);
      ldq4<T>(z + 1 < L.Z ? sz + P : sz, hi);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        az[0][e] = L.cz * (0.5f * (c[e] + lo[e]));
        az[1][e] = L.cz * (0.5f * (c[e] + hi[e]));
        rd[e] = __fdividef(1.f, ax[e] + ax[e + 1] + ay[0][e] + ay[1][e] + az[0][e] + az[1][e]);
      }
    }
  }
};

template <int KIND, class T, bool TOP>
__global__ void __launch_bounds__(kProgThreads) k_subprog(const __grid_constant__ SubProgram<T> P) {
  const SubArgs<T> &a = P.a;
  const int64_t inst = blockIdx.x;
  if (a.active && !a.active[inst]) return;
  extern __shared__ __align__(16) unsigned char sub_smem[];
  float *F = reinterpret_cast<float *>(sub_smem);
  const int nl = a.nlev;
  const SubLevel<T> &L0 = a.lv[0];
  TopQuad<KIND> tq;
  // both fields of every level zero (the ghosts stay so), face arrays, right-hand side of l0
  for (int l = 0; l < nl; ++l) {
    const SubLevel<T> &L = a.lv[l];
    for (int i = threadIdx.x; i < L.o_rhs - L.o_phi; i += kProgThreads) F[L.o_phi + i] = 0.f;
    if (KIND == HFM_OP_SIGMA7 && !(TOP && l == 0)) sub_faces_init<T>(L, inst, F + L.o_face);
  }
  if (TOP) {
    tq.template init<T>(L0, inst, a.rhs);
  } else {
    for (int i = threadIdx.x; i < L0.n; i += kProgThreads) F[L0.o_rhs + i] = St<T>::to(a.rhs[inst * (int64_t)L0.n + i]);
  }
  __syncthreads();
  if (P.phi0) {  // the given iterate of l0, in its first field
    const T *src = P.phi0 + inst * (int64_t)L0.n;
    if (TOP) {
      if (tq.valid) ldq4<T>(src + 4 * threadIdx.x, tq.p);
      tq.store(F + L0.o_phi);
    } else {
      Walk w(threadIdx.x, kProgThreads, L0.Y, L0.X);
      for (int i = threadIdx.x; i < L0.n; i += kProgThreads, w.step(L0.Y, L0.X))
        F[L0.o_phi + pix(w.z, w.y, w.x, L0.Y, L0.X)] = St<T>::to(src[i]);
    }
    __syncthreads();
  }
  unsigned cur = 0;  // bit l: level l's iterate is in tmp
  for (int s = 0; s < P.nsteps; ++s) {
    const int op = P.op[s], l = P.lev[s], cnt = P.cnt[s];
    const SubLevel<T> &L = a.lv[l];
    const SubLevel<T> &Lc = a.lv[l + 1 < nl ? l + 1 : l];
    const int c = (cur >> l) & 1;
    float *ph = F + (c ? L.o_tmp : L.o_phi);    // the iterate
    float *other = F + (c ? L.o_phi : L.o_tmp);
    float *coarse = F + (((cur >> (l + 1)) & 1) ? Lc.o_tmp : Lc.o_phi);
    if (op == SO_COARSE) {
      const int r = prog_coarse<KIND, T>(L, F, a.coarse_omega, cnt);
      cur = (cur & ~(1u << l)) | ((unsigned)r << l);
    } else if (TOP && l == 0) {
      if (op == SO_SWEEP0 || op == SO_SWEEP) {
        for (int k = 0; k < cnt; ++k) {
          if (tq.work) {
            if (op == SO_SWEEP0 && k == 0) {
#pragma unroll
              for (int e = 0; e < 4; ++e) tq.p[e] = a.omega * (tq.f[e] * tq.rdiag(L, e));
            } else {
              float A[4];
              tq.apply(L0, ph, A);
#pragma unroll
              for (int e = 0; e < 4; ++e) tq.p[e] += a.omega * ((tq.f[e] - A[e]) * tq.rdiag(L, e));
            }
            tq.store(other);
          }
          __syncthreads();
          float *t = ph;
          ph = other;
          other = t;
        }
        if (cnt & 1) cur ^= 1u;
      } else if (op == SO_RESTRICT || op == SO_RESTRICT0 || op == SO_RESTRICT_RHS) {
        // x pairs of the quad's residuals, then the four rows of each coarse cell
        float *pairs = F + P.o_top;
        const float scale = op == SO_RESTRICT_RHS ? -1.f : 1.f;  // r = A phi - f, or f itself
        if (tq.work) {
          float A[4] = {0.f, 0.f, 0.f, 0.f};
          if (op == SO_RESTRICT) tq.apply(L0, ph, A);
          if (tq.valid)
            *reinterpret_cast<float2 *>(pairs + 2 * threadIdx.x) =
                make_float2(scale * ((A[0] - tq.f[0]) + (A[1] - tq.f[1])),
                            scale * ((A[2] - tq.f[2]) + (A[3] - tq.f[3])));
        }
        __syncthreads();
        const int Xh = L.X >> 1;
        Walk v(threadIdx.x, kProgThreads, Lc.Y, Lc.X);
        for (int j = threadIdx.x; j < Lc.n; j += kProgThreads, v.step(Lc.Y, Lc.X)) {
          const float *q = pairs + (2 * v.z * L.Y + 2 * v.y) * Xh + v.x;
          const float *q1 = q + L.Y * Xh;
          F[Lc.o_rhs + j] = 0.125f * ((q[0] + q[Xh]) + (q1[0] + q1[Xh]));
        }
        __syncthreads();
      } else {  // SO_CORRECT0, SO_CORRECT, SO_PROLONG
        if (tq.valid) {
          const float sign = op == SO_PROLONG ? 1.f : -1.f;
          const int ic = pix(tq.z >> 1, tq.y >> 1, tq.x0 >> 1, Lc.Y, Lc.X);
          const float c0 = sign * coarse[ic], c1 = sign * coarse[ic + 1];
          const bool z0 = op != SO_CORRECT;
          tq.p[0] = z0 ? c0 : tq.p[0] + c0;
          tq.p[1] = z0 ? c0 : tq.p[1] + c0;
          tq.p[2] = z0 ? c1 : tq.p[2] + c1;
          tq.p[3] = z0 ? c1 : tq.p[3] + c1;
          tq.store(ph);
        }
        __syncthreads();
      }
    } else {
      const float *f = F + L.o_rhs, *Fc = F + L.o_face;
      if (op == SO_SWEEP0 || op == SO_SWEEP) {
        for (int k = 0; k < cnt; ++k) {
          sub_sweep<KIND, T>(L, op == SO_SWEEP0 && k == 0 ? nullptr : ph, Fc, f, other, a.omega, ph);
          float *t = ph;
          ph = other;
          other = t;
        }
        if (cnt & 1) cur ^= 1u << l;
      } else if (op == SO_RESTRICT || op == SO_RESTRICT0) {
        prog_restrict<KIND, T>(L, op == SO_RESTRICT0 ? nullptr : ph, Fc, f, other, Lc, F + Lc.o_rhs);
      } else if (op == SO_RESTRICT_RHS) {
        prog_restrict_rhs<T>(L, f, Lc, F + Lc.o_rhs);
      } else {
        prog_correct<T>(L, ph, Lc, coarse, op == SO_PROLONG ? 1.f : -1.f, op != SO_CORRECT);
      }
    }
  }
  T *out = a.out + inst * (int64_t)L0.n;
  if (TOP) {
    if (tq.valid) stq4<T>(out + 4 * threadIdx.x, tq.p);
  } else {
    const float *res = F + ((cur & 1) ? L0.o_tmp : L0.o_phi);
    Walk w(threadIdx.x, kProgThreads, L0.Y, L0.X);
    for (int i = threadIdx.x; i < L0.n; i += kProgThreads, w.step(L0.Y, L0.X))
      out[i] = St<T>::from(res[pix(w.z, w.y, w.x, L0.Y, L0.X)]);
  }
  if (P.store_all)
    for (int l = 1; l < nl; ++l) {
      const SubLevel<T> &L = a.lv[l];
      const float *res = F + (((cur >> l) & 1) ? L.o_tmp : L.o_phi);
      Walk w(threadIdx.x, kProgThreads, L.Y, L.X);
      for (int i = threadIdx.x; i < L.n; i += kProgThreads, w.step(L.Y, L.X)) {
        P.g_rhs[l][inst * (int64_t)L.n + i] = St<T>::from(F[L.o_rhs + i]);
        P.g_phi[l][inst * (int64_t)L.n + i] = St<T>::from(res[pix(w.z, w.y, w.x, L.Y, L.X)]);
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
// shared memory exactly as k_subcycle does.  Items are numbered step by step, so an item
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
      if (a.kind[s] == SK_SUB) subcycle_body<KIND, T, true>(a.sub, inst, sub_smem);
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

template <int KIND, class T, bool TOP>
int go_subprog(const SubProgram<T> &p, int B, size_t smem, cudaStream_t s) {
  int st = set_max_dynamic_smem((const void *)k_subprog<KIND, T, TOP>, (int)kSubcycleMaxSmem,
                                "cudaFuncSetAttribute(k_subprog)");
  if (st) return st;
  k_subprog<KIND, T, TOP><<<B, kProgThreads, smem, s>>>(p);
  HFM_CHECK_LAUNCH("k_subprog");
  return HFM_OK;
}

template <class T>
int launch_subprogram(int kind, SubProgram<T> &p, int B, cudaStream_t s) {
  const SubLevel<T> &L0 = p.a.lv[0];
  // the quad form: whole quads per row, and at most one quad per thread
  const bool top = (L0.X & 3) == 0 && L0.n <= 4 * kProgThreads;
  size_t smem = layout_sub<T>(kind, p.a);
  if (!smem) return fail(HFM_ERR_BAD_ARG, "subcycle: levels exceed shared memory");
  if (top) {  // level l0 keeps two fields without x ghosts and the pair sums; no faces
    SubLevel<T> &L = p.a.lv[0];
    const int np = (L.Z + 2) * (L.Y + 2) * L.X;
    L.o_phi = 0;
    L.o_tmp = np;
    L.o_rhs = L.o_face = 2 * np;
    p.o_top = 2 * np;
    int off = 2 * np + L.n / 2;
    for (int l = 1; l < p.a.nlev; ++l) {
      SubLevel<T> &q = p.a.lv[l];
      const int shift = off - q.o_phi;
      const int size = (l + 1 < p.a.nlev ? p.a.lv[l + 1].o_phi : (int)(smem / 4)) - q.o_phi;
      q.o_phi += shift;
      q.o_tmp += shift;
      q.o_rhs += shift;
      q.o_face += shift;
      off += size;
    }
    smem = (size_t)off * 4;
    if (smem > kSubcycleMaxSmem) return fail(HFM_ERR_BAD_ARG, "subcycle: levels exceed shared memory");
  }
  switch (kind) {
    case HFM_OP_SIGMA7:
      return top ? go_subprog<HFM_OP_SIGMA7, T, true>(p, B, smem, s) : go_subprog<HFM_OP_SIGMA7, T, false>(p, B, smem, s);
    case HFM_OP_CONST7:
      return top ? go_subprog<HFM_OP_CONST7, T, true>(p, B, smem, s) : go_subprog<HFM_OP_CONST7, T, false>(p, B, smem, s);
    case HFM_OP_K27:
      return top ? go_subprog<HFM_OP_K27, T, true>(p, B, smem, s) : go_subprog<HFM_OP_K27, T, false>(p, B, smem, s);
    default: return fail(HFM_ERR_UNSUPPORTED, "subcycle: operator kind");
  }
}

template int launch_subprogram<float>(int, SubProgram<float> &, int, cudaStream_t);
template int launch_subprogram<__nv_bfloat16>(int, SubProgram<__nv_bfloat16> &, int, cudaStream_t);
template int launch_subprogram<__half>(int, SubProgram<__half> &, int, cudaStream_t);

}  // namespace hfm
