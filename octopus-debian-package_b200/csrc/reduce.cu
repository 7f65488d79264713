// FP64 reductions over a batch: per-state norms and dot products, the
// overlap (Gram) matrix, its Cholesky factor and the triangular update that
// orthonormalises a batch, and the final reduction of the observables the
// stencil pass accumulates.  All sums are compensated (two-sum) and
// deterministic (fixed partial layout, fixed reduction order).
//
// Reference: X(mesh_batch_nrm2) / X(mesh_batch_dotp_vector) /
// X(mesh_batch_dotp_matrix) (src/grid/mesh_batch_inc.F90:20-263, 379-552,
// 970-1167) and the cholesky_serial branch of
// X(states_elec_orthogonalization_full) (src/states/states_elec_calc_inc.F90:66-98).
#include <algorithm>
#include <mutex>

#include "reduce.cuh"

namespace hpsi {

namespace {

template <typename T>
struct C2;
template <>
struct C2<double> {
  using type = double2;
};
template <>
struct C2<float> {
  using type = float2;
};

// ---------------------------------------------------------------------------
// per-state sums: grid (nblk, ceil(ld/SW)); block 256 = SW states x G row groups
// mode 0: sum |a|^2 -> q0 ; mode 1: sum conj(a) b -> (q0, q1)
template <typename T, int MODE>
__global__ void __launch_bounds__(256) state_sum_kernel(const T *a, long long lda, const T *b, long long ldb,
                                                       int np, int nst, double *partial) {
  using V = typename C2<T>::type;
  const int SW = min(nst - int(blockIdx.y) * 256, 256) > 0 ? min(nst - int(blockIdx.y) * 256, 256) : 1;
  const int G = 256 / SW;
  const int t = threadIdx.x;
  const int sl = t % SW, g = t / SW;
  const int s = blockIdx.y * 256 + sl;
  const long long rows_per = (np + gridDim.x - 1) / gridDim.x;
  const long long r0 = blockIdx.x * rows_per;
  const long long r1 = min((long long)np, r0 + rows_per);
  Kahan k0 = {0, 0}, k1 = {0, 0};
  if (g < G && s < nst) {
    for (long long r = r0 + g; r < r1; r += G) {
      const V x = reinterpret_cast<const V *>(a + r * 2 * lda)[s];
      if (MODE == 0) {
        kadd(k0, double(x.x) * double(x.x) + double(x.y) * double(x.y));
      } else {
        const V y = reinterpret_cast<const V *>(b + r * 2 * ldb)[s];
        kadd(k0, double(x.x) * double(y.x) + double(x.y) * double(y.y));
        kadd(k1, double(x.x) * double(y.y) - double(x.y) * double(y.x));
      }
    }
  }
  __shared__ double red[256][4];
  red[t][0] = k0.s;
  red[t][1] = k0.c;
  red[t][2] = k1.s;
  red[t][3] = k1.c;
  __syncthreads();
  if (t < SW && s < nst) {
    Kahan a0 = {0, 0}, a1 = {0, 0};
    for (int gg = 0; gg < G; ++gg) {
      const int u = gg * SW + t;
      kadd(a0, red[u][0]);
      a0.c += red[u][1];
      kadd(a1, red[u][2]);
      a1.c += red[u][3];
    }
    double *o = partial + ((long long)blockIdx.x * nst + s) * 4;
    o[0] = a0.s;
    o[1] = a0.c;
    o[2] = a1.s;
    o[3] = a1.c;
  }
}

// sum partial[nblk][nst][4] over blocks -> out[nst][2] (times scale)
__global__ void state_sum_finalize(const double *partial, int nblk, int nst, double scale, int sqrt_first,
                                   double *out) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nst) return;
  Kahan a0 = {0, 0}, a1 = {0, 0};
  for (int b = 0; b < nblk; ++b) {
    const double *p = partial + ((long long)b * nst + s) * 4;
    kadd(a0, p[0]);
    a0.c += p[1];
    kadd(a1, p[2]);
    a1.c += p[3];
  }
  double v0 = (a0.s + a0.c) * scale;
  if (sqrt_first) v0 = sqrt(v0);
  out[2 * s] = v0;
  out[2 * s + 1] = (a1.s + a1.c) * scale;
}

// ---------------------------------------------------------------------------
// Matrix products of a batch on the FP64 tensor cores (mma.sync.m8n8k4.f64)
// over the batch's real view (lane 2 s = re, 2 s + 1 = im of state s).  They
// run at the FP64 pipe's rate, like plain multiply-adds, but a fragment feeds
// 8 products per value read from shared memory: with 64 x 64 tiles (8 warps of
// 16 x 32) the FP64 pipe is the bound.  Sums stay FP64 for both storage types.
constexpr int GT = 64;   // tile edge (real lanes, rows)
constexpr int GK = 16;   // K step staged at once
constexpr int GST = 4;   // staged steps
constexpr int GFOLD = 8192 / GK;  // K steps summed before they are folded with compensation

__device__ __forceinline__ void dmma(double &d0, double &d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// One complex state (16 bytes FP64, 8 FP32; REALS: FP32 in two pieces of 4) to shared
// memory, zero where !ok.
template <bool REALS = false>
__device__ __forceinline__ void copy_state(double *d, const double *g, bool ok) {
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(d));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(g), "r"(ok ? 16 : 0));
}
template <bool REALS = false>
__device__ __forceinline__ void copy_state(float *d, const float *g, bool ok) {
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(d));
  if constexpr (REALS) {
#pragma unroll
    for (int i = 0; i < 2; ++i)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(s + 4 * i), "l"(g + i), "r"(ok ? 4 : 0));
  } else {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(g), "r"(ok ? 8 : 0));
  }
}
// Row pitch of a staged K x 64 block: the four K rows of a fragment read fall
// into different bank groups (FP64 pitch = 4 mod 16, FP32 = 8 mod 32).
template <typename T>
constexpr int gram_pitch() {
  return sizeof(T) == 8 ? GT + 4 : GT + 8;
}

// Two sums into the partials at `at`, their remainders (Kahan) into oc.
__device__ __forceinline__ void gram_fold(double *o, double *oc, long long at, bool first, const double (&c)[2]) {
  double2 &s = *reinterpret_cast<double2 *>(o + at), &r = *reinterpret_cast<double2 *>(oc + at);
  Kahan x = {0, 0}, y = {0, 0};
  if (!first) x = {s.x, r.x}, y = {s.y, r.y};
  kadd(x, c[0]);
  kadd(y, c[1]);
  s = make_double2(x.s, y.s);
  r = make_double2(x.c, y.c);
}

// Gram matrix of the real views: G[u][v] = sum_p Ar[p][u] Br[p][v], u, v over
// n = 2 nst lanes.  grid (tile pairs, splits over the points); block 256.
// sym: a is b, only the tiles on and above the diagonal are listed (the matrix
// is Hermitian).  Partials [splits][n][n].
// FOLD: for splits of more than 8192 points (many tiles: 3 splits for 512 states,
// one from 660 on): after every GFOLD steps the sums go into the partials with
// compensation, whose remainders follow them ([splits][n][n] again), so that no plain sum
// runs over more than 8192 points.
// 96 states, 267,761 points, FP64: 0.468 ms (one triangle; 78 % of the FP64 rate),
// the update below 0.50 ms; orthonormalisation and overlap together 9.5 -> 1.72 ms
// (before: 2 x 2 register blocks per thread over 32 x 32 tiles, one output of the
// update per thread).
// REALS: rows that start on 4-byte boundaries only (FP32 batches of width 1, the only
// ones whose alignment nothing checks).
template <typename T, bool FOLD, bool REALS = false>
__global__ void __launch_bounds__(256) gram_kernel(const T *a, long long lda, const T *b, long long ldb, int np,
                                                  int n, int tiles, int sym, double *partial) {
  constexpr int PITCH = gram_pitch<T>();
  extern __shared__ __align__(16) unsigned char gsm[];
  T *sa = reinterpret_cast<T *>(gsm);           // [GST][GK][PITCH]
  T *sb = sa + GST * GK * PITCH;
  int tu, tv;
  if (sym) {
    // pair index -> (row, column) of the upper triangle
    int r = 0, i = blockIdx.x;
    while (i >= tiles - r) i -= tiles - r++;
    tu = r;
    tv = r + i;
  } else {
    tu = blockIdx.x / tiles;
    tv = blockIdx.x % tiles;
  }
  const int u0 = tu * GT, v0 = tv * GT;
  const bool same = sym && tu == tv;  // one staged block serves both sides
  const long long per = (np + gridDim.y - 1) / gridDim.y;
  const long long p0 = blockIdx.y * per, p1 = min((long long)np, p0 + per);
  const int nk = p1 > p0 ? int((p1 - p0 + GK - 1) / GK) : 0;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int wu = (warp & 3) * 16, wv = (warp >> 2) * 32;
  auto stage = [&](int k) {
    if (k < nk) {
      const int s = k % GST;
      for (int i = t; i < GK * (GT / 2); i += 256) {
        const int pp = i / (GT / 2), l = 2 * (i % (GT / 2));
        const long long row = p0 + (long long)k * GK + pp;
        const bool in = row < p1;
        const bool ua = in && u0 + l < n, vb = in && v0 + l < n;
        copy_state<REALS>(sa + (s * GK + pp) * PITCH + l, ua ? a + row * 2 * lda + u0 + l : a, ua);
        if (!same) copy_state<REALS>(sb + (s * GK + pp) * PITCH + l, vb ? b + row * 2 * ldb + v0 + l : b, vb);
      }
    }
    cp_async_commit();
  };
  double c[2][4][2] = {};
  for (int k = 0; k < GST - 1; ++k) stage(k);
  for (int k = 0; k < nk; ++k) {
    if constexpr (FOLD) {
      if (k && k % GFOLD == 0) {
        double *o = partial + (long long)blockIdx.y * n * n, *oc = o + (long long)gridDim.y * n * n;
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int u = u0 + wu + 8 * i + (lane >> 2), v = v0 + wv + 8 * j + 2 * (lane & 3);
            if (u < n && v < n) gram_fold(o, oc, (long long)u * n + v, k == GFOLD, c[i][j]);
            c[i][j][0] = c[i][j][1] = 0.0;
          }
      }
    }
    cp_async_wait<GST - 2>();
    __syncthreads();
    stage(k + GST - 1);
    const T *xa = sa + (k % GST) * GK * PITCH, *xb = (same ? sa : sb) + (k % GST) * GK * PITCH;
#pragma unroll
    for (int kk = 0; kk < GK; kk += 4) {
      double fa[2], fb[4];
#pragma unroll
      for (int i = 0; i < 2; ++i) fa[i] = double(xa[(kk + (lane & 3)) * PITCH + wu + 8 * i + (lane >> 2)]);
#pragma unroll
      for (int j = 0; j < 4; ++j) fb[j] = double(xb[(kk + (lane & 3)) * PITCH + wv + 8 * j + (lane >> 2)]);
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) dmma(c[i][j][0], c[i][j][1], fa[i], fb[j]);
    }
  }
  cp_async_wait<0>();
  double *o = partial + (long long)blockIdx.y * n * n;
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int u = u0 + wu + 8 * i + (lane >> 2), v = v0 + wv + 8 * j + 2 * (lane & 3);
      if constexpr (FOLD) {
        if (u < n && v < n)
          gram_fold(o, o + (long long)gridDim.y * n * n, (long long)u * n + v, nk <= GFOLD, c[i][j]);
      } else {
        if (u < n && v < n) *reinterpret_cast<double2 *>(o + (long long)u * n + v) = make_double2(c[i][j][0], c[i][j][1]);
      }
    }
}

// S[i][j] = dV * (conj(a_i) . b_j) from the real Gram G (n = 2 * nst); sym:
// G holds the tiles on and above the diagonal, entries below it are conjugates.
// block (32, 8): 8 slices of the splits per entry, folded in a fixed order.
// FOLD: the partials' remainders follow them.
template <bool FOLD>
__global__ void __launch_bounds__(256) gram_finalize(const double *partial, int splits, int nst, double dv, int sym,
                                                     double *S) {
  __shared__ double red[8][32][4];
  const int i = blockIdx.y, j = blockIdx.x * 32 + threadIdx.x;
  const int n = 2 * nst;
  const bool flip = sym && 2 * i / GT > 2 * j / GT;
  const int r = flip ? j : i, q = flip ? i : j;
  Kahan re = {0, 0}, im = {0, 0};
  if (j < nst) {
#pragma unroll 4
    for (int z = threadIdx.y; z < splits; z += 8) {
      const double2 *G0 = reinterpret_cast<const double2 *>(partial + ((long long)z * n + 2 * r) * n) + q;
      const double2 g0 = G0[0], g1 = G0[nst];  // {rr, ri}, {ir, ii}
      kadd(re, g0.x);
      kadd(re, g1.y);
      kadd(im, g0.y);
      kadd(im, -g1.x);
      if constexpr (FOLD) {
        const double2 *R0 = G0 + (long long)splits * n * nst;
        re.c += R0[0].x + R0[nst].y;
        im.c += R0[0].y - R0[nst].x;
      }
    }
  }
  red[threadIdx.y][threadIdx.x][0] = re.s;
  red[threadIdx.y][threadIdx.x][1] = re.c;
  red[threadIdx.y][threadIdx.x][2] = im.s;
  red[threadIdx.y][threadIdx.x][3] = im.c;
  __syncthreads();
  if (threadIdx.y != 0 || j >= nst) return;
  for (int z = 1; z < 8; ++z) {
    kadd(re, red[z][threadIdx.x][0]);
    re.c += red[z][threadIdx.x][1];
    kadd(im, red[z][threadIdx.x][2]);
    im.c += red[z][threadIdx.x][3];
  }
  const double y = (im.s + im.c) * dv;
  S[2 * ((long long)i * nst + j)] = (re.s + re.c) * dv;
  S[2 * ((long long)i * nst + j) + 1] = flip ? -y : y;
}

// Cholesky S = U^H U (upper) and the inverse of U, one CTA, in global memory:
// for batches whose triangle does not fit shared memory.  S, U, Uinv are
// complex nst x nst row-major (interleaved).  err[0] = 1 if S is not
// positive definite.
__global__ void cholesky_inverse_kernel(const double *S, int nst, double *U, double *Uinv, int *err) {
  const int t = threadIdx.x;
  for (int i = t; i < nst * nst; i += blockDim.x) {
    U[2 * i] = U[2 * i + 1] = 0.0;
    Uinv[2 * i] = Uinv[2 * i + 1] = 0.0;
  }
  __syncthreads();
  __shared__ double djj;
  for (int j = 0; j < nst; ++j) {
    if (t == 0) {
      double d = S[2 * (j * nst + j)];
      for (int k = 0; k < j; ++k) {
        const double ur = U[2 * (k * nst + j)], ui = U[2 * (k * nst + j) + 1];
        d -= ur * ur + ui * ui;
      }
      if (!(d > 0.0)) {
        err[0] = 1;
        d = 1.0;
      }
      djj = sqrt(d);
      U[2 * (j * nst + j)] = djj;
    }
    __syncthreads();
    for (int i = j + 1 + t; i < nst; i += blockDim.x) {
      double sr = S[2 * (j * nst + i)], si = S[2 * (j * nst + i) + 1];
      for (int k = 0; k < j; ++k) {
        const double ar = U[2 * (k * nst + j)], ai = -U[2 * (k * nst + j) + 1];  // conj
        const double br = U[2 * (k * nst + i)], bi = U[2 * (k * nst + i) + 1];
        sr -= ar * br - ai * bi;
        si -= ar * bi + ai * br;
      }
      U[2 * (j * nst + i)] = sr / djj;
      U[2 * (j * nst + i) + 1] = si / djj;
    }
    __syncthreads();
  }
  // Uinv: solve U X = I column by column (thread per column)
  for (int c = t; c < nst; c += blockDim.x) {
    for (int i = c; i >= 0; --i) {
      double xr = (i == c) ? 1.0 : 0.0, xi = 0.0;
      for (int k = i + 1; k <= c; ++k) {
        const double ur = U[2 * (i * nst + k)], ui = U[2 * (i * nst + k) + 1];
        const double vr = Uinv[2 * (k * nst + c)], vi = Uinv[2 * (k * nst + c) + 1];
        xr -= ur * vr - ui * vi;
        xi -= ur * vi + ui * vr;
      }
      const double d = U[2 * (i * nst + i)];
      Uinv[2 * (i * nst + c)] = xr / d;
      Uinv[2 * (i * nst + c) + 1] = xi / d;
    }
  }
}

// The same in shared memory, the upper triangle packed by columns (entry
// (i, j), i <= j, at j (j + 1) / 2 + i): right-looking Cholesky, then the
// triangle inverted in place column by column.  A step's updates are spread
// over the CTA instead of one thread's chain of dependent global loads.
__global__ void __launch_bounds__(512) cholesky_inverse_smem_kernel(const double *S, int nst, double *U, double *Uinv,
                                                                   int *err) {
  extern __shared__ __align__(16) double2 M[];
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31, nw = blockDim.x >> 5;
  auto at = [](int i, int j) { return j * (j + 1) / 2 + i; };
  for (int j = warp; j < nst; j += nw)
    for (int i = lane; i <= j; i += 32)
      M[at(i, j)] = make_double2(S[2 * ((long long)i * nst + j)], S[2 * ((long long)i * nst + j) + 1]);
  __syncthreads();
  double2 *v = M + nst * (nst + 1) / 2;               // a new column of the inverse
  double *rinv = reinterpret_cast<double *>(v + nst);  // 1 / U(j, j)
  for (int j = 0; j < nst; ++j) {
    // one thread takes the root and the reciprocal (every warp's square root
    // would occupy the FP64 pipe for longer than the step's updates)
    if (t == 0) {
      double d = M[at(j, j)].x;
      if (!(d > 0.0)) {
        err[0] = 1;
        d = 1.0;
      }
      const double r = sqrt(d);
      M[at(j, j)] = make_double2(r, 0.0);
      rinv[j] = 1.0 / r;
    }
    __syncthreads();
    const double ri = rinv[j];
    for (int c = j + 1 + t; c < nst; c += blockDim.x) {
      double2 &x = M[at(j, c)];
      x.x *= ri;
      x.y *= ri;
    }
    __syncthreads();
    // trailing update: M(i, c) -= conj(U(j, i)) U(j, c)
    for (int c = j + 1 + warp; c < nst; c += nw) {
      const double2 b = M[at(j, c)];
      for (int i = j + 1 + lane; i <= c; i += 32) {
        const double2 a = M[at(j, i)];
        double2 &x = M[at(i, c)];
        x.x -= a.x * b.x + a.y * b.y;
        x.y -= a.x * b.y - a.y * b.x;
      }
    }
    __syncthreads();
  }
  for (int j = warp; j < nst; j += nw)
    for (int i = lane; i < nst; i += 32) {
      const double2 x = i <= j ? M[at(i, j)] : make_double2(0.0, 0.0);
      U[2 * ((long long)i * nst + j)] = x.x;
      U[2 * ((long long)i * nst + j) + 1] = x.y;
    }
  __syncthreads();
  // column j of the inverse: -X(0..j-1, 0..j-1) U(0..j-1, j) / U(j, j), X the
  // inverse of the leading block (four lanes per row: all rows at once)
  for (int j = 0; j < nst; ++j) {
    const double ri = rinv[j];
    for (int i0 = 0; i0 < j; i0 += blockDim.x / 4) {
      const int i = i0 + t / 4;
      double sr = 0.0, si = 0.0;
      if (i < j) {
#pragma unroll 4
        for (int k = i + (t & 3); k < j; k += 4) {
          const double2 x = M[at(i, k)], u = M[at(k, j)];
          sr += x.x * u.x - x.y * u.y;
          si += x.x * u.y + x.y * u.x;
        }
      }
#pragma unroll
      for (int o = 2; o > 0; o >>= 1) {
        sr += __shfl_xor_sync(0xffffffffu, sr, o);
        si += __shfl_xor_sync(0xffffffffu, si, o);
      }
      if (i < j && (t & 3) == 0) v[i] = make_double2(-sr * ri, -si * ri);
    }
    __syncthreads();
    for (int i = t; i < j; i += blockDim.x) M[at(i, j)] = v[i];
    if (t == 0) M[at(j, j)] = make_double2(ri, 0.0);
    __syncthreads();
  }
  for (int j = warp; j < nst; j += nw)
    for (int i = lane; i < nst; i += 32) {
      const double2 x = i <= j ? M[at(i, j)] : make_double2(0.0, 0.0);
      Uinv[2 * ((long long)i * nst + j)] = x.x;
      Uinv[2 * ((long long)i * nst + j) + 1] = x.y;
    }
}

// psi[p][j] <- sum_{i<=j} psi[p][i] Uinv[i][j], in place: a CTA owns 64 rows
// and takes the 64-lane column tiles from the last to the first, so that a
// tile is written only after every tile that reads it; per tile the rows times
// the real form of Uinv's columns (K up to the tile's end: the matrix is
// triangular) on the FP64 tensor cores.
template <typename T>
__global__ void __launch_bounds__(256) trsm_apply_kernel(T *psi, long long ld, int np, int nst,
                                                        const double *Uinv) {
  constexpr int APITCH = sizeof(T) == 8 ? GK + 4 : GK + 4;  // row pitch of the staged rows
  constexpr int WPITCH = GT + 4;
  extern __shared__ __align__(16) unsigned char gsm[];
  double *sw = reinterpret_cast<double *>(gsm);          // [2][GK][WPITCH]
  T *sx = reinterpret_cast<T *>(sw + 2 * GK * WPITCH);   // [GST][GT][APITCH]
  const int n = 2 * nst;
  const long long r0 = (long long)blockIdx.x * GT;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int wr = (warp & 3) * 16, wv = (warp >> 2) * 32;
  for (int v0 = (n - 1) / GT * GT; v0 >= 0; v0 -= GT) {
    const int kend = min(n, v0 + GT), nk = (kend + GK - 1) / GK;
    auto stage = [&](int k) {
      if (k < nk) {
        for (int i = t; i < GT * (GK / 2); i += 256) {
          const int rr = i / (GK / 2), l = 2 * (i % (GK / 2));
          const bool ok = r0 + rr < np && k * GK + l < kend;
          copy_state(sx + ((k % GST) * GT + rr) * APITCH + l, ok ? psi + (r0 + rr) * 2 * ld + k * GK + l : psi, ok);
        }
      }
      cp_async_commit();
    };
    // one complex entry of Uinv per thread and step: rows 2 i, 2 i + 1 of the
    // real form are {ur, ui}, {-ui, ur}
    const int wi = t / (GT / 2), wj = t % (GT / 2);
    auto entry = [&](int k) {
      const int i = k * (GK / 2) + wi, j = v0 / 2 + wj;
      return k < nk && i < nst && j < nst ? __ldg(reinterpret_cast<const double2 *>(Uinv) + (long long)i * nst + j)
                                          : make_double2(0.0, 0.0);
    };
    double c[2][4][2] = {};
    for (int k = 0; k < GST - 1; ++k) stage(k);
    double2 w = entry(0);
    for (int k = 0; k < nk; ++k) {
      double *swk = sw + (k & 1) * GK * WPITCH;
      *reinterpret_cast<double2 *>(swk + (2 * wi) * WPITCH + 2 * wj) = w;
      *reinterpret_cast<double2 *>(swk + (2 * wi + 1) * WPITCH + 2 * wj) = make_double2(-w.y, w.x);
      w = entry(k + 1);
      cp_async_wait<GST - 2>();
      __syncthreads();
      stage(k + GST - 1);
      const T *xk = sx + (k % GST) * GT * APITCH;
#pragma unroll
      for (int kk = 0; kk < GK; kk += 4) {
        double fa[2], fb[4];
#pragma unroll
        for (int i = 0; i < 2; ++i) fa[i] = double(xk[(wr + 8 * i + (lane >> 2)) * APITCH + kk + (lane & 3)]);
#pragma unroll
        for (int j = 0; j < 4; ++j) fb[j] = swk[(kk + (lane & 3)) * WPITCH + wv + 8 * j + (lane >> 2)];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) dmma(c[i][j][0], c[i][j][1], fa[i], fb[j]);
      }
    }
    cp_async_wait<0>();
    __syncthreads();  // every read of this tile's columns is done
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const long long row = r0 + wr + 8 * i + (lane >> 2);
        const int v = v0 + wv + 8 * j + 2 * (lane & 3);
        if (row < np && v < n) {
          typename C2<T>::type y;
          y.x = T(c[i][j][0]);
          y.y = T(c[i][j][1]);
          *reinterpret_cast<typename C2<T>::type *>(psi + row * 2 * ld + v) = y;
        }
      }
  }
}

// observables: partial [ncta][ld][3][2] -> out[3][nst] (energy, norm2, dipole) * dv,
// then the status word of the passes, so that one copy brings both to the host.
// One CTA per state: its threads take strided slices of the CTA partials
// (compensated sums), then fold them in shared memory.
__global__ void __launch_bounds__(128) obs_finalize_kernel(const double *partial, int ncta, int ld, int nst,
                                                           double dv, const double *ket_partial, int nket,
                                                           const int *status, double *out) {
  const int s = blockIdx.x;
  if (s == 0 && threadIdx.x == 0) out[3 * nst] = double(*status);
  __shared__ double red[3][2][128];
  Kahan a[3] = {{0, 0}, {0, 0}, {0, 0}};
  for (int c = threadIdx.x; c < ncta; c += blockDim.x) {
    const double *p = partial + ((long long)c * ld + s) * 6;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      kadd(a[q], p[2 * q]);
      a[q].c += p[2 * q + 1];
    }
  }
  if (ket_partial)
    for (int c = threadIdx.x; c < nket; c += blockDim.x) {
      const double *p = ket_partial + ((long long)c * ld + s) * 2;
      kadd(a[0], p[0]);
      a[0].c += p[1];
    }
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    red[q][0][threadIdx.x] = a[q].s;
    red[q][1][threadIdx.x] = a[q].c;
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    const int q = threadIdx.x;
    Kahan t = {0, 0};
    for (int i = 0; i < int(blockDim.x); ++i) {
      kadd(t, red[q][0][i]);
      t.c += red[q][1][i];
    }
    out[q * nst + s] = (t.s + t.c) * dv;
  }
}

// rho[ip] (+)= sum_s w[s] |psi_s(ip)|^2 over the np inner points: one warp per
// row, lanes over the states, FP64 sums folded in a fixed order (deterministic).
template <typename T>
__global__ void __launch_bounds__(256) density_kernel(const T *psi, long long ld, int np, int nst, const double *w,
                                                      double *rho, int accumulate) {
  const int lane = threadIdx.x & 31;
  for (long long row = blockIdx.x * 8LL + (threadIdx.x >> 5); row < np; row += gridDim.x * 8LL) {
    const T *r = psi + row * 2 * ld;
    double acc = 0.0;
    for (int s = lane; s < nst; s += 32) {
      const double re = double(r[2 * s]), im = double(r[2 * s + 1]);
      acc += __ldg(w + s) * (re * re + im * im);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if (lane == 0) rho[row] = accumulate ? rho[row] + acc : acc;
  }
}

}  // namespace

template <typename T>
hpsi_status launch_density(const T *psi, long long ld, int np, int nst, const double *w, double *rho, int accumulate,
                           cudaStream_t st) {
  if (np < 1) return HPSI_OK;
  const int grid = std::min((np + 7) / 8, 148 * 16);
  density_kernel<T><<<grid, 256, 0, st>>>(psi, ld, np, nst, w, rho, accumulate);
  HPSI_CHECK_LAUNCH();
  return HPSI_OK;
}
template hpsi_status launch_density<double>(const double *, long long, int, int, const double *, double *, int,
                                            cudaStream_t);
template hpsi_status launch_density<float>(const float *, long long, int, int, const double *, double *, int,
                                           cudaStream_t);

int reduce_blocks(int np) {
  int nb = (np + 4095) / 4096;
  return nb < 1 ? 1 : (nb > 1184 ? 1184 : nb);
}

template <typename T>
hpsi_status launch_state_sum(int mode, const T *a, long long lda, const T *b, long long ldb, int np, int nst,
                             double *partial, int nblk, double scale, int sqrt_first, double *out,
                             cudaStream_t st) {
  dim3 grid(nblk, (nst + 255) / 256);
  if (mode == 0)
    state_sum_kernel<T, 0><<<grid, 256, 0, st>>>(a, lda, b, ldb, np, nst, partial);
  else
    state_sum_kernel<T, 1><<<grid, 256, 0, st>>>(a, lda, b, ldb, np, nst, partial);
  HPSI_CHECK_LAUNCH();
  state_sum_finalize<<<(nst + 127) / 128, 128, 0, st>>>(partial, nblk, nst, scale, sqrt_first, out);
  HPSI_CHECK_LAUNCH();
  return HPSI_OK;
}

// Splits of the points: as many CTAs as the SMs hold at once (three each), at
// least 64 points each, and partial matrices of at most 64 MB (but for one split).
int gram_splits(int np, int nst, bool sym, int num_sms) {
  const long long tiles = (2LL * nst + GT - 1) / GT, pairs = sym ? tiles * (tiles + 1) / 2 : tiles * tiles;
  long long s = std::max<long long>(1, 3LL * num_sms / pairs);
  s = std::min<long long>(s, (np + 63) / 64);
  s = std::min<long long>(s, std::max<long long>(1, (64LL << 20) / (4LL * nst * nst * 8)));
  return int(std::max<long long>(1, std::min<long long>(s, 65535)));
}

// Points of a split: more than 8192 are folded in pieces.
static bool gram_folds(int np, int splits) { return (np + splits - 1) / splits > GFOLD * GK; }

size_t gram_partial_doubles(int np, int nst, int splits) {
  return size_t(splits) * 4 * nst * nst * (gram_folds(np, splits) ? 2 : 1);
}

template <typename T>
hpsi_status launch_gram(const T *a, long long lda, const T *b, long long ldb, int np, int nst, double *partial,
                        int splits, double dv, double *S, cudaStream_t st) {
  const int n = 2 * nst, tiles = (n + GT - 1) / GT;
  const bool sym = a == b && lda == ldb;
  constexpr size_t smem = size_t(2) * GST * GK * gram_pitch<T>() * sizeof(T);
  static std::once_flag once;
  static cudaError_t attr = cudaSuccess;
  std::call_once(once, [&] {
    attr = cudaFuncSetAttribute(gram_kernel<T, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    if (attr == cudaSuccess)
      attr = cudaFuncSetAttribute(gram_kernel<T, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
  });
  HPSI_TRY_CUDA(attr);
  const long long pairs = sym ? (long long)tiles * (tiles + 1) / 2 : (long long)tiles * tiles;
  const bool fold = gram_folds(np, splits);
  auto kern = fold ? gram_kernel<T, true> : gram_kernel<T, false>;
  if constexpr (sizeof(T) == 4) {
    static_assert(smem <= 48 * 1024, "no opt-in shared memory");
    if ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) % 8 != 0)
      kern = fold ? gram_kernel<T, true, true> : gram_kernel<T, false, true>;
  }
  kern<<<dim3(unsigned(pairs), unsigned(splits)), 256, smem, st>>>(a, lda, b, ldb, np, n, tiles, sym, partial);
  HPSI_CHECK_LAUNCH();
  auto fin = fold ? gram_finalize<true> : gram_finalize<false>;
  fin<<<dim3((nst + 31) / 32, nst), dim3(32, 8), 0, st>>>(partial, splits, nst, dv, sym, S);
  HPSI_CHECK_LAUNCH();
  return HPSI_OK;
}

hpsi_status launch_cholesky_inverse(const double *S, int nst, double *U, double *Uinv, int *err, cudaStream_t st) {
  const size_t smem = (size_t(nst) * (nst + 1) / 2 + nst) * sizeof(double2) + size_t(nst) * sizeof(double);
  if (smem <= 226 * 1024) {
    static std::once_flag once;
    static cudaError_t attr = cudaSuccess;
    std::call_once(once, [&] {
      attr = cudaFuncSetAttribute(cholesky_inverse_smem_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024);
    });
    HPSI_TRY_CUDA(attr);
    cholesky_inverse_smem_kernel<<<1, 512, smem, st>>>(S, nst, U, Uinv, err);
  } else {
    cholesky_inverse_kernel<<<1, 256, 0, st>>>(S, nst, U, Uinv, err);
  }
  HPSI_CHECK_LAUNCH();
  return HPSI_OK;
}

template <typename T>
hpsi_status launch_trsm_apply(T *psi, long long ld, int np, int nst, const double *Uinv, cudaStream_t st) {
  constexpr size_t smem = size_t(2) * GK * (GT + 4) * sizeof(double) + size_t(GST) * GT * (GK + 4) * sizeof(T);
  static std::once_flag once;
  static cudaError_t attr = cudaSuccess;
  std::call_once(once, [&] {
    attr = cudaFuncSetAttribute(trsm_apply_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
  });
  HPSI_TRY_CUDA(attr);
  trsm_apply_kernel<T><<<unsigned((np + GT - 1) / GT), 256, smem, st>>>(psi, ld, np, nst, Uinv);
  HPSI_CHECK_LAUNCH();
  return HPSI_OK;
}

hpsi_status launch_obs_finalize(const double *partial, int ncta, int ld, int nst, double dv,
                                const double *ket_partial, int nket, const int *status, double *out,
                                cudaStream_t st) {
  if (nst < 1) return HPSI_OK;
  obs_finalize_kernel<<<nst, 128, 0, st>>>(partial, ncta, ld, nst, dv, ket_partial, nket, status, out);
  HPSI_CHECK_LAUNCH();
  return HPSI_OK;
}

template hpsi_status launch_state_sum<double>(int, const double *, long long, const double *, long long, int, int,
                                              double *, int, double, int, double *, cudaStream_t);
template hpsi_status launch_state_sum<float>(int, const float *, long long, const float *, long long, int, int,
                                             double *, int, double, int, double *, cudaStream_t);
template hpsi_status launch_gram<double>(const double *, long long, const double *, long long, int, int, double *,
                                         int, double, double *, cudaStream_t);
template hpsi_status launch_gram<float>(const float *, long long, const float *, long long, int, int, double *,
                                        int, double, double *, cudaStream_t);
template hpsi_status launch_trsm_apply<double>(double *, long long, int, int, const double *, cudaStream_t);
template hpsi_status launch_trsm_apply<float>(float *, long long, int, int, const double *, cudaStream_t);

}  // namespace hpsi
