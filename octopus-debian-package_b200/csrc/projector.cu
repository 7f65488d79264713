// Kleinman-Bylander projector "bra": projections of a batch on the projector
// spheres, the step X(hamiltonian_elec_base_nlocal_start) performs on the CPU
// as a gather of the sphere points followed by a real GEMM
// (src/hamiltonian/hamiltonian_elec_base_inc.F90:650-780):
//   proj[row0(m) + j][s] = scal[j] * sum_k P_m[k][j] * psi[map_m[k]][s].
// The matching "ket" (add P * proj back onto the covered rows) runs per
// covered row after the stencil pass: one thread per output element, so no
// write races and no colouring are needed.
//
// The contraction runs on the FP64 tensor cores (DMMA,
// mma.sync.m8n8k4.f64) for both storage types: M = 8 real lanes per warp,
// N = 8 projectors per tile, K = 4 sphere points per step, with the gathered
// rows and the projector block staged in shared memory by cp.async.  The SIMT
// kernel below serves matrices with more than 16 projectors and is the
// cross-check of the tensor path.
#include <algorithm>
#include <cstdlib>
#include <mutex>
#include <type_traits>

#include "projector.cuh"

namespace hpsi {

namespace {

constexpr int KB = 32;     // sphere points per staged block
constexpr int LANES = 32;  // real lanes per CTA (16 complex states)
constexpr int APAD = 40;   // padded row length of the staged psi block (doubles)
constexpr int NMAX = 16;   // projectors per matrix served by the DMMA kernel

// 8-byte cp.async that reads `bytes` (8 or 0) and zero-fills the rest
__device__ __forceinline__ void cp_async8_zfill(void *smem, const void *gmem, int bytes) {
  unsigned sa = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(sa), "l"(gmem), "r"(bytes));
}

__device__ __forceinline__ void dmma_m8n8k4(double &d0, double &d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// grid: (nmat, ld2 / LANES, ksplit); block: 128 threads (4 warps x 8 lanes
// each).  Split z sums sphere points [z*npts/ksplit, (z+1)*npts/ksplit) into
// partial[z] (unscaled, FP64); bra_reduce_kernel adds the splits and applies
// scal.  T is the storage type of psi: FP32 rows are staged as stored and
// widened to FP64 when the A fragment is read, so both precisions contract
// in FP64 against the FP64 projector values.
// PHASE: each gathered point is first multiplied by its projector phase
// (lpsi = psi(map) * projector_phases, hamiltonian_elec_base_inc.F90:680-701):
// the phases of a block are staged with it, and a fragment value is rotated
// with its partner lane (2s, 2s + 1: one complex number) when it is read.
template <typename T, bool PHASE>
__global__ void __launch_bounds__(128) bra_dmma_kernel(const ProjArgs p) {
  constexpr int AP = sizeof(T) == 8 ? APAD : 40;  // 40 floats: conflict-free fragment reads
  constexpr int CPR = LANES * int(sizeof(T)) / 16;  // 16-byte copies per staged row
  constexpr int NS = 3;  // staged blocks: two in flight while one is contracted
  __shared__ __align__(16) T sA[NS][KB][AP];
  __shared__ __align__(16) double sB[NS][KB][NMAX];
  __shared__ __align__(16) double2 sP[PHASE ? NS : 1][PHASE ? KB : 1];
  const int m = blockIdx.x;
  const int l0 = blockIdx.y * LANES;
  const int4 md = p.mat[m];  // npoints, nproj, map_off, pt_off
  const int kbeg = int((long long)md.x * blockIdx.z / gridDim.z);
  const int kend = int((long long)md.x * (blockIdx.z + 1) / gridDim.z);
  const int npts = kend - kbeg, npr = md.y;
  const int *map = p.map + md.z + kbeg;
  const double *pt = p.pt64 + md.w + (long long)kbeg * npr;
  const T *psi = static_cast<const T *>(p.psi);
  const long long ld2 = 2 * p.psi_ld;
  const int tid = threadIdx.x, warp = tid >> 5, ln = tid & 31;
  constexpr int EPC = 16 / int(sizeof(T));  // elements per 16-byte copy

  // the map entries of the next staged block are loaded one block ahead into
  // registers, so a row copy never waits for its own index load
  constexpr int NIT = KB * CPR / 128;  // row pieces per thread and block
  static_assert(KB * CPR % 128 == 0, "whole rounds of row pieces");
  int mrow[NIT];
  auto load_map = [&](int k0) {
#pragma unroll
    for (int t = 0; t < NIT; ++t) {
      const int k = (tid + 128 * t) / CPR;
      mrow[t] = k0 + k < npts ? __ldg(map + k0 + k) : 0;
    }
  };
  auto stage = [&](int k0, int b) {
#pragma unroll
    for (int t = 0; t < NIT; ++t) {
      const int i = tid + 128 * t;
      const int k = i / CPR, part = i % CPR;
      T *d = &sA[b][k][part * EPC];
      if (k0 + k < npts && l0 + part * EPC < ld2) {
        cp_async16(d, psi + mrow[t] * ld2 + l0 + part * EPC);
      } else {
        *reinterpret_cast<float4 *>(d) = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
    for (int i = tid; i < KB * NMAX; i += 128) {
      const int k = i / NMAX, j = i % NMAX;
      const bool ok = k0 + k < npts && j < npr;
      cp_async8_zfill(&sB[b][k][j], ok ? pt + (long long)(k0 + k) * npr + j : p.pt64, ok ? 8 : 0);
    }
    if constexpr (PHASE) {
      const double2 *ph = static_cast<const double2 *>(p.phase64) + md.z + kbeg;
      if (tid < KB) {
        if (k0 + tid < npts)
          cp_async16(&sP[b][tid], ph + k0 + tid);
        else
          sP[b][tid] = make_double2(0.0, 0.0);
      }
    }
  };

  double c0[2] = {0.0, 0.0}, c1[2] = {0.0, 0.0};
  const int nblk = (npts + KB - 1) / KB;
  load_map(0);
  if (nblk > 0) stage(0, 0);
  cp_async_commit();
  load_map(KB);
  if (nblk > 1) stage(KB, 1);
  cp_async_commit();
  load_map(2 * KB);
  for (int blk = 0; blk < nblk; ++blk) {
    const int b = blk % NS;
    if (blk + 2 < nblk) stage((blk + 2) * KB, (blk + 2) % NS);
    cp_async_commit();
    load_map((blk + 3) * KB);
    cp_async_wait<2>();
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < KB; kk += 4) {
      double a = double(sA[b][kk + (ln & 3)][warp * 8 + (ln >> 2)]);
      if constexpr (PHASE) {
        const double other = double(sA[b][kk + (ln & 3)][(warp * 8 + (ln >> 2)) ^ 1]);
        const double2 ph = sP[b][kk + (ln & 3)];
        a = ((ln >> 2) & 1) ? other * ph.y + a * ph.x : a * ph.x - other * ph.y;
      }
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        const double bb = sB[b][kk + (ln & 3)][nt * 8 + (ln >> 2)];
        dmma_m8n8k4(c0[nt], c1[nt], a, bb);
      }
    }
    __syncthreads();
  }
  cp_async_wait<0>();
  // C fragment: row (lane) = ln >> 2, cols (projectors) = (ln & 3) * 2 + {0,1}
  const int lane = l0 + warp * 8 + (ln >> 2);
  if (lane >= ld2) return;  // lanes past the batch width (zero-filled above)
  double *out = p.partial + ((long long)blockIdx.z * p.nprojections + p.proj_row[m]) * 2 * p.proj_ld;
#pragma unroll
  for (int nt = 0; nt < 2; ++nt) {
    const int j0 = nt * 8 + (ln & 3) * 2;
    if (j0 < npr) out[(long long)j0 * 2 * p.proj_ld + lane] = c0[nt];
    if (j0 + 1 < npr) out[(long long)(j0 + 1) * 2 * p.proj_ld + lane] = c1[nt];
  }
}

// proj[j][l] = scal[j] * sum_z partial[z][j][l]: block (32, 8), 32 real lanes by
// 8 slices of the splits, folded in a fixed order (FP64 sums, rounded once to
// the storage type).  One thread per lane waited for up to 32 loads in turn.
template <typename T>
__global__ void __launch_bounds__(256) bra_reduce_kernel(const ProjArgs p, int ksplit) {
  __shared__ double red[8][32];
  const long long n = (long long)p.nprojections * 2 * p.proj_ld;
  const long long i = blockIdx.x * 32LL + threadIdx.x;
  double acc = 0.0;
  if (i < n) {
#pragma unroll 4
    for (int z = threadIdx.y; z < ksplit; z += 8) acc += p.partial[(long long)z * n + i];
  }
  red[threadIdx.y][threadIdx.x] = acc;
  __syncthreads();
  if (threadIdx.y != 0 || i >= n) return;
#pragma unroll
  for (int z = 1; z < 8; ++z) acc += red[z][threadIdx.x];
  const int j = int(i / (2 * p.proj_ld));
  static_cast<T *>(p.proj)[i] = T(acc * p.scal64[j]);
}

// SIMT bra: grid (nmat, ceil(ld2/32)); block 128 = 32 lanes x 4 point groups.
// PHASE: each gathered point is first multiplied by its projector phase
// (lpsi = psi(map) * projector_phases, hamiltonian_elec_base_inc.F90:680-701);
// lane pairs (2s, 2s + 1) hold one complex number, exchanged by a shuffle.
template <typename T, bool PHASE>
__global__ void __launch_bounds__(128) bra_simt_kernel(const ProjArgs p) {
  constexpr int MAXP = 32;
  __shared__ T red[4][MAXP][32];
  const int m = blockIdx.x;
  const int ln = threadIdx.x & 31, grp = threadIdx.x >> 5;
  const long long ld2 = 2 * p.psi_ld;
  const int lane = blockIdx.y * 32 + ln;
  const int4 md = p.mat[m];
  const int npts = md.x, npr = md.y;
  const int *map = p.map + md.z;
  const T *pt = static_cast<const T *>(p.pt) + md.w;
  const T *psi = static_cast<const T *>(p.psi);
  T acc[MAXP];
#pragma unroll
  for (int j = 0; j < MAXP; ++j) acc[j] = T(0);
  if constexpr (!PHASE) {
    if (lane < ld2) {
      for (int k = grp; k < npts; k += 4) {
        const T x = psi[__ldg(map + k) * ld2 + lane];
        const T *pk = pt + (long long)k * npr;
#pragma unroll
        for (int j = 0; j < MAXP; ++j)
          if (j < npr) acc[j] += pk[j] * x;
      }
    }
  } else {
    // every lane of the warp runs the loop (the shuffle needs all 32)
    const T *ph = static_cast<const T *>(p.phase) + 2 * (long long)md.z;
    for (int k = grp; k < npts; k += 4) {
      T x = lane < ld2 ? psi[__ldg(map + k) * ld2 + lane] : T(0);
      const T other = __shfl_xor_sync(0xffffffffu, x, 1);
      const T c = ph[2 * k], sn = ph[2 * k + 1];
      x = (ln & 1) ? other * sn + x * c : x * c - other * sn;
      const T *pk = pt + (long long)k * npr;
#pragma unroll
      for (int j = 0; j < MAXP; ++j)
        if (j < npr) acc[j] += pk[j] * x;
    }
  }
#pragma unroll
  for (int j = 0; j < MAXP; ++j) red[grp][j][ln] = acc[j];
  __syncthreads();
  if (grp == 0 && lane < ld2) {
    const T *scal = static_cast<const T *>(p.scal) + p.proj_row[m];
    T *out = static_cast<T *>(p.proj) + (long long)p.proj_row[m] * 2 * p.proj_ld;
    for (int j = 0; j < npr; ++j) {
      const T s = red[0][j][ln] + red[1][j][ln] + red[2][j][ln] + red[3][j][ln];
      out[(long long)j * 2 * p.proj_ld + lane] = s * scal[j];
    }
  }
}

}  // namespace

int bra_ksplit(const ProjArgs &p, int num_sms) {
  const long long ld2 = 2 * p.psi_ld;
  const long long base = (long long)p.nmat * ((ld2 + LANES - 1) / LANES);
  static const long long target = [] {
    const char *e = std::getenv("HPSI_BRA_CTAS_PER_SM");  // tuning override
    return e ? std::max(1, std::atoi(e)) : 32;  // measured: 4 -> 0.196 ms, 16 -> 0.188, 32 -> 0.174 (R = 12 sphere)
  }();
  long long k = (target * num_sms + base - 1) / base;
  k = std::min<long long>(k, std::max(1, p.min_npoints / 128));
  return int(std::max<long long>(1, std::min<long long>(k, 64)));
}

template <typename T>
hpsi_status launch_bra(const ProjArgs &p, bool use_tensor, int ksplit, cudaStream_t st) {
  if (p.nmat == 0) return HPSI_OK;
  const long long ld2 = 2 * p.psi_ld;
  // the staged rows are copied in 16-byte pieces: FP32 needs an even width
  if (use_tensor && p.max_nproj <= NMAX && ld2 % (16 / sizeof(T)) == 0) {
    dim3 grid(p.nmat, unsigned((ld2 + LANES - 1) / LANES), ksplit);
    if (p.phase)
      bra_dmma_kernel<T, true><<<grid, 128, 0, st>>>(p);
    else
      bra_dmma_kernel<T, false><<<grid, 128, 0, st>>>(p);
    HPSI_CHECK_LAUNCH();
    const long long n = (long long)p.nprojections * ld2;
    bra_reduce_kernel<T><<<unsigned((n + 31) / 32), dim3(32, 8), 0, st>>>(p, ksplit);
    HPSI_CHECK_LAUNCH();
    return HPSI_OK;
  }
  if (p.max_nproj > 32) {
    set_error("projector matrices with more than 32 projectors are not supported");
    return HPSI_ERR_UNSUPPORTED;
  }
  dim3 grid(p.nmat, unsigned((ld2 + 31) / 32));
  if (p.phase)
    bra_simt_kernel<T, true><<<grid, 128, 0, st>>>(p);
  else
    bra_simt_kernel<T, false><<<grid, 128, 0, st>>>(p);
  HPSI_CHECK_LAUNCH();
  return HPSI_OK;
}

// ---------------------------------------------------------------------------
// KB ket, one thread per (covered row, complex state): h = sum over the
// row's (matrix, point) entries of P[point][j] * proj[j], then
// out[row] += h (apply) or += a * h (Horner pass), and, if requested, the
// energy partial Re(conj(psi0[row]) h) per state.  Each output element is
// written by exactly one thread, in a fixed order: no atomics, deterministic.
namespace {
// RPW rows per warp: 1 for batches wider than 16 states; narrow batches (at
// most 16 or 8 states) put 2 or 4 rows in a warp, one lane group of 32 / RPW
// lanes per row, so the lanes past the batch width do not idle.
template <typename T, typename C2, bool PHASE, int RPW = 1>
__global__ void __launch_bounds__(256) ket_kernel(const KetArgs k) {
  // each thread serves two states (sb, sb + 32) of its rows: the row's
  // metadata and projector weights are loaded once for both (12 % faster than
  // one state per thread on the R = 12 sphere, 128 states; four states per
  // thread measured 30 % slower, the grid no longer filling the GPU)
  constexpr int L = 32 / RPW;            // lanes per row
  constexpr int SPT = RPW == 1 ? 2 : 1;  // states per thread
  const int lane = threadIdx.x % L, sub = threadIdx.x / L;
  const int sb = blockIdx.x * L * SPT + lane;
  bool act[SPT];
#pragma unroll
  for (int u = 0; u < SPT; ++u) act[u] = sb + L * u < k.nst;
  const T *pt = static_cast<const T *>(k.pt);
  const C2 *proj = static_cast<const C2 *>(k.proj);
  C2 *out = static_cast<C2 *>(k.out);
  const C2 *psi0 = static_cast<const C2 *>(k.psi0);
  Kahan ke[SPT];
#pragma unroll
  for (int u = 0; u < SPT; ++u) ke[u] = {0, 0};
  // each CTA row takes a contiguous range of covered rows: neighbouring rows
  // lie in the same few spheres, so their projections stay in L1
  const int per = (k.nk + gridDim.y - 1) / gridDim.y;
  const int r0 = blockIdx.y * per, r1 = min(k.nk, r0 + per);
  for (int i0 = r0 + threadIdx.y * RPW; i0 < r1; i0 += 8 * RPW) {
    // row of this lane group; density of the final row (the loop bound is
    // the same for the whole warp: the shuffle below is reached by all its
    // lanes, active or not)
    const int i = i0 + sub;
    const bool rv = i < r1;
    double rs = 0.0;
    if (act[0] && rv) {
    const int row = k.krows[i];
    // the output elements are loaded before the sums, so their latency
    // overlaps theirs (prefetching the next row's metadata as well, or four
    // rows per warp, measured slower)
    C2 *o = out + (long long)row * k.out_ld + sb;
    C2 y[SPT], h[SPT];
#pragma unroll
    for (int u = 0; u < SPT; ++u) {
      if (act[u]) y[u] = o[L * u];
      h[u].x = 0;
      h[u].y = 0;
    }
    for (int e = k.kptr[i]; e < k.kptr[i + 1]; ++e) {
      const int4 E = __ldg(k.ent + e);
      const T *pp = pt + E.x;
      const C2 *pr = proj + (long long)E.y * k.proj_ld + sb;
      if constexpr (!PHASE) {
        for (int j = 0; j < E.z; ++j) {
          const T w = pp[j];
#pragma unroll
          for (int u = 0; u < SPT; ++u) {
            if (!act[u]) continue;
            const C2 v = pr[(long long)j * k.proj_ld + L * u];
            h[u].x += w * v.x;
            h[u].y += w * v.y;
          }
        }
      } else {
        // this point's contribution times conj(phase) (the ket of
        // hamiltonian_elec_base_inc.F90:934-1025 with projector phases)
        C2 g[SPT];
#pragma unroll
        for (int u = 0; u < SPT; ++u) g[u].x = g[u].y = 0;
        for (int j = 0; j < E.z; ++j) {
          const T w = pp[j];
#pragma unroll
          for (int u = 0; u < SPT; ++u) {
            if (!act[u]) continue;
            const C2 v = pr[(long long)j * k.proj_ld + L * u];
            g[u].x += w * v.x;
            g[u].y += w * v.y;
          }
        }
        const T *ph = static_cast<const T *>(k.phase) + 2 * (long long)E.w;
        const T c = ph[0], sn = ph[1];
#pragma unroll
        for (int u = 0; u < SPT; ++u) {
          h[u].x += g[u].x * c + g[u].y * sn;
          h[u].y += g[u].y * c - g[u].x * sn;
        }
      }
    }
#pragma unroll
    for (int u = 0; u < SPT; ++u) {
      if (!act[u]) continue;
      if (k.mode == 1) {
        const T ar = T(k.a_re), ai = T(k.a_im);
        y[u].x += ar * h[u].x - ai * h[u].y;
        y[u].y += ar * h[u].y + ai * h[u].x;
      } else {
        y[u].x += h[u].x;
        y[u].y += h[u].y;
      }
      o[L * u] = y[u];
      if (k.rho_ket) rs += k.rho_w[sb + L * u] * (double(y[u].x) * double(y[u].x) + double(y[u].y) * double(y[u].y));
      if (k.obs) {
        const C2 x = psi0[(long long)row * k.psi0_ld + sb + L * u];
        kadd(ke[u], double(x.x) * double(h[u].x) + double(x.y) * double(h[u].y));
      }
    }
    }
    if (k.rho_ket) {
      // sum over the row's lane group (xor offsets below L stay inside it)
      for (int off = L / 2; off > 0; off >>= 1) rs += __shfl_xor_sync(0xffffffffu, rs, off);
      if (lane == 0 && rv) k.rho_ket[(long long)blockIdx.x * k.nk + i] = rs;
    }
  }
  if (k.obs) {
    __shared__ double red[8][32 * SPT][2];
#pragma unroll
    for (int u = 0; u < SPT; ++u) {
      red[threadIdx.y][threadIdx.x + 32 * u][0] = ke[u].s;
      red[threadIdx.y][threadIdx.x + 32 * u][1] = ke[u].c;
    }
    __syncthreads();
    if (threadIdx.y == 0 && sub == 0) {
#pragma unroll
      for (int u = 0; u < SPT; ++u) {
        if (!act[u]) continue;
        Kahan a = {0, 0};
        for (int y = 0; y < 8; ++y)
          for (int q = 0; q < RPW; ++q) {
            kadd(a, red[y][q * L + lane + 32 * u][0]);
            a.c += red[y][q * L + lane + 32 * u][1];
          }
        double *o = k.obs + ((long long)blockIdx.y * k.obs_ld + sb + L * u) * 2;
        o[0] = a.s;
        o[1] = a.c;
      }
    }
  }
}
}  // namespace

// KB ket over blocks of covered rows with the same list of matrices
// (KetArgs::blk, at most 32 rows each): per matrix of the block the CTA stages
// its projections for SW states and the rows' projector values in shared memory
// once, and a thread adds them to RPT rows of one state held in registers.  A
// projection is read from shared memory once for RPT rows; the form above reads
// it through L1 for every row and waits for each load in turn (R = 12 sphere,
// 128 states, FP64: 0.187 ms, here 0.146).  The same terms in the same order per output
// element as above.
namespace {
constexpr int KET_ROWS = 32;
template <typename T, typename C2, bool PHASE, int SW>
__global__ void __launch_bounds__(256, PHASE ? 2 : 4) ket_block_kernel(const KetArgs k) {
  constexpr int HALVES = SW >= 64 ? 2 : 1;           // sweeps over the block's rows: fewer registers, more CTAs per SM
  constexpr int RPT = KET_ROWS * SW / 256 / HALVES;  // rows per thread and sweep
  extern __shared__ __align__(16) unsigned char ksm[];
  C2 *sp = reinterpret_cast<C2 *>(ksm);                  // [nproj][SW]
  T *sw = reinterpret_cast<T *>(sp + k.max_nproj * SW);  // [rows of the block][nproj]
  const int t = threadIdx.x, sl = t % SW;
  const int sbase = blockIdx.x * SW, s = sbase + sl;
  const bool act = s < k.nst;
  const C2 *proj = static_cast<const C2 *>(k.proj);
  C2 *out = static_cast<C2 *>(k.out);
  const C2 *psi0 = static_cast<const C2 *>(k.psi0);
  Kahan ke = {0, 0};
  const int per = (k.nblk + gridDim.y - 1) / gridDim.y;
  const int b0 = blockIdx.y * per, b1 = min(k.nblk, b0 + per);
  for (int b = b0; b < b1; ++b) {
    const int4 D = __ldg(k.blk + b);  // {first row, rows + 256 * entries per row, its first entry, value offset}
    const int cnt = D.y & 255, ne = D.y >> 8;
#pragma unroll 1
    for (int half = 0; half < HALVES; ++half) {
    const int r0 = half * (KET_ROWS / HALVES) + (t / SW) * RPT;
    if (half && cnt <= KET_ROWS / HALVES) break;  // (the same for the whole CTA)
    const T *w = static_cast<const T *>(k.pk) + D.w;
    int row[RPT];
    [[maybe_unused]] int ent0[RPT];  // the rows' first entries
    C2 y[RPT], h[RPT];
#pragma unroll
    for (int q = 0; q < RPT; ++q) {
      const int2 R = r0 + q < cnt ? __ldg(k.brow + D.x + r0 + q) : make_int2(-1, 0);
      row[q] = R.x;
      if constexpr (PHASE) ent0[q] = R.y;
      h[q].x = 0;
      h[q].y = 0;
    }
#pragma unroll
    for (int q = 0; q < RPT; ++q)
      if (act && row[q] >= 0) y[q] = out[(long long)row[q] * k.out_ld + s];
    for (int e = 0; e < ne; ++e) {
      const int4 E = __ldg(k.ent + D.z + e);  // (the first row's entry: projection row and count of the matrix)
      const int np = E.z;
      // one matrix: the second sweep finds it staged
      if (half == 0 || ne > 1) {
        __syncthreads();  // the matrix before has been read
        for (int i = t; i < cnt * np; i += 256) sw[i] = w[i];
        for (int i = t; i < np * SW; i += 256) {
          const int c = sbase + i % SW;
          C2 v;
          v.x = 0;
          v.y = 0;
          if (c < k.nst) v = proj[(long long)(E.y + i / SW) * k.proj_ld + c];
          sp[i] = v;
        }
        __syncthreads();
      }
      if (row[0] >= 0) {
        const T *wr = sw + r0 * np;
        C2 g[RPT];
        if constexpr (PHASE) {
#pragma unroll
          for (int q = 0; q < RPT; ++q) g[q].x = g[q].y = 0;
        }
        for (int j = 0; j < np; ++j) {
          const C2 v = sp[j * SW + sl];
#pragma unroll
          for (int q = 0; q < RPT; ++q) {
            // (rows past the block read another row's value: not used)
            const T a = wr[min(q, cnt - 1 - r0) * np + j];
            C2 &o = PHASE ? g[q] : h[q];
            o.x += a * v.x;
            o.y += a * v.y;
          }
        }
        if constexpr (PHASE) {
          // this matrix's contribution times conj(phase) of each point (the ket
          // of hamiltonian_elec_base_inc.F90:934-1025 with projector phases)
#pragma unroll
          for (int q = 0; q < RPT; ++q) {
            if (row[q] < 0) continue;
            const int pnt = __ldg(k.ent + ent0[q] + e).w;
            const T *ph = static_cast<const T *>(k.phase) + 2 * (long long)pnt;
            const T c = ph[0], sn = ph[1];
            h[q].x += g[q].x * c + g[q].y * sn;
            h[q].y += g[q].y * c - g[q].x * sn;
          }
        }
      }
      w += cnt * np;
    }
#pragma unroll
    for (int q = 0; q < RPT; ++q) {
      if (!act || row[q] < 0) continue;
      if (k.mode == 1) {
        const T ar = T(k.a_re), ai = T(k.a_im);
        y[q].x += ar * h[q].x - ai * h[q].y;
        y[q].y += ar * h[q].y + ai * h[q].x;
      } else {
        y[q].x += h[q].x;
        y[q].y += h[q].y;
      }
      out[(long long)row[q] * k.out_ld + s] = y[q];
      if (k.obs) {
        const C2 x = psi0[(long long)row[q] * k.psi0_ld + s];
        kadd(ke, double(x.x) * double(h[q].x) + double(x.y) * double(h[q].y));
      }
    }
    }
  }
  if (k.obs) {
    __shared__ double red[256][2];
    __syncthreads();
    red[t][0] = ke.s;
    red[t][1] = ke.c;
    __syncthreads();
    if (t < SW && act) {
      Kahan a = {0, 0};
      for (int q = t; q < 256; q += SW) {
        kadd(a, red[q][0]);
        a.c += red[q][1];
      }
      double *o = k.obs + ((long long)blockIdx.y * k.obs_ld + s) * 2;
      o[0] = a.s;
      o[1] = a.c;
    }
  }
}

template <typename T, typename C2, bool PHASE, int SW>
hpsi_status launch_ket_blocks(const KetArgs &k, int rb, cudaStream_t st) {
  const size_t smem = size_t(k.max_nproj) * (SW * sizeof(C2) + KET_ROWS * sizeof(T));
  auto kern = ket_block_kernel<T, C2, PHASE, SW>;
  if (smem > 44 * 1024) {  // (4 KB static)
    static std::once_flag once;
    static cudaError_t attr = cudaSuccess;
    std::call_once(once, [&] { attr = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024); });
    HPSI_TRY_CUDA(attr);
  }
  kern<<<dim3((k.nst + SW - 1) / SW, rb), 256, smem, st>>>(k);
  HPSI_CHECK_LAUNCH();
  return HPSI_OK;
}
template <typename T, typename C2, bool PHASE>
hpsi_status launch_ket_blocks_w(const KetArgs &k, int rb, cudaStream_t st) {
  // states per CTA: the narrowest width that holds the batch, up to 64
  if (k.nst > 32) return launch_ket_blocks<T, C2, PHASE, 64>(k, rb, st);
  if (k.nst > 16) return launch_ket_blocks<T, C2, PHASE, 32>(k, rb, st);
  if (k.nst > 8) return launch_ket_blocks<T, C2, PHASE, 16>(k, rb, st);
  return launch_ket_blocks<T, C2, PHASE, 8>(k, rb, st);
}
}  // namespace

// Whether the blocks are the faster form.  They gain where a block is well filled
// (rows_per_block of at most 32: many overlapping spheres make many lists of a few
// rows each) and where the rows above wait for many projections (wide batches,
// many projectors); with phases their registers halve the CTAs per SM.  Kernel
// alone on a 60^3 mesh at 0.25 bohr, us, rows / blocks (spheres of 2 bohr with 9
// projectors: 32 of them 29.6 rows per block; 400 of 1.2 bohr 9.6; 32 with 18
// projectors 30.4):
//                                   FP64 8 states    32       128     FP32 8     32       128
//   29.6 rows, 9 projectors           25 / 16    44 / 23   94 / 75   18 / 15  34 / 19   60 / 48
//   9.6 rows, 9 projectors            43 / 66   111 / 101 253 / 299  33 / 64  77 / 78  164 / 228
//   29.6 rows, 9 projectors, phases   25 / 24    47 / 32  103 / 130  21 / 19  37 / 29   70 / 91
//   30.4 rows, 18 projectors, phases  26 / 26    71 / 37  168 / 152  23 / 18  55 / 33  108 / 106
//   9.6 rows, 9 projectors, phases    45 / 136  121 / 185 281 / 607  35 / 92  90 / 160 210 / 526
//   31.4 rows, 9 projectors, phases,
//   8,779 rows in all                 13 / 12    16 / 12   27 / 22   13 / 12  15 / 12   24 / 19
// The lines below lie between measured sides of 24 such sets (1 to 32 projectors, 9.6 to
// 31.6 rows, 2 to 128 states).
template <typename T>
static bool ket_blocks_better(const KetArgs &k) {
  const double rows = k.rows_per_block, q = k.nproj_per_point;
  const bool f64 = sizeof(T) == 8;
  if (k.phase) {
    if (k.nst > 32)  // (few rows do not fill the GPU one warp each)
      return rows >= 28 && (q >= (f64 || k.nst <= 64 ? 16 : 24) || (q >= 8 && k.nk <= 16000));
    if (k.nst > 16) return rows >= 25;
    return rows >= 28 && (q >= 16 || (f64 && k.nst > 8 && q >= 8 && rows >= 29));
  }
  if (k.nst > 32) return rows >= 20;
  if (k.nst > 16) return rows >= KET_BLOCK_ROWS;
  if (k.nst > 8) return rows >= (q >= 8 ? 20 : 28);
  return q >= 8 && rows >= (f64 ? 20 : 29);
}

// At most 1024 CTA rows, each over a contiguous range of covered rows: one
// row per thread (up to 65535 CTA rows) measured 45 % slower on the R = 12
// sphere, the projections of neighbouring rows no longer sharing L1.
int ket_row_blocks(int nk) {
  static const int cap = [] {
    const char *e = std::getenv("HPSI_KET_ROW_BLOCKS");  // tuning override
    return e ? std::max(1, std::min(65535, std::atoi(e))) : 1024;
  }();
  return std::max(1, std::min(cap, (nk + 7) / 8));
}

template <typename T>
hpsi_status launch_ket(const KetArgs &k, cudaStream_t st) {
  if (k.nk == 0) return HPSI_OK;
  using C2 = typename std::conditional<sizeof(T) == 8, double2, float2>::type;
  const int rb = k.row_blocks > 0 ? std::min(k.row_blocks, ket_row_blocks(k.nk)) : ket_row_blocks(k.nk);
  // the fused density needs the row's states in one warp (the form above); so
  // do matrices whose projections would not fit shared memory
  if (!k.rho_ket && k.blk && ket_blocks_better<T>(k) && size_t(k.max_nproj) * (64 * sizeof(C2) + KET_ROWS * sizeof(T)) <= 200 * 1024) {
    // a CTA per block, but where the energy partials count the CTA rows or the
    // launch shares the GPU
    const int rows = k.obs || k.row_blocks > 0 ? rb : std::min(k.nblk, 65535);
    return k.phase ? launch_ket_blocks_w<T, C2, true>(k, rows, st) : launch_ket_blocks_w<T, C2, false>(k, rows, st);
  }
  dim3 grid((k.nst + 63) / 64, rb);  // two states per thread
  // narrow batches: several rows per warp
  const int rpw = k.nst <= 8 ? 4 : k.nst <= 16 ? 2 : 1;
  if (k.phase) {
    if (rpw == 4)
      ket_kernel<T, C2, true, 4><<<grid, dim3(32, 8), 0, st>>>(k);
    else if (rpw == 2)
      ket_kernel<T, C2, true, 2><<<grid, dim3(32, 8), 0, st>>>(k);
    else
      ket_kernel<T, C2, true><<<grid, dim3(32, 8), 0, st>>>(k);
  } else {
    if (rpw == 4)
      ket_kernel<T, C2, false, 4><<<grid, dim3(32, 8), 0, st>>>(k);
    else if (rpw == 2)
      ket_kernel<T, C2, false, 2><<<grid, dim3(32, 8), 0, st>>>(k);
    else
      ket_kernel<T, C2, false><<<grid, dim3(32, 8), 0, st>>>(k);
  }
  HPSI_CHECK_LAUNCH();
  return HPSI_OK;
}

template hpsi_status launch_ket<double>(const KetArgs &, cudaStream_t);
template hpsi_status launch_ket<float>(const KetArgs &, cudaStream_t);

template hpsi_status launch_bra<double>(const ProjArgs &, bool, int, cudaStream_t);
template hpsi_status launch_bra<float>(const ProjArgs &, bool, int, cudaStream_t);

void kb_rows(int np, const std::vector<int4> &mat, const std::vector<int> &prow, const int *map, KbRows &o) {
  struct List {
    int len, nproj;   // matrices, projectors of all of them
    int from, next;   // last matrix seen at this list, the list it leads to
    int rows, first;  // rows of the list, place of the next one
  };
  std::vector<List> lists(1, List{0, 0, -1, 0, 0, 0});  // list 0: no matrix
  std::vector<int> id(np, 0);
  for (int i = 0; i < int(mat.size()); ++i)
    for (int k = 0; k < mat[i].x; ++k) {
      int &at = id[map[mat[i].z + k]];
      if (lists[at].from != i) {
        lists[at].from = i;
        lists[at].next = int(lists.size());
        lists.push_back(List{lists[at].len + 1, lists[at].nproj + mat[i].y, -1, 0, 0, 0});
      }
      at = lists[at].next;
    }
  std::vector<int> order;  // lists by their first row
  int nk = 0;
  for (int r = 0; r < np; ++r)
    if (id[r]) {
      if (lists[id[r]].rows++ == 0) order.push_back(id[r]);
      ++nk;
    }
  int at = 0, npk = 0;
  for (int l : order) {
    List &L = lists[l];
    L.first = at;
    for (int i = 0; i < L.rows; i += 32) {
      const int n = std::min(32, L.rows - i);
      o.blk.push_back(make_int4(at + i, n + 256 * L.len, 0, npk));
      npk += n * L.nproj;
    }
    at += L.rows;
  }
  o.krows.reserve(nk);
  o.kptr.reserve(size_t(nk) + 1);
  o.kptr.push_back(0);
  o.brow.resize(nk);
  for (int r = 0; r < np; ++r)
    if (id[r]) {
      List &L = lists[id[r]];
      const int e = o.kptr.back();
      o.brow[L.first++] = make_int2(r, e);
      o.krows.push_back(r);
      o.kptr.push_back(e + L.len);
      id[r] = e;  // place of the row's next entry
    }
  for (int4 &b : o.blk) b.z = o.brow[b.x].y;
  o.ent.resize(o.kptr.back());
  for (int i = 0; i < int(mat.size()); ++i)
    for (int k = 0; k < mat[i].x; ++k)
      o.ent[id[map[mat[i].z + k]]++] = make_int4(mat[i].w + k * mat[i].y, prow[i], mat[i].y, mat[i].z + k);
}

// Tables of the projectors that the device makes itself: the values in FP32,
// the covered rows' numbers (kidx, -1 before) and the values in block order (KetArgs::pk).
namespace {
__global__ void __launch_bounds__(256) kb_layout_kernel(const KbTables t) {
  const long long t0 = blockIdx.x * 256LL + threadIdx.x, step = gridDim.x * 256LL;
  for (long long i = t0; i < t.nval; i += step) t.ptf[i] = float(t.pt[i]);
  for (long long i = t0; i < t.nk; i += step) t.kidx[t.krows[i]] = int(i);
  for (int b = blockIdx.x; b < t.nblk; b += gridDim.x) {
    const int4 D = t.blk[b];
    const int n = D.y & 255, ne = D.y >> 8;
    int w = D.w;
    for (int e = 0; e < ne; ++e) {
      const int q = t.ent[D.z + e].z;
      for (int i = threadIdx.x; i < n * q; i += 256) {
        const double v = t.pt[t.ent[t.brow[D.x + i / q].y + e].x + i % q];
        t.pk[w + i] = v;
        t.pkf[w + i] = float(v);
      }
      w += n * q;
    }
  }
}
}  // namespace

hpsi_status launch_kb_layout(const KbTables &t, int num_sms) {
  HPSI_TRY_CUDA(cudaMemsetAsync(t.kidx, 0xff, size_t(t.np) * sizeof(int), nullptr));
  kb_layout_kernel<<<4 * num_sms, 256>>>(t);
  HPSI_CHECK_LAUNCH();
  HPSI_TRY_CUDA(cudaStreamSynchronize(nullptr));
  return HPSI_OK;
}

}  // namespace hpsi
