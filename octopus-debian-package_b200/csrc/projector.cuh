// KB projector bra kernels (see projector.cu).
#pragma once

#include <vector>

#include "common.cuh"

namespace hpsi {

struct ProjArgs {
  int nmat;
  int max_nproj;
  const int4 *mat;       // per matrix: {npoints, nproj, map offset, projector value offset}
  const int *proj_row;   // per matrix: first projection row
  const int *map;        // sphere point -> mesh row
  const void *pt;        // projector values, projector index fastest per point
  const void *scal;      // per projector scale (storage type)
  const double *pt64;    // the projector values in FP64 (tensor-core path)
  const double *scal64;  // the scales in FP64
  const void *psi;       // batch
  long long psi_ld;
  void *proj;            // projections [nprojections][proj_ld] complex
  long long proj_ld;
  int nprojections;
  int min_npoints;       // smallest sphere (bounds the K split)
  double *partial;       // split-K partials [ksplit][nprojections][proj_ld] complex, FP64
  const void *phase = nullptr;  // per sphere point complex phase (storage type), or null
  const void *phase64 = nullptr;  // the same phases in FP64 (tensor-core path)
};

// Rows per block, on average, from which on the block form of the ket is ever the better
// one (no blocks are made below).
constexpr int KET_BLOCK_ROWS = 14;

struct KetArgs {
  int nk;                // covered rows
  const int *krows;      // covered row -> mesh row
  const int *kptr;       // nk + 1 offsets into ent
  const int4 *ent;       // {projector value offset, projection row, nproj, 0}
  // blocks of at most 32 covered rows with the same list of matrices: {first
  // row in brow, rows + 256 * entries per row, the first row's first entry,
  // offset into pk}; brow: {row, its first entry} in block order; pk: per
  // block and matrix the rows' projector values
  int nblk = 0;
  const int4 *blk = nullptr;
  const int2 *brow = nullptr;
  const void *pk = nullptr;
  int max_nproj = 0;
  double rows_per_block = 0.0, nproj_per_point = 0.0;  // averages, for the choice of the form
  const void *pt;        // projector values
  const void *proj;      // projections [nprojections][proj_ld] complex
  long long proj_ld;
  void *out;             // batch receiving the ket
  long long out_ld;
  int nst;
  int mode;              // 0: out += h; 1: out += a * h
  double a_re, a_im;
  const void *psi0;      // energy partials: Re(conj(psi0) h)
  long long psi0_ld;
  double *obs;           // [ket_row_blocks][obs_ld][2] or null
  int obs_ld;
  const void *phase = nullptr;  // per sphere point complex phase (storage type), or null
  // density of the final rows: rho_ket[blockIdx.x][covered row] = sum over the
  // CTA's states of w_i |out_i(row)|^2, or null
  double *rho_ket = nullptr;
  const double *rho_w = nullptr;
  // CTA rows of the launch, 0: ket_row_blocks(nk) (a launch that has the GPU
  // to itself); a grouped step gives each of its concurrent kets fewer
  int row_blocks = 0;
};

int bra_ksplit(const ProjArgs &p, int num_sms);
int ket_row_blocks(int nk);

template <typename T>
hpsi_status launch_bra(const ProjArgs &p, bool use_tensor, int ksplit, cudaStream_t st);
template <typename T>
hpsi_status launch_ket(const KetArgs &k, cudaStream_t st);

// Covered rows of the projector spheres, in mesh order: krows[nk], kptr[nk + 1],
// ent their entries in matrix order; and in blocks of rows with the same list of
// matrices (KetArgs::blk, brow; lists in the order of their first row).  A
// row's list is a number: matrix i leads from a list to the list with i at its
// end, so that one pass over the points finds them all.
struct KbRows {
  std::vector<int> krows, kptr;
  std::vector<int4> ent, blk;
  std::vector<int2> brow;
};
void kb_rows(int np, const std::vector<int4> &mat, const std::vector<int> &prow, const int *map, KbRows &o);

// Tables of the projectors on the device; launch_kb_layout makes those from ptf on
// (the values in FP32, the covered rows' numbers, the values in block order) and
// waits for them.
struct KbTables {
  const double *pt;
  long long nval;
  const int *krows;
  int nk;
  const int4 *blk;
  int nblk;
  const int2 *brow;
  const int4 *ent;
  float *ptf;
  int *kidx, np;
  double *pk;
  float *pkf;
};
hpsi_status launch_kb_layout(const KbTables &t, int num_sms);

}  // namespace hpsi
