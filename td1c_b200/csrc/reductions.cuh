// reductions.cuh -- argument blocks of the orbital matrix-element and int2e kernels.
#pragma once
#include "common.cuh"

namespace td1c {

struct OrbdotsArgs {
  int nbas, nfun, nent;
  const cplx* orb; const cplx* h0orb; const cplx* h1orb; const cplx* gorb; const cplx* v2orb;
  const int4* ent;   // [nent] (kind, j, i, 0): kind 0 A, 1 B, 2 C, 3 E, 4 GV
  cplx* partial;     // [nchunk][nent]
  cplx* result;      // [nent]
};
int orbdots_nchunk(size_t nbas);  // chunks (CTAs) of the orbdots pass; the partial buffer holds nchunk x nent
int launch_orbdots(const OrbdotsArgs& a, cudaStream_t st);

// Real products over K points of the components (re, im) of a list of complex
// rows, on the FP64 tensor cores (int2e_dmma.cu): S[x][y] = sum_k A_x[k] B_y[k]
// in 8 x 8 tiles.  An item is up to 2 x 4 tiles of one block; the host assigns
// at most I2D_MAXG items to each warp (nm = 0: none).
constexpr int I2D_NW = 8, I2D_MAXG = 2;
// block's first A and B component; tiles mt .. mt + nm - 1, nt .. nt + nn - 1; block's first tile, tiles per row
struct DotProdItem { int compa, compb, mt, nm, nt, nn, tile0, ntile; };
struct DotProdArgs {
  int nrow, nent, nsets;
  size_t K;
  const cplx* const* row;    // [nrow]
  const int* comp;           // row | part << 16
  const DotProdItem* items;  // [nsets][I2D_NW][I2D_MAXG]
  double* partial;           // [nsplit][nent]
  double* sum;               // [nent]
};
int dot_products_nsplit(const DotProdArgs& a, int nsm);
int launch_dot_products(const DotProdArgs& a, int nsplit, cudaStream_t st);

// int2e as FFMA blocks (the no-allocation call) and the entries of the split-TF32 int2e
struct Int2eBlock { int row0, nrow, col0, ncol, ent0, pad0, pad1, pad2; };
struct Int2eArgs {
  int nact, nblocks, nblkent;
  size_t K;                 // Nr * (lmax2 + 1)
  const Int2eBlock* blocks;
  const int* row_pair;      // stored pair index of each block row (ij, i >= j)
  const int2* col_pair;     // (stored pair, conj) of each block column (kl)
  const int4* ent_dst;      // [nblkent] (i, j, k, l) active indices
  const cplx* rho2;         // [npair][K]
  const cplx* v2sph;        // [npair][K]
  cplx* partial;            // [nsplit][nblkent]
  cplx* int2e;              // [nact^4]
};
int launch_int2e(const Int2eArgs& a, int nsplit, cudaStream_t st);

// int2e on the FP64 tensor cores: the products of the stored active pairs' rho2
// and v2sph rows per |Delta m| block, K = Nr (lmax2 + 1)
struct I2dArgs {
  DotProdArgs prod;
  int nact;
  const int4* form;           // [nact^4] entries (RR, RI, IR, II) of each integral, -1: zero
  const unsigned char* flag;  // [nact^4] 1 conjugated column, 2 conjugated integral
  cplx* int2e;                // [nact^4]
};
int launch_int2e_sum_fill(const Int2eArgs& a, int nsplit, cudaStream_t st);
int launch_int2e_dmma(const I2dArgs& d, int nsplit, cudaStream_t st);

// int2e in split TF32 on tcgen05 (the mixed-precision form): every product of
// the P stored active pairs in one 128 x 2NB GEMM per K slice, entries formed
// from it per CTA (the same entry list and partial layout as the DMMA plan).
struct I2tArgs {
  int P, NB;             // stored active pairs (<= 64); B rows per part (>= P, multiple of 16)
  size_t K;
  const int* pair;       // [P] stored pair index of compact pair p
  const int4* ent;       // [nent] (row pair, column pair, conjugated column, 0) of each entry
  int nent;
  const cplx* rho2;
  const cplx* v2sph;
  cplx* partial;         // [nsplit][nent]
  int* status;
};
size_t int2e_tc_smem(const I2tArgs& a);
bool int2e_tc_fits(const I2tArgs& a);
int launch_int2e_tc(const I2tArgs& t, const Int2eArgs& sum, int nsplit, cudaStream_t st);

}  // namespace td1c
