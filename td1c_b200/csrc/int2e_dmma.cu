// int2e_dmma.cu -- MO two-electron integrals (hprod_mkint2_sph.F90:2-100)
// on the FP64 tensor cores.
//
// int2e(i,j,k,l) = sum_x rho2_ij[x] v2sph_kl[x] over x in [0, K), K =
// Nr (lmax2 + 1), for m_i + m_k = m_j + m_l.  Pairs (a, b) and (b, a) are a
// stored field and its conjugate, so every integral is a sign combination of
// the four real products of two stored pairs p, q,
//   RR = sum Re rho_p Re v_q, II, RI = sum Re rho_p Im v_q, IR:
//   v_q plain (RR - II, RI + IR), v_q conjugated (RR + II, IR - RI),
// and the pairs of one |Delta m| need only each other: per |Delta m| one real
// product S = A B^T of the pairs' components (re, im; the diagonal pairs are
// real), on mma.sync.m8n8k4.f64 tiles of 8 x 8 components x 4 points.  For
// CAS(8e,9o) that is 51 tiles where the complex form over ordered pairs
// needed 116 tile products, and each stored row is staged once instead of once
// per order.
//
// One CTA owns a slice of K: the slice of every stored pair's rho2 and v2sph
// rows passes through shared memory in a cp.async ring of NS stages of I2D_KC
// points; each of the 8 warps keeps the accumulators of up to I2D_MAXG items
// (up to 2 x 4 tiles, which share their fragments).  Each CTA writes its
// partial sums; dot_sum_kernel adds them in a fixed order and
// int2e_form_kernel forms the integrals.
//
// What bounds it: staging (90 rows of 16 points a stage for the 45 pairs of
// 9 orbitals, 8 warps waiting for it together) and the tensor pipe in turn.
// Ne, CAS(8e,9o), K = 113905: 93 + 8 us (complex tiles, their sum) -> 42 + 8 + 3
// (products, sum, form); 66 for the products before the item shapes were
// unrolled one by one (dp_item).
#include <algorithm>

#include "common.cuh"
#include "kernels.cuh"
#include "reductions.cuh"

namespace td1c {

constexpr int I2D_KC = 16;                 // points per stage
constexpr int I2D_PITCH = 2 * I2D_KC + 8;  // doubles per staged row: 8 mod 16, so 2 rows x 2 parts x 4 points fall in distinct banks

__device__ __forceinline__ void dmma_8x8x4(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}
__device__ __forceinline__ void cp_async_16(unsigned dst, const void* src, unsigned src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

static size_t dp_smem(int nrow, int ns) { return sizeof(double) * (size_t)ns * nrow * I2D_PITCH; }
// three stages where they fit in shared memory, else two
static int dp_stages(int nrow) { return dp_smem(nrow, 3) <= 224 * 1024 ? 3 : 2; }

// one stage of an item of NM x NN tiles
template <int NM, int NN>
__device__ __forceinline__ void dp_item(const double* sm, const int (&aoff)[2], const int (&boff)[4], double (&acc)[2][4][2]) {
#pragma unroll
  for (int s = 0; s < I2D_KC / 4; ++s) {
    double av[NM], bv[NN];
#pragma unroll
    for (int i = 0; i < NM; ++i) av[i] = sm[aoff[i] + 8 * s];
#pragma unroll
    for (int j = 0; j < NN; ++j) bv[j] = sm[boff[j] + 8 * s];
#pragma unroll
    for (int i = 0; i < NM; ++i)
#pragma unroll
      for (int j = 0; j < NN; ++j) dmma_8x8x4(acc[i][j][0], acc[i][j][1], av[i], bv[j]);
  }
}

// S = A B^T over a slice of K: A and B components (row | part << 16) of the row list, in the items' tiles
template <int NS>
__global__ void __launch_bounds__(I2D_NW * 32, 2) dot_products_kernel(DotProdArgs a) {
  extern __shared__ __align__(16) double i2d_sm[];
  const int nrows = a.nrow;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int gid = lane >> 2, tig = lane & 3;
  const size_t K = a.K;
  const size_t kper = ((K + gridDim.x - 1) / gridDim.x + I2D_KC - 1) / I2D_KC * I2D_KC;
  const size_t k0 = (size_t)blockIdx.x * kper, k1 = min(K, k0 + kper);
  const int nchunk = k1 > k0 ? (int)((k1 - k0 + I2D_KC - 1) / I2D_KC) : 0;
  const unsigned stage_bytes = (unsigned)(sizeof(double) * nrows * I2D_PITCH);
  const unsigned smem0 = (unsigned)__cvta_generic_to_shared(i2d_sm);

  // this thread copies point kk of the rows row0, row0 + NW 32 / KC, ...
  const int kk = tid % I2D_KC, row0 = tid / I2D_KC;
  auto load = [&](int chunk) {
    if (chunk >= nchunk) return;
    const size_t k = k0 + (size_t)chunk * I2D_KC + kk;
    const bool in = k < k1;
    const unsigned dst = smem0 + (unsigned)(chunk % NS) * stage_bytes + (unsigned)(2 * sizeof(double) * kk);
    for (int row = row0; row < nrows; row += I2D_NW * 32 / I2D_KC)
      cp_async_16(dst + (unsigned)(sizeof(double) * I2D_PITCH * row), a.row[row] + (in ? k : 0), in ? 16u : 0u);
  };

  // this warp's items and the lane's fragment offsets (doubles); tiles past the item repeat its first
  int nm[I2D_MAXG], nn[I2D_MAXG], shape[I2D_MAXG], aoff[I2D_MAXG][2], boff[I2D_MAXG][4];
  double acc[I2D_MAXG][2][4][2];
  const DotProdItem* wi = a.items + ((size_t)blockIdx.y * I2D_NW + warp) * I2D_MAXG;
#pragma unroll
  for (int g = 0; g < I2D_MAXG; ++g) {
    const DotProdItem G = wi[g];
    nm[g] = G.nm;
    nn[g] = G.nn;
    shape[g] = G.nm ? 4 * G.nm + G.nn - 1 : 0;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int q = a.comp[G.compa + 8 * (G.mt + (i < G.nm ? i : 0)) + gid];
      aoff[g][i] = (q & 0xffff) * I2D_PITCH + (q >> 16) + 2 * tig;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int q = a.comp[G.compb + 8 * (G.nt + (j < G.nn ? j : 0)) + gid];
      boff[g][j] = (q & 0xffff) * I2D_PITCH + (q >> 16) + 2 * tig;
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[g][i][j][0] = acc[g][i][j][1] = 0.0;
  }

#pragma unroll
  for (int s = 0; s < NS - 1; ++s) { load(s); cp_async_commit(); }
  for (int chunk = 0; chunk < nchunk; ++chunk) {
    cp_async_wait<NS - 2>();
    __syncthreads();  // stage chunk % NS complete for every thread; stage (chunk - 1) % NS free
    load(chunk + NS - 1);
    cp_async_commit();
    const double* sm = i2d_sm + (size_t)(chunk % NS) * nrows * I2D_PITCH;
#pragma unroll
    for (int g = 0; g < I2D_MAXG; ++g) {
      switch (shape[g]) {  // one branch per item and stage
        case 4 * 1 + 0: dp_item<1, 1>(sm, aoff[g], boff[g], acc[g]); break;
        case 4 * 1 + 1: dp_item<1, 2>(sm, aoff[g], boff[g], acc[g]); break;
        case 4 * 1 + 2: dp_item<1, 3>(sm, aoff[g], boff[g], acc[g]); break;
        case 4 * 1 + 3: dp_item<1, 4>(sm, aoff[g], boff[g], acc[g]); break;
        case 4 * 2 + 0: dp_item<2, 1>(sm, aoff[g], boff[g], acc[g]); break;
        case 4 * 2 + 1: dp_item<2, 2>(sm, aoff[g], boff[g], acc[g]); break;
        case 4 * 2 + 2: dp_item<2, 3>(sm, aoff[g], boff[g], acc[g]); break;
        case 4 * 2 + 3: dp_item<2, 4>(sm, aoff[g], boff[g], acc[g]); break;
        default: break;
      }
    }
  }
  cp_async_wait<0>();
  // partial sums: S(row gid, columns 2 tig, 2 tig + 1) of each tile
  double* out = a.partial + (size_t)blockIdx.x * a.nent;
#pragma unroll
  for (int g = 0; g < I2D_MAXG; ++g) {
    const DotProdItem G = wi[g];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (i < nm[g] && j < nn[g])
          *reinterpret_cast<double2*>(out + (size_t)(G.tile0 + (G.mt + i) * G.ntile + G.nt + j) * 64 + gid * 8 + 2 * tig) =
              make_double2(acc[g][i][j][0], acc[g][i][j][1]);
  }
}

// fixed-order sums over the K slices: 32 entries x 32 slice groups per CTA (every load of a thread in
// flight at once; with 8 groups the 37 loads of each took 9 us where the data fits in 1)
__global__ void __launch_bounds__(1024) dot_sum_kernel(const double* __restrict__ partial, int nsplit, int nent,
                                                       double* __restrict__ sum) {
  __shared__ double part[32][33];
  const int lane = threadIdx.x & 31, gq = threadIdx.x >> 5, e = blockIdx.x * 32 + lane;
  double s = 0.0;
  if (e < nent) {
#pragma unroll 10
    for (int c = gq; c < nsplit; c += 32) s += partial[(size_t)c * nent + e];
  }
  part[gq][lane] = s;
  __syncthreads();
  double t = part[lane][gq];  // warp gq adds the groups of entry gq by a fixed tree
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if (lane == 0 && blockIdx.x * 32 + gq < nent) sum[blockIdx.x * 32 + gq] = t;
}

// int2e(i, j, k, l) from the sums: form = (RR, RI, IR, II) entries (-1: zero), flag 1 the column is
// conjugated, flag 2 the integral is the conjugate of int2e(j, i, l, k)
__global__ void int2e_form_kernel(int n4, const int4* __restrict__ form, const unsigned char* __restrict__ flag,
                                  const double* __restrict__ sum, cplx* __restrict__ int2e) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n4) return;
  const int4 f = form[t];
  cplx v = mkc(0, 0);
  if (f.x >= 0) {
    const double rr = sum[f.x], ri = f.y >= 0 ? sum[f.y] : 0.0, ir = f.z >= 0 ? sum[f.z] : 0.0, ii = f.w >= 0 ? sum[f.w] : 0.0;
    const int fl = flag[t];
    v = (fl & 1) ? mkc(rr + ii, ir - ri) : mkc(rr - ii, ri + ir);
    if (fl & 2) v.y = -v.y;
  }
  int2e[t] = v;
}

// K slices: two CTAs per SM where they fit, and at least four stages of points each
int dot_products_nsplit(const DotProdArgs& a, int nsm) {
  const int per = 2 * dp_smem(a.nrow, dp_stages(a.nrow)) <= 224 * 1024 ? 2 : 1;
  return std::max(1, std::min(per * nsm, (int)(a.K / (4 * I2D_KC))));
}

int launch_dot_products(const DotProdArgs& a, int nsplit, cudaStream_t st) {
  if (a.nent <= 0) return 0;
  const int ns = dp_stages(a.nrow);
  const size_t smem = dp_smem(a.nrow, ns);
  if (smem > 227 * 1024 || nsplit < 1) return (int)cudaErrorInvalidValue;
  static bool attr = false;
  if (!attr) {
    cudaFuncSetAttribute(dot_products_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    cudaFuncSetAttribute(dot_products_kernel<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    attr = true;
  }
  const dim3 grid(nsplit, a.nsets);
  if (ns == 3) dot_products_kernel<3><<<grid, I2D_NW * 32, smem, st>>>(a);
  else dot_products_kernel<2><<<grid, I2D_NW * 32, smem, st>>>(a);
  dot_sum_kernel<<<(a.nent + 31) / 32, 1024, 0, st>>>(a.partial, nsplit, a.nent, a.sum);
  return (int)cudaGetLastError();
}

int launch_int2e_dmma(const I2dArgs& d, int nsplit, cudaStream_t st) {
  const int n4 = d.nact * d.nact * d.nact * d.nact;
  if (n4 == 0) return 0;
  const int rc = launch_dot_products(d.prod, nsplit, st);
  if (rc) return rc;
  int2e_form_kernel<<<(n4 + 255) / 256, 256, 0, st>>>(n4, d.form, d.flag, d.prod.sum, d.int2e);
  return (int)cudaGetLastError();
}

}  // namespace td1c
