// legendre_par.cu -- the theta <-> l transforms of legendre_gemm.cu with the
// parity of the Legendre functions folded in.
//
// On a theta grid symmetric about cos(theta) = 0 (Gauss-Legendre nodes)
// P_l^m(-x) = (-1)^(l+m) P_l^m(x), so with t' = nlat - 1 - t the mirror of
// node t and p the parity of l + m
//   l -> theta   E_p[t] = sum_{l of parity p} T[t][l] B[l],  t < h = ceil(nlat / 2)
//                C[t] = E_0[t] + E_1[t],  C[t'] = E_0[t] - E_1[t]
//   theta -> l   S_0[t] = B[t] + B[t'],  S_1[t] = B[t] - B[t'],  t < h
//                C[l] = sum_t T[l][t] S_p(l)[t]
// (the node at cos(theta) = 0 of an odd grid is its own mirror: S_0 = B,
// S_1 = 0, and E_1 = 0 there).  Each transform is two products of half the
// rows and half the depth: half the operations of the dense product, which
// was bound by the FP64 tensor pipe (67 to 75% busy).  The caller checks the
// tables' symmetry when they are bound; other tables keep the dense kernel.
//
// One CTA does both parities of up to 8 MT rows per parity and 32 NT real
// columns: 8 warps = 2 parities x 4 column groups, each warp MT m-tiles x NT
// n-tiles of mma.sync.m8n8k4.f64.  The depth runs in chunks of 16 per parity,
// double-buffered: the tables (stored per parity, rows padded to the chunk)
// and, for l -> theta, the slab rows arrive by cp.async; for theta -> l the
// slab rows t and t' go through registers, where the pair product and the
// fold are formed.  All pitches are 4 mod 16 doubles (conflict-free fragment
// loads).  The l -> theta epilogue swaps half of the accumulators between the
// two parity warps of a column group through shared memory, so that each
// writes both mirrors of its half of the rows.
//
// What bounds it: the FP64 tensor pipe (55% busy) and, between chunks, the
// barrier that frees a buffer.  Measured against the dense kernel (Ne, 1199
// radial points, nlat 95, lmax2 94, 54 pairs): pair densities to l 107.6 -> 64.5
// us, potentials to theta 96 -> 61.4, orbitals to theta 17 -> 11.0, g and v2 to l
// 21.6 -> 16.8; a right-hand side 633 -> 538.  Three m-tiles per warp made the
// right-hand side 11% slower (fewer warps in flight), and 512-thread
// persistent CTAs over the same tiles took 75 and 74 us where this takes 62
// and 59.
#include "common.cuh"
#include "kernels.cuh"

namespace td1c {

constexpr int LP_BK = 16;          // depth of a chunk, per parity
constexpr int LP_LDA = LP_BK + 4;  // pitch of a staged table row (doubles)
constexpr int LP_NT = 256;         // threads

template <int MT, int NT>
__host__ __device__ constexpr size_t lp_smem_bytes() {
  return sizeof(double) * 2 * 2 * ((size_t)8 * MT * LP_LDA + (size_t)LP_BK * (32 * NT + 4));
}

__device__ __forceinline__ void lp_dmma(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}
__device__ __forceinline__ void lp_cp16(double* dst, const double* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(ok ? 16u : 0u)
               : "memory");
}

// M, K: rows and depth of the dense transform; TO_L: theta -> l (K = nlat) or
// l -> theta (M = nlat)
template <int MT, int NT, bool TO_L, bool PAIR>
__global__ void __launch_bounds__(LP_NT) legendre_par_kernel(const LegGemmBatch* __restrict__ batches, int M, int K, int N) {
  constexpr int BM = 8 * MT, BN = 32 * NT, LDB = BN + 4;
  constexpr int NA = (2 * BM * LP_BK / 2 + LP_NT - 1) / LP_NT;  // 16-byte table copies per thread and chunk
  constexpr int NB = LP_BK * BN / 2 / LP_NT;                    // complex slab elements per thread, parity and chunk
  static_assert(NB >= 1 && NB * LP_NT == LP_BK * BN / 2, "slab chunk divides among the threads");
  extern __shared__ __align__(16) double lp_sm[];
  double* As = lp_sm;                          // [2 buffers][2 parities][BM][LDA]
  double* Bs = lp_sm + 2 * 2 * BM * LP_LDA;    // [2 buffers][2 parities][BK][LDB]
  const LegGemmBatch bt = batches[blockIdx.z];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int gid = lane >> 2, tig = lane & 3;
  const int par = warp >> 2, wn = warp & 3;
  const int mpar = bt.mpar;  // |m| mod 2: l of parity p are 2 q + ((mpar + p) & 1)
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int nt = TO_L ? K : M;           // theta points
  const int h = (nt + 1) / 2;            // nodes of the half grid
  const int nl = TO_L ? M : K;           // multipoles
  const int hl = (nl + 1) / 2;           // at most this many of each parity
  const int rows = TO_L ? hl : h, depth = TO_L ? h : hl;
  const int ldp = legendre_ldp(depth);

  auto load_a = [&](int k0, int s) {
    double* as = As + s * 2 * BM * LP_LDA;
#pragma unroll
    for (int q = 0; q < NA; ++q) {
      const int e = tid + LP_NT * q;  // (parity, row, 16-byte column)
      if (NA * LP_NT != BM * LP_BK && e >= BM * LP_BK) break;
      const int r = e / (LP_BK / 2), kk = 2 * (e % (LP_BK / 2));
      const int p = r / BM, mm = r % BM;
      const bool ok = m0 + mm < rows;
      lp_cp16(as + r * LP_LDA + kk, bt.P + (ok ? (size_t)(p * rows + m0 + mm) * ldp + k0 + kk : 0), ok);
    }
  };
  // l -> theta: the slab rows of both parities, copied as they are
  auto load_b = [&](int k0, int s) {
    double* bs = Bs + s * 2 * LP_BK * LDB;
#pragma unroll
    for (int q = 0; q < 2 * NB; ++q) {
      const int e = tid + LP_NT * q;
      const int r = e / (BN / 2), nn = 2 * (e % (BN / 2));
      const int p = r / LP_BK, kk = r % LP_BK;
      const int l = 2 * (k0 + kk) + ((mpar + p) & 1), gn = n0 + nn;
      const bool ok = l < K && gn < N;
      lp_cp16(bs + r * LDB + nn, bt.B0 + (ok ? (size_t)l * bt.ldb + gn : 0), ok);
    }
  };
  // theta -> l: nodes t and t' wait in registers as loaded (the loads of the next chunk are in
  // flight during this chunk's products); the pair product conj(Bj) Bi and the fold are formed
  // on the way to shared memory
  constexpr int NR = PAIR ? 4 : 2;
  cplx raw[NB][NR];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int q = 0; q < NB; ++q) {
      const int e = tid + LP_NT * q;
      const int kk = e / (BN / 2), gn = n0 + 2 * (e % (BN / 2));
      const int t = k0 + kk, u = nt - 1 - t;
      const bool in = t < h && gn < N, mir = in && u != t;
      const size_t ot = (size_t)t * (bt.ldb >> 1) + (gn >> 1), ou = (size_t)u * (bt.ldb >> 1) + (gn >> 1);
      const cplx* b0 = reinterpret_cast<const cplx*>(bt.B0);
      const cplx* b1 = reinterpret_cast<const cplx*>(bt.B1);
      raw[q][0] = in ? __ldg(b0 + ot) : mkc(0, 0);
      raw[q][1] = mir ? __ldg(b0 + ou) : mkc(0, 0);
      if (PAIR) {
        raw[q][2] = in ? __ldg(b1 + ot) : mkc(0, 0);
        raw[q][NR - 1] = mir ? __ldg(b1 + ou) : mkc(0, 0);
      }
    }
  };
  auto store_b = [&](int k0, int s) {
    double* bs = Bs + s * 2 * LP_BK * LDB;
#pragma unroll
    for (int q = 0; q < NB; ++q) {
      const int e = tid + LP_NT * q;
      const int kk = e / (BN / 2), t = k0 + kk;
      const cplx v = PAIR ? cmulc(raw[q][0], raw[q][NR - 2]) : raw[q][0];
      const cplx w = PAIR ? cmulc(raw[q][1], raw[q][NR - 1]) : raw[q][1];
      const int o = kk * LDB + 2 * (e % (BN / 2));
      *reinterpret_cast<cplx*>(bs + o) = cadd(v, w);
      *reinterpret_cast<cplx*>(bs + LP_BK * LDB + o) = 2 * t == nt - 1 ? mkc(0, 0) : csub(v, w);
    }
  };

  double acc[MT][NT][2];
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  const int nchunk = (depth + LP_BK - 1) / LP_BK;
  load_a(0, 0);
  if (TO_L) {
    fetch(0);
    store_b(0, 0);
    if (nchunk > 1) fetch(LP_BK);
  } else {
    load_b(0, 0);
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  for (int c = 0; c < nchunk; ++c) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();  // chunk c is staged for every thread, and the other buffer (chunk c - 1) has been read
    if (c + 1 < nchunk) {
      load_a((c + 1) * LP_BK, (c + 1) & 1);
      if (TO_L) {
        store_b((c + 1) * LP_BK, (c + 1) & 1);
        if (c + 2 < nchunk) fetch((c + 2) * LP_BK);
      } else {
        load_b((c + 1) * LP_BK, (c + 1) & 1);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
    const double* as = As + ((c & 1) * 2 + par) * BM * LP_LDA + gid * LP_LDA + tig;
    const double* bs = Bs + ((c & 1) * 2 + par) * LP_BK * LDB + tig * LDB + wn * 8 * NT + gid;
    const int ksn = min(LP_BK / 4, (depth - c * LP_BK + 3) / 4);
#pragma unroll
    for (int ks = 0; ks < LP_BK / 4; ++ks) {
      if (ks >= ksn) break;
      double a[MT], b[NT];
#pragma unroll
      for (int i = 0; i < MT; ++i) a[i] = as[i * 8 * LP_LDA + 4 * ks];
#pragma unroll
      for (int j = 0; j < NT; ++j) b[j] = bs[4 * ks * LDB + 8 * j];
#pragma unroll
      for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j) lp_dmma(acc[i][j][0], acc[i][j][1], a[i], b[j]);
    }
  }
  // fragment (row gid, columns 2 tig, 2 tig + 1) of each tile
  const int gn0 = n0 + wn * 8 * NT + 2 * tig;
  if (TO_L) {
#pragma unroll
    for (int i = 0; i < MT; ++i) {
      const int l = 2 * (m0 + i * 8 + gid) + ((mpar + par) & 1);
      if (l >= M) continue;
#pragma unroll
      for (int j = 0; j < NT; ++j)
        if (gn0 + 8 * j < N)
          *reinterpret_cast<double2*>(bt.C + (size_t)l * bt.ldc + gn0 + 8 * j) = make_double2(acc[i][j][0], acc[i][j][1]);
    }
  } else {
    // warp (parity p, group wn) keeps the m-tiles i = p mod 2 and hands over the others
    double2* xs = reinterpret_cast<double2*>(lp_sm) + (size_t)wn * MT * NT * 32 + lane;
    static_assert(sizeof(double2) * 4 * MT * NT * 32 <= lp_smem_bytes<MT, NT>(), "exchange buffer");
    __syncthreads();  // the staged chunks have been read
#pragma unroll
    for (int i = 0; i < MT; ++i)
      if ((i & 1) != par)
#pragma unroll
        for (int j = 0; j < NT; ++j) xs[(i * NT + j) * 32] = make_double2(acc[i][j][0], acc[i][j][1]);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < MT; ++i) {
      if ((i & 1) != par) continue;
      const int t = m0 + i * 8 + gid, u = nt - 1 - t;
      if (t >= h) continue;
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        if (gn0 + 8 * j >= N) continue;
        const double2 o = xs[(i * NT + j) * 32];
        const double2 mine = make_double2(acc[i][j][0], acc[i][j][1]);
        const double2 e0 = par ? o : mine, e1 = par ? mine : o;
        *reinterpret_cast<double2*>(bt.C + (size_t)t * bt.ldc + gn0 + 8 * j) = make_double2(e0.x + e1.x, e0.y + e1.y);
        if (u != t)
          *reinterpret_cast<double2*>(bt.C + (size_t)u * bt.ldc + gn0 + 8 * j) = make_double2(e0.x - e1.x, e0.y - e1.y);
      }
    }
  }
}

template <int MT, int NT, bool TO_L, bool PAIR>
static void lp_launch(const LegGemmBatch* d_batches, int nbatch, int M, int K, int N, int rows, cudaStream_t st) {
  constexpr size_t smem = lp_smem_bytes<MT, NT>();
  static bool attr = false;
  if (!attr && smem > 48 * 1024) {
    cudaFuncSetAttribute(legendre_par_kernel<MT, NT, TO_L, PAIR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    attr = true;
  }
  dim3 grid((N + 32 * NT - 1) / (32 * NT), (rows + 8 * MT - 1) / (8 * MT), nbatch);
  legendre_par_kernel<MT, NT, TO_L, PAIR><<<grid, LP_NT, smem, st>>>(d_batches, M, K, N);
}

template <int MT, int NT>
static void lp_launch_kind(const LegGemmBatch* b, int nb, int M, int K, int N, int rows, bool to_l, bool pair, cudaStream_t st) {
  if (!to_l) lp_launch<MT, NT, false, false>(b, nb, M, K, N, rows, st);
  else if (!pair) lp_launch<MT, NT, true, false>(b, nb, M, K, N, rows, st);
  else lp_launch<MT, NT, true, true>(b, nb, M, K, N, rows, st);
}

// mt: at most this many m-tiles per parity (3 or 6; 0 by size)
int launch_legendre_par(const LegGemmBatch* d_batches, int nbatch, int M, int K, int N, bool to_l, bool pair, int mt,
                        cudaStream_t st) {
  if (nbatch <= 0) return 0;
  if (N % 2) return (int)cudaErrorInvalidValue;  // slabs are complex: 16-byte pairs
  const int rows = (M + 1) / 2;
  const int tiles = (rows + 7) / 8;
  const int most = mt == 3 ? 3 : 6;
  const int per = (tiles + (tiles + most - 1) / most - 1) / ((tiles + most - 1) / most);  // m-tiles of one CTA, split evenly
  if (per <= 2) lp_launch_kind<2, 2>(d_batches, nbatch, M, K, N, rows, to_l, pair, st);
  else if (per <= 3) lp_launch_kind<3, 2>(d_batches, nbatch, M, K, N, rows, to_l, pair, st);
  else if (per <= 4) lp_launch_kind<4, 2>(d_batches, nbatch, M, K, N, rows, to_l, pair, st);
  else lp_launch_kind<6, 2>(d_batches, nbatch, M, K, N, rows, to_l, pair, st);
  return (int)cudaGetLastError();
}

}  // namespace td1c
