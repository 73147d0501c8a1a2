// onebody.cu -- one-body part of the orbital RHS on the FEDVR x (l, m) basis.
//
//   h0orb(r,l,i) = sum_{r'} T_l(r,r') orb(r',l,i)           hprod_tprod.F90:152-235
//   h1orb        = length gauge  E r alpha_lm coupling      hprod_zprod.F90:108-135
//                  velocity gauge A (-i alpha)(d/dr, (l+1)/r) hprod_pzprod.F90:114-213
//   frozen core in velocity gauge also gets E r alpha_lm    hprod_htot.F90:120-122
//
// T and the derivative P couple a radial point to the points of its finite
// element, a bridge point to those of both its elements.  One CTA takes one
// element, OB_LC multipoles and one orbital: the element's points and the
// previous element's (for the left bridge, which the element owns) of those
// rows and their l +- 1 neighbours go to shared memory once; T x and P y run
// as DMMA tiles (m8n8k4: rows the owned points, columns (multipole, re | im),
// depth the points), with y = alpha(l-1) x(l-1) + alpha(l) x(l+1), so the
// derivative is taken of the coupled sum instead of every neighbour.  The
// matrices are stored in fragment order (launch_onebody_tables), l = 0 with its
// own kinetic table; the diagonal of T is per (l, r).
//
// The pass runs beside the mean-field chain, so its footprint counts as much as
// its time: 12 KB of shared memory per CTA where the scalar stencil over
// 32-point radial tiles (82 multiply-adds per point and row from shared memory)
// held 110 KB.  What bounds it is the latency of its two loads (points, then table
// fragments).  Ne (60 elements of 21 points, 48 multipoles, 10 orbitals): 61 -> 24 us,
// and 465 -> 450 for a right-hand side.
#include <algorithm>

#include "common.cuh"
#include "kernels.cuh"

namespace td1c {

constexpr int OB_LC = 8, OB_NT = 128;

// tiles of an element: owned points x (its points; the previous element's points for row 0)
__host__ __device__ constexpr int ob_mt(int nd) { return (nd + 7) / 8; }
__host__ __device__ constexpr int ob_ks(int nd) { return (nd + 1 + 3) / 4; }
__host__ __device__ constexpr int ob_kp(int nd) { return (nd + 3) / 4; }
__host__ __device__ constexpr int ob_one(int nd) { return (ob_mt(nd) * ob_ks(nd) + ob_kp(nd)) * 32; }  // one matrix, doubles
size_t onebody_table_size(int nd, int nfe) { return (size_t)3 * ob_one(nd) * nfe; }
// staged row: previous element's nd points, the element's nd + 1; pitch 4 mod 8 (complex): distinct banks
__host__ __device__ constexpr int ob_pitch(int nd) { return (2 * nd + 1 + 3) / 8 * 8 + 4; }

__device__ __forceinline__ void ob_dmma(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

// per element: T (l >= 1), T (l = 0) off the diagonal and P, in fragment order
__global__ void ob_table_kernel(int nfe, int nd, int Nr, const double* __restrict__ radk, const double* __restrict__ radk0,
                                const double* __restrict__ radp, double* __restrict__ tab) {
  const int e = blockIdx.x, which = blockIdx.y, one = ob_one(nd), mt = ob_mt(nd), ks = ob_ks(nd), bw = 2 * nd + 1;
  const double* src = which == 0 ? radk0 : (which == 1 ? radk : radp);
  for (int i = threadIdx.x; i < one; i += blockDim.x) {
    const int lane = i & 31, tile = i >> 5;
    int p, q;  // row point and column point, relative to the left bridge
    if (tile < mt * ks) {
      p = 8 * (tile / ks) + (lane >> 2);
      q = 4 * (tile % ks) + (lane & 3);
      if (q > nd) p = nd;
    } else {
      const int j = 4 * (tile - mt * ks) + (lane & 3);
      p = (lane >> 2) == 0 && j < nd ? 0 : nd;
      q = j - nd;
    }
    const int ip = nd * e + p, iq = nd * e + q;
    const bool in = p < nd && ip >= 1 && ip <= Nr && iq >= 1 && iq <= Nr && (which == 2 || p != q);
    tab[((size_t)e * 3 + which) * one + i] = in ? src[(size_t)bw * ip + nd + q - p] : 0.0;
  }
}
int launch_onebody_tables(int nfe, int nd, int Nr, const double* radk, const double* radk0, const double* radp, double* tab,
                          cudaStream_t st) {
  ob_table_kernel<<<dim3(nfe, 3), 128, 0, st>>>(nfe, nd, Nr, radk, radk0, radp, tab);
  return (int)cudaGetLastError();
}

template <int NDT>
__global__ void __launch_bounds__(OB_NT) onebody_kernel(OneBodyArgs a) {
  extern __shared__ __align__(16) cplx ob_sm[];
  const int Nr = a.Nr, L1 = a.L1, nd = NDT > 0 ? NDT : a.nd;
  constexpr int MT = NDT > 0 ? ob_mt(NDT) : 4, KS = NDT > 0 ? ob_ks(NDT) : 7, KP = NDT > 0 ? ob_kp(NDT) : 7;
  const int mt = ob_mt(nd), ks = ob_ks(nd), kp = ob_kp(nd), one = ob_one(nd), S = ob_pitch(nd), W = 2 * nd + 1;
  cplx* X = ob_sm;                     // [LC + 2][S]: points ir0 - nd .. ir0 + nd
  cplx* Y = X + (OB_LC + 2) * S;       // [LC][S]
  const int e = blockIdx.x, l0 = blockIdx.y * OB_LC, f = blockIdx.z, ir0 = nd * e;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gid = lane >> 2, tig = lane & 3;
  const int m = a.mval[f], am = m < 0 ? -m : m;
  const cplx* __restrict__ orb = a.orb + (size_t)f * L1 * Nr;
  const double* __restrict__ al = a.alph + (size_t)(m + a.mmax1) * L1;
  const double zf = a.lfield[2], ef = a.lfield[5];
  const bool vel = a.igauge == 1;
  for (int q = tid; q < (OB_LC + 2) * W; q += OB_NT) {
    const int lq = q / W, j = q % W, l = l0 - 1 + lq, r = ir0 - nd + j - 1;
    X[lq * S + j] = (l >= 0 && l < L1 && r >= 0 && r < Nr) ? __ldg(orb + (size_t)l * Nr + r) : mkc(0.0, 0.0);
  }
  __syncthreads();
  // the coupled sum y and u = l alpha(l-1) x(l-1) - (l+1) alpha(l) x(l+1) at point j of own row lc
  auto couple = [&](int lc, int j, cplx& y, cplx& u) {
    const int l = l0 + lc;
    y = u = mkc(0, 0);
    if (l - 1 >= am && l < L1) {
      const cplx v = cscale(X[lc * S + j], al[l - 1]);
      y = v;
      u = cscale(v, (double)l);
    }
    if (l >= am && l <= L1 - 2) {
      const cplx v = cscale(X[(lc + 2) * S + j], al[l]);
      y = cadd(y, v);
      u = csub(u, cscale(v, (double)(l + 1)));
    }
  };
  if (vel) {
    for (int q = tid; q < OB_LC * W; q += OB_NT) {
      cplx u;
      couple(q / W, q % W, Y[q / W * S + q % W], u);
    }
    __syncthreads();
  }
  // warp = (matrix, n-tile of 4 multipoles): T x -> h0 in warps 0, 1; P y -> h1 in warps 2, 3
  const bool is_p = warp >= 2;
  const int nt = warp & 1, bl = 4 * nt + (gid >> 1);  // the lane's column: own row bl, part gid & 1
  const double* B = reinterpret_cast<const double*>(is_p ? Y + bl * S : X + (bl + 1) * S) + (gid & 1);
  double c[MT][2], c0[MT][2];
#pragma unroll
  for (int t = 0; t < MT; ++t) c[t][0] = c[t][1] = c0[t][0] = c0[t][1] = 0.0;
  auto product = [&](const double* A, double (&o)[MT][2]) {
#pragma unroll
    for (int k = 0; k < KS; ++k) {
      if (NDT == 0 && k >= ks) break;
      const int q = 4 * k + tig;
      const double b = q <= nd ? B[2 * (nd + q)] : 0.0;
#pragma unroll
      for (int t = 0; t < MT; ++t)
        if (NDT > 0 || t < mt) ob_dmma(o[t][0], o[t][1], __ldg(A + (t * ks + k) * 32 + lane), b);
    }
#pragma unroll
    for (int k = 0; k < KP; ++k) {  // the left bridge's coupling to the previous element
      if (NDT == 0 && k >= kp) break;
      const int j = 4 * k + tig;
      ob_dmma(o[0][0], o[0][1], __ldg(A + (mt * ks + k) * 32 + lane), j < nd ? B[2 * j] : 0.0);
    }
  };
  const double* tab = a.tab + (size_t)e * 3 * one;
  if (!is_p) {
    product(tab, c);
    if (l0 == 0 && nt == 0) product(tab + one, c0);
  } else if (vel) {
    product(tab + 2 * one, c);
  }
  const int lc = 4 * nt + tig, l = l0 + lc;  // the lane's outputs: point 8 t + gid of own row lc
  if (l >= L1) return;
  const double zz = vel ? (f < a.nfcore ? ef : 0.0) : zf;  // length-gauge coupling; E on the frozen core in the velocity gauge
#pragma unroll
  for (int t = 0; t < MT; ++t) {
    const int p = 8 * t + gid, r = ir0 + p - 1;
    if (p >= nd || r < 0 || r >= Nr) continue;
    const size_t o = ((size_t)f * L1 + l) * Nr + r;
    if (!is_p) {
      cplx h = mkc(0, 0);
      if (l >= am) {
        const cplx x = X[(lc + 1) * S + nd + p];
        const double td = a.tdiag[(size_t)l * Nr + r];
        const bool z = l == 0;
        h = mkc(fma(td, x.x, z ? c0[t][0] : c[t][0]), fma(td, x.y, z ? c0[t][1] : c[t][1]));
      }
      a.h0orb[o] = h;
    } else {
      cplx y, u, h = mkc(0, 0);
      couple(lc, nd + p, y, u);
      const double x = a.xrad[r + 1];
      if (vel) {
        const double ri = 1.0 / x;
        h = mkc(zf * (c[t][1] - ri * u.y), zf * (ri * u.x - c[t][0]));
      }
      if (zz != 0.0) { h.x = fma(zz * x, y.x, h.x); h.y = fma(zz * x, y.y, h.y); }
      a.h1orb[o] = h;
    }
  }
}

int launch_onebody(const OneBodyArgs& a, cudaStream_t st) {
  if (a.nd > 25 || (a.Nr + 1) % a.nd) return ST_CONFIG;
  const dim3 grid((a.Nr + 1) / a.nd, (a.L1 + OB_LC - 1) / OB_LC, a.nfun);
  const size_t smem = sizeof(cplx) * (2 * OB_LC + 2) * ob_pitch(a.nd);
  if (a.nd == 20) onebody_kernel<20><<<grid, OB_NT, smem, st>>>(a);
  else onebody_kernel<0><<<grid, OB_NT, smem, st>>>(a);
  return (int)cudaGetLastError();
}

}  // namespace td1c
