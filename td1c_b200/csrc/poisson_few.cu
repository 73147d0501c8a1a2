// poisson_few.cu -- the radial Poisson solve of poisson_cond.cu for up to PS_FEW orbital pairs.
//
// The three passes there stage tiles of 32 pairs x 4 multipoles in shared memory, and the bridge pass runs a
// thread per pair down a chain of 2 (nfe - 1) dependent steps: with one pair, as in He, 31 of 32 staged rows
// are zeros and the chain is the pass.  Here each pass is a product of a small real matrix per (element, l),
// or per l, with columns (pair, re | im), as m8n8k4 DMMA tiles: a warp takes one (element, l) and all pairs,
// loads its B fragments straight from rho2 and its A fragments from tables in fragment order, all loads in
// flight at once, with no shared memory and no barrier; the bridge pass multiplies by the inverse of the
// tridiagonal matrix, formed at set-up.
//
// What bounds it: latency, of the loads within a pass and of the three launches.  He (1 pair, 40 elements of 21
// points, lmax2 46): a right-hand side
// 25.5 -> 19.4 us (calls of several contexts in turn), 8 split steps 2700 -> 2385 us.  From about 20 pairs on the staged passes are as fast
// (21 pairs, 33 elements, lmax2 52: equal) or faster (6 orbitals, 37 elements of 13 points: 57 us a right-hand
// side against 59 here; 55 pairs, 80 elements, lmax2 126: 1.8% less of a split step), since they read each
// operand table once per 32 pairs and leave more of the SM to the kernels beside them.
#include <algorithm>

#include "common.cuh"
#include "kernels.cuh"

namespace td1c {

constexpr int PSW_NT = PS_FEW / 4;  // n-tiles of four pairs
constexpr int PSF_MAXND = 25;       // the condensed factors' largest element

// tiles of the element pass's operand (rows: ni interior points and the left bridge; depth: ni points,
// the two bridge values and t) and of the share pass's (3 rows, nd points), values per (l, element)
__host__ __device__ constexpr int ps_wf_mt(int nd) { return (nd + 7) / 8; }
__host__ __device__ constexpr int ps_wf_ks(int nd) { return (nd + 2 + 3) / 4; }
__host__ __device__ constexpr int ps_sf_ks(int nd) { return (nd + 3) / 4; }
__host__ __device__ constexpr size_t ps_wf_size(int nd) { return (size_t)ps_wf_mt(nd) * ps_wf_ks(nd) * 32; }
__host__ __device__ constexpr size_t ps_sf_size(int nd) { return (size_t)ps_sf_ks(nd) * 32; }

__device__ __forceinline__ void psf_dmma(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

// the records of poisson_cond.cu as DMMA A operands in fragment order: the element pass's rows are the interior
// points and then the left bridge, its depth the interior rho and then x(left), x(right), t; the share pass's
// rows are (t, left share, right share), its depth the owned points
__global__ void ps_few_frag_kernel(PsCond f) {
  const int e = blockIdx.x, l = blockIdx.y, nd = f.nd, ni = f.ni, ks = ps_wf_ks(nd);
  const size_t le = (size_t)l * f.nfe + e;
  const double *er = f.erec + le * f.er, *sr = f.srec + le * f.sr;
  double *wf = f.wfrag + le * ps_wf_size(nd), *sf = f.sfrag + le * ps_sf_size(nd);
  for (int i = threadIdx.x; i < (int)ps_wf_size(nd); i += blockDim.x) {
    const int lane = i & 31, r = 8 * ((i >> 5) / ks) + (lane >> 2), j = 4 * ((i >> 5) % ks) + (lane & 3);
    double v = 0.0;
    if (r < ni) {
      if (j < ni) v = er[j * ni + r];
      else if (j == ni) v = -er[ni * ni + r];
      else if (j == ni + 1) v = -er[ni * ni + ni + r];
      else if (j == ni + 2) v = er[ni * ni + 2 * ni + r];
    } else if (r == ni) {
      if (j == ni) v = er[ni * ni + 3 * ni];
      else if (j == ni + 2) v = er[ni * ni + 3 * ni + 1];
    }
    wf[i] = v;
  }
  for (int i = threadIdx.x; i < (int)ps_sf_size(nd); i += blockDim.x) {
    const int lane = i & 31, r = lane >> 2, j = 4 * (i >> 5) + (lane & 3);
    sf[i] = r < 3 && j < nd ? sr[r * nd + j] : 0.0;
  }
}

// per l: the inverse of the bridge matrix in fragment order (rows and depth the bridges), a column
// per thread from the tridiagonal factors
__global__ void ps_few_binv_kernel(PsCond f) {
  const int l = blockIdx.x, nb = f.nb, c = threadIdx.x + blockIdx.y * blockDim.x;
  const int mt = (nb + 7) / 8, ks = (nb + 3) / 4;
  double* out = f.binv + (size_t)l * mt * ks * 32;
  if (c >= 4 * ks) return;
  auto at = [&](int r) -> double& { return out[((size_t)(r >> 3) * ks + (c >> 2)) * 32 + (r & 7) * 4 + (c & 3)]; };
  for (int r = 0; r < 8 * mt; ++r) at(r) = 0.0;
  if (c >= nb) return;
  const double *tm = f.tm + (size_t)l * nb, *tw = f.tw + (size_t)l * nb, *tu = f.tu + (size_t)l * nb;
  double y = 0.0;
  for (int b = c; b < nb; ++b) {  // forward: zero above the column
    y = b == c ? 1.0 : -tm[b] * y;
    at(b) = y;
  }
  double x = 0.0;
  for (int b = nb - 1; b >= 0; --b) {
    x = (at(b) - tu[b] * x) * tw[b];
    at(b) = x;
  }
}

// ---------------------------------------------------------------------------
// per-RHS passes
// ---------------------------------------------------------------------------
// 1. the element's shares of t and of the bridge right-hand sides
template <int ND>
__global__ void __launch_bounds__(32) ps_few_share_kernel(PsCondArgs a) {
  const PsCond& F = a.f;
  constexpr int KS = ps_sf_ks(ND);
  const int nfe = F.nfe, Nr = a.Nr, L2 = a.L2, npair = a.npair;
  const int lane = threadIdx.x, gid = lane >> 2, tig = lane & 3, nt = (npair + 3) / 4;
  const int e = blockIdx.x, l = blockIdx.y, i0 = ND * e - 1;
  const size_t le = (size_t)l * nfe + e;
  const double* rho = reinterpret_cast<const double*>(a.rho2) + (gid & 1);
  double b[PSW_NT][KS], A[KS];
#pragma unroll
  for (int t = 0; t < PSW_NT; ++t) {
    if (t >= nt) break;
    const int p = 4 * t + (gid >> 1);
    const double* src = rho + 2 * (((size_t)(p < npair ? p : 0) * L2 + l) * Nr);
#pragma unroll
    for (int k = 0; k < KS; ++k) {
      const int i = i0 + 4 * k + tig;  // owned points: the left bridge and the interior
      b[t][k] = (p < npair && 4 * k + tig < ND && i >= 0) ? __ldg(src + 2 * i) : 0.0;
    }
  }
#pragma unroll
  for (int k = 0; k < KS; ++k) A[k] = gid < 3 ? __ldg(F.sfrag + le * ps_sf_size(ND) + k * 32 + lane) : 0.0;
#pragma unroll
  for (int t = 0; t < PSW_NT; ++t) {
    if (t >= nt) break;
    double c0 = 0.0, c1 = 0.0;
#pragma unroll
    for (int k = 0; k < KS; ++k) psf_dmma(c0, c1, A[k], b[t][k]);
    const int p = 4 * t + tig;  // C(row gid, pair tig): re, im
    if (p >= npair || gid > 2) continue;
    if (gid == 0) a.tpart[le * npair + p] = mkc(c0, c1);
    else a.cb[(le * 2 + gid - 1) * npair + p] = mkc(c0, c1);
  }
}

// 2. per l: the bridge values x = S^-1 g with the inverse of the tridiagonal bridge matrix
// (formed at set-up) as DMMA tiles, and t = fac1 sum_e tpart_e in element order.  The substitution
// itself is a chain of 2 (nfe - 1) dependent steps; the product has none.
constexpr int PSB_P = PS_FEW;
constexpr int PSB_LD = 2 * PSB_P + 4;  // pitch of a staged row (doubles): 4 mod 16
constexpr int PSB_T = 256;

constexpr int PSB_KS = 20;         // depth steps of an A row kept in registers

__global__ void __launch_bounds__(PSB_T) ps_few_bridge_kernel(PsCondArgs a) {
  extern __shared__ __align__(16) double psb_sm[];  // [4 ks][PSB_LD] bridge right-hand sides, columns (pair, re | im)
  const PsCond& F = a.f;
  const int l = blockIdx.x, nb = F.nb, nfe = F.nfe, npair = a.npair, tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31, gid = lane >> 2, tig = lane & 3;
  const int mt_n = (nb + 7) / 8, ks_n = (nb + 3) / 4;
  const int np = npair, nt_n = (np + 3) / 4;
  // the warp's first A row is loaded while the right-hand sides arrive
  double A[PSB_KS];
  const double* Ag = F.binv + ((size_t)l * mt_n + warp) * ks_n * 32 + lane;
#pragma unroll
  for (int k = 0; k < PSB_KS; ++k) A[k] = (warp < mt_n && k < ks_n) ? __ldg(Ag + k * 32) : 0.0;
  const cplx* cb = a.cb + ((size_t)l * nfe * 2 + 1) * npair;
#pragma unroll 4
  for (int q = tid; q < 4 * ks_n * PSB_P; q += PSB_T) {
    const int r = q / PSB_P, pc = q % PSB_P;
    cplx g = mkc(0, 0);
    if (r < nb && pc < np) g = cadd(cb[(size_t)2 * r * npair + pc], cb[(size_t)(2 * r + 1) * npair + pc]);  // right share of element r, left of r + 1
    *reinterpret_cast<cplx*>(psb_sm + (size_t)r * PSB_LD + 2 * pc) = g;
  }
  // t: 16 lanes per pair, each every sixteenth element, then a fixed xor tree
  {
    const int pc = tid >> 4, s = tid & 15;
    cplx t = mkc(0, 0);
    if (pc < np)
#pragma unroll 4
      for (int e = s; e < nfe; e += 16) t = cadd(t, a.tpart[((size_t)l * nfe + e) * npair + pc]);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) { t.x += __shfl_xor_sync(0xffffffffu, t.x, o); t.y += __shfl_xor_sync(0xffffffffu, t.y, o); }
    if (s == 0 && pc < np) a.t[(size_t)l * npair + pc] = cscale(t, a.fac1[l]);
  }
  __syncthreads();
  for (int mt = warp; mt < mt_n; mt += PSB_T / 32) {
    if (mt != warp) {
      Ag = F.binv + ((size_t)l * mt_n + mt) * ks_n * 32 + lane;
#pragma unroll
      for (int k = 0; k < PSB_KS; ++k) A[k] = k < ks_n ? __ldg(Ag + k * 32) : 0.0;
    }
    for (int nt = 0; nt < nt_n; nt += 2) {  // two n-tiles at a time
      const double* B = psb_sm + (size_t)tig * PSB_LD + 8 * nt + gid;
      const int two = nt + 1 < nt_n ? 8 : 0;
      double c00 = 0.0, c01 = 0.0, c10 = 0.0, c11 = 0.0;
#pragma unroll
      for (int k = 0; k < PSB_KS; ++k) {
        if (k >= ks_n) break;
        psf_dmma(c00, c01, A[k], B[(size_t)4 * k * PSB_LD]);
        psf_dmma(c10, c11, A[k], B[(size_t)4 * k * PSB_LD + two]);
      }
      for (int k = PSB_KS; k < ks_n; ++k) {
        const double av = __ldg(Ag + k * 32);
        psf_dmma(c00, c01, av, B[(size_t)4 * k * PSB_LD]);
        psf_dmma(c10, c11, av, B[(size_t)4 * k * PSB_LD + two]);
      }
      const int b = 8 * mt + gid, p = 4 * nt + tig;
      if (b < nb) {
        cplx* xb = a.xb + ((size_t)l * nb + b) * npair;
        if (p < np) xb[p] = mkc(c00, c01);
        if (two && p + 4 < np) xb[p + 4] = mkc(c10, c11);
      }
    }
  }
}

// 3. v on the element's owned points: the interior products with the bridge
// values and t as three more depths, the left bridge as one more row; zeros
// for l < |m|
template <int ND>
__global__ void __launch_bounds__(32) ps_few_elem_kernel(PsCondArgs a) {
  const PsCond& F = a.f;
  constexpr int ni = ND - 1, KS = ps_wf_ks(ND), MT = ps_wf_mt(ND);
  const int nfe = F.nfe, nb = F.nb, Nr = a.Nr, L2 = a.L2, npair = a.npair;
  const int lane = threadIdx.x, gid = lane >> 2, tig = lane & 3, nt = (npair + 3) / 4;
  const int e = blockIdx.x, l = blockIdx.y, i0 = ND * e;
  const int part = gid & 1;
  double b[PSW_NT][KS];
#pragma unroll
  for (int t = 0; t < PSW_NT; ++t) {
    if (t >= nt) break;
    const int p = 4 * t + (gid >> 1), pp = p < npair ? p : 0;
    const double* src = reinterpret_cast<const double*>(a.rho2 + ((size_t)pp * L2 + l) * Nr + i0) + part;
#pragma unroll
    for (int k = 0; k < KS; ++k) {
      const int j = 4 * k + tig;
      const double* s = nullptr;
      if (j < ni) s = src + 2 * j;
      else if (j == ni) { if (e >= 1) s = reinterpret_cast<const double*>(a.xb + ((size_t)l * nb + e - 1) * npair + pp) + part; }
      else if (j == ni + 1) { if (e < nb) s = reinterpret_cast<const double*>(a.xb + ((size_t)l * nb + e) * npair + pp) + part; }
      else if (j == ni + 2) s = reinterpret_cast<const double*>(a.t + (size_t)l * npair + pp) + part;
      b[t][k] = (p < npair && s) ? *s : 0.0;
    }
  }
  int zero = 0;  // bit t: l < |m| of the lane's output pair in n-tile t
#pragma unroll
  for (int t = 0; t < PSW_NT; ++t) {
    const int p = 4 * t + tig, m = p < npair ? a.pair_m[p] : 0;
    if (l < (m < 0 ? -m : m)) zero |= 1 << t;
  }
  const double* wf = F.wfrag + ((size_t)l * nfe + e) * ps_wf_size(ND) + lane;
#pragma unroll
  for (int mt = 0; mt < MT; ++mt) {
    double c[PSW_NT][2], A[KS];
#pragma unroll
    for (int k = 0; k < KS; ++k) A[k] = __ldg(wf + (mt * KS + k) * 32);
#pragma unroll
    for (int t = 0; t < PSW_NT; ++t) c[t][0] = c[t][1] = 0.0;
#pragma unroll
    for (int k = 0; k < KS; ++k)
#pragma unroll
      for (int t = 0; t < PSW_NT; ++t)
        if (t < nt) psf_dmma(c[t][0], c[t][1], A[k], b[t][k]);
    const int r = 8 * mt + gid;  // row: interior point, then the left bridge
    if (r > ni || (r == ni && e == 0)) continue;
    const int i = r < ni ? i0 + r : i0 - 1;
#pragma unroll
    for (int t = 0; t < PSW_NT; ++t) {
      const int p = 4 * t + tig;
      if (p < npair) a.v2sph[((size_t)p * L2 + l) * Nr + i] = (zero >> t) & 1 ? mkc(0, 0) : mkc(c[t][0], c[t][1]);
    }
  }
}

void ps_few_sizes(const PsCond& f, size_t* wf, size_t* sf, size_t* bi) {
  *wf = (size_t)f.L2 * f.nfe * ps_wf_size(f.nd);
  *sf = (size_t)f.L2 * f.nfe * ps_sf_size(f.nd);
  *bi = (size_t)f.L2 * ((f.nb + 7) / 8) * ((f.nb + 3) / 4) * 32;
}

// after launch_ps_cond_setup, whose records and bridge factors it rearranges
int launch_ps_few_setup(const PsCond& f, cudaStream_t st) {
  ps_few_frag_kernel<<<dim3(f.nfe, f.L2), 64, 0, st>>>(f);
  if (f.nb > 0) ps_few_binv_kernel<<<dim3(f.L2, (f.nb + 63) / 64 + 1), 64, 0, st>>>(f);
  return (int)cudaGetLastError();
}

// Every element size has its own instance: the rows, depths and their guards are then constants.  One instance with
// loops to the largest size and guards, and this, us a right-hand side of 30 elements, lmax1 20, by points per
// element less one: 9 pairs 5: 67.1, 64.4; 7: 69.7, 65.7; 8: 69.3, 66.3; 10: 71.4, 67.3; 12: 72.7, 68.8; 16: 72.8, 68.9;
// 18: 78.9, 75.4; one pair 8: 44.2, 42.2; 12: 46.2, 45.0; 18: 45.9, 44.2 (7 and 20 within 0.6).
template <int ND>
static int psf_launch(const PsCondArgs& a, cudaStream_t st) {
  if (a.f.nd != ND) {
    if constexpr (ND > 2) return psf_launch<ND - 1>(a, st);
    return ST_CONFIG;
  }
  const dim3 grid(a.f.nfe, a.L2);
  const size_t smem = sizeof(double) * 4 * (size_t)((a.f.nb + 3) / 4) * PSB_LD;
  ps_few_share_kernel<ND><<<grid, 32, 0, st>>>(a);
  ps_few_bridge_kernel<<<a.L2, PSB_T, smem, st>>>(a);
  ps_few_elem_kernel<ND><<<grid, 32, 0, st>>>(a);
  return (int)cudaGetLastError();
}

int launch_ps_few(const PsCondArgs& a, cudaStream_t st) { return psf_launch<PSF_MAXND>(a, st); }

// whether the few-pair passes take these sizes (48 KB of shared memory for the bridge pass)
bool ps_few_fits(const PsCond& f, int npair) {
  return npair <= PS_FEW && f.nd >= 2 && f.nd <= PSF_MAXND && sizeof(double) * 4 * (size_t)((f.nb + 3) / 4) * PSB_LD <= 48 * 1024;
}

}  // namespace td1c
