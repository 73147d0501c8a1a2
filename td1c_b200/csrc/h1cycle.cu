// h1cycle.cu -- the passes of a one-body split step (h1itr_prop.F90:2-175,
// dpade_prod.F90:2-124) with the bridge solve folded into the element pass.
//
// h1prop.cu applies M^-1 = (1 + c T_l)^-1 by static condensation in two
// launches per correction cycle: an element pass and, because a bridge value
// needs the shares of every element, a tridiagonal solve over the nfe - 1
// bridge points (a serial chain of 2 nfe complex steps per orbital).  M is a
// short time step, so the inverse of that tridiagonal matrix falls off fast
// away from its diagonal: by a factor of 1e-4 to 1e-9 per element.  Here the
// columns of the inverse are formed once per factor and a band of half-width w
// of it kept, where every entry outside the band is below 2^-64 of the row's
// diagonal (far below the rounding of the products it would enter); an element's CTA
// then gets its two bridge values as short dot products with the shares of the
// 2 w + 2 elements around it, and a whole cycle is one launch, which also
// decides whether the graph's loop goes on.  A factor whose inverse falls off
// slower (w > H1C_WMAX) keeps the two-launch passes of h1prop.cu.
//
// One CTA per (element e, LC multipoles), 256 threads:
//   1. bridge values left and right of the element for its multipoles and
//      their l +- 1 neighbours; x(I_e) = z - GL x(left) - GR x(right);
//   2. finished corrections into torb and the residual norm (each point once);
//   3. y = the alpha-weighted sum of a row's l +- 1 neighbours;
//   4. the next right-hand side r = a x + b T x + cz V x, with the radial
//      derivative P y (and T x in a first pass) as DMMA tiles: rows the
//      element's points, columns (row, re | im);
//   5. [z; left share; right share] = A' r as DMMA tiles, where A' is the
//      interior inverse with the two rows v_L A^-1 and v_R A^-1 below it (they
//      lie in the padding of the last 8-row tile).
// The matrices of steps 3 and 5 are stored in fragment order, so staging and
// fragment loads are linear; z is [l][element][orbital][point] and the shares
// are [l][element][side][orbital], so everything a CTA stages is contiguous
// per multipole.
//
// What bounds it: the latency of the chain stage, bridge dots, sum, products,
// store within a CTA (three CTAs of 70 KB share an SM).  Measured (Ne, 60
// elements of 21 points, lmax1 47, 10 orbitals): a cycle 52 + 12.3 us (element
// pass + bridge solve) -> 42, a first pass 45 + 12 -> 34; He (40 elements, lmax1 23,
// 1 orbital) a cycle 15 + 9.5 -> 14.  Taking the derivative of every neighbour instead of their
// sum (step 3) took 51 us: more operands in shared memory, two CTAs per SM.
#include <algorithm>

#include "common.cuh"
#include "kernels.cuh"

namespace td1c {

constexpr int H1C_NT = 256;
constexpr int H1C_LC = 3;    // multipoles per CTA
constexpr int H1C_LH = H1C_LC + 2;
constexpr int H1C_TPR = 2;   // torb values of a multipole that a thread holds: nfun nd <= 2 * 256

__device__ __forceinline__ void h1c_dmma(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}
__device__ __forceinline__ void h1c_cp16(void* dst, const void* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(ok ? 16u : 0u)
               : "memory");
}
__device__ __forceinline__ void h1c_cp8(void* dst, const void* src, bool ok) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(ok ? 8u : 0u)
               : "memory");
}

// tile counts of A' (ni + 2 rows, ni deep) and of the band blocks (np x np)
__host__ __device__ constexpr int h1c_mta(int nd) { return (nd + 1 + 7) / 8; }
__host__ __device__ constexpr int h1c_ksa(int nd) { return (nd - 1 + 3) / 4; }
__host__ __device__ constexpr int h1c_mtp(int nd) { return (nd + 1 + 7) / 8; }
__host__ __device__ constexpr int h1c_ksp(int nd) { return (nd + 1 + 3) / 4; }
size_t h1c_af_size(int nd) { return (size_t)h1c_mta(nd) * h1c_ksa(nd) * 32; }   // complex values per (l, element)
size_t h1c_band_size(int nd) { return (size_t)h1c_mtp(nd) * h1c_ksp(nd) * 32; }  // doubles per element

// ---------------------------------------------------------------------------
// set-up
// ---------------------------------------------------------------------------
// per element: P (derivative; the diagonal only at the points the element owns, i.e. not at its right
// bridge) and T (kinetic off-diagonal, l >= 1) over the element's points, in fragment order; 1 / r
__global__ void h1c_band_kernel(int nfe, int nd, int Nr, const double* __restrict__ xrad, const double* __restrict__ radp,
                                const double* __restrict__ radk0, double* __restrict__ rinv, double* __restrict__ pf,
                                double* __restrict__ tf) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k <= Nr + 1; k += gridDim.x * blockDim.x) rinv[k] = k ? 1.0 / xrad[k] : 0.0;
  const int e = blockIdx.x, mt = h1c_mtp(nd), ks = h1c_ksp(nd), bw = 2 * nd + 1;
  for (int i = threadIdx.x; i < mt * ks * 32; i += blockDim.x) {
    const int lane = i & 31, k = (i >> 5) % ks, t = (i >> 5) / ks;
    const int p = 8 * t + (lane >> 2), q = 4 * k + (lane & 3), ip = nd * e + p, iq = nd * e + q;
    const bool in = p <= nd && q <= nd && ip >= 1 && ip <= Nr && iq >= 1 && iq <= Nr;
    const size_t o = in ? (size_t)bw * ip + nd + iq - ip : 0;
    pf[(size_t)e * mt * ks * 32 + i] = in && (p != q || p != nd) ? radp[o] : 0.0;
    tf[(size_t)e * mt * ks * 32 + i] = in && p != q ? radk0[o] : 0.0;
  }
}

// per (element, l): A' in fragment order and (GL, GR) side by side
__global__ void h1c_af_kernel(H1Fac f) {
  const int e = blockIdx.x, l = blockIdx.y, ni = f.ni, nd = f.nd;
  const int mt = h1c_mta(nd), ks = h1c_ksa(nd);
  const size_t le = (size_t)l * f.nfe + e;
  const cplx* ainv = f.ainv + le * ni * ni;  // Ainv(k, j) at [j][k]
  for (int i = threadIdx.x; i < mt * ks * 32; i += blockDim.x) {
    const int lane = i & 31, k = (i >> 5) % ks, t = (i >> 5) / ks;
    const int r = 8 * t + (lane >> 2), j = 4 * k + (lane & 3);
    cplx v = mkc(0, 0);
    if (j < ni) {
      if (r < ni) v = ainv[(size_t)j * ni + r];
      else if (r < ni + 2) {
        const cplx* vv = (r == ni ? f.vl : f.vr) + le * ni;
        for (int q = 0; q < ni; ++q) cfma(v, vv[q], ainv[(size_t)j * ni + q]);
      }
    }
    f.af[le * mt * ks * 32 + i] = v;
  }
  for (int k = threadIdx.x; k < ni; k += blockDim.x) {
    f.glr[le * 2 * ni + k] = f.gl[le * ni + k];
    f.glr[le * 2 * ni + ni + k] = f.gr[le * ni + k];
  }
}

// The inverse of the bridge matrix, a CTA per l and a thread per column (every ncol-th one), from its pivoted LU
// (ZGTTRS algorithm), with the thread's column in the scratch x[l][row][thread].  The band goes to
// sinv[l][row][H1C_BW]; then *w = the largest |row - column| of an entry above 2^-64 of its row's diagonal.  The
// whole inverse is not kept: its size goes with the square of the number of elements.
__global__ void h1c_sinv_kernel(H1Fac f, cplx* __restrict__ scratch, int ncol, int* w) {
  const int l = blockIdx.x, nb = f.nb, j = threadIdx.x;
  const cplx *__restrict__ dl = f.tdl + (size_t)l * nb, *__restrict__ di = f.tdi + (size_t)l * nb;
  const cplx *__restrict__ du = f.tdu + (size_t)l * nb, *__restrict__ du2 = f.tdu2 + (size_t)l * nb;
  const int* __restrict__ ip = f.tpiv + (size_t)l * nb;
  cplx* x = scratch + (size_t)l * nb * ncol + j;  // x[i * ncol]
  cplx* S = f.sinv + (size_t)l * nb * H1C_BW + H1C_WMAX;  // S(r, c) at [r * H1C_BW + c - r]
  auto column = [&](int c) {
    cplx cur = mkc(c == 0 ? 1.0 : 0.0, 0.0);
#pragma unroll 8
    for (int i = 0; i + 1 < nb; ++i) {
      const cplx nxt = mkc(c == i + 1 ? 1.0 : 0.0, 0.0), m = __ldg(dl + i);
      const bool sw = __ldg(ip + i) != i;
      const cplx a = sw ? nxt : cur, b = sw ? cur : nxt;
      x[(size_t)i * ncol] = a;
      cur = csub(b, cmul(m, a));
    }
    cplx x1 = cmul(cur, di[nb - 1]), x2 = mkc(0, 0);
    x[(size_t)(nb - 1) * ncol] = x1;
#pragma unroll 8
    for (int i = nb - 2; i >= 0; --i) {
      cplx v = csub(x[(size_t)i * ncol], cmul(__ldg(du + i), x1));
      if (i + 2 < nb) v = csub(v, cmul(__ldg(du2 + i), x2));
      v = cmul(v, __ldg(di + i));
      x[(size_t)i * ncol] = v;
      x2 = x1;
      x1 = v;
    }
  };
  for (int c = j; c < nb && j < ncol; c += ncol) {
    column(c);
    for (int i = max(0, c - H1C_WMAX); i <= min(nb - 1, c + H1C_WMAX); ++i) S[(size_t)i * H1C_BW + c - i] = x[(size_t)i * ncol];
  }
  __syncthreads();
  int far = 0;
  for (int c = j; c < nb && j < ncol; c += ncol) {
    if (nb > ncol) column(c);  // else the column still stands in x
#pragma unroll 4
    for (int i = 0; i < nb; ++i) {
      const int d = i < c ? c - i : i - c;
      const cplx v = x[(size_t)i * ncol], g = S[(size_t)i * H1C_BW];
      if (d > far && !(fabs(v.x) + fabs(v.y) <= 0x1p-64 * (fabs(g.x) + fabs(g.y)))) far = d;
    }
  }
  if (far) atomicMax(w, far);
}

int launch_h1c_bands(int nfe, int nd, int Nr, const double* xrad, const double* radp, const double* radk0, double* rinv,
                     double* pf, double* tf, cudaStream_t st) {
  h1c_band_kernel<<<nfe, 128, 0, st>>>(nfe, nd, Nr, xrad, radp, radk0, rinv, pf, tf);
  return (int)cudaGetLastError();
}
int launch_h1c_setup(const H1Fac& f, int* w, cudaStream_t st) {
  if (f.nb > 0) {
    // A' is formed last: its place, h1c_af_size >= 32 columns of it, is the scratch
    const int ncol = std::min({f.nb, (int)h1c_af_size(f.nd), 512});
    h1c_sinv_kernel<<<f.L1, (ncol + 31) / 32 * 32, 0, st>>>(f, f.af, ncol, w);
  }
  h1c_af_kernel<<<dim3(f.nfe, f.L1), 128, 0, st>>>(f);
  return (int)cudaGetLastError();
}

// ---------------------------------------------------------------------------
// the passes
// ---------------------------------------------------------------------------
// MODE 0: the first right-hand side of an input vector; 1: a correction cycle (the one after the last
// only adds its correction); 2: the only solve, without cycles, into torb
struct H1CSmem {
  int nd, nf, w, mode;
  bool vel;
  __host__ __device__ int np() const { return nd + 1; }
  __host__ __device__ int ni() const { return nd - 1; }
  __host__ __device__ size_t x() const { return 0; }
  __host__ __device__ size_t y() const { return x() + (size_t)H1C_LH * nf * np(); }  // Y and R; before them, the bridge shares
  __host__ __device__ size_t r() const { return y() + (mode != 2 ? (size_t)H1C_LC * nf * np() : 0); }
  __host__ __device__ size_t af() const {
    const size_t yr = mode != 2 ? 2 * (size_t)H1C_LC * nf * np() : 0, c = mode ? (size_t)H1C_LH * (2 * w + 3) * 2 * nf : 0;
    return y() + (yr > c ? yr : c);
  }
  __host__ __device__ size_t g() const { return af() + (mode != 2 ? (size_t)H1C_LC * h1c_mta(nd) * h1c_ksa(nd) * 32 : 0); }
  __host__ __device__ size_t si() const { return g() + (mode ? (size_t)H1C_LH * 2 * ni() : 0); }
  __host__ __device__ size_t ncplx() const { return si() + (mode ? (size_t)H1C_LH * 2 * (2 * w + 1) : 0); }
  // doubles: P, T fragments, r, 1 / r, diagonal of T, alpha
  __host__ __device__ size_t pf() const { return 2 * ncplx(); }
  __host__ __device__ size_t tf() const { return pf() + (mode != 2 ? (size_t)h1c_mtp(nd) * h1c_ksp(nd) * 32 : 0); }
  __host__ __device__ size_t xr() const { return tf() + (mode == 0 ? (size_t)h1c_mtp(nd) * h1c_ksp(nd) * 32 : 0); }
  __host__ __device__ size_t ri() const { return xr() + np(); }
  __host__ __device__ size_t td() const { return ri() + np(); }
  __host__ __device__ size_t al() const { return td() + (size_t)H1C_LC * np(); }
  __host__ __device__ size_t bytes() const { return sizeof(double) * (al() + (size_t)H1C_LH * nf); }
};

template <int NDT, int MODE>
__global__ void __launch_bounds__(H1C_NT, 3) h1c_kernel(H1CycArgs a) {
  extern __shared__ __align__(16) unsigned char h1c_sm[];
  const H1Fac& F = a.fac;
  const int nd = NDT > 0 ? NDT : F.nd;
  const int np = nd + 1, ni = nd - 1, nfe = F.nfe, nb = F.nb, L1 = a.L1, Nr = a.Nr, nfun = a.nfun, w = F.w;
  const int mta = h1c_mta(nd), ksa = h1c_ksa(nd), mtp = h1c_mtp(nd), ksp = h1c_ksp(nd);
  const int e = blockIdx.x, l0 = blockIdx.y * H1C_LC, tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31, gid = lane >> 2, tig = lane & 3;
  const bool vel = a.igauge == 1;
  const H1CSmem lay{nd, nfun, w, MODE, vel};
  cplx* sm = reinterpret_cast<cplx*>(h1c_sm);
  double* smd = reinterpret_cast<double*>(h1c_sm);
  cplx* X = sm + lay.x();    // [lh][f][np]
  cplx* Y = sm + lay.y();    // [lc][f][np]
  cplx* CB = Y;              // [lh][2w + 3][2][f]: shares of elements e - w - 1 .. e + w + 1
  cplx* R = sm + lay.r();    // [lc][f][np]
  cplx* AF = sm + lay.af();  // [lc][mta][ksa][32]
  cplx* G = sm + lay.g();    // [lh][2][ni]
  cplx* SI = sm + lay.si();  // [lh][2][2w + 1]: rows e - 1 and e of the bridge inverse
  double* PF = smd + lay.pf();
  double* TF = smd + lay.tf();
  double* XR = smd + lay.xr();  // [np] radial coordinate
  double* RI = smd + lay.ri();  // [np] its reciprocal
  double* TD = smd + lay.td();  // [lc][np]
  double* AL = smd + lay.al();  // [f][lh] alpha of l0 - 1 .. l0 + LC
  __shared__ double red[H1C_NT / 32];
  __shared__ int last;
  const int ir0 = nd * e;
  auto valid = [&](int ip) { return ip >= 1 && ip <= Nr; };
  // loops run over the CTA's multipoles outside and over contiguous ranges inside, so the only divisions are
  // by the element's compile-time sizes
  if (MODE == 1 && a.flags[0]) return;  // the residual norm is below thresh
  const int iter = MODE ? a.flags[2] : 0;
  // the tables, which do not depend on the cycle
  if (MODE != 2) {
    const int n = mta * ksa * 32;
    for (int lc = 0; lc < H1C_LC; ++lc)
      if (l0 + lc < L1) {
        const cplx* src = F.af + ((size_t)(l0 + lc) * nfe + e) * n;
        for (int q = tid; q < n; q += H1C_NT) h1c_cp16(AF + lc * n + q, src + q, true);
      }
    const int m = mtp * ksp * 16;  // 16-byte pairs
    if (vel)
      for (int q = tid; q < m; q += H1C_NT) h1c_cp16(PF + 2 * q, a.pf + (size_t)e * 2 * m + 2 * q, true);
    if (MODE == 0) {
      for (int q = tid; q < m; q += H1C_NT) h1c_cp16(TF + 2 * q, a.tf + (size_t)e * 2 * m + 2 * q, true);
      for (int q = tid; q < H1C_LC * np; q += H1C_NT) {
        const int lc = q / np, p = q % np, l = l0 + lc, ip = ir0 + p;
        const bool ok = l < L1 && valid(ip);
        h1c_cp8(TD + q, a.tdiag + (ok ? (size_t)l * Nr + ip - 1 : 0), ok);
      }
    }
    if (tid < np) {
      const bool ok = valid(ir0 + tid);
      h1c_cp8(XR + tid, a.xrad + (ok ? ir0 + tid : 0), ok);
      h1c_cp8(RI + tid, a.rinv + (ok ? ir0 + tid : 0), ok);
    }
    for (int q = tid; q < nfun * H1C_LH; q += H1C_NT) {
      const int f = q / H1C_LH, l = l0 - 1 + q % H1C_LH;
      const bool ok = l >= 0 && l < L1;
      h1c_cp8(AL + q, a.alph + (ok ? (size_t)(a.mv[f] + a.mmax1) * L1 + l : 0), ok);
    }
  }
  // the orbitals of this pass: the first correction also finishes the frozen-core columns (h1itr)
  const int f_lo = MODE == 0 ? a.f_first : (MODE == 1 ? (iter == 0 ? a.f_first : a.nfcore) : a.nfcore);
  const cplx* z_in = a.z[iter & 1];
  const cplx* cb_in = a.cb[iter & 1];
  cplx* z_out = a.z[MODE == 0 ? 0 : (iter + 1) & 1];
  cplx* cb_out = a.cb[MODE == 0 ? 0 : (iter + 1) & 1];
  const bool accumulate = MODE == 1 && iter > 0;
  cplx tv[H1C_LC][H1C_TPR];
  if (MODE == 0) {
    for (int lq = 0; lq < H1C_LH; ++lq) {
      const int l = l0 - 1 + lq;
      const bool lok = l >= 0 && l < L1;
      for (int q = tid; q < nfun * np; q += H1C_NT) {
        const int f = q / np, p = q % np;
        const bool ok = lok && f >= f_lo && valid(ir0 + p);
        h1c_cp16(X + lq * nfun * np + q, a.in + (ok ? ((size_t)f * L1 + l) * Nr + ir0 + p - 1 : 0), ok);
      }
    }
  } else {
    const int bwd = 2 * w + 1, nw = (2 * w + 3) * 2 * nfun, lo = (w + 1 - e) * 2 * nfun, hi = (nfe + w + 1 - e) * 2 * nfun;
    for (int lq = 0; lq < H1C_LH; ++lq) {
      const int l = l0 - 1 + lq;
      const bool lok = l >= 0 && l < L1;
      const size_t le = (size_t)(lok ? l : 0) * nfe + e;
      for (int q = tid; q < nfun * ni; q += H1C_NT) h1c_cp16(X + (lq * nfun + q / ni) * np + 1 + q % ni, z_in + le * nfun * ni + q, lok);
      for (int q = tid; q < nw; q += H1C_NT) {  // elements e - w - 1 .. e + w + 1, contiguous
        const bool ok = lok && q >= lo && q < hi;
        h1c_cp16(CB + lq * nw + q, cb_in + (ok ? le * 2 * nfun + q - (w + 1) * 2 * nfun : 0), ok);
      }
      for (int q = tid; q < 2 * ni; q += H1C_NT) h1c_cp16(G + lq * 2 * ni + q, F.glr + le * 2 * ni + q, lok);
      for (int q = tid; q < 2 * bwd; q += H1C_NT) {
        const int side = q >= bwd, d = q - side * bwd - w, b = e - 1 + side;
        const bool ok = lok && b >= 0 && b < nb && b + d >= 0 && b + d < nb;
        h1c_cp16(SI + lq * 2 * bwd + q, F.sinv + (ok ? ((size_t)l * nb + b) * H1C_BW + H1C_WMAX + d : 0), ok);
      }
    }
#pragma unroll
    for (int lc = 0; lc < H1C_LC; ++lc)
#pragma unroll
      for (int k = 0; k < H1C_TPR; ++k) {
        const int q = tid + k * H1C_NT, f = q / nd, ip = ir0 + q % nd, l = l0 + lc;
        tv[lc][k] = mkc(0, 0);
        if (accumulate && f < nfun && f >= a.nfcore && l < L1 && valid(ip)) tv[lc][k] = a.torb[((size_t)f * L1 + l) * Nr + ip - 1];
      }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  if (MODE) {
    // 1a. bridge values: two lanes per (multipole, orbital, side), each every other term
    const int nv = H1C_LH * nfun * 2;
    for (int q = tid >> 1; q < (nv + 15) / 16 * 16; q += H1C_NT / 2) {
      const int qq = q < nv ? q : 0, lq = qq / (2 * nfun), fs = qq - lq * 2 * nfun, f = fs >> 1, side = fs & 1;
      const int l = l0 - 1 + lq, b = e - 1 + side, m = a.mv[f], am = m < 0 ? -m : m;
      cplx x = mkc(0, 0);
      if (b >= 0 && b < nb && f >= f_lo) {
        const cplx* s = SI + (lq * 2 + side) * (2 * w + 1);
        const cplx* c = CB + (size_t)(lq * (2 * w + 3) + side) * 2 * nfun + f;  // element b - w
        for (int d = tid & 1; d <= 2 * w; d += 2) {
          const cplx gb = cadd(c[(2 * d + 1) * nfun], c[(2 * d + 2) * nfun]);
          if (l >= am) cfma(x, s[d], gb);
          else if (d == w) x = gb;  // channels below |m| pass through
        }
      }
      x.x += __shfl_xor_sync(0xffffffffu, x.x, 1);
      x.y += __shfl_xor_sync(0xffffffffu, x.y, 1);
      if (q < nv && !(tid & 1)) X[(lq * nfun + f) * np + (side ? nd : 0)] = x;
    }
    __syncthreads();
    // 1b, 2. interior points; own rows also go to torb and the norm
    double nrm = 0.0;
    auto interior = [&](int row, int lq, int k) {
      const cplx* x = X + row * np;
      const cplx* g = G + lq * 2 * ni;
      return csub(csub(x[1 + k], cmul(g[k], x[0])), cmul(g[ni + k], x[nd]));
    };
#pragma unroll
    for (int lc = 0; lc < H1C_LC; ++lc)
#pragma unroll
      for (int k = 0; k < H1C_TPR; ++k) {
        const int q = tid + k * H1C_NT, f = q / nd, p = q % nd, l = l0 + lc, row = (lc + 1) * nfun + f;
        if (f < f_lo || f >= nfun || l >= L1 || !valid(ir0 + p)) continue;
        const int m = a.mv[f];
        cplx x = X[row * np + p];
        if (p > 0 && l >= (m < 0 ? -m : m)) X[row * np + p] = x = interior(row, lc + 1, p - 1);
        nrm += cabs2(x);
        if (f >= a.nfcore) a.torb[((size_t)f * L1 + l) * Nr + ir0 + p - 1] = cadd(tv[lc][k], x);
      }
    if (MODE == 2) return;
    if (MODE == 1 && iter >= a.maxcyc) {  // the cycle limit is reached: the last correction is in
      if (a.use_loop && blockIdx.x == 0 && blockIdx.y == 0 && tid == 0) cudaGraphSetConditional(a.loop, 0u);
      return;
    }
    for (int side = 0; side < 2; ++side) {
      const int lq = side ? H1C_LH - 1 : 0, l = l0 - 1 + lq;
      if (l < L1)
        for (int q = tid; q < nfun * ni; q += H1C_NT) {
          const int f = q / ni, k = q % ni, row = lq * nfun + f, m = a.mv[f];
          if (f >= f_lo && l >= (m < 0 ? -m : m)) X[row * np + 1 + k] = interior(row, lq, k);
        }
    }
    for (int o = 16; o > 0; o >>= 1) nrm += __shfl_xor_sync(0xffffffffu, nrm, o);
    if (lane == 0) red[warp] = nrm;
  }
  __syncthreads();
  // the residual norm of the finished correction: the CTA that arrives last decides (its wait
  // overlaps the other CTAs' products; every CTA has read the flags before it arrives)
  if (MODE == 1 && tid == 0) {
    double s = 0.0;
    for (int k = 0; k < H1C_NT / 32; ++k) s += red[k];
    a.partial[blockIdx.y * gridDim.x + blockIdx.x] = s;
    __threadfence();
    last = atomicAdd(a.ticket, 1u) == gridDim.x * gridDim.y - 1;
  }
  const double zf = a.lfield ? a.lfield[2] : 0.0;
  const cplx cz = mkc(a.cz0.x * zf, a.cz0.y * zf);
  const bool do_t = MODE == 0 && (a.b.x != 0.0 || a.b.y != 0.0);
  const bool do_v = cz.x != 0.0 || cz.y != 0.0;
  // 3. y = alpha(l - 1) x(l - 1) + alpha(l) x(l + 1) of the own rows: the laser couples a row to its
  // neighbours through it, -i P y + i u / r in the velocity gauge, with u = l alpha(l - 1) x(l - 1) -
  // (l + 1) alpha(l) x(l + 1), and r y in the length gauge
  auto couple = [&](int f, int lc, int p, cplx& y, cplx& u) {
    const int l = l0 + lc, row = (lc + 1) * nfun + f, m = a.mv[f], am = m < 0 ? -m : m;
    const double* al = AL + f * H1C_LH;  // al[lq] = alpha(l0 - 1 + lq)
    y = u = mkc(0, 0);
    if (l - 1 >= am) {
      const cplx v = cscale(X[(row - nfun) * np + p], al[lc]);
      y = v;
      u = cscale(v, (double)l);
    }
    if (l >= am && l + 1 < L1) {
      const cplx v = cscale(X[(row + nfun) * np + p], al[lc + 1]);
      y = cadd(y, v);
      u = csub(u, cscale(v, (double)(l + 1)));
    }
  };
  if (do_v && vel) {
    for (int lc = 0; lc < H1C_LC; ++lc)
      for (int q = tid; q < nfun * np; q += H1C_NT) {
        cplx y, u;
        couple(q / np, lc, q % np, y, u);
        Y[lc * nfun * np + q] = y;
      }
    __syncthreads();
  }
  // 4. the right-hand side r = a x + b T x + cz V x on the element's points: P y and T x as DMMA tiles (rows
  // the points, columns (orbital row, re | im)), finished where the products come out
  {
    const double *xd = reinterpret_cast<const double*>(X + nfun * np), *yd = reinterpret_cast<const double*>(Y);  // own rows
    const int nrow = H1C_LC * nfun, ntile = (nrow + 3) / 4, fr = MODE == 0 ? a.f_first : a.nfcore;
    for (int nt = warp; nt < ntile; nt += H1C_NT / 32) {
      const int br = 4 * nt + (gid >> 1), bo = (br < nrow ? br : 0) * np * 2 + (gid & 1);
      double c[3][2], d[3][2];
#pragma unroll
      for (int t = 0; t < 3; ++t) c[t][0] = c[t][1] = d[t][0] = d[t][1] = 0.0;
      if (do_v && vel) {
#pragma unroll
        for (int k = 0; k < 6; ++k) {
          if (NDT == 0 && k >= ksp) break;
          const int q = 4 * k + tig;
          const double b = (br < nrow && q < np) ? yd[bo + 2 * q] : 0.0;
#pragma unroll
          for (int t = 0; t < 3; ++t)
            if (NDT > 0 || t < mtp) h1c_dmma(c[t][0], c[t][1], PF[(t * ksp + k) * 32 + lane], b);
        }
      }
      if (do_t) {
#pragma unroll
        for (int k = 0; k < 6; ++k) {
          if (NDT == 0 && k >= ksp) break;
          const int q = 4 * k + tig;
          const double b = (br < nrow && q < np) ? xd[bo + 2 * q] : 0.0;
#pragma unroll
          for (int t = 0; t < 3; ++t)
            if (NDT > 0 || t < mtp) h1c_dmma(d[t][0], d[t][1], TF[(t * ksp + k) * 32 + lane], b);
        }
      }
      const int cr = 4 * nt + tig;
      if (cr >= nrow) continue;
      const int lc = cr / nfun, f = cr - lc * nfun, l = l0 + lc, row = cr + nfun, m = a.mv[f], am = m < 0 ? -m : m;
      const bool dyn = f >= a.nfcore, live = f >= fr && l < L1;  // frozen-core rows take the a-term only
#pragma unroll
      for (int t = 0; t < 3; ++t) {
        const int p = 8 * t + gid, ip = ir0 + p;
        if (p >= np) continue;
        const bool owner = p != nd;  // the right bridge's point-local terms belong to the next element
        cplx r = mkc(0, 0);
        if (live && valid(ip)) {
          if (MODE == 0) {
            const cplx x = X[row * np + p];
            if (owner) r = cmul(a.a, x);
            if (do_t && dyn && l >= am) {
              cplx tx = mkc(d[t][0], d[t][1]);
              if (l == 0) {  // l = 0 has its own table (it differs at the nucleus)
                tx = mkc(0, 0);
                for (int q = 0; q < np; ++q)
                  if (q != p && valid(ir0 + q)) {
                    const double k = a.radk[(size_t)(2 * nd + 1) * ip + nd + q - p];
                    const cplx xq = X[row * np + q];
                    tx.x = fma(k, xq.x, tx.x); tx.y = fma(k, xq.y, tx.y);
                  }
              }
              if (owner) {
                const double td = TD[lc * np + p];
                tx.x = fma(td, x.x, tx.x); tx.y = fma(td, x.y, tx.y);
              }
              cfma(r, a.b, tx);
            }
          }
          if (do_v && dyn) {
            cplx y, u, h = mkc(0, 0);
            couple(f, lc, p, y, u);
            if (vel) {
              h = mkc(c[t][1], -c[t][0]);
              if (owner) { h.x = fma(-RI[p], u.y, h.x); h.y = fma(RI[p], u.x, h.y); }
            } else if (owner) {
              h = cscale(y, XR[p]);
            }
            cfma(r, cz, h);
          }
        }
        R[cr * np + p] = r;
      }
    }
  }
  __syncthreads();
  // 5. z and the bridge shares: A' r with the real and imaginary part of A' as two real products
  //    over the columns (orbital, re | im)
  {
    const double* rd = reinterpret_cast<const double*>(R);
    const int f0 = MODE == 0 ? a.f_first : a.nfcore, nfo = nfun - f0, nto = (nfo + 3) / 4;
    for (int it = warp; it < H1C_LC * mta * nto; it += H1C_NT / 32) {
      const int lc = it / (mta * nto), t = (it / nto) % mta, nt = it % nto, l = l0 + lc;
      if (l >= L1) continue;
      const int fb = f0 + 4 * nt + (gid >> 1);
      const double* B = rd + (size_t)(lc * nfun + (fb < nfun ? fb : 0)) * np * 2 + 2 + (gid & 1);  // interior points
      const cplx* A = AF + (size_t)(lc * mta + t) * ksa * 32 + lane;
      double u0 = 0.0, u1 = 0.0, v0 = 0.0, v1 = 0.0;
#pragma unroll
      for (int k = 0; k < (NDT > 0 ? h1c_ksa(NDT) : 6); ++k) {
        if (NDT == 0 && k >= ksa) break;
        const int j = 4 * k + tig;
        const double b = (fb < nfun && j < ni) ? B[2 * j] : 0.0;
        const cplx av = A[k * 32];
        h1c_dmma(u0, u1, av.x, b);
        h1c_dmma(v0, v1, av.y, b);
      }
      const int f = f0 + 4 * nt + tig, r = 8 * t + gid;
      if (f >= nfun || r >= ni + 2) continue;
      const int m = a.mv[f];
      const bool pass = l < (m < 0 ? -m : m);  // channels below |m| pass through
      const cplx v = mkc(u0 - v1, u1 + v0);
      const cplx* rr = R + (size_t)(lc * nfun + f) * np;
      if (r < ni) {
        z_out[(((size_t)l * nfe + e) * nfun + f) * ni + r] = pass ? rr[1 + r] : v;
      } else {
        const int side = r - ni;
        const cplx rb = rr[side ? nd : 0];
        cb_out[(((size_t)l * nfe + e) * 2 + side) * nfun + f] = pass ? rb : csub(rb, v);
      }
    }
  }
  if (MODE == 0 && blockIdx.x == 0 && blockIdx.y == 0 && tid < 3) a.flags[tid] = 0;  // done, corrections, cycle
  if (MODE == 1 && last) {  // written before the last two barriers
    const int nblk = gridDim.x * gridDim.y;
    __threadfence();
    double s = 0.0;
    for (int b = tid; b < nblk; b += H1C_NT) s += __ldcg(a.partial + b);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) red[warp] = s;
    __syncthreads();
    if (tid == 0) {
      double t = 0.0;
      for (int k = 0; k < H1C_NT / 32; ++k) t += red[k];
      const int fin = sqrt(t / a.norm_div) < a.thresh ? 1 : 0;
      *a.ticket = 0u;
      a.flags[0] = fin;
      if (!fin) a.flags[1] += 1;  // a correction has been solved for
      a.flags[2] = iter + 1;
      if (a.use_loop) cudaGraphSetConditional(a.loop, fin ? 0u : 1u);
    }
  }
}

template <int NDT, int MODE>
static int h1c_launch(const H1CycArgs& a, cudaStream_t st) {
  static size_t cur = 0;
  const size_t smem = H1CSmem{a.fac.nd, a.nfun, a.fac.w, MODE, a.igauge == 1}.bytes();
  if (smem > 48 * 1024 && smem > cur) {
    cudaError_t e = cudaFuncSetAttribute(h1c_kernel<NDT, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    cur = smem;
  }
  h1c_kernel<NDT, MODE><<<dim3(a.fac.nfe, (a.L1 + H1C_LC - 1) / H1C_LC), H1C_NT, smem, st>>>(a);
  return (int)cudaGetLastError();
}

// whether the folded passes take these sizes (the band's width w is known once the factor is built)
bool h1c_fits(int nd, int nfun, int w, int igauge) {
  if (w < 0 || w > H1C_WMAX || nd < 2 || nd > 20 || nfun > 16) return false;
  for (int mode = 0; mode < 3; ++mode)
    if (H1CSmem{nd, nfun, w, mode, igauge == 1}.bytes() > 220 * 1024) return false;
  static_assert(16 * 20 <= H1C_TPR * H1C_NT, "a thread holds H1C_TPR values of torb");
  return true;
}

int launch_h1c(const H1CycArgs& a, int mode, cudaStream_t st) {
  if (a.fac.nd == 20) {  // 21-point Lobatto elements
    return mode == 0 ? h1c_launch<20, 0>(a, st) : (mode == 1 ? h1c_launch<20, 1>(a, st) : h1c_launch<20, 2>(a, st));
  }
  return mode == 0 ? h1c_launch<0, 0>(a, st) : (mode == 1 ? h1c_launch<0, 1>(a, st) : h1c_launch<0, 2>(a, st));
}

}  // namespace td1c
