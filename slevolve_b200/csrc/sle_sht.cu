// Gauss-Legendre spherical-harmonic transform for sm_100a, FP64.
//
// Same transform as the reference (SLEvolve python/slevolve/sht.py:148-343, Fortran spharmt):
//   analysis   U[l,m] = (sum_j P~_lm(mu_j) (S or D by the parity of l-m)_m(j)) / 1.41421356,
//              S/D = (F_north(m) w_j +/- F_south(m) w_j) / nlon, F = rFFT of the grid rows;
//   synthesis  G_north/south(m, j) = 1.41421356 * sum_l U[l,m] P~_lm(mu_j) over even +/- odd l-m,
//              grid rows = unnormalised inverse real FFT of G (Im of m = 0 ignored).
//
// Design (B200):
//   * One block per latitude pair does the row FFTs (radix-8 Stockham in shared memory on
//     nlon/2-point complex sequences, real/complex split) and the north/south fold.
//   * The Legendre functions are regenerated on the fly in FP64 with a two-term recurrence
//     Q_l = mu Q_{l-1} + be_l Q_{l-2} (P~_l = cf_l Q_l) that restarts every SEG degrees from
//     seeds computed once per plan with the reference's own normalised recursion
//     (sht.py:105-144).  Segments are the work units: analysis = one warp per (m, segment),
//     latitudes spread over the lanes (8 per lane at nlat = 512), the latitude sums through shared
//     memory; synthesis = one block per (m, 128 latitudes), its warps dealing out the segments.
//   * (segment, latitude-group) blocks whose |P~| never exceeds 1e-35 (near the poles at high
//     m) are skipped.
#include "sle_internal.cuh"
#include "sle_fft.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <numeric>
#include <vector>

namespace sle {

static thread_local char g_err[1024] = "";

void set_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof g_err, fmt, ap);
  va_end(ap);
}

// --------------------------------------------------------------------------- helpers
// (complex helpers and the Stockham FFT: sle_fft.cuh)

// ------------------------------------------------------------------- plan set-up kernels
// Gauss-Legendre nodes and weights: the Newton iteration of the reference gaulw
// (sht.py:65-101), per node, in the same operation order (no contraction into FMA).
__global__ void k_gauss_nodes(int n, double tol, double* mu, double* w, int* fail) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double pi = 3.141592653589793;  // 4*atan(1) in binary64
  double z = cos(__ddiv_rn(__dmul_rn(pi, __dsub_rn((double)(i + 1), 0.25)), __dadd_rn((double)n, 0.5)));
  double zfin = 0.0, ppfin = 1.0;
  bool done = false;
  for (int sweep = 0; sweep < 10 && !done; ++sweep) {
    double p1 = 1.0, p2 = 0.0;
    for (int k = 1; k <= n; ++k) {
      const double p3 = p2;
      p2 = p1;
      const double a = __dmul_rn(__dmul_rn(__dsub_rn(2.0 * k, 1.0), z), p2);
      const double b = __dmul_rn(__dsub_rn((double)k, 1.0), p3);
      p1 = __ddiv_rn(__dsub_rn(a, b), (double)k);
    }
    const double pp = __ddiv_rn(__dmul_rn((double)n, __dsub_rn(__dmul_rn(z, p1), p2)),
                                __dsub_rn(__dmul_rn(z, z), 1.0));
    const double z1 = z;
    z = __dsub_rn(z1, __ddiv_rn(p1, pp));
    if (fabs(__dsub_rn(z, z1)) < tol) {
      zfin = z;
      ppfin = pp;
      done = true;
    }
  }
  if (!done) atomicExch(fail, 1);
  mu[i] = zfin;
  w[i] = __ddiv_rn(2.0, __dmul_rn(__dmul_rn(__dsub_rn(1.0, __dmul_rn(zfin, zfin)), ppfin), ppfin));
}

// Seeds of every (segment, latitude) and the per-(segment, group) maximum of |P~|.  P~ follows
// the reference LEGEND recursion (sht.py:105-144) operation by operation.  A segment starting at
// degree l0 > m stores (Q_{l0-2}, Q_{l0-1}) in its own scale (P~_l = cf_l Q_l with cf_l0 = 1,
// so Q_{l0-1} = P~_{l0-1} / eps_l0 and Q_{l0-2} = P~_{l0-2} / (eps_l0 eps_{l0-1})); the first
// segment (l0 = m) stores (P~_mm, 0) and uses be_m = 1.  Every degree of every segment then
// follows the same update Q_l = mu Q_{l-1} + be_l Q_{l-2}.
__global__ void k_legendre_tables(sle::ShtDev P, double2* seeds, double* segmax) {
  const int m = blockIdx.x, g = blockIdx.y, lane = threadIdx.x;
  const int j = g * 32 + lane;
  const bool ok = j < P.nh;
  const double x = ok ? P.mu[j] : 0.0;
  const double sinsq = __dsub_rn(1.0, __dmul_rn(x, x));
  double A = 1.0, B = 0.0, prod = 1.0;
  for (int i = 1; i <= m; ++i) {
    A = __dadd_rn(A, 2.0);
    B = __dadd_rn(B, 2.0);
    prod = __ddiv_rn(__dmul_rn(__dmul_rn(prod, sinsq), A), B);
  }
  const int L = P.lmax;
  const double pmm = __dsqrt_rn(__dmul_rn(0.5, prod));
  const double pm1 = __dmul_rn(__dmul_rn(__dsqrt_rn((double)(2 * m + 3)), x), pmm);
  const int np1 = m + 1;
  const double eps_m1 = __dsqrt_rn(__ddiv_rn((double)(np1 * np1 - m * m), (double)(4 * np1 * np1 - 1)));
  double t = __dsub_rn(__dmul_rn(x, pm1), __dmul_rn(eps_m1, pmm));  // x P_{n-1} - eps_{n-1} P_{n-2}
  double prev1 = 0.0, prev2 = 0.0, eps_prev = 0.0;
  double smax = 0.0;
  int seg = P.segoff[m];
  for (int l = m; l <= L; ++l) {
    double pl, eps_l;
    if (l == m) {
      pl = pmm;
      eps_l = 0.0;
    } else if (l == m + 1) {
      pl = pm1;
      eps_l = eps_m1;
    } else {
      eps_l = __dsqrt_rn(__ddiv_rn((double)(l * l - m * m), (double)(4 * l * l - 1)));
      pl = __ddiv_rn(t, eps_l);
      t = __dsub_rn(__dmul_rn(x, pl), __dmul_rn(eps_l, prev1));
    }
    const int r = (l - m) % SEG;
    if (r == 0 && ok) {
      double2 sd;
      if (l == m) {
        sd = make_double2(pmm, 0.0);
      } else {
        sd = make_double2(__ddiv_rn(prev2, __dmul_rn(eps_l, eps_prev)), __ddiv_rn(prev1, eps_l));
      }
      seeds[(size_t)seg * P.nh + j] = sd;
    }
    smax = fmax(smax, ok ? fabs(pl) : 0.0);
    if (r == SEG - 1 || l == L) {
      double v = smax;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
      if (lane == 0) segmax[(size_t)seg * P.ngrp + g] = v;
      smax = 0.0;
      ++seg;
    }
    prev2 = prev1;
    prev1 = pl;
    eps_prev = eps_l;
  }
}

// Recurrence coefficients in segment scale: cf (P~ = cf Q) and be_l = -eps_{l-1}^2 (be_m = 1).
__global__ void k_legendre_coef(sle::ShtDev P, double* be, double* cf) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= P.nseg) return;
  const int m = P.seg_m[s], l0 = P.seg_l0[s];
  const int l1 = min(l0 + SEG, P.lmax + 1);
  const long long base = P.moff[m] + (l0 - m);
  double c = 1.0;
  cf[base] = 1.0;
  if (l0 == m) {
    be[base] = 1.0;  // Q_m = be_m * P~_mm with the first segment's seeds (P~_mm, 0)
  } else {
    const int k = l0 - 1;
    be[base] = -__ddiv_rn((double)(k * k - m * m), (double)(4 * k * k - 1));
  }
  for (int l = l0 + 1; l < l1; ++l) {
    const double eps = __dsqrt_rn(__ddiv_rn((double)(l * l - m * m), (double)(4 * l * l - 1)));
    c = __ddiv_rn(c, eps);
    cf[base + (l - l0)] = c;
    const int k = l - 1;
    be[base + (l - l0)] = -__ddiv_rn((double)(k * k - m * m), (double)(4 * k * k - 1));
  }
}

__global__ void k_istart(sle::ShtDev P, const double* segmax, unsigned char* istart) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= P.nseg) return;
  int g = 0;
  while (g < P.ngrp && segmax[(size_t)s * P.ngrp + g] < SIG_THRESHOLD) ++g;
  istart[s] = (unsigned char)g;
}

// Seeds of the pieces of fseg degrees that the FP64 kernels walk: the recurrence carried through each
// segment with the kernels' own operations, its state (Q_{l0-2}, Q_{l0-1}) stored where a piece starts.
__global__ void k_piece_seeds(sle::ShtDev P, double2* out) {
  const int s = blockIdx.x, m = P.seg_m[s], l0 = P.seg_l0[s];
  const int len = min(SEG, P.lmax + 1 - l0), first = P.leg.fsegoff[m] + (l0 - m) / P.leg.fseg;
  const long long base = P.moff[m] + (l0 - m);
  for (int j = threadIdx.x; j < P.nh; j += blockDim.x) {
    const double mu = P.mu[j];
    const double2 sd = P.seeds[(size_t)s * P.nh + j];
    double qa = sd.x, qb = sd.y;
    for (int t = 0; t < len; ++t) {
      if (t % P.leg.fseg == 0) out[(size_t)(first + t / P.leg.fseg) * P.nh + j] = make_double2(qa, qb);
      const double q = fma(mu, qb, __dmul_rn(P.be[base + t], qa));
      qa = qb;
      qb = q;
    }
  }
}

__global__ void k_lidx(sle::ShtDev P, int* lidx) {
  const int m = blockIdx.x;
  const long long base = P.moff[m];
  for (int l = m + threadIdx.x; l <= P.lmax; l += blockDim.x) lidx[base + (l - m)] = l;
}

struct GridPtrs {
  const double* p[MAXF];
  int kind[MAXF];                  // analysis source (SrcKind)
  const unsigned char* m0[MAXF];
  const unsigned char* m1[MAXF];
};
struct OutGridPtrs {
  double* p[MAXF];
  double* out2[MAXF];        // optional epilogue out2 = grid * mul2
  const double* mul2[MAXF];
};
struct SpecPtrs {
  double2* p[MAXF];
};
struct CSpecPtrs {
  const double2* p[MAXF];
};

// Row rFFT of the north row j and south row nlat-1-j of field blockIdx.y, then the fold
// S = F_N w_j/nlon + F_S w_j/nlon, D = F_N w_j/nlon - F_S w_j/nlon for m <= lmax
// (sht.py:277-287).  X layout [f][0=S,1=D][m][j].  N = nlon/2 complex points per row.
// The row FFTs of one latitude pair for a source kind known at compile time.
template <int N>
struct FoldRows64 {
  const double* g;
  const unsigned char* m0;
  const unsigned char* m1;
  int j, nlat;
  const double2* tw;
  double2* A;
  template <int K>
  __device__ __forceinline__ void operator()() const {
    fft_rows<2, N, false>(TypedPairRows<K>{g, m0, m1, j, nlat, 2 * N}, A, tw, SmemRows<N, double2>{A});
  }
};

template <int N>
__global__ void __launch_bounds__(fft_nt(2, N)) k_fft_fold(sle::ShtDev P, GridPtrs g) {
  extern __shared__ double2 sm[];
  double2* A = sm;
  const int j = blockIdx.x, f = blockIdx.y;
  touch_twiddles<N, fft_nt(2, N)>(P.tw);
  const double wn = P.wn[j], ws = P.ws[j];
  pdl_wait();
  pdl_trigger();
  if (field_gated_off(P, f)) return;
  with_src_kind(g.kind[f], FoldRows64<N>{g.p[f], g.m0[f], g.m1[f], j, P.nlat, P.tw, A});
  const SmemRows<N, double2> Z{A};
  double2* XS = P.X + ((size_t)(f * 2 + 0) * P.nm) * P.nh;
  double2* XD = P.X + ((size_t)(f * 2 + 1) * P.nm) * P.nh;
  for (int m = threadIdx.x; m < P.nm; m += blockDim.x) {
    double2 xr[2];
    const double2 twm = (m > 0 && m < N) ? __ldg(P.tw + m) : make_double2(1.0, 0.0);
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const double2 z0 = Z(r, 0);
      if (m == 0) {
        xr[r] = make_double2(z0.x + z0.y, 0.0);
      } else if (m == N) {
        xr[r] = make_double2(z0.x - z0.y, 0.0);
      } else {
        const double2 zm = Z(r, m);
        const double2 zn = Z(r, N - m);
        const double2 zc = make_double2(zn.x, -zn.y);
        const double2 e = cscale(cadd(zm, zc), 0.5);
        const double2 dz = csub(zm, zc);
        const double2 o = make_double2(0.5 * dz.y, -0.5 * dz.x);  // (zm - zc) / (2i)
        xr[r] = cadd(e, cmul(twm, o));
      }
    }
    const double2 a = cscale(xr[0], wn);
    const double2 b = cscale(xr[1], ws);
    XS[(size_t)m * P.nh + j] = cadd(a, b);
    XD[(size_t)m * P.nh + j] = csub(a, b);
  }
}

// Inverse: north spectrum E + O, south E - O (m <= lmax, 0 above), unnormalised inverse
// real FFT of both rows (sht.py:330-339 with the nlon scaling folded out); field blockIdx.y.
// The half-length complex packing of both rows is formed first, each thread taking a pair of orders
// (m, N - m), so that every (E, O) pair is read once (the packing of an index needs both orders; formed
// while the first pass reads its inputs, per row and index, the same sums were read four times through
// L1 and the blocks waited on those loads); the last pass writes the output rows (and the optional
// epilogue out2 = grid * mul2).  Bound: latency (one latitude pair per block, less than two blocks
// per SM for one field); with the synthesis sums 15.0 -> 8.6 us at
// 256 x 512 and 9.1 -> 4.7 us at 64 x 128, one field.
template <int N>
__global__ void __launch_bounds__(fft_nt(2, N)) k_ifft_unfold(sle::ShtDev P, OutGridPtrs g) {
  extern __shared__ double2 sm[];
  constexpr int NT = fft_nt(2, N);
  double2* A = sm;
  const int j = blockIdx.x, f = blockIdx.y;
  touch_twiddles<N, NT>(P.tw);
  pdl_wait();
  pdl_trigger();
  if (field_gated_off(P, f)) return;
  const int js = P.nlat - 1 - j;
  const double2* G = P.EO + ((size_t)f * P.nh + j) * P.nm * 2;   // (E, O) of each order
  const SmemRows<N, double2> Z{A};
  const double2 zero = make_double2(0.0, 0.0);
  for (int p = threadIdx.x; p < N / 2; p += NT) {
    // the orders a and b of this thread's two outputs (p = 0: the indices 0 and N / 2)
    const int a = p, b = p ? N - p : N / 2;
    const bool ina = a < P.nm, inb = b < P.nm, inn = p == 0 && N < P.nm;
    const double2 ea = ina ? G[2 * a] : zero, oa = ina ? G[2 * a + 1] : zero;
    const double2 eb = inb ? G[2 * b] : zero, ob = inb ? G[2 * b + 1] : zero;
    const double2 en = inn ? G[2 * N] : zero, on = inn ? G[2 * N + 1] : zero;   // the Nyquist order
    const double2 ta = __ldg(P.tw + a), tb = __ldg(P.tw + b);
#pragma unroll
    for (int r = 0; r < 2; ++r) {   // north E + O, south E - O
      const double2 ga = r ? csub(ea, oa) : cadd(ea, oa), gb = r ? csub(eb, ob) : cadd(eb, ob);
      double2 x = ga, y = make_double2(gb.x, -gb.y);
      if (p == 0) {
        x = make_double2(ga.x, 0.0);
        y = make_double2(r ? en.x - on.x : en.x + on.x, 0.0);
      }
      double2 e = cadd(x, y), o = cmul(csub(x, y), make_double2(ta.x, -ta.y));   // exp(+2 pi i m / nlon)
      Z.put(r, a, make_double2(e.x - o.y, e.y + o.x));                           // e + i o
      x = gb;
      y = (p == 0) ? make_double2(gb.x, -gb.y) : make_double2(ga.x, -ga.y);
      e = cadd(x, y);
      o = cmul(csub(x, y), make_double2(tb.x, -tb.y));
      Z.put(r, b, make_double2(e.x - o.y, e.y + o.x));
    }
  }
  __syncthreads();
  const size_t ro = (size_t)j * (2 * N), rso = (size_t)js * (2 * N);
  double* out2 = g.out2[f];
  const double* mul2 = g.mul2[f];
  GridRowsOut sink{reinterpret_cast<double2*>(g.p[f] + ro), reinterpret_cast<double2*>(g.p[f] + rso),
                     out2 ? reinterpret_cast<double2*>(out2 + ro) : nullptr,
                     out2 ? reinterpret_cast<double2*>(out2 + rso) : nullptr,
                     out2 ? reinterpret_cast<const double2*>(mul2 + ro) : nullptr,
                     out2 ? reinterpret_cast<const double2*>(mul2 + rso) : nullptr};
  fft_rows_inplace<2, N, true>(A, P.tw, sink);
}

// ------------------------------------------------------------------ Legendre analysis
// One warp per (order, 64-degree segment): lanes hold latitudes, NA groups of 32 at a time, and
// walk the segment's degrees together.  Per degree and latitude the recurrence costs two FP64
// operations and each field two; the per-lane sums of 16 values are then added up over the warp
// through shared memory (each lane stores its 16 partial sums, a pair of lanes adds the 32 of one
// value), which costs about 6 instructions per degree, where a butterfly with its selects and
// two-word shuffles cost 27.  The totals collect in shared memory and leave scaled and coalesced.
// Bound: FP64 issue while there are warps to issue from; a single field at L = 511 is bound by its
// chains of dependent operations (FP64 pipe active in 42 % of the SMs' active cycles, ten warps per SM,
// blocks for 1.3 waves).  F = 2 shares one recurrence between two fields (6 operations instead of 8 per
// degree and latitude).
// Measured on one field, fold included, back to back in a CUDA graph: 30.3 -> 25.9 us at L = 511
// (16.4 -> 10.3 at L = 255, 13.1 -> 6.4 at L = 63); four fields at L = 511 91.3 -> 64.6 us.
constexpr int ANA_V = 16;             // values per warp reduction
constexpr int ANA_RS = 33;            // row stride of the reduction buffer (bank-conflict free both ways)
constexpr int ANA_WARPS = 2;          // warps (independent segments) per block
constexpr int ANA_NAMAX = 8;          // latitude groups per pass

// Degrees of segment s over the latitude groups g0 .. g0+NA-1 (latitudes at or beyond nh count as
// zero): ANA_V / (2 F) degrees per batch, each advancing the recurrence of the lane's NA latitudes
// and summing its products with the folded input of the degree's parity (segments start at even
// l - m, batches at even degrees).  The staged recurrence coefficients are zero-padded to a whole
// number of batches; the extra degrees are computed and not written.  sacc[(degree F + field) 2 +
// component] receives the sums (added to what is there when `more`).
template <int NA, int F>
__device__ __forceinline__ void ana_pass(const sle::ShtDev& P, int s, int m, int g0, int len,
                                         const double2* const (&Xf)[F], int lane, bool more,
                                         const double* __restrict__ sbe, double* __restrict__ red,
                                         double* __restrict__ sacc) {
  constexpr int TL = ANA_V / (2 * F);
  const int nh = P.nh;
  double mu[NA], qa[NA], qb[NA];
  double2 xs[F][NA], xd[F][NA];
#pragma unroll
  for (int i = 0; i < NA; ++i) {
    const int j = (g0 + i) * 32 + lane;
    const bool ok = j < nh;
    mu[i] = ok ? P.mu[j] : 0.0;
    const double2 sd = ok ? P.leg.fseeds[(size_t)s * nh + j] : make_double2(0.0, 0.0);
    qa[i] = sd.x;
    qb[i] = sd.y;
#pragma unroll
    for (int f = 0; f < F; ++f) {
      xs[f][i] = ok ? Xf[f][(size_t)m * nh + j] : make_double2(0.0, 0.0);
      xd[f][i] = ok ? Xf[f][(size_t)(P.nm + m) * nh + j] : make_double2(0.0, 0.0);
    }
  }
  // this lane's half (lane & 1) of value lane / 2: elements 16 h .., the second half starting eight
  // further on so that the two lanes of a pair read different banks
  const int h = lane & 1;
  const double* rv = red + (lane >> 1) * ANA_RS + 16 * h;
#pragma unroll 1
  for (int off = 0; off < len; off += TL) {
    double v[ANA_V];
#pragma unroll
    for (int t = 0; t < TL; ++t) {
      const double b = sbe[off + t];
#pragma unroll
      for (int i = 0; i < NA; ++i) {
        const double q = fma(mu[i], qb[i], __dmul_rn(b, qa[i]));
        qa[i] = qb[i];
        qb[i] = q;
#pragma unroll
        for (int f = 0; f < F; ++f) {
          const double2 x = (t & 1) ? xd[f][i] : xs[f][i];
          double& re = v[(t * F + f) * 2];
          double& im = v[(t * F + f) * 2 + 1];
          re = (i == 0) ? __dmul_rn(q, x.x) : fma(q, x.x, re);
          im = (i == 0) ? __dmul_rn(q, x.y) : fma(q, x.y, im);
        }
      }
    }
    __syncwarp();   // the previous batch's partial sums are read
#pragma unroll
    for (int u = 0; u < ANA_V; ++u) red[u * ANA_RS + lane] = v[u];
    __syncwarp();
    double p[4];
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      const double r = rv[(u + 8 * h) & 15];
      p[u & 3] = (u < 4) ? r : __dadd_rn(p[u & 3], r);
    }
    double tot = __dadd_rn(__dadd_rn(p[0], p[1]), __dadd_rn(p[2], p[3]));
    tot = __dadd_rn(tot, __shfl_xor_sync(0xffffffffu, tot, 1));
    if (h == 0) {
      double* d = sacc + off * 2 * F + (lane >> 1);
      *d = more ? __dadd_rn(*d, tot) : tot;
    }
  }
}

// Segment s of F fields: the latitude groups from the segment's first significant one (gs) on in
// passes of up to eight groups, then the coefficients (packed, or the dense [l][m] array whose
// order's zeros above the diagonal the first segment writes).
template <int F>
__device__ __forceinline__ void ana_segment(const sle::ShtDev& P, int s, int m, int l0, int gs,
                                            const double2* const (&Xf)[F], double2* const (&Uf)[F], bool dense,
                                            int lane, const double* __restrict__ sbe, const double* __restrict__ scf,
                                            double* __restrict__ red, double* __restrict__ sacc) {
  const int len = min(P.leg.fseg, P.lmax + 1 - l0);
  const long long base = (long long)m * P.nm - (long long)m * (m - 1) / 2 + (l0 - m);
  bool more = false;
  int g = gs;
  while (g < P.ngrp) {
    const int na = min(P.ngrp - g, ANA_NAMAX);
    switch ((na + 1) / 2) {
      case 4: ana_pass<8, F>(P, s, m, g, len, Xf, lane, more, sbe, red, sacc); break;
      case 3: ana_pass<6, F>(P, s, m, g, len, Xf, lane, more, sbe, red, sacc); break;
      case 2: ana_pass<4, F>(P, s, m, g, len, Xf, lane, more, sbe, red, sacc); break;
      default:
        if (na == 2) ana_pass<2, F>(P, s, m, g, len, Xf, lane, more, sbe, red, sacc);
        else ana_pass<1, F>(P, s, m, g, len, Xf, lane, more, sbe, red, sacc);
    }
    g += na;
    more = true;
  }
  __syncwarp();
#pragma unroll
  for (int f = 0; f < F; ++f) {
    for (int e = lane; e < 2 * len; e += 32) {
      const int t = e >> 1, c = e & 1;
      const double val = more ? __dmul_rn(sacc[(t * F + f) * 2 + c], scf[t]) : 0.0;
      const size_t at = dense ? (size_t)(l0 + t) * P.nm + m : (size_t)base + t;
      reinterpret_cast<double*>(Uf[f] + at)[c] = val;
    }
    if (dense && l0 == m)
      for (int l = lane; l < m; l += 32) Uf[f][(size_t)l * P.nm + m] = make_double2(0.0, 0.0);
  }
}

// blockIdx.y: the field (F = 1) or the pair of fields (F = 2; a pair with one field gated off, or
// the last field of an odd number, runs alone with the same arithmetic).  What the plan holds is
// read before the wait for the kernel before (the plan's tables never change).
template <int F>
__global__ void __launch_bounds__(32 * ANA_WARPS, F == 1 ? 6 : 4) k_leg_ana(sle::ShtDev P, SpecPtrs out, int nf, int dense) {
  __shared__ double scoef[ANA_WARPS][2][SEG];
  __shared__ double sred[ANA_WARPS][ANA_V * ANA_RS];
  __shared__ double ssum[ANA_WARPS][2 * SEG * F];
  const int wib = threadIdx.x >> 5;
  const int warp = blockIdx.x * ANA_WARPS + wib;
  const int lane = threadIdx.x & 31;
  if (warp >= P.leg.nfseg) {
    pdl_wait();
    return;
  }
  const int4 item = P.leg.ana_items[warp];   // segment, order, first degree, first significant group
  double* sbe = scoef[wib][0];
  double* scf = scoef[wib][1];
  {
    const int len = min(P.leg.fseg, P.lmax + 1 - item.z);
    const long long base = (long long)item.y * P.nm - (long long)item.y * (item.y - 1) / 2 + (item.z - item.y);
    for (int t = lane; t < P.leg.fseg; t += 32) {
      sbe[t] = (t < len) ? P.be[base + t] : 0.0;
      scf[t] = (t < len) ? __ddiv_rn(P.cf[base + t], SQRT2_LEGACY) : 0.0;
    }
  }
  pdl_wait();
  pdl_trigger();
  __syncwarp();
  const size_t field = (size_t)2 * P.nm * P.nh;
  const int f0 = F * blockIdx.y;
  int first = -1, count = 0;
#pragma unroll
  for (int f = 0; f < F; ++f) {
    if (f0 + f < nf && !field_gated_off(P, f0 + f)) {
      if (first < 0) first = f;
      ++count;
    }
  }
  if (count == 0) return;
  if constexpr (F == 2) {
    if (count == 2) {
      const double2* const X[2] = {P.X + f0 * field, P.X + (f0 + 1) * field};
      double2* const U[2] = {out.p[f0], out.p[f0 + 1]};
      ana_segment<2>(P, item.x, item.y, item.z, item.w, X, U, dense != 0, lane, sbe, scf, sred[wib], ssum[wib]);
      return;
    }
  }
  const double2* const X[1] = {P.X + (f0 + first) * field};
  double2* const U[1] = {out.p[f0 + first]};
  ana_segment<1>(P, item.x, item.y, item.z, item.w, X, U, dense != 0, lane, sbe, scf, sred[wib], ssum[wib]);
}

// ----------------------------------------------------------------- Legendre synthesis
// Block (order m, NA consecutive latitude groups), four warps: warp w sums the segments w, w + 4,
// .. of the order over the block's latitudes (NA per lane, one per group), then the four warps'
// even- and odd-degree sums are added in warp order.  Bound: FP64 issue, two operations per degree and
// latitude for the recurrence and two per field; for a single field at L = 511 its chains and the wait
// for a block's slowest warp (FP64 pipe active in 42 % of the SMs' active cycles, 1.7 waves).  One serial walk over all degrees of
// an order (the form before) had two warps per scheduler waiting on their own recurrences; the
// split over segments gives every scheduler four and more independent walks, and the blocks run
// longest first.  F = 2 shares the recurrence between two fields.  Each (latitude, order) is
// written as one 32-byte (E, O) sector at EO[f][j][m], which the inverse FFT of latitude j reads
// as one contiguous row.  Measured on one field at L = 511: with the inverse FFT, back to back in a
// CUDA graph, 30.2 -> 26.3 us (L = 255: 17.2 -> 8.6, L = 63: 11.5 -> 4.7); four fields at L = 511
// 88.9 -> 61.0 us.  Two or eight warps per block measured slower (32.8 and 31.4 us at that stage
// against 28.0).
constexpr int SYN_WARPS = 4;

// Degrees of one segment, coefficients u (F per degree, scaled) and recurrence factors b staged in
// shared memory, for the lane's latitudes LO .. NA-1.
template <int NA, int LO, int F>
__device__ __forceinline__ void syn_segment(const sle::ShtDev& P, int s, int j0, int len, const double2* __restrict__ su,
                                            const double* __restrict__ sb, double2 (&E)[F][NA], double2 (&O)[F][NA]) {
  double x[NA], qa[NA], qb[NA];
#pragma unroll
  for (int i = LO; i < NA; ++i) {
    const int j = j0 + 32 * i;
    const bool ok = j < P.nh;
    x[i] = ok ? P.mu[j] : 0.0;
    const double2 sd = ok ? P.leg.fseeds[(size_t)s * P.nh + j] : make_double2(0.0, 0.0);
    qa[i] = sd.x;
    qb[i] = sd.y;
  }
#pragma unroll 2
  for (int r = 0; r < len; r += 2) {   // the staged coefficients are zero beyond len
    const double b0 = sb[r], b1 = sb[r + 1];
#pragma unroll
    for (int i = LO; i < NA; ++i) {
      qa[i] = fma(x[i], qb[i], __dmul_rn(b0, qa[i]));   // even degree
      qb[i] = fma(x[i], qa[i], __dmul_rn(b1, qb[i]));   // odd degree
    }
#pragma unroll
    for (int f = 0; f < F; ++f) {
      const double2 u0 = su[r * F + f], u1 = su[(r + 1) * F + f];
#pragma unroll
      for (int i = LO; i < NA; ++i) {
        E[f][i].x = fma(u0.x, qa[i], E[f][i].x);
        E[f][i].y = fma(u0.y, qa[i], E[f][i].y);
        O[f][i].x = fma(u1.x, qb[i], O[f][i].x);
        O[f][i].y = fma(u1.y, qb[i], O[f][i].y);
      }
    }
  }
}

// Warp w of the item's block takes every fourth piece of the two masks' union from the w-th on.
template <int NA, int F>
__device__ __forceinline__ void syn_block(const sle::ShtDev& P, const SynItem& item, const double2* const (&Uf)[F], int f0,
                                          bool dense, double* sm) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m = item.m, hb = item.tile;
  double2* su = reinterpret_cast<double2*>(sm) + (size_t)w * SEG * F;                          // [SEG][F]
  double* sb = sm + (size_t)SYN_WARPS * SEG * F * 2 + (size_t)w * SEG;                         // [SEG]
  double2* part = reinterpret_cast<double2*>(sm + (size_t)SYN_WARPS * SEG * (2 * F + 1));      // partial sums
  const int j0 = 32 * NA * hb + lane;
  const long long moff = (long long)m * P.nm - (long long)m * (m - 1) / 2;
  const int seg0 = P.leg.fsegoff[m];
  double2 E[F][NA], O[F][NA];
#pragma unroll
  for (int f = 0; f < F; ++f)
#pragma unroll
    for (int i = 0; i < NA; ++i) E[f][i] = O[f][i] = make_double2(0.0, 0.0);
  unsigned long long left = item.full | item.half;
  for (int n = 0; left; ++n, left &= left - 1) {
    if ((n & (SYN_WARPS - 1)) != w) continue;
    const int k = __ffsll((long long)left) - 1, s = seg0 + k, l0 = m + P.leg.fseg * k;
    const int len = min(P.leg.fseg, P.lmax + 1 - l0);
    const long long base = moff + P.leg.fseg * k;
    __syncwarp();
    for (int t = lane; t < P.leg.fseg; t += 32) {
      const bool in = t < len;
      const double c = in ? __dmul_rn(P.cf[base + t], SQRT2_LEGACY) : 0.0;
#pragma unroll
      for (int f = 0; f < F; ++f) {
        double2 u = make_double2(0.0, 0.0);
        if (in) u = Uf[f][dense ? (size_t)(l0 + t) * P.nm + m : (size_t)base + t];
        su[t * F + f] = make_double2(__dmul_rn(u.x, c), __dmul_rn(u.y, c));
      }
      sb[t] = in ? P.be[base + t] : 0.0;
    }
    __syncwarp();
    if (NA > 1 && !((item.full >> k) & 1u)) syn_segment<NA, NA / 2, F>(P, s, j0, len, su, sb, E, O);
    else syn_segment<NA, 0, F>(P, s, j0, len, su, sb, E, O);
  }
  // partial sums [warp][field][latitude group][E | O][lane]
  constexpr int PER = F * NA * 2;
#pragma unroll
  for (int f = 0; f < F; ++f)
#pragma unroll
    for (int i = 0; i < NA; ++i) {
      part[((size_t)w * PER + (f * NA + i) * 2 + 0) * 32 + lane] = E[f][i];
      part[((size_t)w * PER + (f * NA + i) * 2 + 1) * 32 + lane] = O[f][i];
    }
  __syncthreads();
  for (int q = w; q < F * NA; q += SYN_WARPS) {
    const int i = q % NA, j = j0 + 32 * i;
    if (j >= P.nh) continue;
    double2 e = part[(size_t)(q * 2) * 32 + lane], o = part[(size_t)(q * 2 + 1) * 32 + lane];
#pragma unroll
    for (int k = 1; k < SYN_WARPS; ++k) {
      const double2 e1 = part[((size_t)k * PER + q * 2) * 32 + lane], o1 = part[((size_t)k * PER + q * 2 + 1) * 32 + lane];
      e = make_double2(__dadd_rn(e.x, e1.x), __dadd_rn(e.y, e1.y));
      o = make_double2(__dadd_rn(o.x, o1.x), __dadd_rn(o.y, o1.y));
    }
    const int f = q / NA;
    double2* dst = P.EO + (((size_t)(f0 + f) * P.nh + j) * P.nm + m) * 2;
    dst[0] = e;
    dst[1] = o;
  }
}

constexpr size_t syn_smem(int na, int f) {
  return (size_t)SYN_WARPS * (SEG * (2 * f + 1) * sizeof(double) + (size_t)f * na * 2 * 32 * sizeof(double2));
}

// blockIdx.x: the item (most work first); blockIdx.y: the field or the pair of fields, as in the
// analysis.
template <int NA, int F>
__global__ void __launch_bounds__(32 * SYN_WARPS, F == 1 ? 4 : 3) k_leg_syn(sle::ShtDev P, CSpecPtrs in, int nf, int dense) {
  extern __shared__ double smd[];
  const SynItem item = P.leg.syn_items[blockIdx.x];
  pdl_wait();
  pdl_trigger();
  const int f0 = F * blockIdx.y;
  int first = -1, count = 0;
#pragma unroll
  for (int f = 0; f < F; ++f) {
    if (f0 + f < nf && !field_gated_off(P, f0 + f)) {
      if (first < 0) first = f;
      ++count;
    }
  }
  if (count == 0) return;
  if constexpr (F == 2) {
    if (count == 2) {
      const double2* const U[2] = {in.p[f0], in.p[f0 + 1]};
      syn_block<NA, 2>(P, item, U, f0, dense != 0, smd);
      return;
    }
  }
  const double2* const U[1] = {in.p[f0 + first]};
  syn_block<NA, 1>(P, item, U, f0 + first, dense != 0, smd);
}

// ---------------------------------------------------------------- dense <-> packed
__global__ void k_pack(sle::ShtDev P, const double2* dense, double2* packed) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long n = (long long)P.nm * P.nm;
  if (i >= n) return;
  const int l = (int)(i / P.nm), m = (int)(i - (long long)l * P.nm);
  if (m <= l) packed[P.moff[m] + (l - m)] = dense[i];
}

__global__ void k_unpack(sle::ShtDev P, const double2* packed, double2* dense) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long n = (long long)P.nm * P.nm;
  if (i >= n) return;
  const int l = (int)(i / P.nm), m = (int)(i - (long long)l * P.nm);
  dense[i] = (m <= l) ? packed[P.moff[m] + (l - m)] : make_double2(0.0, 0.0);
}

// ------------------------------------------------------------------------ launchers
static size_t fft_smem(const ShtDev& d) { return fft_smem_bytes(2, d.n2, sizeof(double2)); }
// Latitude groups per lane of the synthesis (and per block): four from three groups on.
static int syn_na(const ShtDev& d) { return d.ngrp >= 3 ? 4 : d.ngrp; }
// Whether the Legendre kernels take the fields in pairs (one recurrence for two fields): once the
// single-field form has more warps than are resident at once (16 per SM) a pair saves work; below
// that it would only leave schedulers without a warp.  Measured: at L = 255 (640 segments),
// three fields, 20.0 us single against 22.8 us paired; at L = 63, two fields, 6.6 against 8.7 us; from
// L = 511 on every number of fields pairs (two fields 42 us, against twice 26 to 28 us for single ones).
static bool leg_pairs(const sle_sht* plan, int nf) {
  return nf >= 2 && (long long)plan->d.nseg * nf > 16LL * plan->n_sm;
}

// The pieces an analysis of nf fields walks: the short ones while their warps are resident at once (12
// per SM).  Up to there the kernel waits on its own chains, and shorter ones end earlier; beyond, more
// pieces only read more seeds.  The sums over the latitudes do not depend on it.  Fold and analysis of
// one field, segments -> pieces: 6.5 -> 4.5 us at L = 63, 10.5 -> 8.1 at L = 255; three fields at L = 127
// (2112 pieces) 8.9 -> 11.2, so segments there.  The synthesis, whose sums over the degrees are grouped by
// piece, takes the plan's short pieces for every number of fields (a field's result does not depend
// on the others): 4.7 -> 4.0 us at L = 63, 9.3 -> 6.7 for two fields at L = 127.
static const LegSet& ana_set(const sle_sht* plan, int nf) {
  return plan->leg[(long long)plan->leg[1].nfseg * nf <= 12LL * plan->n_sm ? 1 : 0];
}

// The Legendre analysis of nf fields (folded FFTs in d.X).
static int fp64_leg_ana(const sle_sht* plan, ShtDev d, const SpecPtrs& o, int nf, int dense, cudaStream_t st) {
  d.leg = ana_set(plan, nf);
  const unsigned gx = (unsigned)((d.leg.nfseg + ANA_WARPS - 1) / ANA_WARPS);
  if (leg_pairs(plan, nf))
    SLE_CUDA(launch_pdl_if(plan->early, k_leg_ana<2>, dim3(gx, (nf + 1) / 2), dim3(32 * ANA_WARPS), 0, st, d, o, nf, dense));
  else
    SLE_CUDA(launch_pdl_if(plan->early, k_leg_ana<1>, dim3(gx, nf), dim3(32 * ANA_WARPS), 0, st, d, o, nf, dense));
  return SLE_OK;
}

template <int NA>
static int fp64_leg_syn(const sle_sht* plan, ShtDev d, const CSpecPtrs& c, int nf, int dense, cudaStream_t st) {
  d.leg = plan->leg[1];
  const unsigned gx = (unsigned)(d.nm * ((d.ngrp + NA - 1) / NA));
  if (leg_pairs(plan, nf))
    SLE_CUDA(launch_pdl_if(plan->early, k_leg_syn<NA, 2>, dim3(gx, (nf + 1) / 2), dim3(32 * SYN_WARPS), syn_smem(NA, 2), st, d, c, nf, dense));
  else
    SLE_CUDA(launch_pdl_if(plan->early, k_leg_syn<NA, 1>, dim3(gx, nf), dim3(32 * SYN_WARPS), syn_smem(NA, 1), st, d, c, nf, dense));
  return SLE_OK;
}

// One FP64 launch group (1..fp64_group fields, all packed or all dense).
static int fp64_analysis(sle_sht* plan, const FieldSpec* fs, int nf, cudaStream_t st, int prof_cls) {
  ShtDev d = plan->d;
  GridPtrs g{};
  SpecPtrs o{};
  for (int f = 0; f < nf; ++f) {
    g.p[f] = fs[f].grid;
    g.kind[f] = fs[f].kind;
    g.m0[f] = fs[f].m0;
    g.m1[f] = fs[f].m1;
    o.p[f] = fs[f].spec;
    d.gset[f] = fs[f].skip_set;
    d.gclr[f] = fs[f].skip_clear;
  }
  ProfToken t0 = prof_begin(PROF_FFT, nf, st);
#define SLE_LAUNCH_FOLD(NN) \
  SLE_CUDA(launch_pdl_if(plan->early, k_fft_fold<NN>, dim3(d.nh, nf), dim3(fft_threads(2, NN)), fft_smem(d), st, d, g))
  SLE_FFT_SWITCH(d.n2, SLE_LAUNCH_FOLD)
#undef SLE_LAUNCH_FOLD
  prof_end(t0, st);
  ProfToken t1 = prof_begin(prof_cls, nf, st);
  SLE_TRY(fp64_leg_ana(plan, d, o, nf, fs[0].dense, st));
  prof_end(t1, st);
  note_launch(2);
  SLE_CUDA(cudaGetLastError());
  return SLE_OK;
}

static int fp64_synthesis(sle_sht* plan, const FieldSpec* fs, int nf, cudaStream_t st) {
  ShtDev d = plan->d;
  CSpecPtrs c{};
  OutGridPtrs g{};
  for (int f = 0; f < nf; ++f) {
    c.p[f] = fs[f].spec;
    g.p[f] = fs[f].grid;
    g.out2[f] = fs[f].epi_out;
    g.mul2[f] = fs[f].epi_mul;
    d.gset[f] = fs[f].skip_set;
    d.gclr[f] = fs[f].skip_clear;
  }
  ProfToken t0 = prof_begin(PROF_LEG_SYN, nf, st);
  const int na = syn_na(d), dense = fs[0].dense;
  if (na == 4) SLE_TRY(fp64_leg_syn<4>(plan, d, c, nf, dense, st));
  else if (na == 2) SLE_TRY(fp64_leg_syn<2>(plan, d, c, nf, dense, st));
  else SLE_TRY(fp64_leg_syn<1>(plan, d, c, nf, dense, st));
  prof_end(t0, st);
  ProfToken t1 = prof_begin(PROF_IFFT, nf, st);
#define SLE_LAUNCH_IFFT(NN) \
  SLE_CUDA(launch_pdl_if(plan->early, k_ifft_unfold<NN>, dim3(d.nh, nf), dim3(fft_threads(2, NN)), fft_smem(d), st, d, g))
  SLE_FFT_SWITCH(d.n2, SLE_LAUNCH_IFFT)
#undef SLE_LAUNCH_IFFT
  prof_end(t1, st);
  note_launch(2);
  SLE_CUDA(cudaGetLastError());
  return SLE_OK;
}

static MxFieldArgs mx_args(const FieldSpec* fs, int nf) {
  MxFieldArgs a{};
  a.nf = nf;
  for (int f = 0; f < nf; ++f) {
    a.grid[f] = fs[f].grid;
    a.spec[f] = fs[f].spec;
    a.skip_set[f] = fs[f].skip_set;
    a.skip_clear[f] = fs[f].skip_clear;
    a.epi_out[f] = fs[f].epi_out;
    a.epi_mul[f] = fs[f].epi_mul;
    a.kind[f] = fs[f].kind;
    a.m0[f] = fs[f].m0;
    a.m1[f] = fs[f].m1;
  }
  return a;
}

int sht_analysis_list(sle_sht* plan, const FieldSpec* f, int n, cudaStream_t st, int prof_cls) {
  if (n < 1) return SLE_OK;
  const bool mx = plan->precision == SLE_PREC_MIXED;
  const int group = mx ? plan->tune_fpl : plan->fp64_group;
  // equal groups (the tensor-core kernels' cost depends on the launch, not on its width)
  const int ngroups = (n + group - 1) / group;
  for (int g = 0; g < ngroups; ++g) {
    const int lo = (int)((long long)n * g / ngroups), hi = (int)((long long)n * (g + 1) / ngroups);
    if (mx) {
      SLE_TRY(sht_mx_analysis(plan, mx_args(f + lo, hi - lo), plan->mx_status, st, prof_cls));
    } else {
      SLE_TRY(fp64_analysis(plan, f + lo, hi - lo, st, prof_cls));
    }
  }
  return SLE_OK;
}

int sht_synthesis_list(sle_sht* plan, const FieldSpec* f, int n, cudaStream_t st, bool b_ready) {
  if (n < 1) return SLE_OK;
  const bool mx = plan->precision == SLE_PREC_MIXED;
  const int group = mx ? plan->tune_fpl : plan->fp64_group;
  const int ngroups = (n + group - 1) / group;
  for (int g = 0; g < ngroups; ++g) {
    const int lo = (int)((long long)n * g / ngroups), hi = (int)((long long)n * (g + 1) / ngroups);
    if (mx) {
      SLE_TRY(sht_mx_synthesis(plan, mx_args(f + lo, hi - lo), plan->mx_status, st, b_ready && ngroups == 1));
    } else {
      SLE_TRY(fp64_synthesis(plan, f + lo, hi - lo, st));
    }
  }
  return SLE_OK;
}

int sht_pack(sle_sht* plan, const double2* dense, double2* packed, cudaStream_t st) {
  const long long n = (long long)plan->d.nm * plan->d.nm;
  k_pack<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(plan->d, dense, packed);
  note_launch();
  SLE_CUDA(cudaGetLastError());
  return SLE_OK;
}

int sht_unpack(sle_sht* plan, const double2* packed, double2* dense, cudaStream_t st) {
  const long long n = (long long)plan->d.nm * plan->d.nm;
  k_unpack<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(plan->d, packed, dense);
  note_launch();
  SLE_CUDA(cudaGetLastError());
  return SLE_OK;
}

// ---------------------------------------------------------------------- plan create
template <typename T>
static int dalloc(T** p, size_t n) {
  cudaError_t e = cudaMalloc(reinterpret_cast<void**>(p), n * sizeof(T) + 16);
  if (e != cudaSuccess) {
    set_error("cudaMalloc(%zu bytes) failed: %s", n * sizeof(T), cudaGetErrorString(e));
    *p = nullptr;
    return SLE_ERR_OOM;
  }
  return SLE_OK;
}

static void leg_set_free(LegSet& a, const double2* segment_seeds) {
  const void* ptrs[] = {a.fsegoff, a.ana_items, a.syn_items, a.fseeds == segment_seeds ? nullptr : a.fseeds};
  for (const void* q : ptrs)
    if (q) cudaFree(const_cast<void*>(q));
}

static void plan_free(sle_sht* p) {
  if (!p) return;
  if (p->leg[1].fsegoff != p->leg[0].fsegoff) leg_set_free(p->leg[1], p->seeds);
  leg_set_free(p->leg[0], p->seeds);
  void* ptrs[] = {p->mu, p->w, p->wn, p->ws, p->be, p->cf, p->moff, p->lidx, p->segoff,
                  p->seg_m, p->seg_l0, p->seeds, p->tw, p->X, p->istart,
                  p->mx_xf, p->mx_twf, p->mx_gns, p->mx_bsyn, p->mx_s0, p->mx_abort,
                  p->mx_ana_units, p->mx_syn_units, p->mx_syn_seg, p->mx_tab_ana, p->mx_tab_syn,
                  p->mx_ana_cta, p->mx_syn_cta, p->mx_bpos};
  for (void* q : ptrs)
    if (q) cudaFree(q);
  if (p->mx_abort_host) cudaFreeHost(p->mx_abort_host);
  delete p;
}

// Pieces of SEG / split degrees with their seeds (split 1: the segments' own), and the work items of
// the FP64 Legendre kernels over them.
static int leg_set_build(sle_sht* p, LegSet& set, int split, const std::vector<int>& segoff,
                         const std::vector<unsigned char>& ist) {
  ShtDev d = p->d;
  const int L = d.lmax;
  set = LegSet{};
  set.fseg = SEG / split;
  std::vector<int> foff(d.nm + 1), f_m, f_l0, f_ist;
  for (int m = 0; m < d.nm; ++m) {
    foff[m] = (int)f_m.size();
    for (int l0 = m; l0 <= L; l0 += set.fseg) {
      f_m.push_back(m);
      f_l0.push_back(l0);
      f_ist.push_back(ist[segoff[m] + (l0 - m) / SEG]);
    }
  }
  foff[d.nm] = set.nfseg = (int)f_m.size();
  int* off = nullptr;
  SLE_TRY(dalloc(&off, d.nm + 1));
  set.fsegoff = off;
  SLE_CUDA(cudaMemcpy(off, foff.data(), foff.size() * sizeof(int), cudaMemcpyHostToDevice));
  set.fseeds = p->seeds;
  if (split > 1) {
    double2* seeds = nullptr;
    SLE_TRY(dalloc(&seeds, (size_t)set.nfseg * d.nh));
    set.fseeds = seeds;
    d.leg = set;
    k_piece_seeds<<<d.nseg, std::min(256, 32 * d.ngrp)>>>(d, seeds);
    SLE_CUDA(cudaGetLastError());
  }
  const auto by_work = [](const std::vector<long long>& work) {   // most work first
    std::vector<int> order(work.size());
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return work[a] > work[b]; });
    return order;
  };
  const auto upload = [](const auto& items, const std::vector<int>& order, auto** out) -> int {
    auto v = items;
    for (size_t i = 0; i < v.size(); ++i) v[i] = items[order[i]];
    auto* dev = v.data();
    SLE_TRY(dalloc(&dev, v.size()));
    *out = dev;
    SLE_CUDA(cudaMemcpy(dev, v.data(), v.size() * sizeof(v[0]), cudaMemcpyHostToDevice));
    return SLE_OK;
  };
  std::vector<int4> items;
  std::vector<long long> work;
  for (int i = 0; i < set.nfseg; ++i) {
    items.push_back(make_int4(i, f_m[i], f_l0[i], f_ist[i]));
    work.push_back((long long)std::min(set.fseg, L + 1 - f_l0[i]) * (d.ngrp - f_ist[i]));
  }
  SLE_TRY(upload(items, by_work(work), &set.ana_items));
  // synthesis blocks: (order, latitude tile) with the tile's significant pieces
  const int na = syn_na(d), ntile = (d.ngrp + na - 1) / na;
  std::vector<SynItem> tiles;
  work.clear();
  for (int m = 0; m < d.nm; ++m) {
    if (foff[m + 1] - foff[m] > 64) {
      set_error("order %d has %d pieces, more than its work items' masks hold", m, foff[m + 1] - foff[m]);
      return SLE_ERR_BAD_SHAPE;
    }
    for (int t = 0; t < ntile; ++t) {
      const int glo = na * t, ghi = std::min(glo + na, d.ngrp) - 1;
      unsigned long long full = 0, half = 0;
      long long c = 0;
      for (int i = foff[m]; i < foff[m + 1]; ++i) {
        if (f_ist[i] > ghi) continue;
        const bool upper = na > 1 && f_ist[i] >= glo + na / 2;
        (upper ? half : full) |= 1ull << (i - foff[m]);
        c += (long long)std::min(set.fseg, L + 1 - f_l0[i]) * (upper ? 1 : 2);
      }
      tiles.push_back(SynItem{m, t, full, half});
      work.push_back(c);
    }
  }
  return upload(tiles, by_work(work), &set.syn_items);
}

static int plan_build(sle_sht* p, int nlat, int nlon, int lmax) {
  ShtDev& d = p->d;
  d.nlat = nlat;
  d.nlon = nlon;
  d.lmax = lmax;
  d.nh = nlat / 2;
  d.nm = lmax + 1;
  d.n2 = nlon / 2;
  d.log2n2 = 0;
  while ((1 << d.log2n2) < d.n2) ++d.log2n2;
  d.ngrp = (d.nh + 31) / 32;
  d.ncoef = (long long)d.nm * (d.nm + 1) / 2;
  {
    int dev = 0;
    SLE_CUDA(cudaGetDevice(&dev));
    SLE_CUDA(cudaDeviceGetAttribute(&p->n_sm, cudaDevAttrMultiProcessorCount, dev));
    p->n_sm = std::max(1, p->n_sm);
  }
  // host tables: packed offsets, segments
  std::vector<long long> moff(d.nm + 1);
  std::vector<int> segoff(d.nm + 1), seg_m, seg_l0;
  for (int m = 0; m <= d.nm; ++m) moff[m] = (long long)m * (lmax + 1) - (long long)m * (m - 1) / 2;
  for (int m = 0; m < d.nm; ++m) {
    segoff[m] = (int)seg_m.size();
    for (int l0 = m; l0 <= lmax; l0 += SEG) {
      seg_m.push_back(m);
      seg_l0.push_back(l0);
    }
  }
  segoff[d.nm] = (int)seg_m.size();
  d.nseg = (int)seg_m.size();

  SLE_TRY(dalloc(&p->mu, nlat));
  SLE_TRY(dalloc(&p->w, nlat));
  SLE_TRY(dalloc(&p->wn, d.nh));
  SLE_TRY(dalloc(&p->ws, d.nh));
  SLE_TRY(dalloc(&p->moff, d.nm + 1));
  SLE_TRY(dalloc(&p->lidx, d.ncoef));
  SLE_TRY(dalloc(&p->segoff, d.nm + 1));
  SLE_TRY(dalloc(&p->seg_m, d.nseg));
  SLE_TRY(dalloc(&p->seg_l0, d.nseg));
  SLE_TRY(dalloc(&p->seeds, (size_t)d.nseg * d.nh));
  SLE_TRY(dalloc(&p->be, d.ncoef));
  SLE_TRY(dalloc(&p->cf, d.ncoef));
  SLE_TRY(dalloc(&p->istart, d.nseg));
  SLE_TRY(dalloc(&p->tw, tw_table_len(d.n2)));
  {
    // X, EO and packbuf from one allocation: an allocation above 1 MB takes about 0.4 ms whatever its size
    const size_t per = (size_t)2 * d.nm * d.nh;
    p->fp64_group = (int)std::min<size_t>(MAXF, std::max<size_t>(4, FP64_GROUP_BYTES / (per * sizeof(double2))));
    const size_t nx = (p->fp64_group * per + 15) / 16 * 16;   // 256-byte boundaries
    SLE_TRY(dalloc(&p->X, 2 * nx + (size_t)DENSE_MAXF * d.ncoef));
    p->EO = p->X + nx;
    p->packbuf = p->EO + nx;
  }
  double* segmax = nullptr;
  int* fail = nullptr;
  SLE_TRY(dalloc(&segmax, (size_t)d.nseg * d.ngrp));
  SLE_TRY(dalloc(&fail, 1));
  SLE_CUDA(cudaMemset(fail, 0, sizeof(int)));
  SLE_CUDA(cudaMemcpy(p->moff, moff.data(), moff.size() * sizeof(long long), cudaMemcpyHostToDevice));
  SLE_CUDA(cudaMemcpy(p->segoff, segoff.data(), segoff.size() * sizeof(int), cudaMemcpyHostToDevice));
  SLE_CUDA(cudaMemcpy(p->seg_m, seg_m.data(), seg_m.size() * sizeof(int), cudaMemcpyHostToDevice));
  SLE_CUDA(cudaMemcpy(p->seg_l0, seg_l0.data(), seg_l0.size() * sizeof(int), cudaMemcpyHostToDevice));
  // twiddles exp(-2 pi i t / nlon), from long-double sin/cos rounded once, then the same values
  // in the order each FFT pass reads them (layout in sle_fft.cuh)
  std::vector<double2> tw(tw_table_len(d.n2));
  for (int t = 0; t < d.n2; ++t) {
    const long double a = -2.0L * 3.141592653589793238462643383279502884L * (long double)t / (long double)nlon;
    tw[t] = make_double2((double)cosl(a), (double)sinl(a));
  }
  for (int ns = 1, n = d.n2; ns < n;) {
    const int r = n / ns >= 8 ? 8 : n / ns;
    if (ns > 1) {
      for (int u = 1; u < r; ++u) {
        for (int k = 0; k < ns; ++k) {
          const int t = u * k * (2 * n / (ns * r));
          const int at = tw_pass_index(n, ns, u, k);
          if (at >= (int)tw.size() || t >= 2 * n) {
            set_error("twiddle table: index %d of %zu out of range", at, tw.size());
            cudaFree(segmax);
            cudaFree(fail);
            return SLE_ERR_STATE;
          }
          tw[at] = t < n ? tw[t] : make_double2(-tw[t - n].x, -tw[t - n].y);
        }
      }
    }
    ns *= r;
  }
  SLE_CUDA(cudaMemcpy(p->tw, tw.data(), tw.size() * sizeof(double2), cudaMemcpyHostToDevice));

  d.mu = p->mu;
  d.w = p->w;
  d.wn = p->wn;
  d.ws = p->ws;
  d.moff = p->moff;
  d.lidx = p->lidx;
  d.segoff = p->segoff;
  d.seg_m = p->seg_m;
  d.seg_l0 = p->seg_l0;
  d.seeds = p->seeds;
  d.be = p->be;
  d.cf = p->cf;
  d.istart = p->istart;
  d.tw = p->tw;
  d.X = p->X;
  d.EO = p->EO;

  const double tol = std::pow(0.1, 15);  // 0.1**15 as in the reference
  k_gauss_nodes<<<(nlat + 127) / 128, 128>>>(nlat, tol, p->mu, p->w, fail);
  SLE_CUDA(cudaGetLastError());
  // folded weights w/nlon (north rows 0..nh-1, south rows nlat-1 .. nh)
  std::vector<double> mu(nlat), w(nlat), wn(d.nh), ws(d.nh);
  SLE_CUDA(cudaMemcpy(mu.data(), p->mu, nlat * sizeof(double), cudaMemcpyDeviceToHost));
  SLE_CUDA(cudaMemcpy(w.data(), p->w, nlat * sizeof(double), cudaMemcpyDeviceToHost));
  int hfail = 0;
  SLE_CUDA(cudaMemcpy(&hfail, fail, sizeof(int), cudaMemcpyDeviceToHost));
  if (hfail) {
    set_error("gauss nodes: Newton iteration did not converge");
    cudaFree(segmax);
    cudaFree(fail);
    return SLE_ERR_BAD_SHAPE;
  }
  for (int j = 0; j < d.nh; ++j) {
    wn[j] = w[j] / (double)nlon;
    ws[j] = w[nlat - 1 - j] / (double)nlon;
  }
  SLE_CUDA(cudaMemcpy(p->wn, wn.data(), d.nh * sizeof(double), cudaMemcpyHostToDevice));
  SLE_CUDA(cudaMemcpy(p->ws, ws.data(), d.nh * sizeof(double), cudaMemcpyHostToDevice));

  k_lidx<<<d.nm, 128>>>(d, p->lidx);
  k_legendre_tables<<<dim3(d.nm, d.ngrp), 32>>>(d, p->seeds, segmax);
  k_legendre_coef<<<(d.nseg + 127) / 128, 128>>>(d, p->be, p->cf);
  k_istart<<<(d.nseg + 127) / 128, 128>>>(d, segmax, p->istart);
  SLE_CUDA(cudaGetLastError());
  std::vector<unsigned char> ist(d.nseg);
  SLE_CUDA(cudaMemcpy(ist.data(), p->istart, d.nseg, cudaMemcpyDeviceToHost));
  cudaFree(segmax);
  cudaFree(fail);
  long long done = 0, total = 0;
  for (int sg = 0; sg < d.nseg; ++sg) {
    const int len = std::min(SEG, lmax + 1 - seg_l0[sg]);
    done += (long long)len * (d.ngrp - ist[sg]);
    total += (long long)len * d.ngrp;
  }
  p->work_frac = total ? (double)done / (double)total : 1.0;
  SLE_TRY(leg_set_build(p, p->leg[0], 1, segoff, ist));
  // shorter pieces (ana_set): a quarter or half of a segment while that
  // leaves at most 12 warps per SM for one field
  const int split = 4 * d.nseg <= 12 * p->n_sm ? 4 : 2 * d.nseg <= 12 * p->n_sm ? 2 : 1;
  p->leg[1] = p->leg[0];
  if (split > 1) SLE_TRY(leg_set_build(p, p->leg[1], split, segoff, ist));

#define SLE_ATTR_FFT(NN)                                                                              \
  do {                                                                                                \
    SLE_CUDA(cudaFuncSetAttribute(k_fft_fold<NN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fft_smem(d)));    \
    SLE_CUDA(cudaFuncSetAttribute(k_ifft_unfold<NN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fft_smem(d))); \
    SLE_CUDA(cudaFuncSetAttribute(k_fft_fold<NN>, cudaFuncAttributePreferredSharedMemoryCarveout, SMEM_CARVEOUT));               \
    SLE_CUDA(cudaFuncSetAttribute(k_ifft_unfold<NN>, cudaFuncAttributePreferredSharedMemoryCarveout, SMEM_CARVEOUT));            \
  } while (0)
  SLE_FFT_SWITCH(d.n2, SLE_ATTR_FFT)
#undef SLE_ATTR_FFT
#define SLE_CARVE(...) \
  SLE_CUDA(cudaFuncSetAttribute(__VA_ARGS__, cudaFuncAttributePreferredSharedMemoryCarveout, SMEM_CARVEOUT))
  SLE_CARVE(k_leg_ana<1>);
  SLE_CARVE(k_leg_ana<2>);
  SLE_CARVE(k_leg_syn<1, 1>);
  SLE_CARVE(k_leg_syn<1, 2>);
  SLE_CARVE(k_leg_syn<2, 1>);
  SLE_CARVE(k_leg_syn<2, 2>);
  SLE_CARVE(k_leg_syn<4, 1>);
  SLE_CARVE(k_leg_syn<4, 2>);
#undef SLE_CARVE
  SLE_CUDA(cudaDeviceSynchronize());
  return SLE_OK;
}

// ------------------------------------------------------------ allocation-free analysis
// Scratch of sle_sht_analysis_noalloc: the folded row FFT (S and D) of one field for grids of
// up to 512 latitudes and lmax up to 511, 2 x 512 x 256 complex128 = 4 MiB.  It is part of the
// module image, so every GPU that loads this library holds it until the process exits.
constexpr int NOALLOC_MAX_NM = 512;
constexpr int NOALLOC_MAX_NH = 256;
static __device__ __align__(256) double2 g_noalloc_fold[2 * NOALLOC_MAX_NM * NOALLOC_MAX_NH];

}  // namespace sle

// ============================================================================ C ABI
using namespace sle;

namespace {
// Device address of g_noalloc_fold per device, looked up once per device (the host-side name of
// a __device__ array is not a device address and must never be passed to a kernel).
std::mutex g_noalloc_mu;
constexpr int NOALLOC_MAX_DEVICES = 128;
double2* g_noalloc_addr[NOALLOC_MAX_DEVICES] = {};
}  // namespace

extern "C" int sle_abi_version(void) { return SLE_ABI_VERSION; }
extern "C" const char* sle_last_error(void) { return g_err; }

extern "C" int sle_sht_create(int nlat, int nlon, int lmax, sle_sht** out) {
  if (!out) {
    set_error("sle_sht_create: out is NULL");
    return SLE_ERR_BAD_ARG;
  }
  *out = nullptr;
  if (nlat < 2 || nlat % 2 != 0) {
    set_error("nlat must be even");
    return SLE_ERR_BAD_SHAPE;
  }
  if (lmax < 0 || lmax > nlon / 2) {
    set_error("lmax must be <= nlon/2");
    return SLE_ERR_BAD_SHAPE;
  }
  if (nlon < 8 || (nlon & (nlon - 1)) != 0) {
    set_error("nlon must be a power of two >= 8 (got %d)", nlon);
    return SLE_ERR_BAD_SHAPE;
  }
  if (nlat > 2048 || nlon > 4096) {
    set_error("grid %d x %d exceeds the supported maximum 2048 x 4096", nlat, nlon);
    return SLE_ERR_BAD_SHAPE;
  }
  sle_sht* p = new sle_sht();
  std::memset(p, 0, sizeof(sle_sht));
  p->early = true;
  // launch shape of the mixed-precision transforms (sle_sht_set_tuning changes it)
  p->tune_fpl = MX_MAXF;
  p->tune_stages = 4;
  p->tune_fold_rows = 8;
  int rc = plan_build(p, nlat, nlon, lmax);
  if (rc != SLE_OK) {
    plan_free(p);
    return rc;
  }
  *out = p;
  return SLE_OK;
}

extern "C" int sle_sht_destroy(sle_sht* plan) {
  plan_free(plan);
  return SLE_OK;
}

extern "C" int sle_sht_info(const sle_sht* plan, int* nlat, int* nlon, int* lmax, long long* ncoef) {
  if (!plan) {
    set_error("sle_sht_info: NULL plan");
    return SLE_ERR_BAD_ARG;
  }
  if (nlat) *nlat = plan->d.nlat;
  if (nlon) *nlon = plan->d.nlon;
  if (lmax) *lmax = plan->d.lmax;
  if (ncoef) *ncoef = plan->d.ncoef;
  return SLE_OK;
}

extern "C" int sle_sht_work_fraction(const sle_sht* plan, double* frac) {
  if (!plan || !frac) {
    set_error("sle_sht_work_fraction: NULL argument");
    return SLE_ERR_BAD_ARG;
  }
  *frac = plan->work_frac;
  return SLE_OK;
}

extern "C" int sle_sht_gauss(const sle_sht* plan, double* mu_host, double* w_host) {
  if (!plan) {
    set_error("sle_sht_gauss: NULL plan");
    return SLE_ERR_BAD_ARG;
  }
  if (mu_host) SLE_CUDA(cudaMemcpy(mu_host, plan->mu, plan->d.nlat * sizeof(double), cudaMemcpyDeviceToHost));
  if (w_host) SLE_CUDA(cudaMemcpy(w_host, plan->w, plan->d.nlat * sizeof(double), cudaMemcpyDeviceToHost));
  return SLE_OK;
}

static bool aligned16(const void* p) { return p && (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// A mixed-precision kernel that timed out leaves the plan's abort flag raised: report it (the
// check synchronises only on plans that use the tensor-core path).
static int check_abort(sle_sht* plan, cudaStream_t st) {
  if (plan->precision != SLE_PREC_MIXED) return SLE_OK;
  int flag = 0;
  SLE_TRY(sht_mx_abort_flag(plan, &flag, st));
  if (flag) {
    set_error("a tensor-core transform kernel timed out waiting on its pipeline");
    return SLE_ERR_TIMEOUT;
  }
  return SLE_OK;
}

extern "C" int sle_sht_analysis(sle_sht* plan, int nfields, const double* const* grids_dev,
                                void* const* coeffs_dev, int layout, void* stream) {
  if (!plan || !grids_dev || !coeffs_dev) {
    set_error("sle_sht_analysis: NULL argument");
    return SLE_ERR_BAD_ARG;
  }
  const int maxf = (layout == SLE_LAYOUT_PACKED) ? MAX_CALL_FIELDS : DENSE_MAXF;
  if (nfields < 1 || nfields > maxf) {
    set_error("sle_sht_analysis: nfields must be 1..%d for this layout", maxf);
    return SLE_ERR_BAD_ARG;
  }
  for (int f = 0; f < nfields; ++f)
    if (!aligned16(grids_dev[f]) || !aligned16(coeffs_dev[f])) {
      set_error("sle_sht_analysis: device buffers must be non-NULL and 16-byte aligned");
      return SLE_ERR_BAD_ARG;
    }
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  // dense layout: the FP64 kernels write it themselves, the mixed ones go through the packed staging
  const bool staged = layout != SLE_LAYOUT_PACKED && plan->precision == SLE_PREC_MIXED;
  std::vector<FieldSpec> fs(nfields, FieldSpec{});
  for (int f = 0; f < nfields; ++f) {
    fs[f].grid = const_cast<double*>(grids_dev[f]);
    fs[f].spec = staged ? plan->packbuf + (size_t)f * plan->d.ncoef : reinterpret_cast<double2*>(coeffs_dev[f]);
    fs[f].dense = layout != SLE_LAYOUT_PACKED && !staged;
  }
  SLE_TRY(sht_analysis_list(plan, fs.data(), nfields, st));
  SLE_TRY(check_abort(plan, st));
  if (staged)
    for (int f = 0; f < nfields; ++f)
      SLE_TRY(sht_unpack(plan, fs[f].spec, reinterpret_cast<double2*>(coeffs_dev[f]), st));
  return SLE_OK;
}

extern "C" int sle_sht_synthesis(sle_sht* plan, int nfields, const void* const* coeffs_dev, int layout,
                                 double* const* grids_dev, void* stream) {
  if (!plan || !grids_dev || !coeffs_dev) {
    set_error("sle_sht_synthesis: NULL argument");
    return SLE_ERR_BAD_ARG;
  }
  const int maxf = (layout == SLE_LAYOUT_PACKED) ? MAX_CALL_FIELDS : DENSE_MAXF;
  if (nfields < 1 || nfields > maxf) {
    set_error("sle_sht_synthesis: nfields must be 1..%d for this layout", maxf);
    return SLE_ERR_BAD_ARG;
  }
  for (int f = 0; f < nfields; ++f)
    if (!aligned16(grids_dev[f]) || !aligned16(coeffs_dev[f])) {
      set_error("sle_sht_synthesis: device buffers must be non-NULL and 16-byte aligned");
      return SLE_ERR_BAD_ARG;
    }
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  // dense layout: the FP64 kernels read it themselves, the mixed ones go through the packed staging
  const bool staged = layout != SLE_LAYOUT_PACKED && plan->precision == SLE_PREC_MIXED;
  std::vector<FieldSpec> fs(nfields, FieldSpec{});
  for (int f = 0; f < nfields; ++f) {
    double2* in = reinterpret_cast<double2*>(const_cast<void*>(coeffs_dev[f]));
    fs[f].grid = grids_dev[f];
    fs[f].spec = in;
    if (staged) {
      fs[f].spec = plan->packbuf + (size_t)f * plan->d.ncoef;
      SLE_TRY(sht_pack(plan, in, fs[f].spec, st));
    }
    fs[f].dense = layout != SLE_LAYOUT_PACKED && !staged;
  }
  SLE_TRY(sht_synthesis_list(plan, fs.data(), nfields, st));
  return check_abort(plan, st);
}

extern "C" int sle_sht_set_precision(sle_sht* plan, int precision) {
  if (!plan) {
    set_error("sle_sht_set_precision: NULL plan");
    return SLE_ERR_BAD_ARG;
  }
  if (precision != SLE_PREC_FP64 && precision != SLE_PREC_MIXED) {
    set_error("sle_sht_set_precision: unknown precision %d", precision);
    return SLE_ERR_BAD_ARG;
  }
  if (precision == SLE_PREC_MIXED) SLE_TRY(sht_mx_prepare(plan));
  plan->precision = precision;
  return SLE_OK;
}

extern "C" int sle_sht_set_tuning(sle_sht* plan, const sle_mx_tuning* t) {
  if (!plan || !t) {
    set_error("sle_sht_set_tuning: NULL argument");
    return SLE_ERR_BAD_ARG;
  }
  if (t->fields_per_launch < 1 || t->fields_per_launch > MX_MAXF || (t->stages != 2 && t->stages != 4) ||
      (t->fold_rows != 4 && t->fold_rows != 8)) {
    set_error("sle_sht_set_tuning: fields_per_launch 1..%d, stages 2 or 4, fold_rows 4 or 8 (got %d, %d, %d)",
              MX_MAXF, t->fields_per_launch, t->stages, t->fold_rows);
    return SLE_ERR_BAD_ARG;
  }
  plan->tune_fpl = t->fields_per_launch;
  plan->tune_stages = t->stages;
  plan->tune_fold_rows = t->fold_rows;
  return SLE_OK;
}

extern "C" int sle_sht_get_tuning(const sle_sht* plan, sle_mx_tuning* t) {
  if (!plan || !t) {
    set_error("sle_sht_get_tuning: NULL argument");
    return SLE_ERR_BAD_ARG;
  }
  t->fields_per_launch = plan->tune_fpl;
  t->stages = plan->tune_stages;
  t->fold_rows = plan->tune_fold_rows;
  return SLE_OK;
}

extern "C" int sle_sht_pack(sle_sht* plan, const void* dense_dev, void* packed_dev, void* stream) {
  if (!plan || !dense_dev || !packed_dev) {
    set_error("sle_sht_pack: NULL argument");
    return SLE_ERR_BAD_ARG;
  }
  return sht_pack(plan, reinterpret_cast<const double2*>(dense_dev), reinterpret_cast<double2*>(packed_dev),
                  reinterpret_cast<cudaStream_t>(stream));
}

extern "C" int sle_sht_unpack(sle_sht* plan, const void* packed_dev, void* dense_dev, void* stream) {
  if (!plan || !dense_dev || !packed_dev) {
    set_error("sle_sht_unpack: NULL argument");
    return SLE_ERR_BAD_ARG;
  }
  return sht_unpack(plan, reinterpret_cast<const double2*>(packed_dev), reinterpret_cast<double2*>(dense_dev),
                    reinterpret_cast<cudaStream_t>(stream));
}

// One analysis (one field, packed output) whose scratch is the fixed array g_noalloc_fold instead
// of memory from cudaMalloc.  The call launches the same two kernels as sle_sht_analysis; the
// first call on a device looks up the array's device address (cudaGetSymbolAddress) with that
// device current.  No element of the scratch needs clearing: every element the second kernel
// reads is written earlier in the same call by the first.  The FP64 kernels run whatever the
// plan's precision setting is.
extern "C" int sle_sht_analysis_noalloc(sle_sht* plan, const double* grid_dev, void* coeffs_packed_dev,
                                        void* stream) {
  if (!plan) {
    set_error("sle_sht_analysis_noalloc: NULL plan");
    return SLE_ERR_BAD_ARG;
  }
  if (!aligned16(grid_dev) || !aligned16(coeffs_packed_dev)) {
    set_error("sle_sht_analysis_noalloc: device buffers must be non-NULL and 16-byte aligned");
    return SLE_ERR_BAD_ARG;
  }
  if (plan->d.nm > NOALLOC_MAX_NM || plan->d.nh > NOALLOC_MAX_NH) {
    set_error("sle_sht_analysis_noalloc: grid %d x %d with lmax %d exceeds the fixed scratch "
              "(at most 512 latitudes and lmax 511); use sle_sht_analysis",
              plan->d.nlat, plan->d.nlon, plan->d.lmax);
    return SLE_ERR_BAD_SHAPE;
  }
  int dev = -1;
  SLE_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= NOALLOC_MAX_DEVICES) {
    set_error("sle_sht_analysis_noalloc: device ordinal %d out of range", dev);
    return SLE_ERR_BAD_ARG;
  }
  double2* scratch = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (!g_noalloc_addr[dev]) {
      void* p = nullptr;
      SLE_CUDA(cudaGetSymbolAddress(&p, g_noalloc_fold));
      g_noalloc_addr[dev] = reinterpret_cast<double2*>(p);
    }
    scratch = g_noalloc_addr[dev];
  }
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  ShtDev d = plan->d;
  d.X = scratch;
  GridPtrs g{};
  g.p[0] = grid_dev;
  SpecPtrs o{};
  o.p[0] = reinterpret_cast<double2*>(coeffs_packed_dev);
#define SLE_LAUNCH_FOLD1(NN) \
  SLE_CUDA(launch_pdl_if(plan->early, k_fft_fold<NN>, dim3(d.nh, 1), dim3(fft_threads(2, NN)), fft_smem(d), st, d, g))
  SLE_FFT_SWITCH(d.n2, SLE_LAUNCH_FOLD1)
#undef SLE_LAUNCH_FOLD1
  SLE_TRY(fp64_leg_ana(plan, d, o, 1, 0, st));
  SLE_CUDA(cudaGetLastError());
  note_launch(2);
  return SLE_OK;
}
