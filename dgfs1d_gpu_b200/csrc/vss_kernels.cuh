// Fused fast-spectral VSS collision operator of a mixture: one species pair
// (p, q), or every pair of a species, per call.  Reference:
// DGFSBiVSSScatteringModel (dgfs1D/bi/scattering.py:47-321) and
// dgfs1D/bi/kernels/scattering/vss.mako.
//
// Per point and pair the reference computes, with F = FFT(f_p)/n, G = FFT(f_q)/n and
// a_rm(l) = (pi/L) rho_r sigma_m . l:
//   t1 = e^{+i a m_q/(m_p+m_q)} F,  t2 = e^{-i a m_p/(m_p+m_q)} G,
//   Qhat = sum_{r,m} (w_r s_w / n) b_{pq,rm}(l) FFT(IFFT(t1) IFFT(t2)),
//   Q_p += prefac_pq (Re IFFT(Qhat) - f_p Re IFFT(c_pq G)).
// f_p and f_q are real, so (Nyquist planes apart) u = IFFT(t1) and
// v = IFFT(t2) are real and one complex inverse transform of t1 + i t2 gives
// both; the weights b_{pq,rm} depend on both r and m, so every term has its own
// forward transform: two transforms per term instead of three.  For a species
// with itself the product u v is the same for sigma and -sigma, so antipodal
// directions share their transforms.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "cluster_slab.cuh"
#include "fft_reg.cuh"

namespace dgfs {

// Weights of one pair (vss.mako:51-93, launch loop bi/scattering.py:185-204):
//   b_rm(l) = sum_k B_mk fac_b(r) e^{-i mpq s_r sigma'_k . l}
//   c(l)   += sum_r sum_m sum_k B_mk fac_c(r) e^{-i s_r sigma'_k . l}
// with B_mk = (1 + sigma_m . sigma'_k)^eta, s_r = (pi/L) rho_r.  The phases
// are products of per-axis factors; k is processed in chunks so that the
// factor tables of a chunk fit in shared memory.
struct VssSetupArgs {
  const double* Bmk;         // [M][Mpre]
  const double* spre;        // [Mpre][3]
  const double* srho;        // [Nrho] s_r = (pi/L) rho_r
  const double* fac_b;       // [Nrho]
  const double* fac_c;       // [Nrho]
  double mpq;
  int M, Mpre, Nrho;
  double2* b;                // out [Nrho][M][n]
  double2* cpart;            // out [Nrho][n]: the r-th term of c
};

constexpr int kVssKChunk = 16;

template <int N>
__host__ __device__ constexpr int vss_setup_threads() { return N * N < 1024 ? N * N : 1024; }

template <int N>
__global__ void __launch_bounds__(vss_setup_threads<N>())
vss_setup_kernel(VssSetupArgs a) {
  constexpr int n = N * N * N;
  constexpr int NTH = vss_setup_threads<N>();
  const int lx = blockIdx.x, r = blockIdx.y;
  const int t = threadIdx.x;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  // per chunk: x factor [K] (b, c), y/z factors [K][N] (b, c), B [M][K]
  double2* xb = reinterpret_cast<double2*>(smem_raw);
  double2* xc = xb + kVssKChunk;
  double2* yb = xc + kVssKChunk;
  double2* yc = yb + kVssKChunk * N;
  double2* zb = yc + kVssKChunk * N;
  double2* zc = zb + kVssKChunk * N;
  double* Bs = reinterpret_cast<double*>(zc + kVssKChunk * N);
  auto rep = [](int i) { return (double)((i < N / 2) ? i : i - N); };
  constexpr int PTS = (N * N + NTH - 1) / NTH;
  double2 accb[PTS][16];  // M <= 16
  double2 accc[PTS];
#pragma unroll
  for (int k = 0; k < PTS; ++k) {
    accc[k] = make_double2(0, 0);
#pragma unroll
    for (int m = 0; m < 16; ++m) accb[k][m] = make_double2(0, 0);
  }
  const double s = a.srho[r];
  for (int k0 = 0; k0 < a.Mpre; k0 += kVssKChunk) {
    const int kc = min(kVssKChunk, a.Mpre - k0);
    __syncthreads();
    for (int i = t; i < kc * (2 * N + 1); i += blockDim.x) {
      const int k = i / (2 * N + 1), j = i % (2 * N + 1);
      const double* sp = a.spre + 3 * (k0 + k);
      double sn, cs;
      if (j == 0) {
        const double ph = s * sp[0] * rep(lx);
        sincos(a.mpq * ph, &sn, &cs); xb[k] = make_double2(cs, -sn);
        sincos(ph, &sn, &cs); xc[k] = make_double2(cs, -sn);
      } else if (j <= N) {
        const int l = j - 1;
        const double ph = s * sp[1] * rep(l);
        sincos(a.mpq * ph, &sn, &cs); yb[k * N + l] = make_double2(cs, -sn);
        sincos(ph, &sn, &cs); yc[k * N + l] = make_double2(cs, -sn);
      } else {
        const int l = j - 1 - N;
        const double ph = s * sp[2] * rep(l);
        sincos(a.mpq * ph, &sn, &cs); zb[k * N + l] = make_double2(cs, -sn);
        sincos(ph, &sn, &cs); zc[k * N + l] = make_double2(cs, -sn);
      }
    }
    for (int i = t; i < a.M * kc; i += blockDim.x)
      Bs[i] = a.Bmk[(i / kc) * a.Mpre + k0 + i % kc];
    __syncthreads();
#pragma unroll
    for (int p = 0; p < PTS; ++p) {
      const int pt = min(t + p * NTH, N * N - 1);
      const int ly = pt / N, lz = pt % N;
      for (int k = 0; k < kc; ++k) {
        const double2 eb = cmul(cmul(xb[k], yb[k * N + ly]), zb[k * N + lz]);
        const double2 ec = cmul(cmul(xc[k], yc[k * N + ly]), zc[k * N + lz]);
        double bsum = 0;
#pragma unroll
        for (int m = 0; m < 16; ++m) {
          if (m < a.M) {
            const double B = Bs[m * kc + k];
            accb[p][m].x += B * eb.x;
            accb[p][m].y += B * eb.y;
            bsum += B;
          }
        }
        accc[p].x += bsum * ec.x;
        accc[p].y += bsum * ec.y;
      }
    }
  }
#pragma unroll
  for (int p = 0; p < PTS; ++p) {
    const int pt = t + p * NTH;
    if (pt < N * N) {
      const size_t l = (size_t)lx * N * N + pt;
#pragma unroll
      for (int m = 0; m < 16; ++m)
        if (m < a.M) {
          double2 v = accb[p][m];
          v.x *= a.fac_b[r];
          v.y *= a.fac_b[r];
          a.b[((size_t)r * a.M + m) * n + l] = v;
        }
      a.cpart[(size_t)r * n + l] =
          make_double2(a.fac_c[r] * accc[p].x, a.fac_c[r] * accc[p].y);
    }
  }
}

// c(l) = sum_r cpart[r][l], in ascending r.
__global__ void vss_sum_c_kernel(const double2* cpart, int Nrho, size_t n,
                                 double2* c) {
  const size_t l = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (l >= n) return;
  double2 s = make_double2(0, 0);
  for (int r = 0; r < Nrho; ++r) {
    s.x += cpart[(size_t)r * n + l].x;
    s.y += cpart[(size_t)r * n + l].y;
  }
  c[l] = s;
}

// ---------------------------------------------------------------------------
// FP32 mode (no counterpart in the reference, which is FP64 only): the
// Maxwellian split of the VHS operator carried over to a pair.  With
// f_p = M_p + g_p, f_q = M_q + g_q (M from FP64 moments, separable),
//   IFFT(t1) = u_M + X_u,  IFFT(t2) = v_M + X_v,
//   u_M = prod_a IFFT1(e^{+i a_a mq'} mhat_p,a),  v_M likewise with q, -mp',
//   X_u = IFFT3(e^{+i a mq'} F_gp),  X_v = IFFT3(e^{-i a mp'} F_gq)  (FP32),
// and the product splits into u_M v_M, whose 3-D transform is the product of
// the 1-D FP64 transforms H_a = FFT1(u_M,a v_M,a) (vss_maxwell_gain_kernel),
// and the remainder u_M X_v + X_u (v_M + X_v), transformed in FP32
// (vss_terms1_kernel or vss_terms_kernel, one CTA or cluster per (pair, point,
// radial point), summed over the directions in FP32).  The radial sum, the final transform
// and the loss f_p Re IFFT(c G) run in FP64 (prologue and epilogue kernels
// of the VHS operator, with the complex loss kernel c).
// ---------------------------------------------------------------------------
// Grid y: the pairs of the call.
struct VssTablesArgs {
  const double2* mhat_p;   // [E][3][N]
  struct {
    const double2* mhat_q; // [E][3][N]
    const double2* ph;     // [T][2][3][N]
    float2* uv;            // out [E][T][2][3][N]: u_M,a and v_M,a (FP32)
    double2* hh;           // out [E][T][3][N]: FFT1(u_M,a v_M,a)
  } pr[4];
  int T, nevals;
};

template <int N>
__global__ void vss_tables_kernel(const __grid_constant__ VssTablesArgs a) {
  const auto& Pr = a.pr[blockIdx.y];
  const int gid = blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= a.nevals * a.T * 3) return;
  const int ax = gid % 3, term = (gid / 3) % a.T, e = gid / (3 * a.T);
  const double2* mp = a.mhat_p + (size_t)e * 3 * N + ax * N;
  const double2* mq = Pr.mhat_q + (size_t)e * 3 * N + ax * N;
  const double2* pu = Pr.ph + ((size_t)term * 6 + ax) * N;
  const double2* pv = Pr.ph + ((size_t)term * 6 + 3 + ax) * N;
  double2 u[N], v[N];
#pragma unroll
  for (int l = 0; l < N; ++l) {
    u[l] = cmul(mp[l], pu[l]);
    v[l] = cmul(mq[l], pv[l]);
  }
  fft<double, N, +1>(u);
  fft<double, N, +1>(v);
  float2* uv = Pr.uv + ((size_t)e * a.T + term) * 6 * N;
#pragma unroll
  for (int l = 0; l < N; ++l) {
    uv[ax * N + l] = make_float2((float)u[l].x, (float)u[l].y);
    uv[(3 + ax) * N + l] = make_float2((float)v[l].x, (float)v[l].y);
    u[l] = cmul(u[l], v[l]);
  }
  fft<double, N, -1>(u);
  double2* hh = Pr.hh + (((size_t)e * a.T + term) * 3 + ax) * N;
#pragma unroll
  for (int l = 0; l < N; ++l) hh[l] = u[l];
}

// GM[e][l] = sum_r w_r sum_d b_rd(l) prod_a H_a,rd(l_a)   (FP64), d over the
// pair's direction list (merged antipodes share H and add their b).
// Grid (N [lx], N / NYB, pairs ceil(E / EP)), block N NYB: a thread owns the
// wavenumber (lx, ly, lz) of EP points, so that every weight b is read once
// for EP points (one point per thread read b, 32 MB per pair at N=24, from L2
// for each point: 163 us per pair at 18 points).  EP = 3, or the number of points
// if that is less.  The 1-D factors of a chunk of terms are staged in shared
// memory, hx hy folded once per (term, ly).
struct VssGainArgs {
  struct {
    const double2* hh;     // [E][T][3][N]
    const double2* b;      // [T][n]
    double2* GM;           // out [E][n]
    const int2* dirs;
    int nd;
  } pr[4];
  const double* w;         // [Nrho]
  int Nrho, M, nevals;
};
template <int N> struct VssGainGeo {
  static constexpr int NYB = N == 16 ? 16 : 8;   // ly rows per CTA
  static constexpr int NT = N * NYB;
  static constexpr int CH = 12;                  // terms per staged chunk
};

template <int N, int EP>
__global__ void __launch_bounds__(VssGainGeo<N>::NT)
vss_maxwell_gain_kernel(const __grid_constant__ VssGainArgs a) {
  using GG = VssGainGeo<N>;
  constexpr int n = N * N * N, CH = GG::CH, NYB = GG::NYB;
  __shared__ double2 hz[CH][EP][N];
  __shared__ double2 hxy[CH][EP][NYB];
  const int groups = (a.nevals + EP - 1) / EP;
  const int pi = blockIdx.z / groups, nd = a.pr[pi].nd;
  const double2* hh = a.pr[pi].hh;
  const double2* bw = a.pr[pi].b;
  double2* GM = a.pr[pi].GM;
  const int2* dirs = a.pr[pi].dirs;
  const int lx = blockIdx.x, ly0 = blockIdx.y * NYB, e0 = (blockIdx.z % groups) * EP;
  const int t = threadIdx.x, yl = t / N, lz = t % N;
  const size_t l = ((size_t)lx * N + ly0 + yl) * N + lz;
  const int T = a.Nrho * a.M, total = a.Nrho * nd;
  double2 acc[EP];
#pragma unroll
  for (int p = 0; p < EP; ++p) acc[p] = make_double2(0, 0);
  for (int c0 = 0; c0 < total; c0 += CH) {
    const int nc = min(CH, total - c0);
    __syncthreads();
    for (int i = t; i < nc * EP * (N + NYB); i += GG::NT) {
      const int j = i % (N + NYB), p = (i / (N + NYB)) % EP, k = i / (EP * (N + NYB));
      const int e = min(e0 + p, a.nevals - 1), r = (c0 + k) / nd;
      const int term = r * a.M + dirs[(c0 + k) % nd].x;
      const double2* h = hh + ((size_t)e * T + term) * 3 * N;
      if (j < N) {
        hz[k][p][j] = h[2 * N + j];
      } else {
        const double2 x = cmul(h[lx], h[N + ly0 + j - N]);
        const double w = a.w[r];
        hxy[k][p][j - N] = make_double2(w * x.x, w * x.y);
      }
    }
    __syncthreads();
#pragma unroll 4
    for (int k = 0; k < nc; ++k) {
      const int r = (c0 + k) / nd;
      const int2 dir = dirs[(c0 + k) % nd];
      double2 b = bw[(size_t)(r * a.M + dir.x) * n + l];
      if (dir.y >= 0) {
        const double2 q = bw[(size_t)(r * a.M + dir.y) * n + l];
        b.x += q.x; b.y += q.y;
      }
#pragma unroll
      for (int p = 0; p < EP; ++p) {
        const double2 x = cmul(hxy[k][p][yl], hz[k][p][lz]);
        acc[p].x += x.x * b.x; acc[p].x -= x.y * b.y;
        acc[p].y += x.x * b.y; acc[p].y += x.y * b.x;
      }
    }
  }
#pragma unroll
  for (int p = 0; p < EP; ++p)
    if (e0 + p < a.nevals) GM[(size_t)(e0 + p) * n + l] = acc[p];
}

// Pointers of one species pair; a launch covers npair pairs, grid z =
// npair * nevals (pair major).
struct VssTermsPair {
  const void* Fp;          // [E][n] F_p (FP32 mode: F_gp)
  const void* Fq;          // [E][n]
  const void* ph;          // [T][2][3][N] phase factors of u and v
  const float2* uv;        // FP32: [E][T][2][3][N] u_M,a, v_M,a
  const void* b;           // [T][n] weights
  const void* Fnyp;        // [E][3][N][N] Nyquist planes of F_p, F_q
  const void* Fnyq;
  void* rho;               // [E][T][3][N][N] plane transforms (u_i, v_i)
  void* H;                 // out [E][NS][n]
  const int2* dirs;        // [nd] direction and its merged antipode (or -1)
  int nd;
  const double* n2p;       // [E][prologue CTAs] sums |F_p|^2, |F_q|^2
  const double* n2q;
};
struct VssTermsArgs {
  VssTermsPair pr[4];
  const double* w;         // [Nrho]
  int Nrho, M, nevals;
  int NS;                  // radial slices (blockIdx.y): r in [y Nrho/NS, ...)
};

// exp(i N alpha_a) from the phase at the Nyquist index, exp(-i alpha_a N/2)
template <typename T> __device__ __forceinline__ T vss_nu(T ph) {
  T c; c.x = ph.x; c.y = -ph.y;
  return cmul(c, c);
}

// Powers of two that bring F_p and F_q of a point to the same norm.  u and v
// share one complex transform, whose rounding is relative to the larger of the
// two; unscaled, the smaller one (a trace species, or in the FP32 mode the
// species nearer to its Maxwellian) would carry the larger one's absolute
// error.  The smaller is scaled up, by su or sv, and the factor leaves the
// spectral sums through back = 1 / (su sv): every step is exact.  back = 0 if
// either is zero everywhere (u v = 0).
template <typename R> struct VssScale { R su, sv, back; };
__device__ __forceinline__ double pow2(int k) { return __hiloint2double((1023 + k) << 20, 0); }
template <typename R, int N>
__device__ __forceinline__ VssScale<R> vss_scale(const VssTermsPair& Pr, int e) {
  constexpr int NC = prologue_ctas(N);
  double sp = 0, sq = 0;
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    sp += Pr.n2p[(size_t)e * NC + c];
    sq += Pr.n2q[(size_t)e * NC + c];
  }
  // biased exponents; 0x7ff: a sum that is not finite, unscaled.  (The early
  // return also keeps the result in registers: without it the one-CTA kernel at
  // N=24, 18 points, took 517 us instead of 495.)
  constexpr int KMAX = sizeof(R) == 4 ? 60 : 400;
  const int ep = (__double2hiint(sp) >> 20) & 0x7ff, eq = (__double2hiint(sq) >> 20) & 0x7ff;
  if (ep == 0 || eq == 0) return {R(1), R(1), R(0)};
  int k = max(-KMAX, min(KMAX, (eq - ep) / 2));
  if (ep == 0x7ff || eq == 0x7ff) k = 0;
  return {(R)pow2(max(k, 0)), (R)pow2(max(-k, 0)), (R)pow2(-abs(k))};
}

// Plane transforms of one term.  With E the phase factor and f_S as in the
// packed VHS transforms, E F splits on the Nyquist planes into
// E (1 + f_S)/2 F, whose inverse transform is real, and E (1 - f_S)/2 F, whose
// inverse transform is i u_i (i v_i).  This kernel forms u_i + i v_i, the
// inverse transform of -i E_u (1 - f_u)/2 F_p + E_v (1 - f_v)/2 F_q, as three
// 2-D transforms (rows and planes as in vhs_nyq_planes64_kernel), scaled as
// the terms are (vss_scale).
// Grid (terms of the list, 1, npair nevals), 3N threads, one pencil each.
template <typename R, int N>
__global__ void __launch_bounds__(3 * N) vss_planes_kernel(VssTermsArgs a) {
  using T = c2_t<R>;
  constexpr int ROW = N + 1, H = N / 2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* pls = reinterpret_cast<T*>(smem_raw);   // [3][N][ROW] planes of F_p
  T* plq = pls + 3 * N * ROW;                 // of F_q
  T* tb = plq + 3 * N * ROW;                  // [6N] phases
  const int e = blockIdx.z % a.nevals, t = threadIdx.x;
  const VssTermsPair& Pr = a.pr[blockIdx.z / a.nevals];
  const int r = blockIdx.x / a.M, d = blockIdx.x % a.M;
  if (d >= Pr.nd) return;
  const int term = r * a.M + Pr.dirs[d].x;
  const int P = t / N, i = t % N;
  const T* Fp = static_cast<const T*>(Pr.Fnyp) + (size_t)e * 3 * N * N;
  const T* Fq = static_cast<const T*>(Pr.Fnyq) + (size_t)e * 3 * N * N;
  const VssScale<R> sc = vss_scale<R, N>(Pr, e);
#pragma unroll 4
  for (int j = t; j < 3 * N * N; j += 3 * N) {
    pls[(j / N) * ROW + j % N] = Fp[j];
    plq[(j / N) * ROW + j % N] = Fq[j];
  }
  for (int j = t; j < 6 * N; j += 3 * N)
    tb[j] = static_cast<const T*>(Pr.ph)[(size_t)term * 6 * N + j];
  __syncthreads();
  T v[N];
#pragma unroll
  for (int k = 0; k < N; ++k) v[k] = T{R(0), R(0)};
  T* rowp = pls + (P * N + i) * ROW;
  const T* rowq = plq + (P * N + i) * ROW;
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const T* tt = tb + 3 * N * s;
    const T nx = vss_nu(tt[H]), ny = vss_nu(tt[N + H]), nz = vss_nu(tt[2 * N + H]);
    T rowc, f_row, f_rowH;
    const T* tk;
    if (P == 0) {
      rowc = cmul(tt[H], tt[N + i]);
      f_row = (i == H) ? cmul(nx, ny) : nx;
      f_rowH = cmul(f_row, nz);
      tk = tt + 2 * N;
    } else if (P == 1) {
      rowc = cmul(tt[i], tt[N + H]);
      f_row = ny;
      f_rowH = cmul(ny, nz);
      tk = tt + 2 * N;
    } else {
      rowc = cmul(tt[i], tt[2 * N + H]);
      f_row = nz;
      f_rowH = nz;
      tk = tt + N;
    }
    if (P >= 1 && i == H) rowc = T{R(0), R(0)};
    const R ss = s == 0 ? sc.su : sc.sv;
    rowc.x *= ss;
    rowc.y *= ss;
    // (1 - f)/2 rowc
    const T g = cmul(T{R(0.5) * (R(1) - f_row.x), R(-0.5) * f_row.y}, rowc);
    const T gH = (P == 2) ? T{R(0), R(0)}
                          : cmul(T{R(0.5) * (R(1) - f_rowH.x), R(-0.5) * f_rowH.y}, rowc);
    const T* row = s == 0 ? rowp : rowq;
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const T x = cmul(cmul(k == H ? gH : g, tk[k]), row[k]);
      if (s == 0) { v[k].x += x.y; v[k].y -= x.x; }   // -i x
      else { v[k].x += x.x; v[k].y += x.y; }
    }
  }
  fft<R, N, +1>(v);
#pragma unroll
  for (int k = 0; k < N; ++k) rowp[k] = v[k];
  __syncthreads();
#pragma unroll
  for (int k = 0; k < N; ++k) v[k] = pls[(P * N + k) * ROW + i];
  fft<R, N, +1>(v);
  T* rho = static_cast<T*>(Pr.rho) +
           (((size_t)e * a.Nrho * a.M + term) * 3 + P) * N * N;
#pragma unroll
  for (int k = 0; k < N; ++k) rho[(size_t)k * N + i] = v[k];
}

// Terms: one cluster per (pair, point, radial slice), two lanes per pencil
// (half_pencil.cuh), one transform slab A and one receive slab R as in
// vhs_termsh_kernel, whose bound (the exchange through distributed shared
// memory) it shares: two exchanges per term.  Per direction:
//   Z = M_u F_p + i M_v F_q elementwise into A (coalesced reads of F; the row
//   factors of M in a table), z pass, y pass -> exchange into R -> x pass:
//   u_r + i v_r, with the plane transforms u_i + i v_i -> the product h
//   (FP32: u_M X_v + X_u (v_M + X_v)) -> x pass of FFT(h) -> exchange into A
//   -> z pass, y pass, weighted by b into the lane's spectral sums, which stay
//   in registers over all directions of the slice.
// R is free again when the second exchange's barrier completes, and A when
// the first one's does, so a term needs two cluster barriers.
template <typename R, int N, int C> struct VssHGeo {
  using G = HalfGeo<N, C>;
  static constexpr bool SPLIT = sizeof(R) == 4;
  static constexpr int RT = 4 * G::P * N;          // row factors of M_u, M_v
  static constexpr size_t smem =
      (size_t)(G::SLAB + G::P * N * N + RT + (SPLIT ? 6 * N : 0)) * sizeof(c2_t<R>);
  static constexpr int by_smem = (int)((size_t)(228 * 1024) / (smem + 1024));
  // threads per SM by the registers of three arrays of N/2 complex values
  static constexpr int max_threads =
      SPLIT ? (N <= 16 ? 768 : N == 24 ? 576 : 512) : (N <= 16 ? 512 : N == 24 ? 384 : 256);
  static constexpr int by_regs = max_threads / G::NT;
  static constexpr int per_sm =
      by_smem < by_regs ? (by_smem > 0 ? by_smem : 1) : (by_regs > 0 ? by_regs : 1);
};

template <typename R, int N, int C>
__global__ void __launch_bounds__(HalfGeo<N, C>::NT, VssHGeo<R, N, C>::per_sm)
vss_terms_kernel(const __grid_constant__ VssTermsArgs a) {
  using G = HalfGeo<N, C>;
  using T = c2_t<R>;
  constexpr int H = G::H, P = G::P, NT = G::NT;
  constexpr bool SPLIT = sizeof(R) == 4;
  constexpr uint32_t ES = (uint32_t)sizeof(T);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* A = reinterpret_cast<T*>(smem_raw);
  T* Rb = A + G::SLAB;                 // [P][N x][N z]
  T* rt = Rb + P * N * N;              // [u, v][lz != H, lz == H][P N]
  T* uvt = rt + 4 * P * N;             // u_M [3N], v_M [3N] (SPLIT)
  const int t = threadIdx.x, pp = half_pencil(t), h = half_lane(t);
  const unsigned rank = cluster_rank();
  const int e = blockIdx.z % a.nevals;
  const VssTermsPair& Pr = a.pr[blockIdx.z / a.nevals];
  const int r0 = blockIdx.y * a.Nrho / a.NS, r1 = (blockIdx.y + 1) * a.Nrho / a.NS;
  const int nd = Pr.nd, Tt = a.Nrho * a.M;
  const size_t slab0 = (size_t)rank * P * N * N;
  const T* Fp = static_cast<const T*>(Pr.Fp) + (size_t)e * G::n + slab0;
  const T* Fq = static_cast<const T*>(Pr.Fq) + (size_t)e * G::n + slab0;
  const int pl = pp / N, c = pp % N;
  const int lx = rank * P + pl, yy = lx;
  const int rowb = pl * G::PLANE + c * G::ROW, colb = pl * G::PLANE + c;
  const int colr = pl * N * N + c;
  uint32_t rdst[G::GRP];
#pragma unroll
  for (int g = 0; g < G::GRP; ++g)
    rdst[g] = mapa_u32(smem_u32(Rb), (uint32_t)((h * H) / P + g)) +
              ES * (uint32_t)((P > H ? ((h * H) % P) * N * N : 0) + lx * N + c);
  const R sy = (yy & 1) ? R(-1) : R(1), sz = (c & 1) ? R(-1) : R(1);
  const int ez = t % N;                // this thread's lz in the elementwise pass
  T Qh[H];
#pragma unroll
  for (int m = 0; m < H; ++m) Qh[m] = T{R(0), R(0)};
  // (its third part is taken again at the end: it need not stay in registers)
  const VssScale<R> sc = vss_scale<R, N>(Pr, e);
  const R ss = t < P * N ? sc.su : sc.sv;
  // the row factors of a term, scaled: one (field, row) per thread
  auto row_tables = [&](int term) {
    const int f = t / (P * N), row = t % (P * N);
    const int x = rank * P + row / N, y = row % N;
    const T* ph = static_cast<const T*>(Pr.ph) + (size_t)term * 6 * N + f * 3 * N;
    T E = cmul(ph[x], ph[N + y]);
    E.x *= ss;
    E.y *= ss;
    T fx = T{R(1), R(0)};
    if (x == H) fx = vss_nu(ph[H]);
    if (y == H) fx = cmul(fx, vss_nu(ph[N + H]));
    const T fz = cmul(fx, vss_nu(ph[2 * N + H]));
    rt[f * 2 * P * N + row] = cmul(E, T{R(0.5) * (R(1) + fx.x), R(0.5) * fx.y});
    rt[f * 2 * P * N + P * N + row] = cmul(E, T{R(0.5) * (R(1) + fz.x), R(0.5) * fz.y});
    if constexpr (SPLIT) {
      const T* uv = Pr.uv + ((size_t)e * Tt + term) * 6 * N;
      for (int i = t; i < 6 * N; i += NT) uvt[i] = uv[i];
    }
  };
  cluster_sync_all();                  // every CTA runs before remote stores
#pragma unroll 1
  for (int r = r0; r < r1; ++r)
#pragma unroll 1
  for (int d = 0; d < nd; ++d) {
    const int2 dir = Pr.dirs[d];
    const int term = r * a.M + dir.x;
    const T* ph = static_cast<const T*>(Pr.ph) + (size_t)term * 6 * N;
    row_tables(term);
    __syncthreads();                   // tables are in place; A is read
    {
      const T eu = ph[2 * N + ez], ev = ph[5 * N + ez];
      const T* gu = rt + (ez == H ? P * N : 0);
      const T* gv = gu + 2 * P * N;
#pragma unroll
      for (int j = 0; j < H; ++j) {
        const int i = j * NT + t, row = i / N;    // i % N == ez
        const T u = cmul(cmul(gu[row], eu), Fp[i]);
        const T w = cmul(cmul(gv[row], ev), Fq[i]);
        A[row * G::ROW + ez] = T{u.x - w.y, u.y + w.x};
      }
    }
    __syncthreads();
    T v[H];
#pragma unroll
    for (int m = 0; m < H; ++m) v[m] = A[rowb + 2 * m + h];
    fft_half_dit<R, N, +1>(v, h);
#pragma unroll
    for (int m = 0; m < H; ++m) A[rowb + h * H + m] = v[m];
    __syncthreads();
#pragma unroll
    for (int m = 0; m < H; ++m) v[m] = A[colb + (2 * m + h) * G::ROW];
    fft_half_dit<R, N, +1>(v, h);
#pragma unroll
    for (int m = 0; m < H; ++m)
      st_cluster(rdst[P > H ? 0 : m / P] + ES * (uint32_t)((P > H ? m : m % P) * N * N),
                 v[m]);
    cluster_arrive();
    // u_i + i v_i of this lane's points while the exchange completes
    T pi[H];
    {
      const T* rp = static_cast<const T*>(Pr.rho) + ((size_t)e * Tt + term) * 3 * N * N;
      const T rx = rp[yy * N + c];
      const T* rY = rp + N * N + c + h * H * N;
      const T* rZ = rp + 2 * N * N + yy + h * H * N;
#pragma unroll
      for (int m = 0; m < H; ++m) {
        const T ry = rY[m * N], rz = rZ[m * N];
        const R xs = (m & 1) ? R(-1) : R(1);
        pi[m].x = sz * rz.x + (sy * ry.x + xs * rx.x);
        pi[m].y = sz * rz.y + (sy * ry.y + xs * rx.y);
      }
    }
    cluster_wait();
#pragma unroll
    for (int m = 0; m < H; ++m) v[m] = Rb[colr + (2 * m + h) * N];
    fft_half_dit<R, N, +1>(v, h);
    if constexpr (SPLIT) {
      T uyz = cmul(uvt[N + yy], uvt[2 * N + c]);
      T vyz = cmul(uvt[4 * N + yy], uvt[5 * N + c]);
      uyz.x *= sc.su; uyz.y *= sc.su;
      vyz.x *= sc.sv; vyz.y *= sc.sv;
#pragma unroll
      for (int m = 0; m < H; ++m) {
        const T uM = cmul(uvt[h * H + m], uyz), vM = cmul(uvt[3 * N + h * H + m], vyz);
        const T Xu = T{v[m].x, pi[m].x}, Xv = T{v[m].y, pi[m].y};
        const T a1 = cmul(uM, Xv);
        const T a2 = cmul(Xu, T{vM.x + Xv.x, vM.y + Xv.y});
        v[m] = T{a1.x + a2.x, a1.y + a2.y};
      }
    } else {
#pragma unroll
      for (int m = 0; m < H; ++m)
        v[m] = cmul(T{v[m].x, pi[m].x}, T{v[m].y, pi[m].y});
    }
    fft_half_dif<R, N, -1>(v, h);
    {
      const uint32_t a0 = smem_u32(A) + ES * (uint32_t)(yy * G::ROW + c);
#pragma unroll
      for (int m = 0; m < H; ++m) {
        const int l = 2 * m + h;
        st_cluster(mapa_u32(a0, (uint32_t)(l / P)) + ES * (uint32_t)((l % P) * G::PLANE), v[m]);
      }
    }
    cluster_sync_all();
#pragma unroll
    for (int m = 0; m < H; ++m) v[m] = A[rowb + 2 * m + h];
    fft_half_dit<R, N, -1>(v, h);
#pragma unroll
    for (int m = 0; m < H; ++m) A[rowb + h * H + m] = v[m];
    __syncthreads();
#pragma unroll
    for (int m = 0; m < H; ++m) v[m] = A[colb + (2 * m + h) * G::ROW];
    fft_half_dit<R, N, -1>(v, h);
    // lane's points (lx, ly = h H + m, lz = c)
    const size_t o = slab0 + (size_t)pl * N * N + (size_t)h * H * N + c;
    const T* b1 = static_cast<const T*>(Pr.b) + (size_t)term * G::n + o;
    const T* b2 = dir.y >= 0
        ? static_cast<const T*>(Pr.b) + (size_t)(r * a.M + dir.y) * G::n + o : nullptr;
    const R wr = SPLIT ? R(1) : (R)a.w[r];
#pragma unroll
    for (int m = 0; m < H; ++m) {
      T b = b1[(size_t)m * N];
      if (b2) { const T q = b2[(size_t)m * N]; b.x += q.x; b.y += q.y; }
      const T x = cmul(v[m], b);
      Qh[m].x += wr * x.x;
      Qh[m].y += wr * x.y;
    }
  }
  const R back = vss_scale<R, N>(Pr, e).back;
  const R wo = SPLIT ? (R)a.w[r0] * back : back;
  T* Ho = static_cast<T*>(Pr.H) + ((size_t)e * a.NS + blockIdx.y) * G::n + slab0 +
          (size_t)pl * N * N + (size_t)h * H * N + c;
#pragma unroll
  for (int m = 0; m < H; ++m) Ho[(size_t)m * N] = T{wo * Qh[m].x, wo * Qh[m].y};
  cluster_sync_all();  // no CTA leaves while peers may still write into it
}

// Terms with the whole cube in one CTA, for grids that fit (FP32 up to N=24,
// FP64 up to N=16): transform slab A (padded) and the spectral sums Qh in shared
// memory, no exchange.  Passes x (from F_p and F_q, coalesced), y, z; the
// product of a z-pencil and its forward z pass in registers; y; x, weighted by
// b into Qh.  A thread's x pencils of the last pass of a term and the first of
// the next are the same, so a term takes four CTA barriers.  HP: two lanes per
// pencil (N <= 16).
template <typename R, int N> struct Vss1Geo {
  static constexpr bool SPLIT = sizeof(R) == 4;
  static constexpr bool HP = N <= 16;
  static constexpr int V = HP ? N / 2 : N;
  static constexpr int NT = HP ? 2 * N * N : N * N;
  static constexpr int ROW = N + 1, PLANE = N * ROW, n = N * N * N;
  // A, Qh, r_x of the term, u_M and v_M
  static constexpr size_t smem =
      (size_t)(N * PLANE + n + N * ROW + (SPLIT ? 6 * N : 0)) * sizeof(c2_t<R>);
  static constexpr int by_smem = (int)((size_t)(228 * 1024) / (smem + 1024));
  static constexpr int by_regs = (HP ? (SPLIT ? 1024 : 512) : 576) / NT;
  static constexpr int per_sm =
      by_smem < by_regs ? (by_smem > 0 ? by_smem : 1) : (by_regs > 0 ? by_regs : 1);
};

template <typename R, int N>
__global__ void __launch_bounds__(Vss1Geo<R, N>::NT, Vss1Geo<R, N>::per_sm)
vss_terms1_kernel(const __grid_constant__ VssTermsArgs a) {
  using G = Vss1Geo<R, N>;
  using T = c2_t<R>;
  constexpr int V = G::V, NT = G::NT, ROW = G::ROW, PLANE = G::PLANE, H = N / 2;
  constexpr bool HP = G::HP, SPLIT = G::SPLIT;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* A = reinterpret_cast<T*>(smem_raw);     // [N x][N y][ROW z]
  T* Qh = A + N * PLANE;                      // [N][N][N]
  T* rxs = Qh + G::n;                         // [N y][ROW]
  T* uvt = rxs + N * ROW;                     // u_M [3N], v_M [3N] (SPLIT)
  const int t = threadIdx.x, pp = HP ? half_pencil(t) : t, h = HP ? half_lane(t) : 0;
  const int p = pp / N, q = pp % N;
  const int e = blockIdx.z % a.nevals;
  const VssTermsPair& Pr = a.pr[blockIdx.z / a.nevals];
  const int r0 = blockIdx.y * a.Nrho / a.NS, r1 = (blockIdx.y + 1) * a.Nrho / a.NS;
  const int nd = Pr.nd, Tt = a.Nrho * a.M;
  const T* Fp = static_cast<const T*>(Pr.Fp) + (size_t)e * G::n + pp;
  const T* Fq = static_cast<const T*>(Pr.Fq) + (size_t)e * G::n + pp;
  auto in = [&](int m) { return HP ? 2 * m + h : m; };
  auto out = [&](int m) { return HP ? h * H + m : m; };
  auto inv = [&](T* v) {
    if constexpr (HP) fft_half_dit<R, N, +1>(v, h);
    else fft<R, N, +1>(v);
  };
  auto fwd = [&](T* v) {
    if constexpr (HP) fft_half_dit<R, N, -1>(v, h);
    else fft<R, N, -1>(v);
  };
  const VssScale<R> sc = vss_scale<R, N>(Pr, e);
  for (int i = t; i < G::n; i += NT) Qh[i] = T{R(0), R(0)};
  __syncthreads();
#pragma unroll 1
  for (int r = r0; r < r1; ++r)
#pragma unroll 1
  for (int d = 0; d < nd; ++d) {
    const int2 dir = Pr.dirs[d];
    const int term = r * a.M + dir.x;
    const T* rp = static_cast<const T*>(Pr.rho) + ((size_t)e * Tt + term) * 3 * N * N;
    T v[V];
    {  // x pass, (ly, lz) = (p, q): Z = M_u F_p + i M_v F_q
      T g[2], gx[2];
      const T* ph = static_cast<const T*>(Pr.ph) + (size_t)term * 6 * N;
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const T* f = ph + 3 * N * s;
        T E = cmul(f[N + p], f[2 * N + q]);
        const R ss = s == 0 ? sc.su : sc.sv;
        E.x *= ss;
        E.y *= ss;
        T fy = T{R(1), R(0)};
        if (p == H) fy = vss_nu(f[N + H]);
        if (q == H) fy = cmul(fy, vss_nu(f[2 * N + H]));
        const T fx = cmul(fy, vss_nu(f[H]));
        g[s] = cmul(E, T{R(0.5) * (R(1) + fy.x), R(0.5) * fy.y});
        gx[s] = cmul(E, T{R(0.5) * (R(1) + fx.x), R(0.5) * fx.y});
      }
#pragma unroll
      for (int m = 0; m < V; ++m) {
        const int x = in(m);
        const bool nyq = HP ? (2 * m == H && h == 0) : m == H;
        const T u = cmul(cmul(nyq ? gx[0] : g[0], ph[x]), Fp[x * N * N]);
        const T w = cmul(cmul(nyq ? gx[1] : g[1], ph[3 * N + x]), Fq[x * N * N]);
        v[m] = T{u.x - w.y, u.y + w.x};
      }
      inv(v);
#pragma unroll
      for (int m = 0; m < V; ++m) A[out(m) * PLANE + p * ROW + q] = v[m];
    }
    __syncthreads();
    // tables of the product, read two barriers later at the earliest
    for (int i = t; i < N * N; i += NT) rxs[(i / N) * ROW + i % N] = rp[i];
    if constexpr (SPLIT) {
      const T* uv = Pr.uv + ((size_t)e * Tt + term) * 6 * N;
      for (int i = t; i < 6 * N; i += NT) uvt[i] = uv[i];
    }
#pragma unroll
    for (int m = 0; m < V; ++m) v[m] = A[p * PLANE + in(m) * ROW + q];   // (x, z)
    inv(v);
#pragma unroll
    for (int m = 0; m < V; ++m) A[p * PLANE + out(m) * ROW + q] = v[m];
    const T rz = rp[2 * N * N + p * N + q];
    __syncthreads();
#pragma unroll
    for (int m = 0; m < V; ++m) v[m] = A[p * PLANE + q * ROW + in(m)];   // (x, y)
    inv(v);
    {
      const R sx = (p & 1) ? R(-1) : R(1), sy = (q & 1) ? R(-1) : R(1);
      const T* rY = rp + N * N + p * N;
      T uxy{}, vxy{};
      if constexpr (SPLIT) {
        uxy = cmul(uvt[p], uvt[N + q]);
        vxy = cmul(uvt[3 * N + p], uvt[4 * N + q]);
        uxy.x *= sc.su; uxy.y *= sc.su;
        vxy.x *= sc.sv; vxy.y *= sc.sv;
      }
#pragma unroll
      for (int m = 0; m < V; ++m) {
        const int z = out(m);
        const T rx = rxs[q * ROW + z], ry = rY[z];
        const R zs = (m & 1) ? R(-1) : R(1);
        const T Xu = T{v[m].x, sx * rx.x + (sy * ry.x + zs * rz.x)};
        const T Xv = T{v[m].y, sx * rx.y + (sy * ry.y + zs * rz.y)};
        if constexpr (SPLIT) {
          const T uM = cmul(uxy, uvt[2 * N + z]), vM = cmul(vxy, uvt[5 * N + z]);
          const T a1 = cmul(uM, Xv);
          const T a2 = cmul(Xu, T{vM.x + Xv.x, vM.y + Xv.y});
          v[m] = T{a1.x + a2.x, a1.y + a2.y};
        } else {
          v[m] = cmul(Xu, Xv);
        }
      }
    }
    if constexpr (HP) fft_half_dif<R, N, -1>(v, h);    // out() -> in()
    else fft<R, N, -1>(v);
#pragma unroll
    for (int m = 0; m < V; ++m) A[p * PLANE + q * ROW + in(m)] = v[m];
    __syncthreads();
#pragma unroll
    for (int m = 0; m < V; ++m) v[m] = A[p * PLANE + in(m) * ROW + q];
    fwd(v);
#pragma unroll
    for (int m = 0; m < V; ++m) A[p * PLANE + out(m) * ROW + q] = v[m];
    __syncthreads();
#pragma unroll
    for (int m = 0; m < V; ++m) v[m] = A[in(m) * PLANE + p * ROW + q];
    fwd(v);
    const T* b1 = static_cast<const T*>(Pr.b) + (size_t)term * G::n + pp;
    const T* b2 = dir.y >= 0
        ? static_cast<const T*>(Pr.b) + (size_t)(r * a.M + dir.y) * G::n + pp : nullptr;
    const R wr = SPLIT ? R(1) : (R)a.w[r];
#pragma unroll
    for (int m = 0; m < V; ++m) {
      const int j = out(m) * N * N;
      T b = b1[j];
      if (b2) { const T c = b2[j]; b.x += c.x; b.y += c.y; }
      const T x = cmul(v[m], b);
      T s = Qh[j + pp];
      s.x += wr * x.x;
      s.y += wr * x.y;
      Qh[j + pp] = s;
    }
    // (HP: the pencil's other lane still reads A[in()] of this pass, and both
    // lanes' next stores follow the shuffles of the next transform)
  }
  const R wo = SPLIT ? (R)a.w[r0] * sc.back : sc.back;
  T* Ho = static_cast<T*>(Pr.H) + ((size_t)e * a.NS + blockIdx.y) * G::n + pp;
#pragma unroll
  for (int m = 0; m < V; ++m) {
    const int j = out(m) * N * N;
    const T s = Qh[j + pp];
    Ho[j] = T{wo * s.x, wo * s.y};
  }
}

}  // namespace dgfs
