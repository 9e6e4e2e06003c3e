// Heterodyne grid search: het_space (QuickCBC.c:4570-4910) with limits (4275-4385),
// Fisher_All (2695-2817), FisherEvec (2449-2530), efix (4387-4567) and diff (4913-4964).
//
// The control logic (the eigen-directions of the Fisher matrix, the bracketing/secant search of efix, the
// flattening of the grid to J = 2 regions) runs on the host in FP64, restated from the reference.  The
// device computes the waveforms and everything that runs over bins: the band limits from the SNR
// accumulation, the Fisher sums over the reference set's 22 central-difference neighbours, the distances
// of each round of efix trial points (all directions search in step), the ratios of the 11 scaled steps to
// the reference, and the adaptive grid walk.  Only those results cross to the host, through pinned memory.
//
// Differences from the reference, on purpose: no diagnostic files (fspace.dat, df.dat,
// df_flat.dat, ratio.dat) and no printing; the grid is copied out before its scratch is released
// (the reference reads it after free, QuickCBC.c:4866-4893).
#include <cuda_runtime.h>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <algorithm>
#include <functional>
#include <string>
#include <vector>

#include "qcbc_hetspace.h"

namespace qcbc {
namespace {

constexpr int NP = 11;
constexpr double kEtaMin = 0.05;                       // ConstCBC.h:57
constexpr double kTPIr = 6.2831853071795862319959269370884;   // TPI, ConstCBC.h:4
constexpr double kPIr = 3.1415926535897931159979634685442;    // PI, Constants.h:2
constexpr double kEps = 1.0e-5;                        // Fisher_All step, QuickCBC.c:2723

// Final-state fit of the ringdown frequency (Utilities.c:313-360), masses in seconds.
double fqnm(double m1, double m2, double chi1, double chi2) {
  const double p0 = 0.04827, p1 = 0.01707;
  const double k00 = -3.82, k01 = -1.2019, k02 = -1.20764, k10 = 3.79245, k11 = 1.18385, k12 = 4.90494;
  const double scri = 0.41616;
  double q = m1 < m2 ? m1 / m2 : m2 / m1;
  double eta = q / ((1.0 + q) * (1.0 + q));
  double atot = (chi1 + q * q * chi2) / ((1.0 + q) * (1.0 + q));
  double aeff = atot + scri * eta * (chi1 + chi2);
  double Z1 = 1.0 + pow((1.0 - aeff * aeff), (1. / 3.)) * (pow((1. + aeff), (1. / 3.)) + pow((1. - aeff), (1. / 3.)));
  double Z2 = sqrt(3.0 * aeff * aeff + Z1 * Z1);
  double risco = 3.0 + Z2 - (aeff / (fabs(aeff) + 1.0e-20)) * sqrt((3.0 - Z1) * (3.0 + Z1 + 2.0 * Z2));
  double Eisco = sqrt(1.0 - 2. / (3.0 * risco));
  double Lisco = (2. / (3.0 * sqrt(3.))) * (1. + 2.0 * sqrt(3.0 * risco - 2.0));
  double Mf = (1.0 - eta * (1.0 - Eisco) - 4.0 * eta * eta * (4.0 * p0 + 16.0 * p1 * atot * (atot + 1.0) + Eisco - 1.0)) *
              (m1 + m2);
  double af = atot + eta * (Lisco - 2 * atot * (Eisco - 1.0)) + k00 * eta * eta + k01 * eta * eta * aeff +
              k02 * eta * eta * aeff * aeff + k10 * eta * eta * eta + k11 * eta * eta * eta * aeff +
              k12 * eta * eta * eta * aeff * aeff;
  return (1.5251 - 1.1568 * pow((1.0 - af), 0.1292)) / (kTPIr * Mf);
}

// Utilities.c:567-585
double fringdown(const double* p) {
  const double Msun = 1.988546954961461467461011951140572744e30, Tsun = 4.92569043916e-6;
  double Mc = exp(p[0]) / Msun * Tsun, M = exp(p[1]) / Msun * Tsun;
  double eta = pow((Mc / M), (5.0 / 3.0));
  if (eta > 0.25) eta = 0.25;
  double dm = sqrt(1.0 - 4.0 * eta);
  return fqnm(M * (1.0 + dm) / 2.0, M * (1.0 - dm) / 2.0, p[2], p[3]);
}

// Cyclic Jacobi rotations for the symmetric eigenproblem (Golub & Van Loan, Matrix Computations
// 8.5): A is overwritten; V gets the eigenvectors as columns; eigenvalues on the diagonal.
void jacobi_eigen(double (&A)[NP][NP], double (&V)[NP][NP], double* eval) {
  for (int i = 0; i < NP; i++)
    for (int j = 0; j < NP; j++) V[i][j] = i == j ? 1.0 : 0.0;
  for (int sweep = 0; sweep < 100; sweep++) {
    double off = 0.0, tot = 0.0;
    for (int i = 0; i < NP; i++)
      for (int j = 0; j < NP; j++) {
        tot += A[i][j] * A[i][j];
        if (i != j) off += A[i][j] * A[i][j];
      }
    if (off <= 1e-30 * tot || off == 0.0) break;
    for (int p = 0; p + 1 < NP; p++)
      for (int q = p + 1; q < NP; q++) {
        const double apq = A[p][q];
        if (apq == 0.0) continue;
        const double theta = (A[q][q] - A[p][p]) / (2.0 * apq);
        const double t = (theta >= 0 ? 1.0 : -1.0) / (fabs(theta) + sqrt(theta * theta + 1.0));
        const double c = 1.0 / sqrt(t * t + 1.0), s = t * c;
        for (int k = 0; k < NP; k++) {
          const double akp = A[k][p], akq = A[k][q];
          A[k][p] = c * akp - s * akq;
          A[k][q] = s * akp + c * akq;
        }
        for (int k = 0; k < NP; k++) {
          const double apk = A[p][k], aqk = A[q][k];
          A[p][k] = c * apk - s * aqk;
          A[q][k] = s * apk + c * aqk;
        }
        for (int k = 0; k < NP; k++) {
          const double vkp = V[k][p], vkq = V[k][q];
          V[k][p] = c * vkp - s * vkq;
          V[k][q] = s * vkp + c * vkq;
        }
      }
  }
  for (int i = 0; i < NP; i++) eval[i] = A[i][i];
}

// FisherEvec (QuickCBC.c:2449-2530): eigenvalues in ascending |value| as 1-sigma jump sizes
// 1/sqrt(max(value, 10)); ev[i] = eigenvector i.  A vanishing diagonal gives unit directions.
void fisher_evec(const double (&F)[NP][NP], double* ej, double (&ev)[NP][NP]) {
  bool small = false;
  for (int i = 0; i < NP; i++)
    if (fabs(F[i][i]) < 1.0e-16) small = true;
  if (small) {
    for (int i = 0; i < NP; i++) {
      ej[i] = 10000.0;
      for (int j = 0; j < NP; j++) ev[i][j] = i == j ? 1.0 : 0.0;
    }
    return;
  }
  double A[NP][NP], V[NP][NP], val[NP];
  memcpy(A, F, sizeof(A));
  jacobi_eigen(A, V, val);
  for (int i = 0; i + 1 < NP; i++) {            // ascending |value|, columns follow
    int best = i;
    for (int j = i + 1; j < NP; j++)
      if (fabs(val[j]) < fabs(val[best])) best = j;
    if (best != i) {
      std::swap(val[i], val[best]);
      for (int k = 0; k < NP; k++) std::swap(V[k][i], V[k][best]);
    }
  }
  for (int i = 0; i < NP; i++) {
    ej[i] = val[i];
    for (int j = 0; j < NP; j++) ev[i][j] = V[j][i];
  }
  for (int i = 0; i < NP; i++) {
    if (ej[i] < 10.0) ej[i] = 10.0;
    ej[i] = 1.0 / sqrt(ej[i]);
  }
}

// A step from params along direction (eval e_i): sign flipped if it leaves eta <= 1/4, angles
// wrapped, clamped to the prior box, eta kept in [etamin, 0.2499] (QuickCBC.c:4414-4450).
void step_point(const double* params, double a, const double* e, const double* pmin, const double* pmax, double* px) {
  for (int j = 0; j < NP; ++j) px[j] = params[j] + a * e[j];
  double leta = (5.0 / 3.0) * (px[0] - px[1]);
  if (exp(leta) > 0.25)
    for (int j = 0; j < NP; ++j) px[j] = params[j] - a * e[j];
  double x = px[4] / kTPIr;
  px[4] = (x - floor(x)) * kTPIr;
  if (x < 0.0) px[4] += 1.0;
  x = px[7] / kTPIr;
  px[7] = (x - floor(x)) * kTPIr;
  if (x < 0.0) px[7] += 1.0;
  x = px[9] / kPIr;
  px[9] = (x - floor(x)) * kPIr;
  if (x < 0.0) px[9] += 1.0;
  while (px[4] > kTPIr) px[4] -= kTPIr;
  while (px[4] < 0.0) px[4] += kTPIr;
  while (px[7] > kTPIr) px[7] -= kTPIr;
  while (px[7] < 0.0) px[7] += kTPIr;
  while (px[9] > kPIr) px[9] -= kPIr;
  while (px[9] < 0.0) px[9] += kPIr;
  for (int j = 0; j < NP; ++j) if (px[j] > pmax[j]) px[j] = pmax[j];
  for (int j = 0; j < NP; ++j) if (px[j] < pmin[j]) px[j] = pmin[j];
  leta = (5.0 / 3.0) * (px[0] - px[1]);
  const double eta = exp(leta);
  if (eta > 0.25) px[0] = px[1] + 3.0 / 5.0 * log(0.2499);
  if (eta < kEtaMin) px[0] = px[1] + 3.0 / 5.0 * log(kEtaMin);
}

#define HS_CU(x)                                                                   \
  do {                                                                             \
    cudaError_t e_ = (x);                                                          \
    if (e_ != cudaSuccess) {                                                       \
      err = std::string(#x) + ": " + cudaGetErrorString(e_);                       \
      return -3;                                                                   \
    }                                                                              \
  } while (0)

// Device scratch of the grid searches of one host thread, kept from call to call (grow-only, per
// device).  The Fisher waves are (2 NP + 1) nifo doubles twice per in-band bin and their terms 66 nifo, about
// 350 MB together at 128 s and 4096 Hz, and allocating and releasing them on every call cost up to a second.  A search ends with
// its stream synchronised, so the next search of the thread may reuse the buffers.  They are
// released with the process.
struct ScratchCache {
  std::vector<void*> p[16];
  std::vector<size_t> cap[16];
  void *h[16] = {}, *m[16] = {};     // pinned host block and its device address
  size_t hcap[16] = {};
};
thread_local ScratchCache tls_scratch;

// Hands out the cached buffers in the order a search asks for them; on every exit path the search's
// stream is drained before the buffers can be handed out again.
struct Scratch {
  int device = 0;
  size_t next = 0;
  cudaStream_t stream;
  explicit Scratch(cudaStream_t s) : stream(s) { cudaGetDevice(&device); }
  ~Scratch() { cudaStreamSynchronize(stream); }
  template <class T>
  cudaError_t alloc(T** out, size_t n) {
    std::vector<void*>& p = tls_scratch.p[device];
    std::vector<size_t>& cap = tls_scratch.cap[device];
    const size_t bytes = n * sizeof(T) > 0 ? n * sizeof(T) : 1;
    if (next == p.size()) {
      p.push_back(nullptr);
      cap.push_back(0);
    }
    if (cap[next] < bytes) {
      cudaFree(p[next]);
      p[next] = nullptr;
      cap[next] = 0;
      cudaError_t e = cudaMalloc(&p[next], bytes);
      if (e != cudaSuccess) return e;
      cap[next] = bytes;
    }
    *out = static_cast<T*>(p[next++]);
    return cudaSuccess;
  }
  // the thread's pinned host block as a T, and the device's view of it
  template <class T>
  cudaError_t host(T** h, T** m) {
    ScratchCache& c = tls_scratch;
    if (c.hcap[device] < sizeof(T)) {
      cudaFreeHost(c.h[device]);
      c.h[device] = nullptr;
      c.hcap[device] = 0;
      cudaError_t e = cudaMallocHost(&c.h[device], sizeof(T));
      if (e == cudaSuccess) e = cudaHostGetDevicePointer(&c.m[device], c.h[device], 0);
      if (e != cudaSuccess) return e;
      c.hcap[device] = sizeof(T);
    }
    *h = static_cast<T*>(c.h[device]);
    *m = static_cast<T*>(c.m[device]);
    return cudaSuccess;
  }
};

}  // namespace

void fisher_evec_11(const double (&F)[11][11], double* ej, double (&ev)[11][11]) { fisher_evec(F, ej, ev); }

int efix_run(const double* params, const double* pmin, const double* pmax, double* eval, const double (&evec)[11][11],
             double zs, const std::function<int(const double*, int, double*)>& dist) {
  const double zmx = zs * 2.0, zmn = zs / 2.0;
  struct Search {
    double e[NP], dzmin = 1.0e20, alpham = 1.0, alpha0 = 1.0, alpha = 0.0, z0 = 0.0;
    int k = 0;
    bool secant = false, done = false;
  } dir[NP];
  for (int i = 0; i < NP; i++)
    for (int j = 0; j < NP; j++) dir[i].e[j] = eval[i] * evec[i][j];
  for (;;) {
    double px[NP * NP], z[NP];
    int who[NP], n = 0;
    for (int i = 0; i < NP; i++) {
      if (dir[i].done) continue;
      step_point(params, dir[i].secant ? dir[i].alpha : dir[i].alpha0, dir[i].e, pmin, pmax, px + (size_t)n * NP);
      who[n++] = i;
    }
    if (n == 0) break;
    if (int rc = dist(px, n, z)) return rc;
    for (int q = 0; q < n; q++) {
      Search& d = dir[who[q]];
      const double dz = fabs(z[q] - zs);
      if (!d.secant) {                                // bracket: double or divide until within a factor of two
        d.z0 = z[q];
        if (dz < d.dzmin) { d.dzmin = dz; d.alpham = d.alpha0; }
        if (d.z0 < zmn) d.alpha0 *= 2.0;
        if (d.z0 > zmx) d.alpha0 /= 1.9;
        d.k++;
        if (!((d.z0 > zmx || d.z0 < zmn) && d.k < 15 && fabs(d.alpha0 < 1.0e4))) {
          d.alpha = d.alpha0 * 1.1;
          d.k = 0;
          d.secant = true;
        }
      } else {
        double next;
        if (d.alpha > d.alpha0) next = d.alpha0 + (zs - d.z0) / (z[q] - d.z0) * (d.alpha - d.alpha0);
        else next = d.alpha + (zs - z[q]) / (d.z0 - z[q]) * (d.alpha0 - d.alpha);
        if (dz < d.dzmin) { d.dzmin = dz; d.alpham = d.alpha; }
        d.z0 = z[q];
        d.alpha0 = d.alpha;
        d.alpha = next;
        d.k++;
        if (!(fabs(z[q] - zs) > 0.2 && d.k < 10 && fabs(d.alpha < 1.0e4))) d.done = true;
      }
    }
  }
  for (int i = 0; i < NP; i++) {
    if (dir[i].dzmin / zs > 1.0) dir[i].alpham = 0.0;  // kill any failed direction
    eval[i] *= dir[i].alpham;
  }
  return 0;
}

int het_space_run(const HetSpaceIn& in, const double* params, const double* pmin, const double* pmax,
                  HetSpaceOut& out, std::string& err) {
  const NetGeom& g = in.g;
  const int nifo = g.nifo, N = in.N, N2 = N / 2;
  const double Tobs = in.Tobs;
  const int ss = in.sn_stride;
  cudaStream_t s = in.stream;
  Scratch sc(s);
  constexpr int kSets = 2 * NP + 1, kChunks = 148, kHostGrid = 4096;
  double *d_freq, *d_S, *d_amp, *d_ph, *d_dS, *d_bsum;
  PhdRec* d_rec;
  int* d_st;
  HsLimits* d_lim;
  int imin = (int)(Tobs * in.fmin), imax = (int)(Tobs * in.fmax);   // band of the Fisher matrix
  if (imax > N2) imax = N2;
  const int nfish = imax > imin ? imax - imin : 0;
  HS_CU(sc.alloc(&d_rec, (size_t)kSets));
  HS_CU(sc.alloc(&d_st, (size_t)kSets));
  HS_CU(sc.alloc(&d_amp, (size_t)nifo * N2));                       // the reference set's waves
  HS_CU(sc.alloc(&d_ph, (size_t)nifo * N2));
  HS_CU(sc.alloc(&d_dS, (size_t)N2));
  HS_CU(sc.alloc(&d_bsum, (size_t)N2 / 1024 + 1));
  HS_CU(sc.alloc(&d_lim, 1));
  HS_CU(sc.alloc(&d_freq, in.d_freq ? 1 : (size_t)N2));
  HS_CU(sc.alloc(&d_S, in.d_S ? 1 : (size_t)nifo * ss));
  // pinned host memory the kernels read and write: parameters, limits, distances, the Fisher matrix, the grid
  struct Pinned {
    HsLimits lim;
    double par[kSets * NP], part[NP * kChunks], fish[NP * NP];
    int count, grid[kHostGrid];
  }*h, *m;
  HS_CU(sc.host(&h, &m));
  if (!in.d_freq) HS_CU(cudaMemcpyAsync(d_freq, in.h_freq, sizeof(double) * N2, cudaMemcpyHostToDevice, s));
  if (!in.d_S) HS_CU(cudaMemcpyAsync(d_S, in.h_S, sizeof(double) * nifo * ss, cudaMemcpyHostToDevice, s));
  const double *freq = in.d_freq ? in.d_freq : d_freq, *S = in.d_S ? in.d_S : d_S;
  int launches = 0;

  // records of `nset` parameter sets (host rows of NP); the stream has been waited for since the last
  auto records = [&](const double* par, int nset) {
    memcpy(h->par, par, sizeof(double) * NP * nset);
    launch_setup(m->par, nset, g, in.qnm, d_rec, d_st, s);
    launches += 1;
  };

  // ---- limits (QuickCBC.c:4275-4385)
  double fstop = 2.0 * fringdown(params);
  if (fstop < 64.0) fstop = 64.0;
  int M = (int)(fstop * Tobs);
  if (M > N2) M = N2;
  if (M < 2) { err = "het_space: signal band below two bins"; return -2; }
  records(params, 1);                                 // the reference set, its waves kept for diff and the ratios
  launch_waves(d_rec, 1, g, freq, M, d_amp, d_ph, s);
  launch_hs_limits(d_rec, d_amp, nifo, M, S, ss, in.fmin, Tobs, d_dS, d_bsum, d_lim, &m->lim, s);
  launches += 3;
  HS_CU(cudaGetLastError());
  HS_CU(cudaStreamSynchronize(s));
  const int MN = h->lim.MN, MM = h->lim.MM, J = 2;
  const double tol = 0.003;
  if (MM <= MN) { err = "het_space: empty signal band"; return -2; }
  int rc;

  // ---- Fisher_All (QuickCBC.c:2695-2817) and FisherEvec
  double F[NP][NP];
  for (int i = 0; i < NP; i++)
    for (int j = 0; j < NP; j++) F[i][j] = i == j ? 1.0e4 : 0.0;
  if (fabs(params[2]) < 0.9999 && fabs(params[3]) < 0.9999) {
    std::vector<double> P((size_t)kSets * NP);
    for (int k = 0; k < kSets; k++) memcpy(&P[(size_t)k * NP], params, NP * sizeof(double));
    for (int i = 0; i < NP; i++) {
      P[(size_t)(1 + 2 * i) * NP + i] += kEps;
      P[(size_t)(2 + 2 * i) * NP + i] -= kEps;
    }
    double *fa, *fp, *d_fparts;
    HS_CU(sc.alloc(&fa, (size_t)kSets * nifo * std::max(nfish, 1)));
    HS_CU(sc.alloc(&fp, (size_t)kSets * nifo * std::max(nfish, 1)));
    double* d_terms;
    HS_CU(sc.alloc(&d_terms, (size_t)NP * (NP + 1) / 2 * nifo * std::max(nfish, 1)));
    HS_CU(sc.alloc(&d_fparts, (size_t)NP * (NP + 1) / 2 * 8));
    records(P.data(), kSets);
    launch_waves(d_rec, kSets, g, freq + imin, nfish, fa, fp, s);
    launch_fisher_full(fa, fp, g, nfish, S + imin, ss, kEps, d_terms, d_fparts, m->fish, s);
    launches += 4;
    HS_CU(cudaGetLastError());
    HS_CU(cudaStreamSynchronize(s));
    const double* G = h->fish;
    for (int i = 0; i < NP; i++)
      for (int j = i; j < NP; j++) F[i][j] = F[j][i] = G[i * NP + j];
  }
  double eval[NP], evec[NP][NP];
  fisher_evec(F, eval, evec);

  // ---- efix (QuickCBC.c:4387-4567), zs = 30, diff on the full grid
  auto dist = [&](const double* px, int n, double* z) -> int {
    records(px, n);
    launch_wave_diff(d_rec, n, g, freq, d_amp, d_ph, M, h->lim.jmin, M, S, ss, kChunks, m->part, s);
    launches += 1;
    HS_CU(cudaGetLastError());
    HS_CU(cudaStreamSynchronize(s));
    for (int q = 0; q < n; q++) {
      z[q] = 0.0;
      for (int c = 0; c < kChunks; c++) z[q] += h->part[q * kChunks + c];
    }
    return 0;
  };
  rc = efix_run(params, pmin, pmax, eval, evec, 30.0, dist);
  if (rc != 0) return rc;

  // ---- grid walk (QuickCBC.c:4624-4765): the 11 steps' waves as ratios to the reference's, and the walk
  std::vector<double> P((size_t)NP * NP);
  for (int i = 0; i < NP; ++i) {
    double e[NP];
    for (int j = 0; j < NP; j++) e[j] = eval[i] * evec[i][j];
    step_point(params, 1.0, e, pmin, pmax, &P[(size_t)i * NP]);
  }
  records(P.data(), NP);
  const int W = MM - MN, per = NP * nifo;
  double *d_Cs, *d_Sn;
  int *d_grid, *d_first;
  HS_CU(sc.alloc(&d_Cs, (size_t)per * W));
  HS_CU(sc.alloc(&d_Sn, (size_t)per * W));
  HS_CU(sc.alloc(&d_grid, (size_t)W + 2));
  HS_CU(sc.alloc(&d_first, 3));
  launch_hs_ratios(d_rec, NP, g, freq, d_amp, d_ph, M, MN, MM, d_Cs, d_Sn, s);
  const int djmax = (int)(100.0 * Tobs);                 // maximum spacing
  HS_CU(launch_hs_walk(d_Cs, d_Sn, d_dS, d_lim, per, MN, MM, djmax, tol, W + 2, d_first, d_grid, m->grid,
                       kHostGrid, &m->count, s));
  launches += 2;
  HS_CU(cudaStreamSynchronize(s));
  const int count = h->count;
  if (count < 1) { err = "het_space: grid walk did not finish"; return -2; }
  std::vector<int> fgrid((size_t)count);
  if (count <= kHostGrid) memcpy(fgrid.data(), h->grid, sizeof(int) * count);
  else HS_CU(cudaMemcpy(fgrid.data(), d_grid, sizeof(int) * count, cudaMemcpyDeviceToHost));
  const int Mr = (int)fgrid.size() - 1;

  // ---- spacing per bin and the flattened grid with J = 2 points per region (QuickCBC.c:4767-4864).  The
  // spacing is constant between grid points (100 outside them), so its smallest value over a range of bins
  // is found over the few stretches that overlap the range.
  struct Stretch { int lo, hi, d; };                     // bins [lo, hi)
  std::vector<Stretch> st;
  st.push_back({0, fgrid[0], 100});
  for (int i = 0; i < Mr; i++) st.push_back({fgrid[i], fgrid[i + 1], fgrid[i + 1] - fgrid[i]});
  st.push_back({fgrid[Mr], MM, MM - fgrid[Mr]});
  st.push_back({MM, N2, 100});
  auto spacing_min = [&](int a, int b, int least) {      // smallest spacing of bins [a, b] within [0, N/2)
    size_t lo = 0, hi = st.size();
    while (lo < hi) {                                    // first stretch that ends beyond a
      const size_t mid = (lo + hi) / 2;
      if (st[mid].hi > a) hi = mid; else lo = mid + 1;
    }
    for (; lo < st.size() && st[lo].lo <= b; lo++)
      if (st[lo].hi > st[lo].lo && st[lo].d < least) least = st[lo].d;
    return least;
  };
  std::vector<int> fg;
  fg.reserve(1024);
  int j = MN, k = 0, ii = 0;
  fg.push_back(j);
  do {
    int jm = spacing_min(j, j, 2147483647);
    bool flag;
    do {
      k = j + jm * J;
      const int least = spacing_min(j, k, jm);
      flag = least < jm && k < N2;                       // a range that leaves the bins is not tried again
      jm = least;
    } while (flag);
    j = k;
    for (int i = 0; i < J; ++i) {
      ii++;
      fg.push_back(fg[ii - 1] + jm);
    }
    if (ii > N2) { err = "het_space: grid does not terminate"; return -2; }
  } while (j < MM);
  {
    const int jm = (MM - fg[ii - J]) / J;                // fix the last section so it ends at MM
    if (jm >= 1) {
      ii -= J;
      for (int i = 0; i < J; ++i) {
        ii++;
        fg[ii] = fg[ii - 1] + jm;
      }
    }
  }
  out.MN = MN;
  out.MM = MM;
  out.J = J;
  out.M = ii + 1;
  out.NR = ii / J;
  out.fgrid.assign(fg.begin(), fg.begin() + out.M);
  out.launches = launches;
  return 0;
}

}  // namespace qcbc
