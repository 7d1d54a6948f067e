// Reference-point selection (host).
//
// Reference counterpart: createRPArray, src/utils.cu:66-281, which draws 2k
// uniform points in [0,1)^d with glibc rand(), keeps the k/2 whose distances
// over a 1% sample have the largest spread, and adds "box corner" points;
// buildNodeNet then scores 32 such candidates per layer
// (src/nodes.cu:168-222).  The goal is the same here — reference points whose
// distance fields spread the data over many ε-wide bins — reached directly:
// the k points sit far outside the data along its k leading principal axes
// (sample covariance, orthogonal iteration), so each distance field behaves
// like a projection on one principal axis and successive fields are nearly
// uncorrelated.  MISTIC_RP_BOX reproduces the plain "uniform in the bounding
// box" choice with a seeded generator; MISTIC_RP_USER takes the caller's.
#include <math.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "internal.cuh"

namespace mistic {

namespace {

// SplitMix64: small deterministic generator for seeded choices.
struct SplitMix {
  uint64_t s;
  explicit SplitMix(uint64_t seed) : s(seed) {}
  uint64_t next() {
    uint64_t z = (s += 0x9e3779b97f4a7c15ull);
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
  }
  double uniform() { return (next() >> 11) * (1.0 / 9007199254740992.0); }
  double normal() {
    double u1 = uniform(), u2 = uniform();
    if (u1 < 1e-300) u1 = 1e-300;
    return sqrt(-2.0 * log(u1)) * cos(6.283185307179586 * u2);
  }
};

// Sum of a_i b_i in four independent chains (one chain is bound by the FMA
// latency, not by its throughput).
double dot(const double* a, const double* b, uint32_t d) {
  double s0 = 0, s1 = 0, s2 = 0, s3 = 0;
  uint32_t i = 0;
  for (; i + 4 <= d; i += 4) {
    s0 += a[i] * b[i];
    s1 += a[i + 1] * b[i + 1];
    s2 += a[i + 2] * b[i + 2];
    s3 += a[i + 3] * b[i + 3];
  }
  for (; i < d; ++i) s0 += a[i] * b[i];
  return (s0 + s1) + (s2 + s3);
}

// Modified Gram-Schmidt on the k columns of V (d x k, column-major); returns
// the sum of the columns' norms before they were scaled.
double orthonormalise(std::vector<double>& V, uint32_t d, uint32_t k, SplitMix& rng, int passes) {
  double sum = 0;
  for (uint32_t c = 0; c < k; ++c) {
    double* v = &V[(size_t)c * d];
    for (int pass = 0; pass < passes; ++pass) {
      for (uint32_t p = 0; p < c; ++p) {
        const double* u = &V[(size_t)p * d];
        const double t = dot(u, v, d);
        for (uint32_t i = 0; i < d; ++i) v[i] -= t * u[i];
      }
    }
    const double nrm = sqrt(dot(v, v, d));
    if (nrm < 1e-300) {  // degenerate direction: replace with a random one
      for (uint32_t i = 0; i < d; ++i) v[i] = rng.normal();
      --c;  // redo this column
      continue;
    }
    sum += nrm;
    for (uint32_t i = 0; i < d; ++i) v[i] /= nrm;
  }
  return sum;
}

// W = cov V for the k columns of V (both d x k, column-major), eight columns
// and two rows of cov at a time: 16 sums in registers per pass over a row.
void cov_times(const std::vector<double>& cov, uint32_t d, uint32_t k, const std::vector<double>& V,
               std::vector<double>& W, std::vector<double>& T) {
  T.resize((size_t)d * 8);
  for (uint32_t c0 = 0; c0 < k; c0 += 8) {
    const uint32_t nc = std::min(8u, k - c0);
    for (uint32_t b = 0; b < d; ++b)
      for (uint32_t c = 0; c < 8; ++c) T[(size_t)b * 8 + c] = c < nc ? V[(size_t)(c0 + c) * d + b] : 0.0;
    for (uint32_t a = 0; a < d; a += 2) {
      const double* r0 = &cov[(size_t)a * d];
      const double* r1 = a + 1 < d ? r0 + d : r0;
      double s0[8] = {0, 0, 0, 0, 0, 0, 0, 0}, s1[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      const double* t = T.data();
      for (uint32_t b = 0; b < d; ++b, t += 8) {
        const double x0 = r0[b], x1 = r1[b];
        for (int c = 0; c < 8; ++c) {
          s0[c] += x0 * t[c];
          s1[c] += x1 * t[c];
        }
      }
      for (uint32_t c = 0; c < nc; ++c) {
        W[(size_t)(c0 + c) * d + a] = s0[c];
        if (a + 1 < d) W[(size_t)(c0 + c) * d + a + 1] = s1[c];
      }
    }
  }
}

// Eigenvectors of the symmetric k x k matrix H (row-major, destroyed) by
// cyclic Jacobi rotations (the textbook method), as the columns of Q.
void jacobi(std::vector<double>& H, uint32_t k, std::vector<double>& Q) {
  Q.assign((size_t)k * k, 0.0);
  for (uint32_t i = 0; i < k; ++i) Q[(size_t)i * k + i] = 1.0;
  for (int sweep = 0; sweep < 30; ++sweep) {
    double off = 0, diag = 0;
    for (uint32_t p = 0; p < k; ++p)
      for (uint32_t q = 0; q < k; ++q) (p == q ? diag : off) += H[(size_t)p * k + q] * H[(size_t)p * k + q];
    if (!(off > 1e-24 * diag)) break;
    for (uint32_t p = 0; p < k; ++p)
      for (uint32_t q = p + 1; q < k; ++q) {
        const double hpq = H[(size_t)p * k + q];
        if (hpq == 0.0) continue;
        const double th = (H[(size_t)q * k + q] - H[(size_t)p * k + p]) / (2.0 * hpq);
        const double t = (th >= 0 ? 1.0 : -1.0) / (fabs(th) + sqrt(th * th + 1.0));
        const double c = 1.0 / sqrt(t * t + 1.0), s = t * c;
        for (uint32_t i = 0; i < k; ++i) {
          const double x = H[(size_t)i * k + p], y = H[(size_t)i * k + q];
          H[(size_t)i * k + p] = c * x - s * y;
          H[(size_t)i * k + q] = s * x + c * y;
        }
        for (uint32_t i = 0; i < k; ++i) {
          const double x = H[(size_t)p * k + i], y = H[(size_t)q * k + i];
          H[(size_t)p * k + i] = c * x - s * y;
          H[(size_t)q * k + i] = s * x + c * y;
        }
        for (uint32_t i = 0; i < k; ++i) {
          const double x = Q[(size_t)i * k + p], y = Q[(size_t)i * k + q];
          Q[(size_t)i * k + p] = c * x - s * y;
          Q[(size_t)i * k + q] = s * x + c * y;
        }
      }
  }
}

}  // namespace

void select_reference_points(const mistic_opts& o, uint32_t d, uint32_t k, const std::vector<double>& mean,
                             const std::vector<double>& mn, const std::vector<double>& mx,
                             const std::vector<double>& cov, std::vector<double>& rps) {
  rps.assign((size_t)k * d, 0.0);
  if (k == 0) return;
  if (o.rp_mode == MISTIC_RP_USER) {
    if (!o.rp_user) throw Error(MISTIC_ERR_INVALID_ARG, "rp_mode USER needs opts.rp_user");
    for (size_t i = 0; i < (size_t)k * d; ++i) {
      if (!std::isfinite(o.rp_user[i])) throw Error(MISTIC_ERR_INVALID_ARG, "rp_user has a non-finite value");
      rps[i] = o.rp_user[i];
    }
    return;
  }
  SplitMix rng(o.seed ^ 0x6d69737469637270ull);
  if (o.rp_mode == MISTIC_RP_BOX || cov.empty()) {
    for (uint32_t j = 0; j < k; ++j)
      for (uint32_t i = 0; i < d; ++i) rps[(size_t)j * d + i] = mn[i] + (mx[i] - mn[i]) * rng.uniform();
    return;
  }
  // PCA: orthogonal iteration on a few columns more than wanted until the
  // variance they capture stands still, then the eigenvectors of cov within
  // their span (Rayleigh-Ritz).  The spare columns take up the slow
  // convergence between neighbouring eigenvalues, and the index's candidate
  // count depends on the captured variance only.  Orthogonal iteration on the
  // wanted columns alone, a fixed 200 (d <= 64) or 60 times with one long
  // chain per sum, took 0.4 ms at d = 18, 2.2 ms at d = 57, 46 ms at d = 384.
  const uint32_t kk = std::min(k, d), L = std::min((kk + 15) & ~7u, d);
  std::vector<double> V((size_t)L * d), W((size_t)L * d), T;
  for (auto& v : V) v = rng.normal();
  orthonormalise(V, d, L, rng, 1);
  double var = 0;
  for (int it = 0; it < 60; ++it) {
    cov_times(cov, d, L, V, W, T);
    std::swap(V, W);
    const double v2 = orthonormalise(V, d, L, rng, 1);
    if (it >= 2 && fabs(v2 - var) <= 5e-3 * v2) break;
    var = v2;
  }
  orthonormalise(V, d, L, rng, 1);
  cov_times(cov, d, L, V, W, T);
  std::vector<double> H((size_t)L * L), Q;
  for (uint32_t p = 0; p < L; ++p)
    for (uint32_t q = p; q < L; ++q)
      H[(size_t)p * L + q] = H[(size_t)q * L + p] = dot(&V[(size_t)p * d], &W[(size_t)q * d], d);
  jacobi(H, L, Q);
  std::vector<std::pair<double, uint32_t>> rq(L);  // largest eigenvalue first
  for (uint32_t c = 0; c < L; ++c) {
    rq[c] = {-H[(size_t)c * L + c], c};
    double* w = &W[(size_t)c * d];
    std::fill(w, w + d, 0.0);
    for (uint32_t p = 0; p < L; ++p) {
      const double f = Q[(size_t)p * L + c];
      const double* v = &V[(size_t)p * d];
      for (uint32_t i = 0; i < d; ++i) w[i] += f * v[i];
    }
  }
  std::swap(V, W);
  std::sort(rq.begin(), rq.end());
  double diam = 0;
  for (uint32_t i = 0; i < d; ++i) diam += (mx[i] - mn[i]) * (mx[i] - mn[i]);
  diam = sqrt(diam);
  if (!(diam > 0)) diam = 1.0;
  const double far = 64.0 * diam;
  for (uint32_t j = 0; j < k; ++j) {
    double* r = &rps[(size_t)j * d];
    if (j < kk) {
      const double* v = &V[(size_t)rq[j].second * d];
      for (uint32_t i = 0; i < d; ++i) r[i] = mean[i] - far * v[i];
    } else {  // more reference points than dimensions: seeded box points
      for (uint32_t i = 0; i < d; ++i) r[i] = mn[i] + (mx[i] - mn[i]) * rng.uniform();
    }
  }
}

// Scored reference points (MISTIC_RP_SCORED): the reference's per-layer
// selection, buildNodeNet's candidate scoring (src/nodes.cu:168-222) over
// createRPArray's candidate sets (src/utils.cu:66-136), restated: layer by
// layer, every candidate point bins a sample of the data into eps-wide
// distance fields, and the candidate that leaves the fewest sample pairs
// within one field of each other on every layer chosen so far (the
// neighbour relation of the join) is kept.  Candidates: far points along the
// sample's leading principal axes on both sides, sample points, and seeded
// box points.
void select_reference_points_scored(const mistic_opts& o, uint32_t d, uint32_t k, double eps,
                                    const std::vector<double>& mean, const std::vector<double>& mn,
                                    const std::vector<double>& mx, const std::vector<double>& cov,
                                    const std::vector<double>& sample, uint32_t S, std::vector<double>& rps) {
  rps.assign((size_t)k * d, 0.0);
  if (k == 0) return;
  // candidate pool
  const uint32_t na = std::min<uint32_t>(2 * k, d);
  std::vector<double> pca;
  {
    mistic_opts o2 = o;
    o2.rp_mode = MISTIC_RP_PCA;
    select_reference_points(o2, d, na, mean, mn, mx, cov, pca);  // far points on one side of each axis
  }
  std::vector<double> cand;
  for (uint32_t a = 0; a < na; ++a) {
    const double* p = &pca[(size_t)a * d];
    for (int side = 0; side < 2; ++side)
      for (uint32_t i = 0; i < d; ++i) cand.push_back(side == 0 ? p[i] : 2.0 * mean[i] - p[i]);
  }
  SplitMix rng(o.seed ^ 0x73636f7265647270ull);
  for (int c = 0; c < 8 && S > 0; ++c) {
    const uint32_t r = (uint32_t)(rng.next() % S);
    for (uint32_t i = 0; i < d; ++i) cand.push_back(sample[(size_t)r * d + i]);
  }
  for (int c = 0; c < 8; ++c)
    for (uint32_t i = 0; i < d; ++i) cand.push_back(mn[i] + (mx[i] - mn[i]) * rng.uniform());
  const uint32_t C = (uint32_t)(cand.size() / d);
  // scoring sample: up to 1024 of the sample rows, evenly spaced
  const uint32_t T = std::min<uint32_t>(S, 1024);
  std::vector<uint32_t> rows(T);
  for (uint32_t t = 0; t < T; ++t) rows[t] = (uint32_t)((uint64_t)t * S / std::max(1u, T));
  const double w = eps > 0 ? eps : 1.0;
  std::vector<int64_t> fld((size_t)C * T);
  for (uint32_t c = 0; c < C; ++c)
    for (uint32_t t = 0; t < T; ++t) {
      const double* x = &sample[(size_t)rows[t] * d];
      const double* r = &cand[(size_t)c * d];
      double s2 = 0;
      for (uint32_t i = 0; i < d; ++i) s2 += (x[i] - r[i]) * (x[i] - r[i]);
      fld[(size_t)c * T + t] = (int64_t)std::floor(std::sqrt(s2) / w);
    }
  // surviving sample pairs (a < b), as a flat bitmap
  const size_t NP = (size_t)T * (T - (T > 0)) / 2;
  std::vector<uint8_t> alive(NP, 1);
  std::vector<uint8_t> used(C, 0);
  for (uint32_t j = 0; j < k; ++j) {
    uint32_t best = UINT32_MAX;
    size_t best_n = SIZE_MAX;
    for (uint32_t c = 0; c < C; ++c) {
      if (used[c]) continue;
      const int64_t* f = &fld[(size_t)c * T];
      size_t cnt = 0, pi = 0;
      for (uint32_t a = 0; a < T; ++a)
        for (uint32_t b = a + 1; b < T; ++b, ++pi)
          if (alive[pi] && std::llabs(f[a] - f[b]) <= 1) ++cnt;
      if (cnt < best_n) {
        best_n = cnt;
        best = c;
      }
    }
    if (best == UINT32_MAX) break;
    used[best] = 1;
    const int64_t* f = &fld[(size_t)best * T];
    size_t pi = 0;
    for (uint32_t a = 0; a < T; ++a)
      for (uint32_t b = a + 1; b < T; ++b, ++pi)
        if (alive[pi] && std::llabs(f[a] - f[b]) > 1) alive[pi] = 0;
    for (uint32_t i = 0; i < d; ++i) rps[(size_t)j * d + i] = cand[(size_t)best * d + i];
  }
}

}  // namespace mistic
