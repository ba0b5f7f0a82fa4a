// Order >=2: contraction of axial-basis source moments with band-folded RTE
// kernels (reference _shower_basis.py:894-1050, apply_multi_spectral
// :1126-1198, shower/ge2.py:99-119).
//
// For an OM d and a basis point c at distance r (interval j of the log-r
// grid, offset t) the reference sums, per band lambda and frequency w,
//
//   N_d(w) += s_lambda(r) e^{i w r / v_lambda}
//             sum_l sum_a rot_l[a](w) * sum_p D_p[a] cubic_{lambda j l p}(t, w),
//   rot_l[a](w) = sum_b erow_l[a][b] ch_lambda[c][l, b](w).
//
// Exchanging the sums over a and b gives
//
//   N_d(w) += s e^{i w r/v} sum_l sum_b ch[c][l,b](w) sum_p F_l[b][p] cubic_{j l p}(t, w),
//   F_l[b][p] = sum_a erow_l[a][b] D_p[a],
//
// where F (nch x pairs real numbers per (d, c)) carries all the geometry:
// Wigner small-d rotation, azimuthal rotation, detector harmonics and the
// acceptance coefficients. ge2_geometry_kernel forms F in float64 once per
// (d, c); ge2_apply_kernel runs the float32 contraction with one thread per
// (band, frequency); ge2_reduce_kernel sums the point chunks in a fixed order
// (identical results alone or in a batch) and applies the emission-time phase.
#include <algorithm>

#include "lh_common.cuh"
#include "lh_timing.cuh"
#include "lh_harmonics.cuh"

namespace lh {

constexpr int kGe2Degree = 16;   // source/kernel degree bound
constexpr int kGe2Out = 4;       // acceptance (detector) degree bound
constexpr int kGe2M = 4;         // azimuthal degree bound
constexpr int kGe2Chunk = 32;    // points per partial sum

// Radius, interval, band scales and F of every (OM, point). A CTA takes a block of
// consecutive pairs through three steps in shared memory: one thread per pair
// forms the pair's angles, harmonics and scales; one thread per (pair, nu, mu)
// runs that Wigner chain over the degrees; one thread per (pair, channel row)
// forms the row's F. With one thread per pair the Wigner table (675 float64 at
// degree 8) sat in local memory: 0.22 ms for 61k pairs and 0.105 ms for 8k, most
// of it latency; now 0.139 and 0.041 ms.
constexpr int kGe2GeoThreads = 128;
constexpr size_t kGe2GeoSmem = 46 * 1024;

// float64 values of shared memory: the recurrence factors, then per pair the
// Wigner table, cosine, half-angle cosine and sine, cos/sin(n phi), and the
// detector weight of each (lambda, +mu) and (lambda, -mu).
__host__ __device__ inline int ge2_geo_wigner(const lh_ge2_table& T) {
  return (T.degree + 1) * (2 * T.acc_degree + 1) * (T.max_m + 1);
}
__host__ __device__ inline int ge2_geo_pair_values(const lh_ge2_table& T) {
  return ge2_geo_wigner(T) + 3 + 2 * (T.max_m + 1) + 2 * T.n_pairs;
}
// Pairs per CTA: as many as fit, at most 32.
__host__ __device__ inline int ge2_geo_pairs(const lh_ge2_table& T) {
  const int left = (int)(kGe2GeoSmem / sizeof(double)) - 2 * ge2_geo_wigner(T);
  const int fit = left / ge2_geo_pair_values(T);
  return fit < 32 ? fit : 32;
}
static size_t ge2_geo_smem(const lh_ge2_table& T) {
  return sizeof(double) * (2 * (size_t)ge2_geo_wigner(T) +
                           (size_t)ge2_geo_pairs(T) * ge2_geo_pair_values(T));
}

static unsigned ge2_geo_blocks(const lh_ge2_table& T, int64_t pairs) {
  const int per = ge2_geo_pairs(T);
  return (unsigned)((pairs + per - 1) / per);
}

// Entry (q, n) of the real rotation row block of degree l: detector order q and
// source order n, from the Wigner table (_shower_basis.py:957-977).
LH_DEVICE double ge2_rotation(const double* wig, int l, int A, int M, const double* cosn,
                              const double* sinn, int q, int n) {
  const double root2 = sqrt(2.0);
  const int W = 2 * A + 1, k = abs(n), pp = abs(q);
  auto w = [&](int nu, int mu) { return wig[(l * W + nu + A) * (M + 1) + mu]; };
  if (q == 0) {
    if (n == 0) return w(0, 0);
    const double base = root2 * par(k) * w(0, k);
    return n > 0 ? base * cosn[k] : base * sinn[k];
  }
  if (n == 0) return q > 0 ? root2 * par(pp) * w(pp, 0) : 0.0;
  const double cross = par(pp) * w(pp, k), straight = w(-pp, k);
  if (q > 0) {
    const double cc = par(k) * (cross + straight);
    return n > 0 ? cc * cosn[k] : cc * sinn[k];
  }
  const double ss = par(k) * (cross - straight);
  return n > 0 ? -ss * sinn[k] : ss * cosn[k];
}

LH_DEVICE void ge2_geometry_body(const lh_ge2_table& T, const lh_ge2_problem& P, int64_t block,
                                 int* g_j, float* g_t, double* g_r, float* g_scale, float* g_F) {
  extern __shared__ double s_geo[];
  __shared__ int s_inside[32];
  const int64_t total = (int64_t)P.n_om * P.n_points;
  const int per_block = ge2_geo_pairs(T);
  const int64_t first = block * per_block;
  if (first >= total) return;
  const int count = (int)min((int64_t)per_block, total - first);
  const int L = T.degree, A = T.acc_degree, M = T.max_m, W = 2 * A + 1, NP = T.n_pairs;
  const int chains = W * (M + 1), n_wig = ge2_geo_wigner(T), values = ge2_geo_pair_values(T);
  double* s_lower = s_geo;          // [l][chain]: (l + 1) sqrt((l^2 - mu^2)(l^2 - nu^2))
  double* s_upper = s_geo + n_wig;  // [l][chain]: l sqrt(((l+1)^2 - mu^2)((l+1)^2 - nu^2))
  double* s_pair = s_geo + 2 * n_wig;
  for (int e = threadIdx.x; e < L * chains; e += blockDim.x) {
    const int l = e / chains, chain = e - l * chains, nu = chain / (M + 1) - A,
              mu = chain % (M + 1);
    double lower = (double)(l * l - mu * mu) * (double)(l * l - nu * nu);
    lower = lower > 0.0 ? sqrt(lower) : 0.0;
    const double upper = sqrt((double)((l + 1) * (l + 1) - mu * mu) *
                              (double)((l + 1) * (l + 1) - nu * nu));
    s_lower[e] = (l + 1) * lower;
    s_upper[e] = l * upper;
  }
  for (int k = threadIdx.x; k < count; k += blockDim.x) {
    const int64_t idx = first + k;
    const int d = (int)(idx / P.n_points), c = (int)(idx % P.n_points);
    const double dx = P.receivers[3 * d] - P.points[3 * c];
    const double dy = P.receivers[3 * d + 1] - P.points[3 * c + 1];
    const double dz = P.receivers[3 * d + 2] - P.points[3 * c + 2];
    const double radius = sqrt(dx * dx + dy * dy + dz * dz);
    g_r[idx] = radius;
    const bool inside = radius >= P.radial_low && radius <= P.radial_high;
    s_inside[k] = inside;
    if (!inside) {
      g_j[idx] = -1;
      continue;
    }
    double* pair = s_pair + k * values + n_wig;
    double* cosn = pair + 3;
    double* sinn = cosn + M + 1;
    double* weight = sinn + M + 1;
    double cosine = dz / radius;
    cosine = cosine > 1.0 ? 1.0 : (cosine < -1.0 ? -1.0 : cosine);
    const double phi = atan2(dy, dx);
    const double tr = sqrt(dx * dx + dy * dy);
    const double sine = tr / radius;
    const double cp = tr == 0.0 ? 1.0 : dx / tr;
    const double sp = tr == 0.0 ? 0.0 : dy / tr;
    pair[0] = cosine;
    pair[1] = sqrt((1.0 + cosine) / 2.0);
    pair[2] = sqrt((1.0 - cosine) / 2.0);
    for (int n = 0; n <= M; ++n) {
      cosn[n] = cos(n * phi);
      sinn[n] = sin(n * phi);
    }
    const double lx = P.looks[3 * d], ly = P.looks[3 * d + 1], lz = P.looks[3 * d + 2];
    const double a1 = cosine * cp * lx + cosine * sp * ly - sine * lz;
    const double a2 = -sp * lx + cp * ly;
    const double a3 = sine * cp * lx + sine * sp * ly + cosine * lz;
    double det[(kGe2Out + 1) * (kGe2Out + 1)];
    real_harmonics(a1, a2, a3, A, det);
    // pair weights: alpha_lam Y[lam, +mu], alpha_lam Y[lam, -mu]
    for (int p = 0; p < NP; ++p) {
      const int lam = T.pair_lambda[p], mup = T.pair_mu[p], centre = lam * lam + lam;
      weight[2 * p] = T.alpha[lam] * det[centre + mup];
      weight[2 * p + 1] = mup ? T.alpha[lam] * det[centre - mup] : 0.0;
    }
    const double logr = log(radius);
    int j = bin_right(T.log_r, T.n_intervals + 1, logr);
    j = j < 0 ? 0 : (j > T.n_intervals - 1 ? T.n_intervals - 1 : j);
    g_j[idx] = j;
    g_t[idx] = (float)(logr - T.log_r[j]);
    for (int lam = 0; lam < T.n_bands; ++lam)
      g_scale[(int64_t)lam * total + idx] =
          (float)(P.out_scale[(int64_t)lam * P.n_om + d] * exp(-T.absorption[lam] * radius) /
                  (4 * kPi * radius * radius));
  }
  __syncthreads();
  // Wigner d^l_(mu nu), mu = 0..M, by recurrence in l (:51-87)
  for (int e = threadIdx.x; e < count * chains; e += blockDim.x) {
    const int k = e / chains, chain = e - k * chains, nu = chain / (M + 1) - A,
              mu = chain % (M + 1);
    const int start = abs(nu) > mu ? abs(nu) : mu;
    if (!s_inside[k] || start > L) continue;
    double* wig = s_pair + k * values;
    const double cosine = wig[n_wig], hc = wig[n_wig + 1], hs = wig[n_wig + 2];
    double prev = 0.0, cur = wigner_start(start, mu, nu, hc, hs, T.start_norm, T.jmax);
    wig[start * chains + chain] = cur;
    for (int l = start; l < L; ++l) {
      double value;
      if (l == 0) value = cosine * cur;
      else
        value = ((2 * l + 1) * (l * (l + 1) * cosine - mu * nu) * cur -
                 s_lower[l * chains + chain] * prev) / s_upper[l * chains + chain];
      prev = cur;
      cur = value;
      wig[(l + 1) * chains + chain] = cur;
    }
  }
  __syncthreads();
  // F_l[b][p] for every kept source channel (row = starts[l] + keep + n)
  const int rows = T.starts[L] + 2 * min(L, M) + 1;
  for (int e = threadIdx.x; e < count * rows; e += blockDim.x) {
    const int k = e / rows, row = e - k * rows;
    if (!s_inside[k]) continue;
    int l = 0;
    while (l < L && T.starts[l + 1] <= row) ++l;
    const int keep = l < M ? l : M, top_p = l < A ? l : A;
    const int n = row - T.starts[l] - keep;
    const double* wig = s_pair + k * values;
    const double* cosn = wig + n_wig + 3;
    const double* sinn = cosn + M + 1;
    const double* weight = sinn + M + 1;
    float* F = g_F + ((first + k) * (int64_t)T.nch + row) * NP;
    for (int p = 0; p < NP; ++p) {
      const int mup = T.pair_mu[p];
      double f = 0.0;
      if (mup <= top_p && n <= keep) {
        const double pos = weight[2 * p], neg = weight[2 * p + 1];
        if (neg != 0.0) f += ge2_rotation(wig, l, A, M, cosn, sinn, -mup, n) * neg;
        if (pos != 0.0) f += ge2_rotation(wig, l, A, M, cosn, sinn, mup, n) * pos;
      }
      F[p] = (float)f;
    }
  }
}

// Grid (OM, point chunk); thread = (band, frequency). Partial sums per chunk.
LH_DEVICE void ge2_apply_body(const lh_ge2_table& T, const lh_ge2_problem& P, int d, int chunk,
                              int chunks, const int* g_j, const float* g_t, const double* g_r,
                              const float* g_scale, const float* g_F, double2* partial) {
  extern __shared__ float s_F[];  // [kGe2Chunk][nch*NP] for the chunk's points
  const int c0 = chunk * kGe2Chunk;
  const int c1 = min(P.n_points, c0 + kGe2Chunk);
  const int NP = T.n_pairs, nch = T.nch, Wn = P.n_omega;
  const int64_t total = (int64_t)P.n_om * P.n_points;
  const int64_t base = (int64_t)d * P.n_points;
  const int fsz = nch * NP;
  for (int i = threadIdx.x; i < (c1 - c0) * fsz; i += blockDim.x)
    s_F[i] = g_F[(base + c0) * fsz + i];
  __syncthreads();
  const int items = T.n_bands * Wn;
  if (2 * items <= (int)blockDim.x) {
    // few (band, frequency) items (zero-frequency applies): one thread per
    // (point, item), the chunk's point values summed in point order
    float2* s_val = reinterpret_cast<float2*>(s_F + kGe2Chunk * fsz);  // [point][item]
    const int n = c1 - c0;
    for (int k = threadIdx.x; k < n * items; k += blockDim.x) {
      const int u = k / items, item = k - u * items;
      const int lam = item / Wn, w = item % Wn;
      const int64_t idx = base + c0 + u;
      const int j = g_j[idx];
      float2 value = make_float2(0.f, 0.f);
      if (j >= 0) {
        const float t = g_t[idx];
        const float* F = s_F + u * fsz;
        const float2* ch = reinterpret_cast<const float2*>(P.channels) +
                           (((int64_t)lam * P.n_points + c0 + u) * nch) * P.n_omega_channels;
        float pr = 0.f, pi = 0.f;
        for (int l = 0; l <= T.degree; ++l) {
          float rr[8], ri[8];
          const float2* cf = reinterpret_cast<const float2*>(T.coef) +
                             ((((int64_t)lam * T.n_intervals + j) * (T.degree + 1) + l) * NP * 4) *
                                 T.n_omega + w;
          for (int p = 0; p < NP; ++p) {
            const float2 k0 = cf[(p * 4 + 0) * T.n_omega], k1 = cf[(p * 4 + 1) * T.n_omega];
            const float2 k2 = cf[(p * 4 + 2) * T.n_omega], k3 = cf[(p * 4 + 3) * T.n_omega];
            rr[p] = fmaf(fmaf(fmaf(k0.x, t, k1.x), t, k2.x), t, k3.x);
            ri[p] = fmaf(fmaf(fmaf(k0.y, t, k1.y), t, k2.y), t, k3.y);
          }
          const int keep = l < T.max_m ? l : T.max_m;
          for (int row = T.starts[l]; row < T.starts[l] + 2 * keep + 1; ++row) {
            float gr = 0.f, gi = 0.f;
            for (int p = 0; p < NP; ++p) {
              const float f = F[row * NP + p];
              gr = fmaf(f, rr[p], gr);
              gi = fmaf(f, ri[p], gi);
            }
            const float2 x = ch[row * P.n_omega_channels + w];
            pr += x.x * gr - x.y * gi;
            pi += x.x * gi + x.y * gr;
          }
        }
        const float sc = g_scale[(int64_t)lam * total + idx];
        float sv = 0.f, cv = 1.f;
        if (T.flight) {
          const double turns = T.omega[w] * g_r[idx] / T.speed[lam] * (1.0 / (2 * kPi));
          sincospif(2.f * (float)(turns - rint(turns)), &sv, &cv);
        }
        value = make_float2(sc * (pr * cv - pi * sv), sc * (pr * sv + pi * cv));
      }
      s_val[u * items + item] = value;
    }
    __syncthreads();
    for (int item = threadIdx.x; item < items; item += blockDim.x) {
      const int lam = item / Wn, w = item % Wn;
      float acc_re = 0.f, acc_im = 0.f;
      for (int u = 0; u < n; ++u) {
        acc_re += s_val[u * items + item].x;
        acc_im += s_val[u * items + item].y;
      }
      partial[(((int64_t)d * chunks + chunk) * T.n_bands + lam) * Wn + w] =
          make_double2(acc_re, acc_im);
    }
    return;
  }
  for (int item = threadIdx.x; item < items; item += blockDim.x) {
    const int lam = item / Wn, w = item % Wn;
    const double om = T.omega[w];
    float acc_re = 0.f, acc_im = 0.f;
    for (int c = c0; c < c1; ++c) {
      const int64_t idx = base + c;
      const int j = g_j[idx];
      if (j < 0) continue;
      const float t = g_t[idx];
      const float* F = s_F + (c - c0) * fsz;
      const float2* ch = reinterpret_cast<const float2*>(P.channels) +
                         (((int64_t)lam * P.n_points + c) * nch) * P.n_omega_channels;
      float pr = 0.f, pi = 0.f;
      for (int l = 0; l <= T.degree; ++l) {
        // radial cubic of every pair at (lam, j, l, w)
        float rr[8], ri[8];
        const float2* cf = reinterpret_cast<const float2*>(T.coef) +
                           ((((int64_t)lam * T.n_intervals + j) * (T.degree + 1) + l) * NP * 4) *
                               T.n_omega + w;
        for (int p = 0; p < NP; ++p) {
          const float2 k0 = cf[(p * 4 + 0) * T.n_omega], k1 = cf[(p * 4 + 1) * T.n_omega];
          const float2 k2 = cf[(p * 4 + 2) * T.n_omega], k3 = cf[(p * 4 + 3) * T.n_omega];
          rr[p] = fmaf(fmaf(fmaf(k0.x, t, k1.x), t, k2.x), t, k3.x);
          ri[p] = fmaf(fmaf(fmaf(k0.y, t, k1.y), t, k2.y), t, k3.y);
        }
        const int keep = l < T.max_m ? l : T.max_m;
        for (int row = T.starts[l]; row < T.starts[l] + 2 * keep + 1; ++row) {
          float gr = 0.f, gi = 0.f;
          for (int p = 0; p < NP; ++p) {
            const float f = F[row * NP + p];
            gr = fmaf(f, rr[p], gr);
            gi = fmaf(f, ri[p], gi);
          }
          const float2 x = ch[row * P.n_omega_channels + w];
          pr += x.x * gr - x.y * gi;
          pi += x.x * gi + x.y * gr;
        }
      }
      // band scale and flight phase e^{i w r / v}
      const float sc = g_scale[(int64_t)lam * total + idx];
      float sv = 0.f, cv = 1.f;
      if (T.flight) {
        const double turns = om * g_r[idx] / T.speed[lam] * (1.0 / (2 * kPi));
        sincospif(2.f * (float)(turns - rint(turns)), &sv, &cv);
      }
      acc_re += sc * (pr * cv - pi * sv);
      acc_im += sc * (pr * sv + pi * cv);
    }
    partial[(((int64_t)d * chunks + chunk) * T.n_bands + lam) * Wn + w] =
        make_double2(acc_re, acc_im);
  }
}

// result[d][w] = e^{i w ref} * sum over chunks and bands, fixed order.
LH_DEVICE void ge2_reduce_body(const lh_ge2_table& T, const lh_ge2_problem& P, int64_t idx,
                               int chunks, const double2* partial) {
  const int Wn = P.n_omega;
  if (idx >= (int64_t)P.n_om * Wn) return;
  const int d = (int)(idx / Wn), w = (int)(idx % Wn);
  double re = 0.0, im = 0.0;
  for (int ch = 0; ch < chunks; ++ch)
    for (int lam = 0; lam < T.n_bands; ++lam) {
      const double2 v = partial[(((int64_t)d * chunks + ch) * T.n_bands + lam) * Wn + w];
      re += v.x;
      im += v.y;
    }
  const double ang = T.omega[w] * P.reference_ns;
  const double c = cos(ang), s = sin(ang);
  P.result[2 * idx] = re * c - im * s;
  P.result[2 * idx + 1] = re * s + im * c;
}

// One problem: grids over its own sizes.
__global__ void ge2_geometry_kernel(lh_ge2_table T, lh_ge2_problem P, int* g_j, float* g_t,
                                    double* g_r, float* g_scale, float* g_F) {
  ge2_geometry_body(T, P, blockIdx.x, g_j, g_t, g_r, g_scale,
                    g_F);
}

__global__ void __launch_bounds__(256, 4)
ge2_apply_kernel(lh_ge2_table T, lh_ge2_problem P, const int* g_j,
                                 const float* g_t, const double* g_r, const float* g_scale,
                                 const float* g_F, double2* partial) {
  ge2_apply_body(T, P, blockIdx.x, blockIdx.y, gridDim.y, g_j, g_t, g_r, g_scale, g_F, partial);
}

__global__ void ge2_reduce_kernel(lh_ge2_table T, lh_ge2_problem P, int chunks,
                                  const double2* partial) {
  ge2_reduce_body(T, P, blockIdx.x * (int64_t)blockDim.x + threadIdx.x, chunks, partial);
}

// Many problems (events) in one launch: blockIdx.z (or .y) selects the problem,
// whose workspace regions start at its pair / partial offsets.
struct Ge2Slot {
  lh_ge2_problem P;
  int64_t pair_offset;     // sum of n_om * n_points of the earlier problems
  int64_t partial_offset;  // sum of n_om * chunks * n_bands * n_omega of the earlier problems
  int32_t chunks;
};

struct Ge2Arrays {
  int* g_j;
  float* g_t;
  double* g_r;
  float* g_scale;  // [problem][band][pairs]
  float* g_F;
  double2* partial;
};

__global__ void ge2_geometry_batch_kernel(lh_ge2_table T, const Ge2Slot* slots, Ge2Arrays A) {
  const Ge2Slot& S = slots[blockIdx.y];
  const int64_t o = S.pair_offset;
  ge2_geometry_body(T, S.P, blockIdx.x, A.g_j + o, A.g_t + o,
                    A.g_r + o, A.g_scale + o * T.n_bands, A.g_F + o * T.nch * T.n_pairs);
}

__global__ void __launch_bounds__(256, 4)
ge2_apply_batch_kernel(lh_ge2_table T, const Ge2Slot* slots, Ge2Arrays A) {
  const Ge2Slot& S = slots[blockIdx.z];
  if ((int)blockIdx.x >= S.P.n_om || (int)blockIdx.y >= S.chunks) return;
  const int64_t o = S.pair_offset;
  ge2_apply_body(T, S.P, blockIdx.x, blockIdx.y, S.chunks, A.g_j + o, A.g_t + o, A.g_r + o,
                 A.g_scale + o * T.n_bands, A.g_F + o * T.nch * T.n_pairs,
                 A.partial + S.partial_offset);
}

__global__ void ge2_reduce_batch_kernel(lh_ge2_table T, const Ge2Slot* slots, Ge2Arrays A) {
  const Ge2Slot& S = slots[blockIdx.y];
  ge2_reduce_body(T, S.P, blockIdx.x * (int64_t)blockDim.x + threadIdx.x, S.chunks,
                  A.partial + S.partial_offset);
}

int ge2_chunks(const lh_ge2_problem& P) { return (P.n_points + kGe2Chunk - 1) / kGe2Chunk; }

// Shared memory of the apply kernels (256 threads): the chunk's F rows, then
// the point values of the few-item path when a problem takes it (at most 128
// (band, frequency) items).
size_t ge2_apply_smem(const lh_ge2_table& T, int items) {
  return (size_t)kGe2Chunk * T.nch * T.n_pairs * sizeof(float) +
         (2 * items <= 256 ? (size_t)kGe2Chunk * items * sizeof(float2) : 0);
}

size_t ge2_workspace(const lh_ge2_table& T, const lh_ge2_problem& P) {
  const size_t pairs = (size_t)P.n_om * P.n_points;
  const size_t chunks = (size_t)ge2_chunks(P);
  auto up = [](size_t x) { return (x + 255) & ~size_t(255); };
  return up(pairs * 4) + up(pairs * 4) + up(pairs * 8) + up(pairs * T.n_bands * 4) +
         up(pairs * T.nch * T.n_pairs * 4) +
         up((size_t)P.n_om * chunks * T.n_bands * P.n_omega * sizeof(double2));
}

int ge2_launch(const lh_ge2_table& T, const lh_ge2_problem& P, void* ws, cudaStream_t s) {
  const size_t pairs = (size_t)P.n_om * P.n_points;
  auto up = [](size_t x) { return (x + 255) & ~size_t(255); };
  uint8_t* p = static_cast<uint8_t*>(ws);
  int* g_j = reinterpret_cast<int*>(p); p += up(pairs * 4);
  float* g_t = reinterpret_cast<float*>(p); p += up(pairs * 4);
  double* g_r = reinterpret_cast<double*>(p); p += up(pairs * 8);
  float* g_scale = reinterpret_cast<float*>(p); p += up(pairs * T.n_bands * 4);
  float* g_F = reinterpret_cast<float*>(p); p += up(pairs * T.nch * T.n_pairs * 4);
  double2* partial = reinterpret_cast<double2*>(p);
  ge2_geometry_kernel<<<ge2_geo_blocks(T, (int64_t)pairs), kGe2GeoThreads, ge2_geo_smem(T), s>>>(T, P, g_j, g_t, g_r, g_scale, g_F);
  const int chunks = ge2_chunks(P);
  const size_t smem = ge2_apply_smem(T, T.n_bands * P.n_omega);
  if (smem > 48 * 1024)
    cudaFuncSetAttribute(ge2_apply_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  ge2_apply_kernel<<<dim3(P.n_om, chunks), 256, smem, s>>>(T, P, g_j, g_t, g_r, g_scale, g_F,
                                                            partial);
  const int64_t outs = (int64_t)P.n_om * P.n_omega;
  ge2_reduce_kernel<<<(unsigned)((outs + 255) / 256), 256, 0, s>>>(T, P, chunks, partial);
  return cudaGetLastError() == cudaSuccess ? LH_OK : LH_ECUDA;
}

size_t ge2_slot_size() { return sizeof(Ge2Slot); }

size_t ge2_batch_workspace(const lh_ge2_table& T, const lh_ge2_problem* P, int32_t n) {
  size_t pairs = 0, partial = 0;
  for (int i = 0; i < n; ++i) {
    pairs += (size_t)P[i].n_om * P[i].n_points;
    partial += (size_t)P[i].n_om * ge2_chunks(P[i]) * T.n_bands * P[i].n_omega;
  }
  auto up = [](size_t x) { return (x + 255) & ~size_t(255); };
  return up(sizeof(Ge2Slot) * (size_t)n) + up(pairs * 4) + up(pairs * 4) + up(pairs * 8) +
         up(pairs * T.n_bands * 4) + up(pairs * T.nch * T.n_pairs * 4) +
         up(partial * sizeof(double2));
}

// The slot table is staged in `host_slots` (caller memory, pinned when the call
// should not wait) and copied to the workspace on the stream.
int ge2_batch_launch(const lh_ge2_table& T, const lh_ge2_problem* P, int32_t n, void* ws,
                     void* host_slots, cudaStream_t s) {
  auto up = [](size_t x) { return (x + 255) & ~size_t(255); };
  Ge2Slot* hs = static_cast<Ge2Slot*>(host_slots);
  size_t pairs = 0, partial = 0;
  int max_om = 0, max_chunks = 0;
  int64_t max_pairs = 0, max_outs = 0;
  for (int i = 0; i < n; ++i) {
    hs[i].P = P[i];
    hs[i].pair_offset = (int64_t)pairs;
    hs[i].partial_offset = (int64_t)partial;
    hs[i].chunks = ge2_chunks(P[i]);
    const int64_t pp = (int64_t)P[i].n_om * P[i].n_points;
    pairs += pp;
    partial += (size_t)P[i].n_om * hs[i].chunks * T.n_bands * P[i].n_omega;
    max_om = std::max(max_om, P[i].n_om);
    max_chunks = std::max(max_chunks, hs[i].chunks);
    max_pairs = std::max(max_pairs, pp);
    max_outs = std::max(max_outs, (int64_t)P[i].n_om * P[i].n_omega);
  }
  uint8_t* p = static_cast<uint8_t*>(ws);
  Ge2Slot* slots = reinterpret_cast<Ge2Slot*>(p); p += up(sizeof(Ge2Slot) * (size_t)n);
  Ge2Arrays A;
  A.g_j = reinterpret_cast<int*>(p); p += up(pairs * 4);
  A.g_t = reinterpret_cast<float*>(p); p += up(pairs * 4);
  A.g_r = reinterpret_cast<double*>(p); p += up(pairs * 8);
  A.g_scale = reinterpret_cast<float*>(p); p += up(pairs * T.n_bands * 4);
  A.g_F = reinterpret_cast<float*>(p); p += up(pairs * T.nch * T.n_pairs * 4);
  A.partial = reinterpret_cast<double2*>(p);
  if (cudaMemcpyAsync(slots, hs, sizeof(Ge2Slot) * (size_t)n, cudaMemcpyHostToDevice, s) !=
      cudaSuccess)
    return LH_ECUDA;
  if (max_outs == 0) return LH_OK;
  if (max_pairs > 0) {  // problems without points reduce nothing: their results are zero
    ge2_geometry_batch_kernel<<<dim3(ge2_geo_blocks(T, max_pairs), n), kGe2GeoThreads,
                                ge2_geo_smem(T), s>>>(T, slots, A);
    size_t smem = 0;
    for (int i = 0; i < n; ++i) smem = std::max(smem, ge2_apply_smem(T, T.n_bands * P[i].n_omega));
    if (smem > 48 * 1024)
      cudaFuncSetAttribute(ge2_apply_batch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)smem);
    {
      lh::TimedLaunch timed_launch(LH_KT_GE2_APPLY, s);
      ge2_apply_batch_kernel<<<dim3(max_om, max_chunks, n), 256, smem, s>>>(T, slots, A);
    }
  }
  ge2_reduce_batch_kernel<<<dim3((unsigned)((max_outs + 255) / 256), n), 256, 0, s>>>(T, slots, A);
  return cudaGetLastError() == cudaSuccess ? LH_OK : LH_ECUDA;
}


// ------------------------------------------------------------------ tensor cores
// The contraction on tcgen05 (BF16 operands, FP32 accumulation in TMEM). In
// the split mode every operand is the sum of three BF16 parts (hi + mid + lo,
// 24 significant bits, as float32) and six products are accumulated: hi hi,
// hi mid, mid hi, hi lo, lo hi, mid mid (the rest lie below float32's
// rounding); the single mode multiplies the hi parts.
//
// For interval j and kernel degree l the band-folded coefficients form a real
// matrix A_jl[(band, w, part)][(pair p, power q)] (part: real or imaginary
// coefficient; K = 4 x pairs <= 32), and a (OM, point) pair of interval j
// forms B[(channel row r of degree l)][(p, q)] = F[r][p] t^(3 - q). The
// product X = A_jl B^T holds, for every source channel row of the pair and
// every (band, w), the row's F contracted with the cubic radial kernels. The
// epilogue multiplies each X entry by the row's source channel (complex, per
// band and frequency) and sums rows and degrees in registers; then the pair's
// band scale and flight phase give its spectrum, written per pair and summed
// over points by ge2_tc_reduce_kernel in a fixed order.
//
// Layout: M = (band, w) rows in H <= 2 halves of 128 TMEM lanes, each half as
// a real and an imaginary accumulator; N = channel row x pair columns
// (column r * P + i for pair i of a group of P pairs). Pairs are bucketed by
// interval (counting sort); a CTA takes work items (tile of up to three groups
// of one interval, half) and runs them as a pipeline of warp roles:
//   MMA       one warp bulk-copies each degree's coefficients of the half into a
//             ring of kTcAStages stages (48 KB each with three BF16 parts) and
//             issues the products of (degree, group) into a ring of kTcSlots
//             TMEM slots (real and imaginary accumulator, 2 x kTcCols columns);
//   builders  form the B tile of (degree, group) from F and t, three parts, in
//             a ring of kTcBStages tiles;
//   epilogue  four warps (TMEM lane quarters) per group multiply its columns by
//             the channels and keep its pairs' sums in registers across the
//             degrees.
// So the MMAs of one (degree, group), 24 of N = 80, run while others are drained
// and the next coefficients arrive. Measured on 61k pairs (8 showers x 48 OMs,
// degree 8): 0.77 ms against 2.83 ms for a CTA that built, multiplied and drained
// sub-tiles of 8 pairs one after another (two such CTAs per SM: issue 26 %,
// long-scoreboard 7.7 per issue). What bounds it: the epilogue alone takes 0.56 ms
// (its channel loads 0.2 ms of that), the MMAs and their hand-over 0.5 ms (~50
// cycles per MMA whatever its N, as each reads 4 KB of A from shared memory), the
// pipeline without either 0.33 ms. Twenty warps of 96 registers (four groups) spilled in
// the epilogue's row loop and took 1.1 ms; both halves in one CTA read twice the
// coefficients (432 KB per work item now) and took 1.3 ms.
constexpr int kTcK = 32;                                  // K columns (pairs x 4 <= 32)
constexpr uint32_t kTcTileBytes = 128u * kTcK * 2u;       // one 128 x 32 BF16 operand tile
constexpr int kTcParts = 3;                               // BF16 parts of a split operand
constexpr int kTcCols = 80;         // columns of an accumulator: rows x pairs, padded to 16
constexpr int kTcSlots = 3;         // TMEM slots of 2 x kTcCols columns (480 of 512)
constexpr int kTcAStages = 3;
constexpr int kTcBStages = 4;
constexpr int kTcGroups = 3;                  // most pair groups per tile
constexpr int kTcEpiWarps = 4 * kTcGroups;    // one warp per group and lane quarter
constexpr int kTcBuildWarps = 3;
constexpr int kTcThreads = 32 * (kTcEpiWarps + kTcBuildWarps + 1);  // 16 warps: 128 registers each
constexpr size_t kTcSmem = 227 * 1024;        // most shared memory of a CTA

// One (OM, point) pair in range.
struct __align__(16) Ge2TcEntry {
  const char* rows;      // the point's channel block: band 0, row 0, w 0
  int64_t band_bytes;    // between bands
  int32_t pair;          // global pair id
  float t;               // offset in the interval
  int32_t pad[2];
};

struct Ge2TcArgs {
  Ge2Arrays A;
  const uint8_t* packed;        // [interval][degree] blocks: [hi, lo][half][re, im] tiles
  const Ge2TcEntry* entries;    // the pairs in range, bucketed by interval
  const int4* tiles;            // interval, first entry, pairs, groups
  const int32_t* n_tiles;
  float2* partial;              // [global pair][band * n_omega + w]
  int32_t* status;
  int passes;                   // 6 split-BF16, 1 BF16
  int halves;                   // H: ceil(bands x omega / 128)
  size_t row_bytes;             // between channel rows, the same in every problem
};

size_t ge2_tc_smem_bytes(int pairs, int n_bands, int parts);

// Shared memory of ge2_tc_tiles_kernel: the starts of the intervals' pairs and tiles.
static size_t ge2_tc_tiles_smem(int n_intervals) {
  return sizeof(int32_t) * 2 * ((size_t)n_intervals + 1);
}

// Whether a table takes the tensor-core path; `pairs` per group: 16 where the
// widest degree's rows x 16 fit an accumulator's columns, else 8 (up to 9 rows).
// The rings and the table of the pairs' channels, 8 bytes per pair and band, have to
// fit shared memory (up to 60 bands with 16 pairs, 121 with 8), and so do the starts
// of the intervals (up to 29000); other tables take the CUDA cores.
bool ge2_tc_supported(const lh_ge2_table& T, int& halves, int& pairs) {
  const int M = T.n_bands * T.n_omega;
  const int rows_max = 2 * std::min(T.degree, T.max_m) + 1;
  halves = (M + 127) / 128;
  pairs = rows_max * 16 <= kTcCols ? 16 : 8;
  return M <= 256 && 4 * T.n_pairs <= kTcK && ((rows_max * pairs + 15) & ~15) <= kTcCols &&
         ge2_tc_smem_bytes(pairs, T.n_bands, kTcParts) <= kTcSmem &&
         ge2_tc_tiles_smem(T.n_intervals) <= kTcSmem - 64;  // one static int beside it
}

size_t ge2_tc_block_bytes(const lh_ge2_table& T, int halves) {
  (void)T;
  return (size_t)kTcParts * halves * 2 * kTcTileBytes;
}

// x = hi + mid + lo, each BF16 (24 significant bits together).
LH_DEVICE void split3_bf16(float x, __nv_bfloat16& hi, __nv_bfloat16& mid, __nv_bfloat16& lo) {
  hi = __float2bfloat16_rn(x);
  const float r = x - __bfloat162float(hi);
  mid = __float2bfloat16_rn(r);
  lo = __float2bfloat16_rn(r - __bfloat162float(mid));
}

// Two values' parts, packed (the first in the low half): split3_bf16 of each.
LH_DEVICE void split3_bf16x2(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  auto pack = [](float x, float y) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(x, y);
    return *reinterpret_cast<const uint32_t*>(&v);
  };
  auto low = [](uint32_t v) { return __uint_as_float(v << 16); };
  auto high = [](uint32_t v) { return __uint_as_float(v & 0xffff0000u); };
  hi = pack(a, b);
  a -= low(hi);
  b -= high(hi);
  mid = pack(a, b);
  lo = pack(a - low(mid), b - high(mid));
}

// Packs the folded coefficients into the operand tiles (no swizzle, K-major
// 8 x 16-byte core matrices), hi, mid and lo parts.
__global__ void ge2_tc_pack_kernel(const lh_ge2_table T, int halves, __nv_bfloat16* out) {
  const int L1 = T.degree + 1, W = T.n_omega, M = T.n_bands * W;
  const int64_t per_block = (int64_t)halves * 2 * 128 * kTcK;
  const int64_t total = (int64_t)T.n_intervals * L1 * per_block;
  const int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (idx >= total) return;
  const int k = (int)(idx % kTcK);
  const int m = (int)((idx / kTcK) % 128);
  const int part = (int)((idx / (kTcK * 128)) % 2);
  const int h = (int)((idx / (kTcK * 256)) % halves);
  const int64_t jl = idx / per_block;
  const int l = (int)(jl % L1), j = (int)(jl / L1);
  const int flat = h * 128 + m;
  float v = 0.f;
  if (flat < M && k < 4 * T.n_pairs) {
    const int lam = flat / W, w = flat % W, pp = k >> 2, q = k & 3;
    const float2 c = reinterpret_cast<const float2*>(T.coef)
        [((((int64_t)lam * T.n_intervals + j) * L1 + l) * T.n_pairs * 4 + pp * 4 + q) * W + w];
    v = part ? c.y : c.x;
  }
  __nv_bfloat16 hi, mid, lo;
  split3_bf16(v, hi, mid, lo);
  const int64_t tile = (int64_t)(h * 2 + part) * 128 * kTcK;
  const int64_t at = jl * kTcParts * per_block + tile + tile_offset(m, k);
  out[at] = hi;
  out[at + per_block] = mid;
  out[at + 2 * per_block] = lo;
}

// Bucket pass 1 and 3 over every pair of every problem, points outermost so
// that a bucket lists the OMs of one point together: count per interval, then
// place (warp-aggregated atomics).
__global__ void ge2_tc_bucket_kernel(const Ge2Slot* slots, Ge2Arrays A, int nch, int32_t* counts,
                                     Ge2TcEntry* entries) {
  const Ge2Slot& S = slots[blockIdx.y];
  const int64_t total = (int64_t)S.P.n_om * S.P.n_points;
  const int64_t rounded = (total + 31) & ~(int64_t)31;
  const int lane = threadIdx.x & 31;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < rounded;
       t += (int64_t)gridDim.x * blockDim.x) {
    int j = -1;
    int64_t idx = 0, c = 0;
    if (t < total) {
      c = t / S.P.n_om;
      idx = (t - c * S.P.n_om) * S.P.n_points + c;
      j = A.g_j[S.pair_offset + idx];
    }
    const unsigned peers = __match_any_sync(0xffffffffu, j);
    const int leader = __ffs(peers) - 1;
    int base = 0;
    if (lane == leader && j >= 0) base = atomicAdd(counts + j, __popc(peers));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (entries && j >= 0) {
      Ge2TcEntry e;
      const int64_t point_bytes = (int64_t)nch * S.P.n_omega_channels * (int64_t)sizeof(float2);
      e.rows = reinterpret_cast<const char*>(S.P.channels) + c * point_bytes;
      e.band_bytes = S.P.n_points * point_bytes;
      e.pair = (int32_t)(S.pair_offset + idx);
      e.t = A.g_t[S.pair_offset + idx];
      e.pad[0] = e.pad[1] = 0;
      entries[base + __popc(peers & ((1u << lane) - 1u))] = e;
    }
  }
}

// One CTA: the fill cursors (bucket starts) and the tiles. A tile takes as many
// groups as still leave every SM two work items (tile, half): more groups share
// their coefficients, fewer spread a small problem over the SMs.
__global__ void __launch_bounds__(256)
ge2_tc_tiles_kernel(int n_intervals, int group_pairs, int halves, int32_t* counts, int4* tiles,
                    int32_t* n_tiles, unsigned long long* units) {
  extern __shared__ int32_t s_scan[];  // [n_intervals + 1] bucket starts, then tile starts
  int32_t* s_start = s_scan;
  int32_t* s_tile = s_scan + n_intervals + 1;
  __shared__ int s_per;
  for (int j = threadIdx.x; j < n_intervals; j += blockDim.x) s_start[j + 1] = counts[j];
  __syncthreads();
  if (threadIdx.x == 0) {
    int32_t at = 0, tile = 0;
    for (int j = 0; j < n_intervals; ++j) {
      const int32_t c = s_start[j + 1];
      s_start[j] = at;
      at += c;
    }
    s_start[n_intervals] = at;
    int per = kTcGroups * group_pairs;
    while (per > group_pairs && (int64_t)at * halves < 2 * 148 * (int64_t)per) per -= group_pairs;
    for (int j = 0; j < n_intervals; ++j) {
      s_tile[j] = tile;
      tile += (s_start[j + 1] - s_start[j] + per - 1) / per;
    }
    s_tile[n_intervals] = tile;
    s_per = per;
    *n_tiles = tile;
    if (units) atomicAdd(units, (unsigned long long)at);  // (OM, point) pairs in range
  }
  __syncthreads();
  const int per = s_per;
  for (int j = threadIdx.x; j < n_intervals; j += blockDim.x) counts[j] = s_start[j];
  for (int k = threadIdx.x; k < s_tile[n_intervals]; k += blockDim.x) {
    int lo = 0, hi = n_intervals;  // the bucket: last j with s_tile[j] <= k
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (s_tile[mid] <= k) lo = mid; else hi = mid;
    }
    const int first = s_start[lo] + (k - s_tile[lo]) * per;
    const int count = min(per, s_start[lo + 1] - first);
    tiles[k] = make_int4(lo, first, count, (count + group_pairs - 1) / group_pairs);
  }
}

// A work item: half h of a tile, the tile's interval and its entries (the same on
// every caller).
struct Ge2TcTile {
  int h, j, first, count, groups;
};

LH_DEVICE Ge2TcTile ge2_tc_tile(const Ge2TcArgs& G, int item) {
  const int tile = item / G.halves;
  const int4 v = __ldg(G.tiles + tile);
  return Ge2TcTile{item - tile * G.halves, v.x, v.y, v.z, v.w};
}

constexpr uint32_t kTcLboA = 128u * 16u, kTcLboB = (uint32_t)kTcCols * 16u;

// The products of one step, the real and the imaginary accumulator in turn (two
// chains of dependent MMAs instead of one). Descriptors of the parts and K steps
// are the stage's plus constants (addresses in 16-byte units).
template <int kPasses>
LH_DEVICE void ge2_tc_issue(uint32_t d, uint64_t da0, uint64_t db0, uint32_t idesc) {
  // (A part, B part) of each product of the split mode, largest first
  constexpr int pass_a[6] = {0, 0, 1, 0, 2, 1}, pass_b[6] = {0, 1, 0, 2, 0, 1};
#pragma unroll
  for (int pass = 0; pass < kPasses; ++pass)
#pragma unroll
    for (int kk = 0; kk < kTcK / 16; ++kk)
#pragma unroll
      for (int part = 0; part < 2; ++part) {
        const uint64_t da = da0 + (uint64_t)(((pass_a[pass] * 2 + part) * kTcTileBytes +
                                              kk * 2 * kTcLboA) >> 4);
        const uint64_t db = db0 + (uint64_t)((pass_b[pass] * kTcCols * kTcK * 2 +
                                              kk * 2 * kTcLboB) >> 4);
        tc_mma_bf16(d + (uint32_t)(part * kTcCols), da, db, idesc, pass + kk ? 1u : 0u);
      }
}

// One lane of a converged warp (always the same one).
LH_DEVICE bool elect_one() {
  uint32_t mine;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(mine));
  return mine != 0;
}

struct Ge2TcBars {
  uint64_t a_full[kTcAStages], a_empty[kTcAStages];
  uint64_t b_full[kTcBStages], b_empty[kTcBStages];
  // per group, for even and odd steps: its columns are in TMEM / have been read.
  // At most two steps of a group are in flight, so a parity names the phase.
  uint64_t t_full[kTcGroups][2], t_empty[kTcGroups][2];
  uint64_t drain;
};

// P pairs per group; Offset holds the byte offsets in a point's channel block (64-bit
// ones take 1 % longer: 0.778 against 0.770 ms for 61k pairs). Each role walks the same
// sequence of (work item, degree, group) and counts its stages itself; a wait that runs
// into its time limit ends that role, and the roles waiting for it then end the same way.
template <int P, typename Offset>
__global__ void __launch_bounds__(kTcThreads, 1)
ge2_tc_kernel(const lh_ge2_table T, const Ge2TcArgs G) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const int H = G.halves;
  const int parts = G.passes > 1 ? kTcParts : 1;
  const uint32_t a_bytes = (uint32_t)parts * 2u * kTcTileBytes;  // one half's coefficients
  constexpr int kBElems = kTcCols * kTcK;
  const uint32_t b_bytes = (uint32_t)parts * kBElems * 2u;
  uint8_t* s_a = smem;
  uint8_t* s_b = s_a + kTcAStages * a_bytes;
  // each pair's channel block per band: [group][band][pair]
  const char** s_ch = reinterpret_cast<const char**>(s_b + kTcBStages * b_bytes);
  Ge2TcBars* bars = reinterpret_cast<Ge2TcBars*>(s_ch + kTcGroups * P * T.n_bands);
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(bars + 1);

  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  if (tid == 0) {
    for (int i = 0; i < kTcAStages; ++i) mbar_init(bars->a_full + i, 1), mbar_init(bars->a_empty + i, 1);
    for (int i = 0; i < kTcBStages; ++i)
      mbar_init(bars->b_full + i, kTcBuildWarps), mbar_init(bars->b_empty + i, 1);
    for (int i = 0; i < 2 * kTcGroups; ++i)
      mbar_init(&bars->t_full[0][0] + i, 1), mbar_init(&bars->t_empty[0][0] + i, 4);
    mbar_init(&bars->drain, 1);
    fence_barrier_init();
  }
  if (warp == 0) {
    tmem_alloc(s_tmem, 512);
    tmem_relinquish();
  }
  // K columns past 4 n_pairs stay zero in every B tile
  for (int e = tid; e < kTcBStages * (int)b_bytes / 16; e += kTcThreads)
    reinterpret_cast<uint4*>(s_b)[e] = make_uint4(0u, 0u, 0u, 0u);
  fence_proxy_async();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *s_tmem;
  const int L1 = T.degree + 1, W = T.n_omega, NB = T.n_bands, M = NB * W;
  const int n_items = *G.n_tiles * H;
  bool failed = false;

  if (warp < kTcEpiWarps) {
    // ---- epilogue: group g, TMEM lanes quarter * 32 + lane
    const int quarter = warp & 3, g = warp >> 2;
    const uint32_t lane_base = tmem + ((uint32_t)(quarter * 32) << 16);
    const int rows = T.starts[T.degree] + 2 * min(T.degree, T.max_m) + 1;  // over all degrees
    const char** table = s_ch + g * P * NB;
    uint32_t before = 0;  // (degree, group) steps of the items before
    uint32_t taken = 0;   // this group's steps so far
    for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
      const Ge2TcTile t = ge2_tc_tile(G, item);
      const int cnt = min(P, t.count - g * P);
      if (cnt > 0) {
        const int m0 = t.h * 128 + quarter * 32, m = m0 + lane;
        const bool m_ok = m < M;
        const bool reads = m0 < M;  // warps without a row read no TMEM
        const int lam = m_ok ? m / W : 0, wq = m_ok ? m % W : 0;
        // the table of the item before has been read; a wait that gave up ends
        // all four warps here
        if (group_sync_or<128>(g, failed)) { failed = true; break; }
        for (int e = quarter * 32 + lane; e < P * NB; e += 128) {
          // places past the last pair repeat the first: computed, not written
          const int band = e / P, i = e - band * P;
          const Ge2TcEntry& q = G.entries[t.first + g * P + (i < cnt ? i : 0)];
          table[e] = q.rows + band * q.band_bytes;
        }
        group_sync_or<128>(g, false);
        const char* const* mine = table + lam * P;
        const uint32_t wq_bytes = (uint32_t)wq * (uint32_t)sizeof(float2);
        float acc_re[P], acc_im[P];
#pragma unroll
        for (int i = 0; i < P; ++i) acc_re[i] = acc_im[i] = 0.f;
        // The rows of all degrees in order. The channels of eight pairs are loaded
        // one row ahead (two with 8 pairs per group): each of the two buffers is
        // filled again as soon as it has been used, across degrees too, so that a
        // warp keeps 8 to 16 loads in flight.
        constexpr int kRows = 16 / P;  // rows per turn of the loop: two buffers
        float2 ch[2][8];
        auto fetch = [&](float2 (&to)[8], int row, int c) {
          const Offset at = (Offset)min(row, rows - 1) * (Offset)G.row_bytes + wq_bytes;
#pragma unroll
          for (int i = 0; i < 8; ++i)
            to[i] = __ldg(reinterpret_cast<const float2*>(mine[c * 8 + i] + at));
        };
        if (reads) {
          fetch(ch[0], 0, 0);
          fetch(ch[1], P == 16 ? 0 : 1, P == 16 ? 1 : 0);
        }
        int l = 0, r = 0, nr = 1;
        uint32_t base = 0;
        for (int row0 = 0; row0 < rows && !failed; row0 += kRows) {
#pragma unroll
          for (int u = 0; u < kRows; ++u) {
            if (row0 + u >= rows || failed) continue;  // the same for the whole warp
            if (r == 0) {  // a degree's columns
              const uint32_t step = before + (uint32_t)(l * t.groups + g);
              base = lane_base + (step % kTcSlots) * 2u * kTcCols;
              if (!warp_wait(&bars->t_full[g][taken & 1u], (taken >> 1) & 1u)) {
                failed = true;
                continue;
              }
              tc_fence_after();
            }
            if (reads) {
#pragma unroll
              for (int c = 0; c < P / 8; ++c) {
                if (c * 8 >= cnt) continue;
                float2 (&x)[8] = ch[P == 16 ? c : u];
#pragma unroll
                for (int i0 = 0; i0 < 8; i0 += 4) {
                  float xr[4], xi[4];
                  tmem_ld4x2(base + (uint32_t)(r * P + c * 8 + i0),
                             base + (uint32_t)(kTcCols + r * P + c * 8 + i0), xr, xi);
#pragma unroll
                  for (int i = 0; i < 4; ++i) {
                    acc_re[c * 8 + i0 + i] += x[i0 + i].x * xr[i] - x[i0 + i].y * xi[i];
                    acc_im[c * 8 + i0 + i] += x[i0 + i].x * xi[i] + x[i0 + i].y * xr[i];
                  }
                }
                fetch(x, row0 + u + kRows, c);
              }
            }
            if (++r == nr) {
              tc_fence_before();
              __syncwarp();
              if (lane == 0) mbar_arrive(&bars->t_empty[g][taken & 1u]);
              ++taken;
              ++l;
              r = 0;
              nr = 2 * min(l, T.max_m) + 1;
            }
          }
        }
        // the pairs' sums; ge2_tc_reduce_kernel applies their scale and flight phase
        if (!failed && m_ok) {
#pragma unroll
          for (int i = 0; i < P; ++i)
            if (i < cnt)
              G.partial[(int64_t)G.entries[t.first + g * P + i].pair * M + m] =
                  make_float2(acc_re[i], acc_im[i]);
        }
      }
      before += (uint32_t)(L1 * t.groups);
    }
  } else if (warp < kTcEpiWarps + kTcBuildWarps) {
    // ---- builders: B[n = r * P + i][k = 4 p + q] = F[r][p] t^(3 - q), split in parts
    const int b0 = (warp - kTcEpiWarps) * 32;
    const int NP = T.n_pairs;
    const uint32_t inv_np = 65536u / NP + 1u;  // x / NP = x inv_np >> 16 for x < 2^16 / NP
    uint32_t seq = 0;
    for (int item = blockIdx.x; item < n_items && !failed; item += gridDim.x) {
      const Ge2TcTile t = ge2_tc_tile(G, item);
      // lane k holds pairs k and 32 + k of the tile (at most kTcGroups x P = 48)
      const Ge2TcEntry& e_lo = G.entries[t.first + min(lane, t.count - 1)];
      const Ge2TcEntry& e_hi = G.entries[t.first + min(lane + 32, t.count - 1)];
      const int id_lo = e_lo.pair, id_hi = e_hi.pair;
      const float t_lo = e_lo.t, t_hi = e_hi.t;
      for (int l = 0; l < L1 && !failed; ++l) {
        const int nr = 2 * min(l, T.max_m) + 1, row0 = T.starts[l], per = nr * NP;
        const uint32_t inv_per = 65536u / per + 1u;  // exact: P x per^2 < 2^16
        for (int g = 0; g < t.groups; ++g, ++seq) {
          const int total = min(P, t.count - g * P) * per;
          const uint32_t stage = seq % kTcBStages;
          if (!warp_wait(bars->b_empty + stage, ((seq / kTcBStages) & 1u) ^ 1u)) {
            failed = true;
            break;
          }
          uint8_t* out = s_b + stage * b_bytes;
          const bool upper = g * P >= 32;
          constexpr int kAhead = 5;  // elements whose F is on its way per thread
          for (int e0 = b0; e0 < total; e0 += 32 * kTcBuildWarps * kAhead) {
            float f[kAhead], t1[kAhead];
            int at[kAhead];
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
              const int e = e0 + u * 32 * kTcBuildWarps + lane;
              const bool ok = e < total;
              const int i = ok ? (int)(((uint32_t)e * inv_per) >> 16) : 0;
              const int rp = ok ? e - i * per : 0;
              const int r = (int)(((uint32_t)rp * inv_np) >> 16), p = rp - r * NP;
              const int src = (g * P + i) & 31;
              const int id = __shfl_sync(0xffffffffu, upper ? id_hi : id_lo, src);
              t1[u] = __shfl_sync(0xffffffffu, upper ? t_hi : t_lo, src);
              at[u] = ok ? ((p >> 1) * kTcCols + r * P + i) * 16 + (p & 1) * 8 : -1;
              f[u] = ok ? __ldg(G.A.g_F + ((int64_t)id * T.nch + row0) * NP + rp) : 0.f;
            }
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
              if (at[u] < 0) continue;
              const float t2 = t1[u] * t1[u];
              const float v[4] = {f[u] * (t2 * t1[u]), f[u] * t2, f[u] * t1[u], f[u]};
              uint2 part[kTcParts];
              split3_bf16x2(v[0], v[1], part[0].x, part[1].x, part[2].x);
              split3_bf16x2(v[2], v[3], part[0].y, part[1].y, part[2].y);
#pragma unroll
              for (int k = 0; k < kTcParts; ++k)
                if (k < parts) *reinterpret_cast<uint2*>(out + at[u] + k * kBElems * 2) = part[k];
            }
          }
          fence_proxy_async();  // generic-proxy smem writes -> visible to the tensor core
          __syncwarp();
          if (lane == 0) mbar_arrive(bars->b_full + stage);
        }
      }
    }
  } else {
    // ---- one warp loads the coefficients (one bulk copy per part) and issues the
    // MMAs: the load of stage n + 2 goes out after the MMAs of stage n, once those
    // of stage n - 1 have left its place. The whole warp walks the loops and one
    // elected lane issues, so that addresses and descriptors are uniform values
    // (tcgen05.mma takes them from uniform registers: issued from a branch of one
    // lane, each MMA took ~50 cycles of register moves whatever its N).
    const unsigned full = 0xffffffffu;
    const bool leader = elect_one();
    const uint32_t tmem_u = __shfl_sync(full, tmem, 0);
    const size_t block_bytes = (size_t)kTcParts * H * 2u * kTcTileBytes;
    int ld_item = blockIdx.x, ld_l = 0;  // the next stage to load
    const uint8_t* ld_from = nullptr;
    uint32_t loaded = 0;
    auto load_next = [&]() {
      if (ld_item >= n_items) return;
      if (ld_l == 0) {
        const Ge2TcTile t = ge2_tc_tile(G, ld_item);
        ld_from = G.packed + (size_t)t.j * L1 * block_bytes + (size_t)t.h * 2 * kTcTileBytes;
      }
      const uint32_t as = loaded % kTcAStages;
      if (!warp_wait(bars->a_empty + as, ((loaded / kTcAStages) & 1u) ^ 1u)) {
        failed = true;
        return;
      }
      if (leader) {
        mbar_expect_tx(bars->a_full + as, a_bytes);
        for (int k = 0; k < parts; ++k)
          bulk_g2s(s_a + as * a_bytes + (size_t)k * 2 * kTcTileBytes,
                   ld_from + (size_t)k * H * 2 * kTcTileBytes, 2 * kTcTileBytes,
                   bars->a_full + as);
      }
      __syncwarp();
      ++loaded;
      ld_from += block_bytes;
      if (++ld_l == L1) {
        ld_l = 0;
        ld_item += gridDim.x;
      }
    };
    for (int k = 0; k < kTcAStages - 1; ++k) load_next();
    const uint64_t desc_a = smem_desc_kmajor(s_a, kTcLboA, 128);
    const uint64_t desc_b = smem_desc_kmajor(s_b, kTcLboB, 128);
    uint32_t step = 0, a_seq = 0;
    // Steps issued and drained per group, modulo 256, one byte per group, and each
    // slot's last user and its step: packed in registers (arrays indexed at run
    // time would sit in local memory, behind an L1 that the channels stream
    // through).
    uint32_t issued = 0, drained = 0, slot_user = 0, slot_step = 0, slot_used = 0;
    auto byte_of = [](uint32_t v, int k) { return (v >> (8 * k)) & 0xffu; };
    auto set_byte = [](uint32_t v, int k, uint32_t x) {
      return (v & ~(0xffu << (8 * k))) | ((x & 0xffu) << (8 * k));
    };
    // the group's steps up to `upto` (exclusive) have been read
    auto drain_group = [&](int g, uint32_t upto) {
      uint32_t n = byte_of(drained, g);
      while ((int8_t)(upto - n) > 0) {
        if (!warp_wait(&bars->t_empty[g][n & 1u], (n >> 1) & 1u)) return false;
        n = (n + 1) & 0xffu;
      }
      drained = set_byte(drained, g, n);
      return true;
    };
    for (int item = blockIdx.x; item < n_items && !failed; item += gridDim.x) {
      const int groups = __shfl_sync(full, ge2_tc_tile(G, item).groups, 0);
      for (int l = 0; l < L1 && !failed; ++l, ++a_seq) {
        const int nr = 2 * min(l, T.max_m) + 1, n_pad = (nr * P + 15) & ~15;
        const uint32_t idesc = instr_desc_bf16_f32(128, n_pad);
        const uint32_t as = a_seq % kTcAStages;
        if (!warp_wait(bars->a_full + as, (a_seq / kTcAStages) & 1u)) { failed = true; break; }
        const uint64_t da0 = desc_a + ((as * a_bytes) >> 4);
        for (int g = 0; g < groups; ++g, ++step) {
          const uint32_t bs = step % kTcBStages, slot = step % kTcSlots;
          const uint32_t mine = byte_of(issued, g);
          // the group's step before last and the slot's last step have been read
          if (!(drain_group(g, mine - 1) &&
                (!((slot_used >> slot) & 1u) ||
                 drain_group((int)byte_of(slot_user, slot), byte_of(slot_step, slot) + 1)) &&
                warp_wait(bars->b_full + bs, (step / kTcBStages) & 1u))) {
            failed = true;
            break;
          }
          slot_used |= 1u << slot;
          slot_user = set_byte(slot_user, slot, (uint32_t)g);
          slot_step = set_byte(slot_step, slot, mine);
          tc_fence_after();
          const uint64_t db0 = desc_b + ((bs * b_bytes) >> 4);
          const uint32_t d = tmem_u + slot * 2u * kTcCols;
          if (leader) {
            if (G.passes > 1) ge2_tc_issue<6>(d, da0, db0, idesc);
            else ge2_tc_issue<1>(d, da0, db0, idesc);
            tc_commit(&bars->t_full[g][mine & 1u]);
            tc_commit(bars->b_empty + bs);
            if (g == groups - 1) tc_commit(bars->a_empty + as);
          }
          __syncwarp();
          issued = set_byte(issued, g, mine + 1);
        }
        if (!failed) load_next();
      }
    }
    // nothing in flight outlives the shared memory and the TMEM allocation:
    // copies that were never waited for (a role gave up), then the MMAs
    for (; a_seq < loaded; ++a_seq)
      warp_wait(bars->a_full + a_seq % kTcAStages, (a_seq / kTcAStages) & 1u);
    if (leader) tc_commit(&bars->drain);
    __syncwarp();
    warp_wait(&bars->drain, 0);
  }
  if (failed && lane == 0) atomicOr(reinterpret_cast<unsigned*>(G.status), LH_STATUS_TIMEOUT);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 512);
}

// result[d][w] = e^{i w ref} * sum over points and bands of s e^{i w r / v} times the
// pairs' sums (float32 each, added in float64). A CTA takes one OM and 32
// frequencies; its kTcReduceParts warps take every kTcReduceParts-th point and
// their sums are added in order, so that the result is the same alone and in a
// batch. With one thread per (OM, frequency) over all points the chains of
// loads took 190 us for 384 OMs x 160 points.
constexpr int kTcReduceParts = 16;

__global__ void __launch_bounds__(32 * kTcReduceParts)
ge2_tc_reduce_kernel(const lh_ge2_table T, const Ge2Slot* slots, Ge2Arrays A,
                     const float2* partial) {
  __shared__ double2 s_sum[kTcReduceParts][32];
  __shared__ double s_inv_speed[256];  // at most 256 (band, frequency) rows
  for (int lam = threadIdx.x; lam < T.n_bands; lam += blockDim.x)
    s_inv_speed[lam] = 1.0 / T.speed[lam];
  __syncthreads();
  const Ge2Slot& S = slots[blockIdx.y];
  const int W = S.P.n_omega, M = T.n_bands * T.n_omega;
  const int blocks_w = (W + 31) / 32;
  const int d = blockIdx.x / blocks_w;
  if (d >= S.P.n_om) return;
  const int lane = threadIdx.x & 31, part = threadIdx.x >> 5;
  const int w = (blockIdx.x - d * blocks_w) * 32 + lane;
  double re = 0.0, im = 0.0;
  if (w < W) {
    const double omega = T.omega[w];
    const int64_t pairs = (int64_t)S.P.n_om * S.P.n_points;
    for (int c = part; c < S.P.n_points; c += kTcReduceParts) {
      const int64_t idx = (int64_t)d * S.P.n_points + c, g = S.pair_offset + idx;
      if (A.g_j[g] < 0) continue;
      const double r = A.g_r[g];
      for (int lam = 0; lam < T.n_bands; ++lam) {
        const float2 v = partial[g * M + lam * T.n_omega + w];
        const float sc = A.g_scale[S.pair_offset * T.n_bands + lam * pairs + idx];
        float sv = 0.f, cv = 1.f;
        if (T.flight) {
          const double turns = omega * r * s_inv_speed[lam] * (1.0 / (2 * kPi));
          sincospif(2.f * (float)(turns - rint(turns)), &sv, &cv);
        }
        re += (double)(sc * fmaf(v.x, cv, -(v.y * sv)));
        im += (double)(sc * fmaf(v.y, cv, v.x * sv));
      }
    }
  }
  s_sum[part][lane] = make_double2(re, im);
  __syncthreads();
  if (part != 0 || w >= W) return;
  for (int k = 1; k < kTcReduceParts; ++k) {
    re += s_sum[k][lane].x;
    im += s_sum[k][lane].y;
  }
  const double ang = T.omega[w] * S.P.reference_ns;
  const double c = cos(ang), s = sin(ang);
  const int64_t idx = (int64_t)d * W + w;
  S.P.result[2 * idx] = re * c - im * s;
  S.P.result[2 * idx + 1] = re * s + im * c;
}

size_t ge2_tc_smem_bytes(int pairs, int n_bands, int parts) {
  return (size_t)kTcAStages * parts * 2 * kTcTileBytes +
         (size_t)kTcBStages * parts * kTcCols * kTcK * 2 +
         sizeof(char*) * kTcGroups * pairs * n_bands + sizeof(Ge2TcBars) + 16;
}

size_t ge2_tc_pack_bytes(const lh_ge2_table& T) {
  int halves, group_pairs;
  if (!ge2_tc_supported(T, halves, group_pairs)) return 0;
  return (size_t)T.n_intervals * (T.degree + 1) * ge2_tc_block_bytes(T, halves);
}

int ge2_tc_pack(const lh_ge2_table& T, void* packed, cudaStream_t s) {
  int halves, group_pairs;
  if (!ge2_tc_supported(T, halves, group_pairs)) return LH_EUNSUPPORTED;
  const int64_t total = (int64_t)T.n_intervals * (T.degree + 1) * halves * 2 * 128 * kTcK;
  ge2_tc_pack_kernel<<<(unsigned)((total + 255) / 256), 256, 0, s>>>(
      T, halves, static_cast<__nv_bfloat16*>(packed));
  return cudaGetLastError() == cudaSuccess ? LH_OK : LH_ECUDA;
}

// Workspace of the tensor-core batch: the batch layout of ge2_batch_workspace,
// then the bucket arrays, the pair entries and the per-pair spectra.
size_t ge2_tc_workspace(const lh_ge2_table& T, const lh_ge2_problem* P, int32_t n) {
  size_t pairs = 0;
  for (int i = 0; i < n; ++i) pairs += (size_t)P[i].n_om * P[i].n_points;
  auto up = [](size_t x) { return (x + 255) & ~size_t(255); };
  int halves, group_pairs;
  if (!ge2_tc_supported(T, halves, group_pairs)) return 0;
  return ge2_batch_workspace(T, P, n) + 2 * up(sizeof(int32_t) * (T.n_intervals + 1)) +
         up(sizeof(int4) * (pairs / group_pairs + T.n_intervals + 1)) +
         up(sizeof(Ge2TcEntry) * pairs) + up(sizeof(float2) * pairs * T.n_bands * T.n_omega);
}

// The problems whose channel rows have `stride` (n_omega_channels), with their
// slots from `first_slot` on; the number of them comes back in `count`.
static int ge2_tc_class_launch(const lh_ge2_table& T, const lh_ge2_problem* P, int32_t n,
                               int32_t stride, int32_t first_slot, int32_t& count, int passes,
                               const void* packed, void* ws, void* host_slots, int32_t* status,
                               cudaStream_t s) {
  int halves, group_pairs;
  if (!ge2_tc_supported(T, halves, group_pairs)) return LH_EUNSUPPORTED;
  auto up = [](size_t x) { return (x + 255) & ~size_t(255); };
  Ge2Slot* hs = static_cast<Ge2Slot*>(host_slots) + first_slot;
  size_t pairs = 0;
  int64_t max_pairs = 0;
  int max_om = 0;
  count = 0;
  for (int i = 0; i < n; ++i) {
    if (P[i].n_omega_channels != stride) continue;
    Ge2Slot& S = hs[count++];
    S.P = P[i];
    S.pair_offset = (int64_t)pairs;
    S.partial_offset = 0;
    S.chunks = 0;
    const int64_t pp = (int64_t)P[i].n_om * P[i].n_points;
    pairs += pp;
    max_pairs = std::max(max_pairs, pp);
    max_om = std::max(max_om, P[i].n_om);
  }
  uint8_t* p = static_cast<uint8_t*>(ws);
  Ge2Slot* slots = reinterpret_cast<Ge2Slot*>(p); p += up(sizeof(Ge2Slot) * (size_t)n);
  Ge2Arrays A;
  A.g_j = reinterpret_cast<int*>(p); p += up(pairs * 4);
  A.g_t = reinterpret_cast<float*>(p); p += up(pairs * 4);
  A.g_r = reinterpret_cast<double*>(p); p += up(pairs * 8);
  A.g_scale = reinterpret_cast<float*>(p); p += up(pairs * T.n_bands * 4);
  A.g_F = reinterpret_cast<float*>(p); p += up(pairs * T.nch * T.n_pairs * 4);
  A.partial = nullptr;
  // the CUDA-core path's chunk partials are not used here
  p = static_cast<uint8_t*>(ws) + ge2_batch_workspace(T, P, n);
  int32_t* counts = reinterpret_cast<int32_t*>(p); p += up(sizeof(int32_t) * (T.n_intervals + 1));
  int32_t* n_tiles = reinterpret_cast<int32_t*>(p); p += up(sizeof(int32_t) * (T.n_intervals + 1));
  int4* tiles = reinterpret_cast<int4*>(p);
  p += up(sizeof(int4) * (pairs / group_pairs + T.n_intervals + 1));
  Ge2TcEntry* entries = reinterpret_cast<Ge2TcEntry*>(p); p += up(sizeof(Ge2TcEntry) * pairs);
  float2* partial = reinterpret_cast<float2*>(p);
  slots += first_slot;
  if (cudaMemcpyAsync(slots, hs, sizeof(Ge2Slot) * (size_t)count, cudaMemcpyHostToDevice, s) !=
      cudaSuccess)
    return LH_ECUDA;
  if (max_om == 0) return LH_OK;
  if (max_pairs == 0) {  // no points anywhere: every result is zero
    for (int i = 0; i < count; ++i)
      cudaMemsetAsync(hs[i].P.result, 0, sizeof(double) * 2 * (size_t)hs[i].P.n_om * T.n_omega, s);
    return cudaGetLastError() == cudaSuccess ? LH_OK : LH_ECUDA;
  }
  ge2_geometry_batch_kernel<<<dim3(ge2_geo_blocks(T, max_pairs), count), kGe2GeoThreads,
                              ge2_geo_smem(T), s>>>(T, slots, A);
  cudaMemsetAsync(counts, 0, sizeof(int32_t) * (T.n_intervals + 1), s);
  const unsigned bucket_blocks = (unsigned)std::min<int64_t>((max_pairs + 255) / 256, 148 * 4);
  ge2_tc_bucket_kernel<<<dim3(bucket_blocks, count), 256, 0, s>>>(slots, A, T.nch, counts, nullptr);
  const size_t tiles_smem = ge2_tc_tiles_smem(T.n_intervals);
  if (tiles_smem > 47 * 1024 &&  // a static int lies beside it
      cudaFuncSetAttribute(ge2_tc_tiles_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)tiles_smem) != cudaSuccess)
    return LH_ECUDA;
  ge2_tc_tiles_kernel<<<1, 256, tiles_smem, s>>>(
      T.n_intervals, group_pairs, halves, counts, tiles, n_tiles,
      kernel_units() ? kernel_units() + LH_KT_GE2_TC : nullptr);
  ge2_tc_bucket_kernel<<<dim3(bucket_blocks, count), 256, 0, s>>>(slots, A, T.nch, counts, entries);
  Ge2TcArgs G;
  G.A = A;
  G.packed = static_cast<const uint8_t*>(packed);
  G.entries = entries;
  G.tiles = tiles;
  G.n_tiles = n_tiles;
  G.row_bytes = (size_t)stride * sizeof(float2);
  G.partial = partial;
  G.status = status;
  G.passes = passes;
  G.halves = halves;
  const size_t smem = ge2_tc_smem_bytes(group_pairs, T.n_bands, passes > 1 ? kTcParts : 1);
  // rows too far apart for 32-bit offsets (channels cut from far wider buffers)
  const bool wide = T.nch * G.row_bytes > UINT32_MAX;
  auto* kernel = group_pairs == 16
                     ? (wide ? ge2_tc_kernel<16, uint64_t> : ge2_tc_kernel<16, uint32_t>)
                     : (wide ? ge2_tc_kernel<8, uint64_t> : ge2_tc_kernel<8, uint32_t>);
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
      cudaSuccess)
    return LH_ECUDA;
  // persistent CTAs, one per SM; work items beyond the grid are taken in turn
  const int64_t item_bound = ((int64_t)(pairs + group_pairs - 1) / group_pairs + T.n_intervals) * halves;
  const unsigned grid = (unsigned)std::max<int64_t>(1, std::min<int64_t>(item_bound, 148));
  {
    lh::TimedLaunch timed_launch(LH_KT_GE2_TC, s);
    kernel<<<grid, kTcThreads, smem, s>>>(T, G);
  }
  ge2_tc_reduce_kernel<<<dim3((unsigned)(max_om * ((T.n_omega + 31) / 32)), count),
                         32 * kTcReduceParts, 0, s>>>(T, slots, A, partial);
  return cudaGetLastError() == cudaSuccess ? LH_OK : LH_ECUDA;
}

// The epilogue takes one channel row stride per launch (the route's problems all
// have the table's): problems of other strides follow in launches of their own
// over the same workspace, each class with its own slots.
int ge2_tc_batch_launch(const lh_ge2_table& T, const lh_ge2_problem* P, int32_t n, int passes,
                        const void* packed, void* ws, void* host_slots, int32_t* status,
                        cudaStream_t s) {
  for (int i = 0; i < n; ++i)
    if (P[i].n_omega != T.n_omega) return LH_EINVAL;  // full spectra only
  int32_t done = 0;
  for (int i = 0; i < n && done < n; ++i) {
    bool seen = false;
    for (int k = 0; k < i && !seen; ++k) seen = P[k].n_omega_channels == P[i].n_omega_channels;
    if (seen) continue;
    int32_t count = 0;
    const int rc = ge2_tc_class_launch(T, P, n, P[i].n_omega_channels, done, count, passes, packed,
                                       ws, host_slots, status, s);
    if (rc != LH_OK) return rc;
    done += count;
  }
  return LH_OK;
}

}  // namespace lh
