// Order >=2 source compile: axial-slice basis of a shower's node bands.
//
// Reference: node_sources (shower/ge2.py:35-67) -> compile_axial_slices
// (_shower_basis.py:188-645) with the shower basis (0.25 m slices, cubic
// Lagrange axial weights, 5-moment transverse stencil of half-width 0.2 m
// for slices wider than 0.03 m, linear deposit on a 0.02 ns time lattice,
// stencil points on the axis), _cone_harmonics (:81-99) and the harmonics of
// axial_fast._harmonics_into / _layout.
//
// For element node e (chord midpoint, or two Gauss nodes on long chords) at
// axial coordinate z, transverse (x, y), time t, direction u and cone cosine
// mu_C in band b, with slice lattice zl = (z - z0)/h_z and tick lattice
// tl = (t - t_ref)/dt:
//   D[b][zb + j][tb + d][k][c] += w_j(zl - zb) w_d(tl - tb) F_k P_l(mu_C) Y_c(u)
// with F = photons_b (1, x, y, x^2, y^2) x node weight, j = -1..2 (cubic),
// d = 0, 1 (linear). Per slice the time lattice is transformed,
//   V[b][s][k][c](w) = sum_tick D[b][s][tick][k][c] e^{i w tick dt},
// and the slice's points carry V (thin slice, one point at the field-0
// centroid) or the stencil combination of its five moments (wide slice).
//
// B200 layout: one thread per node forms the node's link weights, band factors,
// harmonics and Legendre values once and counts it under its base lattice key
// (zb, tb); the occupied keys are listed as they are first met. Ticks are stored
// for each slice's own range only, one row of [band][moment][channel] per (slice,
// tick). One CTA per occupied key adds its nodes' products, eight links in
// registers per (moment, channel) thread, to the rows; one CTA per (slice, band,
// block of frequencies) runs the time-lattice transform with rotating phasors and
// writes the points' channels.
// Measured on 6637 elements (2700 keys, 39 channels, 65 frequencies), before and
// after: key scan 45 us (one CTA over every lattice key) -> 3 us; clearing 42 us
// (203 MB of lattice, mostly never read) -> 8 us; keys 121 us (one thread per node
// forming its harmonics inside the key's CTA) -> 25 us; layout 51 us (one
// thread) -> 3 us; transform 143 us (one frequency per thread, no copies ahead) ->
// 97 us, bound by the float64 chain of two CTAs per SM. The node pass takes 24 us.
#include <algorithm>

#include "lh_common.cuh"
#include "lh_timing.cuh"

namespace lh {

constexpr int kSrcMaxBands = 8;
constexpr int kSrcMaxNch = 153;       // degree 16, azimuthal degree 4
constexpr int kSrcChunk = 32;         // most nodes staged per pass
constexpr size_t kSrcStageBytes = 40 * 1024;  // of a pass's nodes

// Float64 values of a node: harmonics [nch], Legendre values [band][degree + 1],
// link weights [8], axial weights [4], factors [band][5].
struct SrcRow {
  int legendre, link, axial, factor, size;
};
__host__ __device__ inline SrcRow src_row(const lh_source_problem& P) {
  SrcRow r;
  r.legendre = P.nch;
  r.link = r.legendre + P.n_bands * (P.degree + 1);
  r.axial = r.link + 8;
  r.factor = r.axial + 4;
  r.size = r.factor + P.n_bands * 5;
  return r;
}
__host__ __device__ inline int src_chunk(const lh_source_problem& P) {
  const int fit = (int)(kSrcStageBytes / sizeof(double)) / src_row(P).size;
  return fit < kSrcChunk ? fit : kSrcChunk;
}

// Cubic Lagrange weights of shifts -1, 0, 1, 2 at offset r (_shower_basis.py:112-118)
LH_DEVICE void src_axial_weights(double r, double* w) {
  w[0] = -r * (r - 1) * (r - 2) / 6;
  w[1] = (r + 1) * (r - 1) * (r - 2) / 2;
  w[2] = -(r + 1) * r * (r - 2) / 2;
  w[3] = (r + 1) * r * (r - 1) / 6;
}

// Real orthonormal harmonics of direction (x, y, z) into out[kept channel]
// (axial_fast._harmonics_into)
LH_DEVICE void src_harmonics(double x, double y, double z, const lh_source_problem& P, double* out) {
  const double radius = sqrt(x * x + y * y + z * z);
  const double mu = z / radius;
  const double transverse = sqrt(x * x + y * y);
  const double sine = transverse / radius;
  const double cp = transverse == 0.0 ? 1.0 : x / transverse;
  const double sp = transverse == 0.0 ? 0.0 : y / transverse;
  double cm = 1.0, sm = 0.0;
  double diagonal = 1.0 / sqrt(4 * kPi);
  const int degree = P.degree, max_m = P.max_m;
  for (int m = 0; m <= max_m; ++m) {
    if (m) {
      diagonal *= sqrt((2.0 * m + 1) / (2.0 * m)) * sine;
      const double c2 = cm * cp - sm * sp, s2 = sm * cp + cm * sp;
      cm = c2;
      sm = s2;
    }
    double v0 = diagonal, v1 = 0.0;
    for (int ell = m; ell <= degree; ++ell) {
      double value;
      if (ell == m) {
        value = v0;
      } else if (ell == m + 1) {
        value = sqrt(2.0 * m + 3) * mu * v0;
        v1 = value;
      } else {
        value = P.aa[ell * (max_m + 1) + m] * mu * v1 - P.bb[ell * (max_m + 1) + m] * v0;
        v0 = v1;
        v1 = value;
      }
      const int centre = P.starts[ell] + min(ell, max_m);
      if (m == 0) {
        out[centre] = value;
      } else {
        out[centre - m] = sqrt(2.0) * value * sm;
        out[centre + m] = sqrt(2.0) * value * cm;
      }
    }
  }
}

struct SrcWorkspace {
  int64_t* key;        // [node], -1 outside the lattice
  double* rows;        // [node][SrcRow]
  int32_t *counts, *offsets, *cursor;  // [lattice key]
  int32_t* order;      // nodes by key
  int64_t* groups;     // occupied keys, in no order
  int32_t* n_groups;   // [4]: occupied keys, nodes listed, occupied slices
  int32_t *slice_lo, *slice_hi;        // tick range, hi < 0: empty
  int64_t* slice_row;  // [n_slices + 1] first deposit row of each slice
  int32_t *slice_point, *slice_wide;
  double *deposit, *zero;
  size_t bytes;
};

// One thread per (element, node): lattice coordinates, the node's row of values,
// counts and first meeting of its base key, each slice's tick range.
__global__ void __launch_bounds__(64)
src_nodes_kernel(const lh_source_problem P, const SrcWorkspace W, int32_t* status) {
  const int64_t total = (int64_t)P.n_el * P.element_order;
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const unsigned full = 0xffffffffu;
  long long key = -1;
  if (k < total) {
    const int e = (int)(k / P.element_order);
    const int n = (int)(k - (int64_t)e * P.element_order);
    const double f = P.node_fraction[n];
    const double px = P.start[3 * e] + f * P.length[e] * P.direction[3 * e];
    const double py = P.start[3 * e + 1] + f * P.length[e] * P.direction[3 * e + 1];
    const double pz = P.start[3 * e + 2] + f * P.length[e] * P.direction[3 * e + 2];
    const double ox = px - P.centre[0], oy = py - P.centre[1], oz = pz - P.centre[2];
    const double z = ox * P.axis[0] + oy * P.axis[1] + oz * P.axis[2];
    const double tx = ox - z * P.axis[0], ty = oy - z * P.axis[1], tz = oz - z * P.axis[2];
    const double x = tx * P.first[0] + ty * P.first[1] + tz * P.first[2];
    const double y = tx * P.second[0] + ty * P.second[1] + tz * P.second[2];
    const double t = P.t0[e] + f * (P.t1[e] - P.t0[e]);
    const double zl = (z - P.z_origin) / P.cell_m;
    const double zbf = floor(zl);
    const double tl = (t - P.reference_ns) / P.time_step_ns;
    const double tbf = floor(tl);
    const long long zb = (long long)zbf, tb = (long long)tbf;
    if (zb < 1 || zb + 2 >= P.n_slices || tb < 0 || tb + 1 >= P.kmax) {
      atomicOr(reinterpret_cast<unsigned*>(status), LH_STATUS_OVERFLOW);
    } else {
      key = zb * P.kmax + tb;
      for (int j = -1; j <= 2; ++j) {
        atomicMin(W.slice_lo + zb + j, (int)tb);
        atomicMax(W.slice_hi + zb + j, (int)tb + 1);
      }
      const SrcRow R = src_row(P);
      double* row = W.rows + k * R.size;
      const double ux = P.direction[3 * e], uy = P.direction[3 * e + 1], uz = P.direction[3 * e + 2];
      // the direction in (first, second, axis)
      src_harmonics(ux * P.first[0] + uy * P.first[1] + uz * P.first[2],
                    ux * P.second[0] + uy * P.second[1] + uz * P.second[2],
                    ux * P.axis[0] + uy * P.axis[1] + uz * P.axis[2], P, row);
      double wz[4];
      const double zr = zl - zbf, tr = tl - tbf;
      src_axial_weights(zr, wz);
      const double wt[2] = {1 - tr, tr};
      for (int j = 0; j < 4; ++j) {
        row[R.axial + j] = wz[j];
        for (int d = 0; d < 2; ++d) row[R.link + 2 * j + d] = wz[j] * wt[d];
      }
      for (int b = 0; b < P.n_bands; ++b) {
        // signed band field C0/lambda^2 + C2/(lambda n)^2 times the chord node weight
        const double g = (P.c0[e] * P.band_s0[b] + P.c2[e] * P.band_s2[b]) * P.node_weight[n];
        double* factor = row + R.factor + 5 * b;
        factor[0] = g;
        factor[1] = g * x;
        factor[2] = g * y;
        factor[3] = g * x * x;
        factor[4] = g * y * y;
        const double mu = 1.0 / (P.beta[e] * P.band_phase[b]);
        double* legendre = row + R.legendre + b * (P.degree + 1);
        double prev = 1.0, cur = mu;
        for (int ell = 0; ell <= P.degree; ++ell) {
          double p;
          if (ell == 0) p = 1.0;
          else if (ell == 1) p = cur;
          else {
            p = ((2 * ell - 1) * mu * cur - (ell - 1) * prev) / ell;
            prev = cur;
            cur = p;
          }
          legendre[ell] = p;
        }
      }
    }
    W.key[k] = key;
  }
  const bool fresh = key >= 0 && atomicAdd(W.counts + key, 1) == 0;
  const unsigned news = __ballot_sync(full, fresh);
  if (news) {
    const int lane = threadIdx.x & 31;
    int at = 0;
    if (lane == __ffs(news) - 1) at = atomicAdd(W.n_groups, __popc(news));
    at = __shfl_sync(full, at, __ffs(news) - 1);
    if (fresh) W.groups[at + __popc(news & ((1u << lane) - 1u))] = key;
  }
}

// CTA 0: the first deposit row of each slice. The others: each occupied key's
// place in the node list (in no order).
__global__ void __launch_bounds__(256)
src_rows_kernel(const lh_source_problem P, const SrcWorkspace W) {
  if (blockIdx.x > 0) {
    const int total = W.n_groups[0];
    for (int g = (blockIdx.x - 1) * blockDim.x + threadIdx.x; g < total;
         g += (gridDim.x - 1) * blockDim.x) {
      const int64_t key = W.groups[g];
      const int at = atomicAdd(W.n_groups + 1, W.counts[key]);
      W.offsets[key] = at;
      W.cursor[key] = at;
    }
    return;
  }
  __shared__ long long warp_sum[8];
  __shared__ int occupied;
  if (threadIdx.x == 0) occupied = 0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  long long carry = 0;
  int mine = 0;
  for (int64_t first = 0; first < P.n_slices; first += blockDim.x) {
    const int64_t s = first + threadIdx.x;
    const int hi = s < P.n_slices ? W.slice_hi[s] : -1;
    const long long n = hi >= 0 ? hi - W.slice_lo[s] + 1 : 0;
    mine += hi >= 0;
    long long v = n;
    for (int off = 1; off < 32; off <<= 1) {
      const long long up = __shfl_up_sync(0xffffffffu, v, off);
      if (lane >= off) v += up;
    }
    __syncthreads();
    if (lane == 31) warp_sum[warp] = v;
    __syncthreads();
    long long before = carry;
    for (int w = 0; w < 8; ++w) {
      if (w < warp) before += warp_sum[w];
      carry += warp_sum[w];
    }
    if (s < P.n_slices) W.slice_row[s] = before + v - n;
  }
  atomicAdd(&occupied, mine);
  __syncthreads();
  if (threadIdx.x == 0) {
    W.slice_row[P.n_slices] = carry;
    W.n_groups[2] = occupied;
  }
}

// Lists the nodes by key and clears the deposit rows in use.
__global__ void src_scatter_kernel(const lh_source_problem P, const SrcWorkspace W) {
  const int64_t first = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t total = (int64_t)P.n_el * P.element_order;
  for (int64_t k = first; k < total; k += stride) {
    const int64_t key = W.key[k];
    if (key >= 0) W.order[atomicAdd(W.cursor + key, 1)] = (int32_t)k;
  }
  const int64_t values = W.slice_row[P.n_slices] * P.n_bands * 5 * P.nch;
  double2* pairs = reinterpret_cast<double2*>(W.deposit);
  for (int64_t k = first; k < (values + 1) / 2; k += stride) pairs[k] = make_double2(0.0, 0.0);
}

// One CTA per occupied base key, one thread per (moment, channel): the nodes'
// products of a band summed over the eight links in registers, then added to the
// links' rows.
__global__ void src_group_kernel(const lh_source_problem P, const SrcWorkspace W) {
  extern __shared__ __align__(16) double s_node[];  // [node of the pass][SrcRow]
  const SrcRow R = src_row(P);
  const int NB = P.n_bands, nch = P.nch, chunk = src_chunk(P);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int k = threadIdx.x / nch, c = threadIdx.x - k * nch;
  const bool mine = k < 5;
  const int ell = mine ? P.channel_degree[c] : 0;
  const int total_groups = W.n_groups[0];
  for (int gi = blockIdx.x; gi < total_groups; gi += gridDim.x) {
    const int64_t key = W.groups[gi];
    const int begin = W.offsets[key], count = W.counts[key];
    const long long zb = key / P.kmax, tb = key - zb * P.kmax;
    auto stage = [&](int from, int nn) {
      __syncthreads();
      for (int q = warp; q < nn; q += warps) {
        const double* row = W.rows + (int64_t)W.order[begin + from + q] * R.size;
        for (int i = lane; i < R.size; i += 32) s_node[q * R.size + i] = row[i];
      }
      __syncthreads();
    };
    const bool once = count <= chunk;
    for (int b = 0; b < NB; ++b) {
      double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0}, sum = 0.0;
      // the field moments of the slices: thread (axial shift, moment)
      const bool zeroth = threadIdx.x < 20;
      const int shift = threadIdx.x / 5, moment = threadIdx.x - 5 * shift;
      for (int from = 0; from < count; from += chunk) {
        const int nn = min(chunk, count - from);
        if (!once || b == 0) stage(from, nn);
        if (mine)
          for (int q = 0; q < nn; ++q) {
            const double* row = s_node + q * R.size;
            const double v = row[R.factor + 5 * b + k] *
                             (row[c] * row[R.legendre + b * (P.degree + 1) + ell]);
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[j] += row[R.link + j] * v;
          }
        if (zeroth)
          for (int q = 0; q < nn; ++q)
            sum += s_node[q * R.size + R.axial + shift] *
                   s_node[q * R.size + R.factor + 5 * b + moment];
      }
      if (mine) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if (acc[j] == 0.0) continue;
          const long long slice = zb + (j >> 1) - 1;
          const int64_t at = W.slice_row[slice] + tb + (j & 1) - W.slice_lo[slice];
          atomicAdd(W.deposit + ((at * NB + b) * 5 + k) * nch + c, acc[j]);
        }
      }
      if (zeroth) atomicAdd(W.zero + ((zb + shift - 1) * NB + b) * 5 + moment, sum);
    }
  }
}

// One warp per band: point layout (_shower_basis.py:375-420, 466-475): occupied
// slices in order, then the +x, -x, +y, -y stencil points of the wide slices; thin
// slices sit at their field-0 centroid, wide ones on the axis.
__global__ void src_layout_kernel(const lh_source_problem P, const SrcWorkspace W,
                                  lh_source_output O) {
  const int NB = P.n_bands, b = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned full = 0xffffffffu, lower = (1u << lane) - 1u;
  const int64_t S = P.n_slices;
  const double h = P.stencil_m;
  int occ = 0, wide_count = 0;
  for (int64_t first = 0; first < S; first += 32) {
    const int64_t s = first + lane;
    const bool used = s < S && W.slice_hi[s] >= 0;
    bool wide = false;
    double cx = 0.0, cy = 0.0;
    if (used) {
      const double* zm = W.zero + (s * NB + b) * 5;
      const double mass = zm[0];
      const double safe = mass != 0.0 ? mass : 1.0;
      // absolute values by comparison: nvcc 12.9 at -O3 dropped fabs() of this
      // select (fabs(safe) came back negative for a negative mass)
      const double num = zm[3] + zm[4];
      const double spread = sqrt((num < 0.0 ? -num : num) / (safe < 0.0 ? -safe : safe));
      wide = spread > P.stencil_threshold_m;
      cx = wide ? 0.0 : zm[1] / safe;
      cy = wide ? 0.0 : zm[2] / safe;
    }
    const unsigned used_mask = __ballot_sync(full, used), wide_mask = __ballot_sync(full, wide);
    if (s < S) {
      const int point = occ + __popc(used_mask & lower);
      W.slice_point[b * S + s] = used ? point : -1;
      W.slice_wide[b * S + s] = wide ? wide_count + __popc(wide_mask & lower) : -1;
      if (used) {
        double* pt = O.points + ((int64_t)b * O.capacity + point) * 3;
        pt[0] = P.z_origin + (double)s * P.cell_m;
        pt[1] = cx;
        pt[2] = cy;
      }
    }
    occ += __popc(used_mask);
    wide_count += __popc(wide_mask);
  }
  __syncwarp();
  // stencil points: offsets (h,0), (-h,0), (0,h), (0,-h) in wide-slice order
  for (int64_t s = lane; s < S; s += 32) {
    const int w = W.slice_wide[b * S + s];
    if (w < 0) continue;
    for (int o = 0; o < 4; ++o) {
      double* pt = O.points + ((int64_t)b * O.capacity + occ + o * wide_count + w) * 3;
      pt[0] = P.z_origin + (double)s * P.cell_m;
      pt[1] = o == 0 ? h : (o == 1 ? -h : 0.0);
      pt[2] = o == 2 ? h : (o == 3 ? -h : 0.0);
    }
  }
  if (lane == 0) O.n_points[b] = occ + 4 * wide_count;
}

// One CTA per (slice, band, block of 2 `pairs` frequencies): time-lattice
// transform and the slice's points (_shower_basis.py:577-611). One thread per
// (channel, two frequencies) walks the slice's ticks with two rotating phasors, so
// that a value read from shared memory is used four times; the CTA stages the
// deposit rows of kSrcTransformBytes worth of ticks at a time (coalesced,
// independent loads).
constexpr int kSrcPairs = 8;
constexpr int kSrcTransformBytes = 48 * 1024;

// The sums of kMoments moments over the slice's ticks; `deposit` is the band's first
// row, `stride` float64 values from tick to tick.
template <int kMoments>
LH_DEVICE void src_transform_ticks(const double* deposit, int64_t stride, int ticks, int nch,
                                   double* s_dep, bool mine, int c, double (&pc)[2],
                                   double (&ps)[2], const double (&dc)[2], const double (&ds)[2],
                                   double (&re)[2][5], double (&im)[2][5]) {
  // two buffers: the next ticks' rows are on their way while these are used
  const int row = kMoments * nch;  // staged doubles per tick
  const int room = (int)(kSrcTransformBytes / sizeof(double)) / 2;
  const int chunk = max(1, min(64, room / row));
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  auto fetch = [&](int t0, double* to) {
    const int n_t = min(chunk, ticks - t0);
    for (int tt = warp; tt < n_t; tt += warps) {
      const double* from = deposit + (t0 + tt) * stride;
      for (int r = lane; r < row; r += 32) copy_async8(to + tt * row + r, from + r);
    }
    copy_async_commit();
  };
  fetch(0, s_dep);
  for (int t0 = 0, buf = 0; t0 < ticks; t0 += chunk, buf ^= 1) {
    const int n_t = min(chunk, ticks - t0);
    if (t0 + chunk < ticks) {
      fetch(t0 + chunk, s_dep + (buf ^ 1) * room);
      copy_async_wait<1>();
    } else {
      copy_async_wait<0>();
    }
    __syncthreads();
    const double* rowp = s_dep + buf * room + c;
    for (int tt = 0; tt < (mine ? n_t : 0); ++tt, rowp += row) {
#pragma unroll
      for (int k = 0; k < kMoments; ++k) {
        const double v = rowp[k * nch];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          re[u][k] += v * pc[u];
          im[u][k] += v * ps[u];
        }
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const double npc = pc[u] * dc[u] - ps[u] * ds[u], nps = ps[u] * dc[u] + pc[u] * ds[u];
        pc[u] = npc;
        ps[u] = nps;
      }
    }
    __syncthreads();  // the buffer is filled again
  }
}

__global__ void __launch_bounds__(512)
src_transform_kernel(const lh_source_problem P, const SrcWorkspace Wk, lh_source_output O,
                     int pairs) {
  extern __shared__ double s_dep[];  // [tick][moment][channel]
  const int64_t s = blockIdx.x;
  const int b = blockIdx.y;
  const int NB = P.n_bands, nch = P.nch, W = P.n_omega;
  if (Wk.slice_hi[s] < 0) return;
  const int lo = Wk.slice_lo[s], hi = Wk.slice_hi[s];
  const int64_t S = P.n_slices, row0 = Wk.slice_row[s];
  const int point = Wk.slice_point[b * S + s];
  const int wide = Wk.slice_wide[b * S + s];
  const int occ = Wk.n_groups[2];
  const int wide_count = (O.n_points[b] - occ) / 4;
  const double h = P.stencil_m, h2 = h * h;
  const double scale = P.band_scale[b];
  const int i = threadIdx.x;
  const int c = i % nch, w0 = blockIdx.z * 2 * pairs + i / nch;
  const bool mine = i < nch * pairs && w0 < W;
  double ps[2], pc[2], ds[2], dc[2];
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const double om = mine ? P.omega[min(w0 + u * pairs, W - 1)] : 0.0;
    sincos(om * lo * P.time_step_ns, &ps[u], &pc[u]);
    sincos(om * P.time_step_ns, &ds[u], &dc[u]);
  }
  double re[2][5] = {}, im[2][5] = {};
  const double* deposit = Wk.deposit + (row0 * NB + b) * 5 * (int64_t)nch;
  const int64_t stride = (int64_t)NB * 5 * nch;
  if (wide >= 0)
    src_transform_ticks<5>(deposit, stride, hi - lo + 1, nch, s_dep, mine, c, pc, ps, dc, ds, re, im);
  else
    src_transform_ticks<1>(deposit, stride, hi - lo + 1, nch, s_dep, mine, c, pc, ps, dc, ds, re, im);
  if (!mine) return;
  float2* out = reinterpret_cast<float2*>(O.channels);
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int w = w0 + u * pairs;
    if (w >= W) continue;
    const double* r = re[u];
    const double* m = im[u];
    auto put = [&](int p, double vr, double vi) {
      out[(((int64_t)b * O.capacity + p) * nch + c) * W + w] =
          make_float2((float)(scale * vr), (float)(scale * vi));
    };
    if (wide < 0) {
      put(point, r[0], m[0]);
    } else {
      // m0, mx, my, mxx, myy -> centre, +x, -x, +y, -y
      put(point, r[0] - (r[3] + r[4]) / h2, m[0] - (m[3] + m[4]) / h2);
      put(occ + 0 * wide_count + wide, 0.5 * (r[3] / h2 + r[1] / h), 0.5 * (m[3] / h2 + m[1] / h));
      put(occ + 1 * wide_count + wide, 0.5 * (r[3] / h2 - r[1] / h), 0.5 * (m[3] / h2 - m[1] / h));
      put(occ + 2 * wide_count + wide, 0.5 * (r[4] / h2 + r[2] / h), 0.5 * (m[4] / h2 + m[2] / h));
      put(occ + 3 * wide_count + wide, 0.5 * (r[4] / h2 - r[2] / h), 0.5 * (m[4] / h2 - m[2] / h));
    }
  }
}

static size_t src_align(size_t x) { return (x + 255) & ~(size_t)255; }

static SrcWorkspace src_layout(const lh_source_problem& P, unsigned char* base) {
  SrcWorkspace W{};
  size_t off = 0;
  auto take = [&](size_t bytes) {
    unsigned char* p = base ? base + off : nullptr;
    off += src_align(bytes);
    return p;
  };
  const int64_t n_nodes = (int64_t)P.n_el * P.element_order;
  const int64_t n_keys = P.n_slices * P.kmax;
  const int NB = P.n_bands;
  // cleared together: counts, n_groups, zero
  W.counts = reinterpret_cast<int32_t*>(take(sizeof(int32_t) * n_keys));
  W.n_groups = reinterpret_cast<int32_t*>(take(sizeof(int32_t) * 4));
  W.zero = reinterpret_cast<double*>(take(sizeof(double) * P.n_slices * NB * 5));
  W.slice_lo = reinterpret_cast<int32_t*>(take(sizeof(int32_t) * P.n_slices));
  W.slice_hi = reinterpret_cast<int32_t*>(take(sizeof(int32_t) * P.n_slices));
  W.key = reinterpret_cast<int64_t*>(take(sizeof(int64_t) * n_nodes));
  W.rows = reinterpret_cast<double*>(take(sizeof(double) * src_row(P).size * n_nodes));
  W.offsets = reinterpret_cast<int32_t*>(take(sizeof(int32_t) * n_keys));
  W.cursor = reinterpret_cast<int32_t*>(take(sizeof(int32_t) * n_keys));
  W.order = reinterpret_cast<int32_t*>(take(sizeof(int32_t) * n_nodes));
  W.groups = reinterpret_cast<int64_t*>(take(sizeof(int64_t) * std::min(n_keys, n_nodes)));
  W.slice_row = reinterpret_cast<int64_t*>(take(sizeof(int64_t) * (P.n_slices + 1)));
  W.slice_point = reinterpret_cast<int32_t*>(take(sizeof(int32_t) * P.n_slices * NB));
  W.slice_wide = reinterpret_cast<int32_t*>(take(sizeof(int32_t) * P.n_slices * NB));
  W.deposit = reinterpret_cast<double*>(take(sizeof(double) * n_keys * NB * 5 * P.nch));
  W.bytes = off;
  return W;
}

static bool src_valid(const lh_source_problem* P) {
  if (!P) return false;
  if (P->n_el < 1 || !P->start || !P->direction || !P->length || !P->c0 || !P->c2 || !P->beta ||
      !P->t0 || !P->t1)
    return false;
  if (P->n_bands < 1 || P->n_bands > kSrcMaxBands) return false;
  if (P->degree < 0 || P->degree > 16 || P->max_m < 0 || P->max_m > 4 || P->max_m > P->degree ||
      P->nch < 1 || P->nch > kSrcMaxNch)
    return false;
  if (P->element_order < 1 || P->element_order > 2) return false;
  if (!(P->cell_m > 0) || !(P->stencil_m > 0) || !(P->time_step_ns > 0)) return false;
  if (P->n_slices < 4 || P->kmax < 2 || P->n_slices * P->kmax > (1ll << 30)) return false;
  if (P->n_omega < 1 || !P->omega) return false;
  return true;
}

}  // namespace lh

extern "C" size_t lh_source_workspace_bytes(const lh_source_problem* P) {
  if (!lh::src_valid(P)) return 0;
  return lh::src_layout(*P, nullptr).bytes;
}

extern "C" int lh_source_compile(const lh_source_problem* P, const lh_source_output* O,
                                 void* workspace, size_t workspace_bytes, int32_t* status,
                                 void* stream) {
  if (!lh::src_valid(P) || !O || !O->points || !O->channels || !O->n_points || !status)
    return LH_EINVAL;
  if (O->capacity < P->n_slices * 5) return LH_EINVAL;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  lh::SrcWorkspace W = lh::src_layout(*P, static_cast<unsigned char*>(workspace));
  if (!workspace || workspace_bytes < W.bytes) return LH_ENOMEM;
  const int64_t n_nodes = (int64_t)P->n_el * P->element_order;
  const int NB = P->n_bands;
  const int threads = ((5 * P->nch + 31) / 32) * 32;  // of the group kernel: at most 768
  const size_t gsmem = sizeof(double) * lh::src_row(*P).size * (size_t)lh::src_chunk(*P);
  cudaMemsetAsync(W.counts, 0, reinterpret_cast<unsigned char*>(W.slice_lo) -
                                   reinterpret_cast<unsigned char*>(W.counts), s);
  cudaMemsetAsync(W.slice_lo, 0x7f, sizeof(int32_t) * P->n_slices, s);
  cudaMemsetAsync(W.slice_hi, 0xff, sizeof(int32_t) * P->n_slices, s);
  cudaMemsetAsync(O->channels, 0, sizeof(float) * 2 * NB * O->capacity * P->nch * P->n_omega, s);
  lh::src_nodes_kernel<<<(unsigned)((n_nodes + 63) / 64), 64, 0, s>>>(*P, W, status);
  const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((n_nodes + 255) / 256, 148 * 4));
  lh::src_rows_kernel<<<1 + blocks, 256, 0, s>>>(*P, W);
  lh::src_scatter_kernel<<<148 * 8, 256, 0, s>>>(*P, W);
  {
    lh::TimedLaunch timed_launch(LH_KT_SRC_GROUP, s);
    lh::src_group_kernel<<<148 * 8, threads, gsmem, s>>>(*P, W);
  }
  lh::src_layout_kernel<<<1, 32 * NB, 0, s>>>(*P, W, *O);
  const int pairs = std::max(1, std::min(lh::kSrcPairs, 512 / P->nch));
  dim3 grid((unsigned)P->n_slices, (unsigned)NB,
            (unsigned)((P->n_omega + 2 * pairs - 1) / (2 * pairs)));
  {
    lh::TimedLaunch timed_launch(LH_KT_SRC_TRANSFORM, s);
    lh::src_transform_kernel<<<grid, ((P->nch * pairs + 31) / 32) * 32, lh::kSrcTransformBytes,
                               s>>>(*P, W, *O, pairs);
  }
  return cudaGetLastError() == cudaSuccess ? LH_OK : LH_ECUDA;
}
