// Isotropic calibration flashes, all scattering orders, on the device.
//
// Reference: TransportKernel._transport_isotropic (transport.py:1061-1164) with
// ResponseCache.acceptance_spectrum / moments_at (cache.py:294-436) and
// readout_bins (readout.py:43-72), for a monochromatic flash and the
// centre-ray receiver.
//
// Work decomposition: a tile is 64 (flash, OM) pairs = 128 readout rows
// (orders 1 and 2 of each pair).
//  1. pair setup (float64, one thread per pair): distance, head-on cosine,
//     acceptance, the OM clock time_origin_ns, the order-0 bin, the radial
//     interval of the log-r spline and the safety bound of transport.py:1115;
//  2. spectrum (float32, one thread per (pair, omega)): cubic in log r of the
//     detrended multipole moments, contracted with alpha_l P_l(cos)/(4 pi),
//     times attenuation and the flight phase; writes the absolute spectrum and
//     the demodulated (relative) spectrum of orders 1 and 2 as readout rows;
//  3. readout of the rows (see lh_readout.cu) and the order-0 bin rows,
//     charge (spectrum at the first frequency) and the active mask.
// flash_tc_kernel and flash_step_kernel fuse 1-3 in one persistent kernel: the readout
// rows are written straight into shared memory as the tensor-core A tile.
#include "lh_common.cuh"
#include "lh_readout.cuh"

namespace lh {

constexpr int kFlashPairs = 64;  // pairs per tile -> 128 readout rows
constexpr int kMaxAcc = 8;       // highest acceptance degree handled
constexpr int kFlashThreads = 256;    // plain path
constexpr int kFlashTcThreads = 512;  // fused path; with roles 11 warps of spectra, 4 of drain, 1 of MMAs
// A tile of the fused path: K-major, no swizzle, [k/8][row][k%8] with each
// 8-column chunk of the 128 rows padded by 16 bytes (2064 B apart, the MMA's
// leading byte offset). A warp stores 32 consecutive columns of one row: the
// padding puts their four chunks in different banks (2048 B apart they shared
// four banks: 4-way conflicts on every A-tile store).
constexpr int kAChunk = 128 * 8 + 8;   // elements per 8-column chunk
LH_DEVICE int a_offset(int row, int k) { return (k >> 3) * kAChunk + row * 8 + (k & 7); }

struct FlashPair {
  double origin;  // time_origin_ns of the OM for this flash
  double t12;     // r / speed: flight time of the spectrum phase (orders 1, 2)
  double t0;      // absolute order-0 phase time (r / speed inside, t + r / speed outside)
  double q0;      // order-0 bin weight
  double c12, c0, cr;  // t12, t0 and t12 - origin in turns per (rad/ns): t / (2 pi)
  int64_t pair;   // flash * n_om + OM
  float tt;       // offset in the log-r interval
  float amp12;    // photons * area * efficiency * exp(-mu_a r) / (4 pi r^2)
  float amp0;     // order-0 amplitude
  int j;          // log-r interval, -1 outside the table's radial range
  int bin0;       // order-0 bin, -1 outside the window
  uint8_t valid;  // pair exists
  uint8_t inside;
  uint8_t flags;  // bit 1: unsafe (outside range, bound above threshold); bit 2: coincident
  float w[kMaxAcc + 1];  // alpha_l P_l(cos) / (4 pi)
  float charge[3];
};

// Flashes in this launch: the device count when given (graph replay), else n_flash.
LH_DEVICE int flash_count(const lh_flash_batch& b) {
  if (b.n_flash_device) {
    const int n = *b.n_flash_device;
    return n < 0 ? 0 : (n > b.n_flash ? b.n_flash : n);
  }
  return b.n_flash;
}

// Step 1 for one pair.
LH_DEVICE void flash_pair_setup(const lh_flash_problem& p, const lh_flash_batch& b, int64_t pair,
                                FlashPair& s) {
  const int n_om = p.n_om;
  const int64_t f = pair / n_om;
  const int d = (int)(pair % n_om);
  const double sx = b.pos[3 * f], sy = b.pos[3 * f + 1], sz = b.pos[3 * f + 2];
  const double px = p.om_pos[3 * d], py = p.om_pos[3 * d + 1], pz = p.om_pos[3 * d + 2];
  // displacement = positions - source; radii = |displacement| (transport.py:1069-1070)
  const double dx = __dsub_rn(px, sx), dy = __dsub_rn(py, sy), dz = __dsub_rn(pz, sz);
  const double r = sqrt(dot3_rn(dx, dy, dz, dx, dy, dz));
  s.flags = 0;
  if (r == 0.0) {
    atomicOr(reinterpret_cast<unsigned*>(b.status), LH_STATUS_COINCIDENT);
    s.flags |= 4;
  }
  // head_on_cosine (model.py:158-162): toward = (source - position) / |.|
  const double tx = __dsub_rn(sx, px), ty = __dsub_rn(sy, py), tz = __dsub_rn(sz, pz);
  const double tn = sqrt(dot3_rn(tx, ty, tz, tx, ty, tz));
  const double cosine = dot3_rn(p.om_look[3 * d], p.om_look[3 * d + 1], p.om_look[3 * d + 2],
                                tx / tn, ty / tn, tz / tn);
  // Legendre P_l(cos): acceptance A = sum alpha_l (2l+1) P_l / (4 pi) (cache.py:509-521)
  // and contraction weights alpha_l P_l / (4 pi) (cache.py:416-418)
  double pl_prev = 1.0, pl = cosine, acc = 0.0;
  for (int l = 0; l <= p.acc_top; ++l) {
    double P;
    if (l == 0) P = 1.0;
    else if (l == 1) P = cosine;
    else {
      P = ((2 * l - 1) * cosine * pl - (l - 1) * pl_prev) / l;
      pl_prev = pl;
      pl = P;
    }
    acc += p.alpha[l] * (2 * l + 1) * P / (4 * kPi);
    s.w[l] = (float)(P * p.alpha[l] / (4 * kPi));
  }
  const double area = p.om_area[d];
  const double photons = b.photons[f];
  const double t_src = b.time_ns[f];
  const double scale = photons * area * p.efficiency;
  const double four_pi_r2 = 4 * kPi * r * r;
  s.q0 = scale * acc * exp(-p.mu_t * r) / four_pi_r2;
  s.inside = (r >= p.r_low) && (r <= p.r_high);
  const double upper = photons * area * p.efficiency * acc * exp(-p.mu_a * r) / four_pi_r2;
  if (!s.inside && 10 * upper >= p.threshold) {
    s.flags |= 2;
    atomicOr(reinterpret_cast<unsigned*>(b.status), LH_STATUS_UNSAFE);
    atomicAdd(b.status + 1, 1);
    atomicMax(reinterpret_cast<unsigned long long*>(b.status + 2),
              (unsigned long long)__double_as_longlong(r));
  }
  const double arrival = t_src + r / p.speed;
  s.origin = t_src + r / p.origin_speed;
  const int bin = bin_right(p.edges, p.n_edges, arrival - s.origin);
  s.bin0 = (bin >= 0 && bin < p.n_edges - 1) ? bin : -1;
  if (s.inside) {
    const double logr = log(r);
    int j = bin_right(p.log_r, p.n_radii, logr);
    j = j < 0 ? 0 : (j > p.n_radii - 2 ? p.n_radii - 2 : j);
    s.j = j;
    s.tt = (float)(logr - p.log_r[j]);
    s.amp12 = (float)(scale * (exp(-p.mu_a * r) / four_pi_r2));
    s.amp0 = (float)(scale * acc * (exp(-p.mu_t * r) / four_pi_r2));
    s.t12 = r / p.speed;
    s.t0 = r / p.speed;
  } else {
    s.j = -1;
    s.tt = 0.f;
    s.amp12 = 0.f;
    s.amp0 = (float)s.q0;
    s.t12 = 0.0;
    s.t0 = arrival;
  }
  const double inv2pi = 1.0 / (2 * kPi);
  s.c12 = s.t12 * inv2pi;
  s.c0 = s.t0 * inv2pi;
  s.cr = (s.t12 - s.origin) * inv2pi;
  s.valid = 1;
}

// exp(2 pi i turns): the turns reduced in float64 to (-1/2, 1/2], the angle in
// float32 on the SFU (absolute error ~1e-6, far inside the 1e-4 bar of the
// spectra and bins).
LH_DEVICE float2 phase_turns(double turns) {
  const float frac = (float)(turns - rint(turns));
  float sv, cv;
  __sincosf((float)(2 * kPi) * frac, &sv, &cv);
  return make_float2(cv, sv);
}

LH_DEVICE float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// One degree's cubic coefficients of orders 1 and 2 at one frequency.
struct FlashCoef {
  float2 a0, a1, a2, a3;  // order 1: c0..c3
  float2 b0, b1, b2, b3;  // order 2
};

// [interval][degree][order][power][omega]: the lanes of a warp (consecutive
// omega) read consecutive float2, one coalesced segment per coefficient.
LH_DEVICE FlashCoef flash_coef(const lh_flash_problem& p, int j, int l, int w) {
  const int W = p.n_omega;
  const float2* c = reinterpret_cast<const float2*>(p.coef) +
                    ((int64_t)j * (p.acc_top + 1) + l) * 8 * W + w;
  return FlashCoef{__ldg(c),         __ldg(c + W),     __ldg(c + 2 * W), __ldg(c + 3 * W),
                   __ldg(c + 4 * W), __ldg(c + 5 * W), __ldg(c + 6 * W), __ldg(c + 7 * W)};
}

LH_DEVICE void flash_degree(const FlashCoef& c, float t, float wl, float2& s1, float2& s2) {
  float vr = fmaf(fmaf(fmaf(c.a0.x, t, c.a1.x), t, c.a2.x), t, c.a3.x);
  float vi = fmaf(fmaf(fmaf(c.a0.y, t, c.a1.y), t, c.a2.y), t, c.a3.y);
  s1.x = fmaf(wl, vr, s1.x);
  s1.y = fmaf(wl, vi, s1.y);
  vr = fmaf(fmaf(fmaf(c.b0.x, t, c.b1.x), t, c.b2.x), t, c.b3.x);
  vi = fmaf(fmaf(fmaf(c.b0.y, t, c.b1.y), t, c.b2.y), t, c.b3.y);
  s2.x = fmaf(wl, vr, s2.x);
  s2.y = fmaf(wl, vi, s2.y);
}

// Step 2 for one (pair, omega) from its contracted spectra s1, s2 (zero outside the
// table): returns the relative spectra of orders 1, 2 through rel1/rel2 and writes
// the absolute spectrum of all orders.
LH_DEVICE void flash_item(const lh_flash_problem& p, const lh_flash_batch& b, int w, double om,
                          FlashPair& s, float2 s1, float2 s2, float2& rel1, float2& rel2) {
  if (s.j >= 0) {
    s1.x *= s.amp12; s1.y *= s.amp12;
    s2.x *= s.amp12; s2.y *= s.amp12;
  }
  const float2 e12 = phase_turns(om * s.c12);
  const float2 e0 = (s.t0 == s.t12) ? e12 : phase_turns(om * s.c0);
  const float2 r12 = s.j >= 0 ? phase_turns(om * s.cr) : make_float2(1.f, 0.f);
  const float2 o0 = make_float2(s.amp0 * e0.x, s.amp0 * e0.y);
  const float2 o1 = cmul(s1, e12), o2 = cmul(s2, e12);
  if (s.valid) {
    float2* out = reinterpret_cast<float2*>(b.spectrum) + (s.pair * p.n_omega + w) * 3;
    out[0] = o0;
    out[1] = o1;
    out[2] = o2;
    if (w == 0) {
      s.charge[0] = o0.x;
      s.charge[1] = o1.x;
      s.charge[2] = o2.x;
    }
  }
  rel1 = cmul(s1, r12);
  rel2 = cmul(s2, r12);
}

// Step 3 (order 0 and the mask) for the tile's pairs.
// The calling thread is number `index` of the `stride` (at least 64) that take part.
LH_DEVICE void flash_tile_order0(const lh_flash_problem& p, const lh_flash_batch& b,
                                 const FlashPair* sp, int n_bins, int index, int stride) {
  if ((n_bins & 3) == 0) {  // rows are 16-byte aligned: four bins per store
    const int quads = n_bins >> 2;
    for (int i = index; i < kFlashPairs * quads; i += stride) {
      const int lp = i / quads, bin = (i % quads) * 4;
      const FlashPair& s = sp[lp];
      if (!s.valid) continue;
      const float q = (float)s.q0;
      const float4 v = make_float4(bin == s.bin0 ? q : 0.f, bin + 1 == s.bin0 ? q : 0.f,
                                   bin + 2 == s.bin0 ? q : 0.f, bin + 3 == s.bin0 ? q : 0.f);
      *reinterpret_cast<float4*>(b.components + (s.pair * 3) * n_bins + bin) = v;
    }
  } else {
    for (int i = index; i < kFlashPairs * n_bins; i += stride) {
      const int lp = i / n_bins, bin = i % n_bins;
      const FlashPair& s = sp[lp];
      if (!s.valid) continue;
      b.components[(s.pair * 3) * n_bins + bin] = (bin == s.bin0) ? (float)s.q0 : 0.f;
    }
  }
  if (index < kFlashPairs) {
    const FlashPair& s = sp[index];
    if (s.valid) {
      const int64_t pair = s.pair;
      const double q = ((double)s.charge[0] + (double)s.charge[1]) + (double)s.charge[2];
      for (int o = 0; o < 3; ++o) b.charge[pair * 3 + o] = (double)s.charge[o];
      b.origin[pair] = s.origin;
      const bool active = p.threshold == 0.0 ? s.inside : (s.inside && q >= p.threshold);
      b.active[pair] = (uint8_t)((active ? 1 : 0) | s.flags);
    }
  }
}

LH_DEVICE void flash_slot_setup(const lh_flash_problem& p, const lh_flash_batch& b, FlashPair& s,
                                int64_t pair, int64_t n_pairs) {
  s.pair = pair;
  if (pair < n_pairs) {
    flash_pair_setup(p, b, pair, s);
  } else {
    s.valid = 0;
    s.j = -1;
    s.amp12 = s.amp0 = 0.f;
    s.t12 = s.t0 = s.origin = 0.0;
    s.c12 = s.c0 = s.cr = 0.0;
    s.inside = 0;
    s.flags = 0;
  }
  s.charge[0] = s.charge[1] = s.charge[2] = 0.f;
}

LH_DEVICE void flash_tile_setup(const lh_flash_problem& p, const lh_flash_batch& b, FlashPair* sp,
                                int64_t base, int64_t n_pairs) {
  if (threadIdx.x < kFlashPairs)
    flash_slot_setup(p, b, sp[threadIdx.x], base + threadIdx.x, n_pairs);
}

// ---------------------------------------------------------------- plain path
// One block per tile; readout rows go to a row-major fp32 workspace that
// readout_fp32_kernel consumes.
// A launch of few flashes is one chain of coefficient loads per thread: kPlainDegrees
// degrees' loads are on their way together (one flash of 3 degrees: 42.2 us with the
// loads of one degree at a time, 39.2 with four; 30 flashes 175 and 171).
constexpr int kPlainDegrees = 4;
__global__ void __launch_bounds__(kFlashThreads)
flash_plain_kernel(lh_flash_problem p, lh_flash_batch b, int kpad, int n_bins, float* a_rows) {
  __shared__ FlashPair sp[kFlashPairs];
  const int64_t n_pairs = (int64_t)flash_count(b) * p.n_om;
  const int64_t base = (int64_t)blockIdx.x * kFlashPairs;
  flash_tile_setup(p, b, sp, base, n_pairs);
  __syncthreads();
  const int nw = p.n_omega;
  // Every row the readout reads (2 per pair of the host count, whose grid
  // follows) is written in full here: pairs past the device count get zero
  // rows (flash_item yields zero spectra for them), and the padding columns
  // 2 nw .. kpad-1 are zeroed whatever their number.
  const int64_t host_pairs = (int64_t)b.n_flash * p.n_om;
  for (int i = threadIdx.x; i < kFlashPairs * nw; i += blockDim.x) {
    const int lp = i / nw, w = i % nw;
    FlashPair& pair = sp[lp];
    float2 s1 = make_float2(0.f, 0.f), s2 = make_float2(0.f, 0.f), r1, r2;
    if (pair.j >= 0)
      for (int l0 = 0; l0 <= p.acc_top; l0 += kPlainDegrees) {
        FlashCoef c[kPlainDegrees];
#pragma unroll
        for (int k = 0; k < kPlainDegrees; ++k)
          if (l0 + k <= p.acc_top) c[k] = flash_coef(p, pair.j, l0 + k, w);
#pragma unroll
        for (int k = 0; k < kPlainDegrees; ++k)
          if (l0 + k <= p.acc_top) flash_degree(c[k], pair.tt, pair.w[l0 + k], s1, s2);
      }
    flash_item(p, b, w, p.omega[w], pair, s1, s2, r1, r2);
    if (base + lp < host_pairs) {
      float* row1 = a_rows + (2 * (base + lp)) * (int64_t)kpad;
      float* row2 = row1 + kpad;
      row1[w] = r1.x;
      row1[nw + w] = r1.y;
      row2[w] = r2.x;
      row2[nw + w] = r2.y;
      for (int c = 2 * nw + w; c < kpad; c += nw) {
        row1[c] = 0.f;
        row2[c] = 0.f;
      }
    }
  }
  __syncthreads();
  flash_tile_order0(p, b, sp, n_bins, threadIdx.x, blockDim.x);
}

// ---------------------------------------------------------------- fused tcgen05 path
// One CTA per SM, each over its share of consecutive pairs. B (the readout
// operator, hi and lo parts) is loaded once per CTA. The CTA sorts up to
// kFlashSort pairs at a time by radial interval and takes them in tiles of 64 as a
// pipeline of warp roles: the first warps hold the cubic coefficients of their
// frequency in registers, run over neighbouring pairs (reading coefficients only
// where the interval changes) and write A (bf16 hi/lo) into shared memory; the last
// warp issues the MMAs into one of two accumulators; four warps write the order-0
// rows, drain the accumulator and set up the pairs of the tile after next, while the
// first warps compute the next tile. They wait only for the MMAs, since A is there
// once. A share of few pairs (a single flash) spreads over the SMs pair by pair.
// kDegrees: acceptance degrees whose coefficients a thread holds, two or three (four or
// more would not fit beside the rest in the 128 registers of a thread; flash_step_kernel
// takes those).
//
// What bounds it: the outputs (65 frequencies x 24 bytes and 480 bins x 4 bytes a
// pair) take 0.10 ms for 4096 flashes of 48 OMs. The launch took 0.380 ms with
// coefficients read for every pair (192 bytes a pair and frequency through L1), 0.345
// with pairs sorted and all warps in step, 0.304 with roles: now the spectra (11
// warps of latency chains, 40 % of the issue slots) and the drains take about as long
// as each other. 576 threads leave 96 registers each (0.376), eight draining warps
// leave three groups of frequencies (0.293, but 0.166 for 3 x 501 flashes against
// 0.148). One flash: 21.8 us on one SM, now 13.9 on 48. 137 flashes: 25.4, now 22.2.
constexpr int kFlashSort = 2048;        // pairs sorted at a time
constexpr int kFlashMaxBuckets = 1024;  // radial intervals the sort tells apart
constexpr int kFlashDense = 2;          // pairs per interval from which runs share them

// The pair's radial interval for the sort, in float32: where it is off by one the
// pair only sits between neighbours of another interval.
LH_DEVICE int flash_bucket(const lh_flash_problem& p, const lh_flash_batch& b, int64_t pair,
                           int buckets) {
  const int64_t f = pair / p.n_om;
  const int d = (int)(pair - f * p.n_om);
  const float dx = (float)(p.om_pos[3 * d] - b.pos[3 * f]),
              dy = (float)(p.om_pos[3 * d + 1] - b.pos[3 * f + 1]),
              dz = (float)(p.om_pos[3 * d + 2] - b.pos[3 * f + 2]);
  const int j = bin_right(p.log_r, p.n_radii, 0.5f * __logf(dx * dx + dy * dy + dz * dz)) + 1;
  return min(max(j, 0), buckets - 1);
}

// One (pair, frequency) from its contracted spectra: the outputs and the A rows of
// orders 1 and 2, K columns (Re, Im) per frequency, one bf16x2 store per row and part.
LH_DEVICE void flash_rows(const lh_flash_problem& p, const lh_flash_batch& b, int w, double om,
                          FlashPair& s, float2 s1, float2 s2, int lp, __nv_bfloat16* s_ahi,
                          __nv_bfloat16* s_alo) {
  float2 r1, r2;
  flash_item(p, b, w, om, s, s1, s2, r1, r2);
  const __nv_bfloat162 h1 = __floats2bfloat162_rn(r1.x, r1.y);
  const __nv_bfloat162 l1 = __floats2bfloat162_rn(r1.x - __low2float(h1),
                                                  r1.y - __high2float(h1));
  const __nv_bfloat162 h2 = __floats2bfloat162_rn(r2.x, r2.y);
  const __nv_bfloat162 l2 = __floats2bfloat162_rn(r2.x - __low2float(h2),
                                                  r2.y - __high2float(h2));
  const int o1 = a_offset(2 * lp, 2 * w), o2 = a_offset(2 * lp + 1, 2 * w);
  *reinterpret_cast<__nv_bfloat162*>(s_ahi + o1) = h1;
  *reinterpret_cast<__nv_bfloat162*>(s_alo + o1) = l1;
  *reinterpret_cast<__nv_bfloat162*>(s_ahi + o2) = h2;
  *reinterpret_cast<__nv_bfloat162*>(s_alo + o2) = l2;
}

// A tile's spectra, written as A rows (order 1, order 2 of each pair), by the first
// `team` threads, each one frequency of a range of pairs: the thread's `group` of the
// `groups` that the team makes (formed once per launch). kDegrees: acceptance degrees
// whose coefficients a thread holds, reading them again where the interval changes (0:
// any number, read for every pair).
template <int kDegrees>
LH_DEVICE void flash_tile_spectra(const lh_flash_problem& p, const lh_flash_batch& b,
                                  FlashPair* sp, __nv_bfloat16* s_ahi, __nv_bfloat16* s_alo,
                                  int count, int team, int groups, int group) {
  const int tid = threadIdx.x, nw = p.n_omega;
  if (group >= groups) return;
  const int first = group * count / groups, last = (group + 1) * count / groups;
  for (int w = tid - group * nw; w < nw; w += team) {
    const double om = p.omega[w];
    constexpr int kHeld = kDegrees > 0 ? kDegrees : 1;
    FlashCoef held[kHeld];
    int j_held = -1;
    for (int lp = first; lp < last; ++lp) {
      FlashPair& s = sp[lp];
      float2 s1 = make_float2(0.f, 0.f), s2 = make_float2(0.f, 0.f);
      if (s.j >= 0) {
        if (kDegrees > 0) {
          if (s.j != j_held) {
            j_held = s.j;
#pragma unroll
            for (int l = 0; l < kHeld; ++l) held[l] = flash_coef(p, j_held, l, w);
          }
#pragma unroll
          for (int l = 0; l < kHeld; ++l) flash_degree(held[l], s.tt, s.w[l], s1, s2);
        } else {
          for (int l = 0; l <= p.acc_top; ++l)
            flash_degree(flash_coef(p, s.j, l, w), s.tt, s.w[l], s1, s2);
        }
      }
      flash_rows(p, b, w, om, s, s1, s2, lp, s_ahi, s_alo);
    }
  }
}

// The same for any number of degrees, by runs of kRun neighbouring pairs and one
// frequency: a degree's coefficients are read once for the run's pairs of one interval.
template <int kRun>
LH_DEVICE void flash_tile_runs(const lh_flash_problem& p, const lh_flash_batch& b, FlashPair* sp,
                               __nv_bfloat16* s_ahi, __nv_bfloat16* s_alo, int count, int team) {
  const int nw = p.n_omega, runs = (count + kRun - 1) / kRun;
  for (int i = threadIdx.x; i < runs * nw; i += team) {
    const int run = i / nw, w = i - run * nw;
    FlashPair* q = sp + run * kRun;
    // slots past the count hold no pair; only with a run of 3 may they pass the tile's 64
    const int n = kFlashPairs % kRun ? min(kRun, kFlashPairs - run * kRun) : kRun;
    float2 s1[kRun], s2[kRun];
#pragma unroll
    for (int k = 0; k < kRun; ++k) s1[k] = s2[k] = make_float2(0.f, 0.f);
    for (int l = 0; l <= p.acc_top; ++l) {
      FlashCoef c;
      int j_held = -1;
#pragma unroll
      for (int k = 0; k < kRun; ++k) {
        if (k >= n || q[k].j < 0) continue;
        if (q[k].j != j_held) {
          j_held = q[k].j;
          c = flash_coef(p, j_held, l, w);
        }
        flash_degree(c, q[k].tt, q[k].w[l], s1[k], s2[k]);
      }
    }
    const double om = p.omega[w];
#pragma unroll
    for (int k = 0; k < kRun; ++k)
      if (k < n) flash_rows(p, b, w, om, q[k], s1[k], s2[k], run * kRun + k, s_ahi, s_alo);
  }
}

// The spectra warps' way through a chunk's tiles.
template <int kDegrees>
LH_DEVICE void flash_spectra(const lh_flash_problem& p, const lh_flash_batch& b,
                             FlashPair* sp_buf, __nv_bfloat16* s_ahi, __nv_bfloat16* s_alo,
                             uint64_t* bar_pairs, uint64_t* bar_a, uint64_t* bar_mma, int workers,
                             int n_bins, int in_chunk, int64_t tiles_before, bool& failed) {
  const int tid = threadIdx.x, nw = p.n_omega;
  const int groups = max(1, workers / nw), group = tid / nw;
  const int tiles = (in_chunk + kFlashPairs - 1) / kFlashPairs;
  for (int tile = 0; tile < tiles; ++tile) {
    const int64_t at = tiles_before + tile;
    FlashPair* sp = sp_buf + (at & 1) * kFlashPairs;
    const int count = min(kFlashPairs, in_chunk - tile * kFlashPairs);
    // this tile's pairs are there, and the tensor core has read the last tile's A
    bool ok = warp_wait(bar_pairs + (at & 1), (uint32_t)(at >> 1) & 1u);
    if (ok && at > 0) ok = warp_wait(bar_mma + ((at - 1) & 1), (uint32_t)((at - 1) >> 1) & 1u);
    if (!ok) {
      failed = true;
      return;
    }
    flash_tile_spectra<kDegrees>(p, b, sp, s_ahi, s_alo, count, workers, groups, group);
    fence_proxy_async();  // generic-proxy smem writes -> visible to the tensor core
    __syncwarp();
    if ((tid & 31) == 0) mbar_arrive(bar_a + (at & 1));
    if (tile + 1 == tiles) {  // nothing left to compute: the order-0 rows of the last tile
      if (!warp_wait(bar_a + (at & 1), (uint32_t)(at >> 1) & 1u)) failed = true;
      else flash_tile_order0(p, b, sp, n_bins, tid, workers);
    }
  }
}

// One tile's MMAs (one thread): hi x hi, hi x lo, lo x hi over the K steps.
LH_DEVICE void flash_mma(uint32_t d, const __nv_bfloat16* s_ahi, const __nv_bfloat16* s_alo,
                         const __nv_bfloat16* s_bhi, const __nv_bfloat16* s_blo, int kpad,
                         int n_tile, int passes) {
  const uint32_t idesc = instr_desc_bf16_f32(128, n_tile);
  const int ksteps = kpad / 16;
  const uint32_t lbo_a = kAChunk * 2u, lbo_b = (uint32_t)n_tile * 16u;
  int first = 1;
  for (int pass = 0; pass < passes; ++pass) {
    const __nv_bfloat16* pa = (pass == 2) ? s_alo : s_ahi;
    const __nv_bfloat16* pb = (pass == 1) ? s_blo : s_bhi;
    for (int kk = 0; kk < ksteps; ++kk) {
      uint64_t da = smem_desc_kmajor(reinterpret_cast<const uint8_t*>(pa) + kk * 2 * lbo_a,
                                     lbo_a, 128);
      uint64_t db = smem_desc_kmajor(reinterpret_cast<const uint8_t*>(pb) + kk * 2 * lbo_b,
                                     lbo_b, 128);
      tc_mma_bf16(d, da, db, idesc, first ? 0u : 1u);
      first = 0;
    }
  }
}

// One warp's 32 rows and columns [begin, end) of the accumulator -> components. Four lanes exchange their
// rows' 16 bins, so that they store one row's 64 bytes together and a store
// instruction covers eight rows in whole sectors instead of 32 rows in parts.
LH_DEVICE void flash_drain(const lh_flash_batch& b, const FlashPair* sp, uint32_t d, int quarter,
                           int n_bins, int begin, int end) {
  const int lane = threadIdx.x & 31;
  const int row = quarter * 32 + lane;
  if (!__any_sync(0xffffffffu, sp[row >> 1].valid)) return;
  const uint32_t addr = d + ((uint32_t)(quarter * 32) << 16);
  const bool vec = (n_bins & 3) == 0;
  const bool upper = lane & 2, odd = lane & 1;
  for (int c = begin; c < end; c += 16) {
    float v[16];
    tmem_ld16(addr + (uint32_t)c, v);
    if (vec && c + 16 <= n_bins) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {  // parts 2, 3 of the lower lanes <-> 0, 1 of the upper
        const float got = __shfl_xor_sync(0xffffffffu, upper ? v[i] : v[8 + i], 2);
        if (upper) v[i] = got; else v[8 + i] = got;
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {  // parts 1, 3 of the even lanes <-> 0, 2 of the odd
        const float got0 = __shfl_xor_sync(0xffffffffu, odd ? v[i] : v[4 + i], 1);
        const float got1 = __shfl_xor_sync(0xffffffffu, odd ? v[8 + i] : v[12 + i], 1);
        if (odd) { v[i] = got0; v[8 + i] = got1; } else { v[4 + i] = got0; v[12 + i] = got1; }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {  // part lane & 3 of row 4 (lane / 4) + j
        const int r = quarter * 32 + (lane & ~3) + j;
        const FlashPair& s = sp[r >> 1];
        if (s.valid)
          *reinterpret_cast<float4*>(b.components + (s.pair * 3 + 1 + (r & 1)) * (int64_t)n_bins +
                                     c + 4 * (lane & 3)) =
              make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
      }
    } else if (sp[row >> 1].valid) {
      float* dst = b.components + (sp[row >> 1].pair * 3 + 1 + (row & 1)) * (int64_t)n_bins;
#pragma unroll
      for (int i = 0; i < 16; ++i)
        if (c + i < n_bins) dst[c + i] = v[i];
    }
  }
}

// Shared memory of a fused CTA.
struct FlashSmem {
  uint32_t b_bytes;
  __nv_bfloat16 *ahi, *alo, *bhi, *blo;
  FlashPair* pairs;  // two tiles' pairs
  // operator loaded; then for even and odd tiles: pairs set up, A written, accumulators
  // complete. Each completes once per tile, and only after all its waiters of the tile
  // two before.
  uint64_t *bar_b, *bar_pairs, *bar_a, *bar_mma;
  uint32_t* tmem;
  uint16_t *order, *bucket;  // pairs of the share by interval
  int* count;                // [buckets]
};

LH_DEVICE FlashSmem flash_smem(uint8_t* smem, int kpad, int n_tile) {
  FlashSmem S;
  const uint32_t a_bytes = (uint32_t)(kpad / 8) * kAChunk * 2u;
  S.b_bytes = (uint32_t)n_tile * kpad * 2u;
  S.ahi = reinterpret_cast<__nv_bfloat16*>(smem);
  S.alo = reinterpret_cast<__nv_bfloat16*>(smem + a_bytes);
  S.bhi = reinterpret_cast<__nv_bfloat16*>(smem + 2 * a_bytes);
  S.blo = reinterpret_cast<__nv_bfloat16*>(smem + 2 * a_bytes + S.b_bytes);
  S.pairs = reinterpret_cast<FlashPair*>(smem + 2 * a_bytes + 2 * S.b_bytes);
  S.bar_b = reinterpret_cast<uint64_t*>(S.pairs + 2 * kFlashPairs);
  S.bar_pairs = S.bar_b + 1;
  S.bar_a = S.bar_b + 3;
  S.bar_mma = S.bar_b + 5;
  S.tmem = reinterpret_cast<uint32_t*>(S.bar_b + 7);
  S.order = reinterpret_cast<uint16_t*>(S.bar_b + 8);
  S.bucket = S.order + kFlashSort;
  S.count = reinterpret_cast<int*>(S.bucket + kFlashSort);
  return S;
}

// The whole CTA: lists the `in_chunk` pairs from `chunk` on by radial interval. The
// barriers are the CTA's whether it sorts or not.
LH_DEVICE void flash_sort(const lh_flash_problem& p, const lh_flash_batch& b, const FlashSmem& S,
                          int64_t chunk, int in_chunk, bool sorted) {
  const int tid = threadIdx.x, lane = tid & 31;
  const int buckets = min(p.n_radii + 1, kFlashMaxBuckets);
  for (int i = tid; sorted && i < buckets; i += blockDim.x) S.count[i] = 0;
  __syncthreads();
  for (int i = tid; sorted && i < in_chunk; i += blockDim.x) {
    const int j = flash_bucket(p, b, chunk + i, buckets);
    S.bucket[i] = (uint16_t)j;
    atomicAdd(S.count + j, 1);
  }
  __syncthreads();
  if (sorted && tid < 32) {  // exclusive prefix sums
    int carry = 0;
    for (int first = 0; first < buckets; first += 32) {
      const int v = first + lane < buckets ? S.count[first + lane] : 0;
      int sum = v;
      for (int off = 1; off < 32; off <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, sum, off);
        if (lane >= off) sum += up;
      }
      if (first + lane < buckets) S.count[first + lane] = carry + sum - v;
      carry += __shfl_sync(0xffffffffu, sum, 31);
    }
  }
  __syncthreads();
  for (int i = tid; sorted && i < in_chunk; i += blockDim.x)
    S.order[atomicAdd(S.count + S.bucket[i], 1)] = (uint16_t)i;
  __syncthreads();
}

template <int kDegrees>
__global__ void __launch_bounds__(kFlashTcThreads, 1)
flash_tc_kernel(lh_flash_problem p, lh_flash_batch b, const __nv_bfloat16* __restrict__ g_bhi,
                const __nv_bfloat16* __restrict__ g_blo, int kpad, int n_bins, int n_tile,
                int passes, int sorted) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const FlashSmem S = flash_smem(smem, kpad, n_tile);
  const uint32_t b_bytes = S.b_bytes;
  __nv_bfloat16 *s_ahi = S.ahi, *s_alo = S.alo, *s_bhi = S.bhi, *s_blo = S.blo;
  // a tile's drain sets up the pairs of the tile after next
  FlashPair* sp_buf = S.pairs;
  uint64_t *bar_b = S.bar_b, *bar_pairs = S.bar_pairs, *bar_a = S.bar_a, *bar_mma = S.bar_mma;
  uint32_t* s_tmem = S.tmem;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // roles: spectra (the first warps), drain (four warps), MMA (the last warp)
  const int mma_warp = (int)(blockDim.x >> 5) - 1, drain_warp = mma_warp - 4;
  const int workers = 32 * drain_warp;
  const bool need_lo_b = passes >= 2;
  if (tid == 0) {
    mbar_init(bar_b, 1);
    for (int k = 0; k < 2; ++k) {
      mbar_init(bar_pairs + k, 4);
      mbar_init(bar_a + k, drain_warp);
      mbar_init(bar_mma + k, 1);
    }
    fence_barrier_init();
  }
  const uint32_t d_stride = n_tile <= 128 ? 128u : 256u;  // TMEM columns between accumulators
  if (warp == 0) {
    tmem_alloc(s_tmem, 2 * d_stride);
    tmem_relinquish();
  }
  const int64_t n_pairs = (int64_t)flash_count(b) * p.n_om;
  const int nw = p.n_omega;
  const int padw = kpad - 2 * nw;
  for (int i = tid; i < 128 * padw; i += blockDim.x) {  // columns that no spectrum fills
    const int off = a_offset(i / padw, 2 * nw + i % padw);
    s_ahi[off] = __float2bfloat16_rn(0.f);
    s_alo[off] = __float2bfloat16_rn(0.f);
  }
  fence_proxy_async();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *s_tmem;
  if (tid == 0) {
    mbar_expect_tx(bar_b, b_bytes * (need_lo_b ? 2u : 1u));
    bulk_g2s(s_bhi, g_bhi, b_bytes, bar_b);
    if (need_lo_b) bulk_g2s(s_blo, g_blo, b_bytes, bar_b);
  }
  bool b_ready = false, failed = false;
  int64_t issued = -1;  // the MMA warp's last tile

  // this CTA's share of the pairs
  const int64_t share = (n_pairs + gridDim.x - 1) / gridDim.x;
  const int64_t share_begin = min(n_pairs, (int64_t)blockIdx.x * share);
  const int64_t share_end = min(n_pairs, share_begin + share);
  int64_t tiles_before = 0;  // tiles of the chunks before: the barriers' phases go on
  for (int64_t chunk = share_begin; chunk < share_end && !failed; chunk += kFlashSort) {
    const int in_chunk = (int)min((int64_t)kFlashSort, share_end - chunk);
    flash_sort(p, b, S, chunk, in_chunk, sorted);
    // the pair at place k of the sorted chunk, past its end none
    auto pair_at = [&](int k) {
      return k < in_chunk ? chunk + (sorted ? (int)S.order[k] : k) : n_pairs;
    };
    const int tiles = (in_chunk + kFlashPairs - 1) / kFlashPairs;
    // the first two tiles' pairs
    if (tid < 2 * kFlashPairs && tid / kFlashPairs < tiles)
      flash_slot_setup(p, b,
                       sp_buf[((tiles_before + tid / kFlashPairs) & 1) * kFlashPairs +
                              tid % kFlashPairs],
                       pair_at(tid), n_pairs);
    __syncthreads();
    if (warp < drain_warp) {
      flash_spectra<kDegrees>(p, b, sp_buf, s_ahi, s_alo, bar_pairs, bar_a, bar_mma, workers,
                              n_bins, in_chunk, tiles_before, failed);
    } else if (warp == mma_warp) {
      for (int tile = 0; tile < tiles && !failed; ++tile) {
        const int64_t at = tiles_before + tile;
        const uint32_t parity = (uint32_t)(at >> 1) & 1u;
        if (!b_ready) {
          b_ready = true;
          if (!warp_wait(bar_b, 0)) failed = true;
        }
        if (!failed && !warp_wait(bar_a + (at & 1), parity)) failed = true;
        if (failed) break;
        tc_fence_after();
        if (lane == 0) {
          flash_mma(tmem + (uint32_t)(at & 1) * d_stride, s_ahi, s_alo, s_bhi, s_blo, kpad,
                    n_tile, passes);
          tc_commit(bar_mma + (at & 1));
        }
        __syncwarp();
        issued = at;
      }
    } else {
      const int index = tid - 32 * drain_warp;
      if (lane == 0)
        for (int k = 0; k < min(2, tiles); ++k) mbar_arrive(bar_pairs + ((tiles_before + k) & 1));
      for (int tile = 0; tile < tiles; ++tile) {
        const int64_t at = tiles_before + tile;
        const uint32_t parity = (uint32_t)(at >> 1) & 1u;
        FlashPair* sp = sp_buf + (at & 1) * kFlashPairs;
        bool ok = warp_wait(bar_pairs + (at & 1), parity) && warp_wait(bar_a + (at & 1), parity);
        if (ok && tile + 1 < tiles) flash_tile_order0(p, b, sp, n_bins, index, 128);
        ok = ok && warp_wait(bar_mma + (at & 1), parity);
        if (ok) {
          tc_fence_after();
          flash_drain(b, sp, tmem + (uint32_t)(at & 1) * d_stride, warp & 3, n_bins, 0, n_tile);
          tc_fence_before();
        }
        if (group_sync_or<128>(0, !ok)) {  // all four warps are done with the pairs, or none goes on
          failed = true;
          break;
        }
        if (tile + 2 < tiles) {
          if (index < kFlashPairs)
            flash_slot_setup(p, b, sp[index], pair_at((tile + 2) * kFlashPairs + index), n_pairs);
          __syncwarp();
          if (lane == 0) mbar_arrive(bar_pairs + (at & 1));
        }
      }
    }
    failed = __syncthreads_or(failed);
    tiles_before += tiles;
  }
  if (failed && tid == 0) atomicOr(reinterpret_cast<unsigned*>(b.status), LH_STATUS_TIMEOUT);
  if (warp == mma_warp) {  // nothing in flight when the CTA ends
    if (issued >= 0) mbar_wait(bar_mma + (issued & 1), (uint32_t)(issued >> 1) & 1u);
    if (!b_ready) mbar_wait(bar_b, 0);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 2 * d_stride);
}

// The CTA in step: all warps but the last form a tile's spectra (the last sets up the
// next tile's pairs meanwhile, then issues the MMAs), all write its order-0 rows and all
// drain it. It stays for what the roles slow down:
//  * CTAs of 256 threads, where the roles leave three warps for the spectra: 4000 flashes
//    of 48 OMs with 3 degrees take 0.339 ms against 0.507 (2: 0.305, 0.490), 137 flashes
//    25.6 us against 36.3;
//  * degrees that are not held, whose spectra outweigh the drains: 4000 flashes with 5
//    degrees take 0.392 ms against 0.466 (9: 0.525, 0.673), with 256 threads 0.513 against
//    1.25; 137 flashes with 4 degrees 26.4 us against 28.4.
// Degrees not held are read for every pair, or once per run of pairs where an interval
// has kFlashDense pairs or more on average: with 5 degrees and 512 threads 29.1 against
// 31.1 us at one pair per interval (137 flashes), 46.0 and 45.7 at two (300), 89.4 and
// 81.9 at 4.7 (700). Runs of 3 make three rounds of 480 threads over a tile, runs of 4 five
// of 224: the fewest (512 threads with runs of 4: 84.8).
template <int kDegrees>
__global__ void __launch_bounds__(kFlashTcThreads, 1)
flash_step_kernel(lh_flash_problem p, lh_flash_batch b, const __nv_bfloat16* __restrict__ g_bhi,
                  const __nv_bfloat16* __restrict__ g_blo, int kpad, int n_bins, int n_tile,
                  int passes, int sorted) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const FlashSmem S = flash_smem(smem, kpad, n_tile);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int workers = blockDim.x - 32;
  if (tid == 0) {
    mbar_init(S.bar_b, 1);
    mbar_init(S.bar_mma, 1);
    fence_barrier_init();
  }
  const uint32_t columns = n_tile <= 128 ? 128u : 256u;
  if (warp == 0) {
    tmem_alloc(S.tmem, columns);
    tmem_relinquish();
  }
  const int padw = kpad - 2 * p.n_omega;
  for (int i = tid; i < 128 * padw; i += blockDim.x) {  // columns that no spectrum fills
    const int off = a_offset(i / padw, 2 * p.n_omega + i % padw);
    S.ahi[off] = __float2bfloat16_rn(0.f);
    S.alo[off] = __float2bfloat16_rn(0.f);
  }
  fence_proxy_async();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *S.tmem;
  if (tid == 0) {
    mbar_expect_tx(S.bar_b, S.b_bytes * (passes >= 2 ? 2u : 1u));
    bulk_g2s(S.bhi, g_bhi, S.b_bytes, S.bar_b);
    if (passes >= 2) bulk_g2s(S.blo, g_blo, S.b_bytes, S.bar_b);
  }
  const int64_t n_pairs = (int64_t)flash_count(b) * p.n_om;
  const int64_t share = (n_pairs + gridDim.x - 1) / gridDim.x;
  const int64_t share_begin = min(n_pairs, (int64_t)blockIdx.x * share);
  const int64_t share_end = min(n_pairs, share_begin + share);
  // the drain: warp w reads TMEM lanes 32 (w % 4).., the warps of one lane quarter
  // split the 16-column pieces between them
  const int pieces = (n_tile / 16 + (int)blockDim.x / 128 - 1) / ((int)blockDim.x / 128) * 16;
  const int c_begin = min((warp >> 2) * pieces, n_tile), c_end = min(c_begin + pieces, n_tile);
  const int groups = max(1, workers / p.n_omega), group = tid / p.n_omega;
  bool b_ready = false, failed = false, issued = false;
  uint32_t phase = 0;  // of the accumulator: one tile each
  for (int64_t chunk = share_begin; chunk < share_end && !failed; chunk += kFlashSort) {
    const int in_chunk = (int)min((int64_t)kFlashSort, share_end - chunk);
    flash_sort(p, b, S, chunk, in_chunk, sorted);
    auto pair_at = [&](int k) {
      return k < in_chunk ? chunk + (sorted ? (int)S.order[k] : k) : n_pairs;
    };
    const int tiles = (in_chunk + kFlashPairs - 1) / kFlashPairs;
    const bool dense = sorted && in_chunk >= kFlashDense * p.n_radii;
    if (tid < kFlashPairs) flash_slot_setup(p, b, S.pairs[tid], pair_at(tid), n_pairs);
    __syncthreads();
    for (int tile = 0; tile < tiles; ++tile) {
      FlashPair* sp = S.pairs + (tile & 1) * kFlashPairs;
      const int count = min(kFlashPairs, in_chunk - tile * kFlashPairs);
      if (tid >= workers) {
        if (tile + 1 < tiles)
          for (int k = lane; k < kFlashPairs; k += 32)
            flash_slot_setup(p, b, S.pairs[((tile + 1) & 1) * kFlashPairs + k],
                             pair_at((tile + 1) * kFlashPairs + k), n_pairs);
      } else if (kDegrees > 0 || !dense) {
        flash_tile_spectra<kDegrees>(p, b, sp, S.ahi, S.alo, count, workers, groups, group);
      } else if (workers >= 256) {
        flash_tile_runs<3>(p, b, sp, S.ahi, S.alo, count, workers);
      } else {
        flash_tile_runs<4>(p, b, sp, S.ahi, S.alo, count, workers);
      }
      fence_proxy_async();  // generic-proxy smem writes -> visible to the tensor core
      __syncthreads();
      if (tid >= workers) {
        if (!b_ready) {
          b_ready = true;
          if (!warp_wait(S.bar_b, 0)) failed = true;
        }
        if (!failed) {
          tc_fence_after();
          if (lane == 0) {
            flash_mma(tmem, S.ahi, S.alo, S.bhi, S.blo, kpad, n_tile, passes);
            tc_commit(S.bar_mma);
          }
          __syncwarp();
          issued = true;
        }
      } else {
        flash_tile_order0(p, b, sp, n_bins, tid, workers);
      }
      failed = __syncthreads_or(failed);
      if (failed) break;  // nothing was issued for this tile
      failed = __syncthreads_or(!mbar_wait(S.bar_mma, phase));
      if (failed) break;
      issued = false;
      phase ^= 1u;
      tc_fence_after();
      flash_drain(b, sp, tmem, warp & 3, n_bins, c_begin, c_end);
      tc_fence_before();
      __syncthreads();
    }
  }
  if (failed && tid == 0) atomicOr(reinterpret_cast<unsigned*>(b.status), LH_STATUS_TIMEOUT);
  if (warp == (int)(blockDim.x >> 5) - 1) {  // nothing in flight when the CTA ends
    if (issued) mbar_wait(S.bar_mma, phase);
    if (!b_ready) mbar_wait(S.bar_b, 0);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, columns);
}

// ---------------------------------------------------------------- broadband
// out[i] = the nodes' values in node order, four at a time where every array is
// 16-byte aligned. What bounds it is the copy of (nodes + 1) arrays: one float per
// thread and step kept too few loads on their way (0.175 ms for 337 MB, 501
// flashes of three nodes; 0.052 ms now, 6.4 TB/s).
LH_DEVICE void flash_sum_nodes(const float* const* from, int n_nodes, float* out, int64_t n,
                               int64_t first, int64_t stride) {
  bool aligned = (reinterpret_cast<uintptr_t>(out) & 15) == 0;
  for (int k = 0; k < n_nodes; ++k) aligned &= (reinterpret_cast<uintptr_t>(from[k]) & 15) == 0;
  int64_t done = 0;
  if (aligned) {
    const int64_t quads = n >> 2;
    done = quads << 2;
    constexpr int kAhead = 4;  // steps on their way per thread
    for (int64_t i0 = first; i0 < quads; i0 += kAhead * stride) {
      float4 v[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; ++u) v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int k = 0; k < n_nodes; ++k) {
        const float4* src = reinterpret_cast<const float4*>(from[k]);
        float4 x[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
          if (i0 + u * stride < quads) x[u] = __ldcs(src + i0 + u * stride);
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
          if (i0 + u * stride < quads) {
            v[u].x += x[u].x;
            v[u].y += x[u].y;
            v[u].z += x[u].z;
            v[u].w += x[u].w;
          }
      }
#pragma unroll
      for (int u = 0; u < kAhead; ++u)
        if (i0 + u * stride < quads) reinterpret_cast<float4*>(out)[i0 + u * stride] = v[u];
    }
  }
  for (int64_t i = done + first; i < n; i += stride) {
    float v = 0.f;
    for (int k = 0; k < n_nodes; ++k) v += from[k][i];
    out[i] = v;
  }
}

// Sum of the node runs of a broadband flash and the mask and range check of
// the sum (transport.py:1088-1164). Grid-stride over the spectrum and bins
// (node order fixed: identical results alone or in a batch), then one thread
// per pair: charge, the absorption-only estimate over the nodes, flags.
__global__ void __launch_bounds__(256)
flash_combine_kernel(const __grid_constant__ lh_flash_problem p,
                     const __grid_constant__ lh_flash_nodes nd,
                     const __grid_constant__ lh_flash_batch b) {
  const int64_t n_pairs = (int64_t)flash_count(b) * p.n_om;
  const int nb = p.n_edges - 1;
  const int64_t first = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  flash_sum_nodes(nd.spectrum, nd.n_nodes, b.spectrum, n_pairs * p.n_omega * 6, first, stride);
  flash_sum_nodes(nd.components, nd.n_nodes, b.components, n_pairs * 3 * nb, first, stride);
  for (int64_t pair = first; pair < n_pairs; pair += stride) {
    double q[3] = {0.0, 0.0, 0.0};
    for (int n = 0; n < nd.n_nodes; ++n)
      for (int o = 0; o < 3; ++o) q[o] += nd.charge[n][pair * 3 + o];
    for (int o = 0; o < 3; ++o) b.charge[pair * 3 + o] = q[o];
    // geometry and acceptance as flash_pair_setup
    const int64_t f = pair / p.n_om;
    const int d = (int)(pair % p.n_om);
    const double sx = b.pos[3 * f], sy = b.pos[3 * f + 1], sz = b.pos[3 * f + 2];
    const double px = p.om_pos[3 * d], py = p.om_pos[3 * d + 1], pz = p.om_pos[3 * d + 2];
    const double dx = __dsub_rn(px, sx), dy = __dsub_rn(py, sy), dz = __dsub_rn(pz, sz);
    const double r = sqrt(dot3_rn(dx, dy, dz, dx, dy, dz));
    int flags = 0;
    if (r == 0.0) {
      atomicOr(reinterpret_cast<unsigned*>(b.status), LH_STATUS_COINCIDENT);
      flags |= 4;
    }
    const double tx = __dsub_rn(sx, px), ty = __dsub_rn(sy, py), tz = __dsub_rn(sz, pz);
    const double tn = sqrt(dot3_rn(tx, ty, tz, tx, ty, tz));
    const double cosine = dot3_rn(p.om_look[3 * d], p.om_look[3 * d + 1], p.om_look[3 * d + 2],
                                  tx / tn, ty / tn, tz / tn);
    double pl_prev = 1.0, pl = cosine, acc = 0.0;
    for (int l = 0; l <= p.acc_top; ++l) {
      double P;
      if (l == 0) P = 1.0;
      else if (l == 1) P = cosine;
      else {
        P = ((2 * l - 1) * cosine * pl - (l - 1) * pl_prev) / l;
        pl_prev = pl;
        pl = P;
      }
      acc += p.alpha[l] * (2 * l + 1) * P / (4 * kPi);
    }
    const double four_pi_r2 = 4 * kPi * r * r;
    double upper = 0.0;
    for (int n = 0; n < nd.n_nodes; ++n)
      upper += nd.photons[n][f] * p.om_area[d] * nd.efficiency[n] * acc *
               exp(-nd.absorption[n] * r) / four_pi_r2;
    const bool inside = (r >= p.r_low) && (r <= p.r_high);
    if (!inside && 10 * upper >= p.threshold) {
      flags |= 2;
      atomicOr(reinterpret_cast<unsigned*>(b.status), LH_STATUS_UNSAFE);
      atomicAdd(b.status + 1, 1);
      atomicMax(reinterpret_cast<unsigned long long*>(b.status + 2),
                (unsigned long long)__double_as_longlong(r));
    }
    const double total = (q[0] + q[1]) + q[2];
    const bool active = p.threshold == 0.0 ? inside : (inside && total >= p.threshold);
    b.active[pair] = (uint8_t)((active ? 1 : 0) | flags);
  }
}

size_t flash_tc_smem_bytes(int kpad, int n_tile, bool sorted) {
  return 2ull * (kpad / 8) * kAChunk * 2 + 2ull * n_tile * kpad * 2 +
         2 * sizeof(FlashPair) * kFlashPairs + 64 +
         (sorted ? 2 * sizeof(uint16_t) * kFlashSort + sizeof(int) * kFlashMaxBuckets : 0);
}

// The instance for a CTA of `threads` and `degrees` acceptance degrees: roles where two
// or three degrees are held by a CTA of 512, else in step.
FlashTcKernel flash_tc_kernel_of(int degrees, int threads) {
  switch (degrees) {
    case 2: return threads == 512 ? flash_tc_kernel<2> : flash_step_kernel<2>;
    case 3: return threads == 512 ? flash_tc_kernel<3> : flash_step_kernel<3>;
    default: return flash_step_kernel<0>;
  }
}

}  // namespace lh
