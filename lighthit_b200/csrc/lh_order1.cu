// Order 1 (single scattering) of spectral elements, grouped pencils.
//
// Reference: transport_prompt's grouped order 1 (prompt.py:1020-1258) with
//   stage A  compress (prompt.py:1317-1402): subsegment_cells,
//            compress_subsegments, finish_pencils (_prompt_numba.py:1094-1232,
//            2247-2354): every element is cut into ceil(L / a_step)
//            sub-segments, each sub-segment's Cherenkov ring is sampled at
//            `ring_nodes` azimuths, and the nodes are summed into
//            (0.5 m position cell, cube-sphere direction pixel) pencils that
//            carry 23 moments (weights, mean position/time/direction and their
//            covariances);
//   stage B  grouped_pencils_order1 (_prompt_numba.py:1750-2086): for each OM
//            the pencils are merged into (tau, log r, hemisphere, theta) groups
//            carrying acceptance moments; the groups of one (tau, r) batch
//            share a path grid in asinh((S - r) / sigma), their single-
//            scattering profile is summed on it, and the profile is deposited
//            per wavelength band as exact exp x quadratic panels into the bins
//            (_batch_grid, _batch_add_moments, _batch_deposit, _deposit_panel,
//            _finalize: _prompt_numba.py:157-632).
//
// B200 layout. Stage A: one thread per ring node writes its moments into a
// global open-addressing table keyed by (cell, pixel) with float64 atomics;
// one thread per occupied slot then forms the pencil. Stage B: one thread per
// (OM, pencil) computes the pencil's geometry against the OM and adds its
// moments into that OM's group table (atomics); one CTA per OM sorts its
// group keys in shared memory (bitonic) and emits its batches; a persistent
// grid of warps takes batches from the global list, builds each batch's path
// grid and profile and deposits its panels (batches too long for a warp go to
// CTAs); one CTA per OM finishes the bins by prefix scans. Everything is float64, as the
// deposit's global quadratic coefficients in t cancel strongly.
#include <algorithm>

#include "lh_common.cuh"
#include "lh_timing.cuh"

namespace lh {

constexpr int kO1MaxNodes = 2048;
constexpr int kO1MaxMono = 10;
constexpr int kO1MaxValues = 2 * kO1MaxMono + 6;
constexpr int kO1MaxBands = 8;
constexpr int kO1MaxGauss = 64;
constexpr int kO1Moments = 23;
constexpr int kO1SmemSort = 16384;  // group tables up to this size sort in shared memory
constexpr int kO1BatchThreads = 128;

LH_DEVICE uint64_t o1_mix(uint64_t v) {
  v = (v ^ (v >> 30)) * 0xbf58476d1ce4e5b9ull;
  v = (v ^ (v >> 27)) * 0x94d049bb133111ebull;
  return v ^ (v >> 31);
}

// A slot whose claiming thread is still zeroing its row holds its key with
// this bit set (keys stay below 2^62).
constexpr long long kO1Busy = 1ll << 62;
constexpr long long kO1ClaimWaitNs = 100000000ll;  // a wait for a claimed row gives up after 0.1 s

// Insert `key` (>= 0) into an open-addressing table of `capacity` (power of
// two) slots holding -1 when free, whose rows of `n` doubles at `rows` are
// not cleared beforehand: the thread that claims a free slot marks it busy,
// zeroes the slot's row, then publishes the key; a thread that finds its key
// still busy waits for the publication (bounded: past kO1ClaimWaitNs it sets
// LH_STATUS_TIMEOUT and returns -1). Returns the slot, or -1 when the table
// is full (LH_STATUS_OVERFLOW); `fresh` tells whether this call claimed it.
// Only the rows of published slots are ever read.
LH_DEVICE int64_t o1_insert(long long* keys, int64_t capacity, long long key, double* rows,
                            int n, bool& fresh, int32_t* status, bool ordered = false) {
  const uint64_t mask = (uint64_t)capacity - 1;
  uint64_t slot = (ordered ? (uint64_t)key : o1_mix((uint64_t)key)) & mask;
  fresh = false;
  unsigned long long* word = reinterpret_cast<unsigned long long*>(keys);
  for (int64_t probe = 0; probe < capacity; ++probe) {
    const long long prev = (long long)atomicCAS(word + slot, (unsigned long long)(-1ll),
                                                (unsigned long long)(key | kO1Busy));
    if (prev == -1ll) {
      double* row = rows + (int64_t)slot * n;
      for (int k = 0; k < n; ++k) row[k] = 0.0;
      __threadfence();  // the zeros reach the device before the key does
      atomicExch(word + slot, (unsigned long long)key);
      fresh = true;
      return (int64_t)slot;
    }
    if (prev == key) return (int64_t)slot;
    if (prev == (key | kO1Busy)) {
      const unsigned long long began = global_ns();
      for (int poll = 0;; ++poll) {
        if ((long long)atomicAdd(word + slot, 0ull) == key) {
          __threadfence();  // the row's zeros before this thread's additions
          return (int64_t)slot;
        }
        if ((poll & 63) == 63 && (long long)(global_ns() - began) > kO1ClaimWaitNs) {
          atomicOr(reinterpret_cast<unsigned*>(status), LH_STATUS_TIMEOUT);
          return -1;
        }
      }
    }
    slot = (slot + 1) & mask;
  }
  atomicOr(reinterpret_cast<unsigned*>(status), LH_STATUS_OVERFLOW);
  return -1;
}

// ------------------------------------------------------------------ stage A

// Pixel row of a face coordinate u in [-1, 1]: (atan(u) + pi/4) / (pi/2) * n_face,
// truncated and clamped. The float32 arctangent of the float32 quotient decides it
// wherever that is further than 1e-3 from a whole number (its error is below 3e-4
// for up to 512 pixels), the float64 expression elsewhere, so the result is the
// float64 one.
LH_DEVICE int o1_pixel_row(double num, double den, int n_face) {
  constexpr float quarter_f = 0.78539816f, scale_f = 0.63661977f;  // pi / 4, 2 / pi
  const float v = (atanf(__fdividef((float)num, (float)den)) + quarter_f) * (scale_f * n_face);
  const float f = floorf(v), part = v - f;
  int i;
  if (n_face <= 512 && part > 1e-3f && part < 1.0f - 1e-3f) {
    i = (int)f;
  } else {
    const double quarter = 0.25 * kPi;
    i = (int)((atan(num / den) + quarter) / (2.0 * quarter) * n_face);
  }
  return min(max(i, 0), n_face - 1);
}

// Equi-angular cube-sphere pixel (_prompt_numba.py:1015-1043)
LH_DEVICE int o1_pixel(double sx, double sy, double sz, int n_face) {
  const double ax = fabs(sx), ay = fabs(sy), az = fabs(sz);
  int face;
  double u, v, major;
  if (ax >= ay && ax >= az) {
    face = sx > 0 ? 0 : 1; u = sy; v = sz; major = ax;
  } else if (ay >= az) {
    face = sy > 0 ? 2 : 3; u = sx; v = sz; major = ay;
  } else {
    face = sz > 0 ? 4 : 5; u = sx; v = sy; major = az;
  }
  return (face * n_face + o1_pixel_row(u, major, n_face)) * n_face +
         o1_pixel_row(v, major, n_face);
}

struct O1Subseg {
  double px, py, pz, t;
};

LH_DEVICE O1Subseg o1_subseg(const lh_order1_elements& E, int64_t i, int64_t ia, int64_t n_a) {
  const double frac = (ia + 0.5) / n_a;
  O1Subseg s;
  s.px = E.start[3 * i] + frac * E.length[i] * E.direction[3 * i];
  s.py = E.start[3 * i + 1] + frac * E.length[i] * E.direction[3 * i + 1];
  s.pz = E.start[3 * i + 2] + frac * E.length[i] * E.direction[3 * i + 2];
  s.t = E.t0[i] + frac * (E.t1[i] - E.t0[i]);
  return s;
}

// Warp-level sums by key: every lane writes its n values to its row of the
// warp's staging area (`stage`, 32 rows of n doubles in shared memory), and
// each group of lanes with equal keys (`group`, a __match_any_sync mask; its
// lowest lane the `leader`, holding the group's `row`) adds its members' rows
// in lane order with one atomic per value. The warp takes several groups at a
// time (five of 18 values, four of 23: a lane sums three values of one group),
// so that an atomic instruction covers whole sectors of a few rows. With each
// leader adding its own group's values instead, which warps of more than 16
// groups did, every atomic instruction touched as many sectors as groups: the
// ring stage of 1.3M nodes (about 20 groups per warp) took 0.255 ms, now 0.13 ms.
LH_DEVICE void o1_warp_group_add(double* stage, int n, unsigned group, bool leader, double* row) {
  __syncwarp();
  const unsigned full = 0xffffffffu;
  unsigned leaders = __ballot_sync(full, leader && row != nullptr);
  const int lane = threadIdx.x & 31;
  const int per = (n + 2) / 3, at_once = min(32 / per, 5);  // lanes per group, groups at a time
  const int place = lane / per, k = lane - place * per;
  while (leaders) {
    int src = __ffs(leaders) - 1;
    leaders &= leaders - 1;
    bool mine = place == 0;
#pragma unroll
    for (int i = 1; i < 5; ++i)
      if (i < at_once && leaders) {  // the same for the whole warp
        const int next = __ffs(leaders) - 1;
        leaders &= leaders - 1;
        if (place == i) {
          src = next;
          mine = true;
        }
      }
    unsigned members = __shfl_sync(full, group, src);
    double* target = reinterpret_cast<double*>(
        __shfl_sync(full, reinterpret_cast<unsigned long long>(row), src));
    if (!mine) continue;
    const bool third = k + 2 * per < n;
    const double* from = stage + k;
    double sum0 = 0.0, sum1 = 0.0, sum2 = 0.0;
    for (; members; members &= members - 1) {
      const double* value = from + (__ffs(members) - 1) * n;
      sum0 += value[0];
      sum1 += value[per];
      if (third) sum2 += value[2 * per];
    }
    atomicAdd(target + k, sum0);
    atomicAdd(target + k + per, sum1);
    if (third) atomicAdd(target + k + 2 * per, sum2);
  }
  __syncwarp();
}

constexpr int kO1RingBlock = 4;     // ring nodes per thread
constexpr int kO1RingThreads = 256;

// One thread per (sub-segment, block of kO1RingBlock ring nodes):
// compress_subsegments (_prompt_numba.py:1122-1232) with the ring rotation
// evaluated directly. The lanes of a warp hold consecutive sub-segments and
// take the same ring node together, so nodes that land in the same (cell,
// pixel) (neighbouring steps of a track or shower) are summed in registers
// first: one hash insert and one set of moment atomics per distinct key and warp.
__global__ void __launch_bounds__(kO1RingThreads, 3)
o1_ring_kernel(const lh_order1_config C, const lh_order1_elements E,
                               const int64_t* subseg_offset, int64_t n_subseg,
                               long long* keys, int64_t capacity, double* rows,
                               int32_t* status) {
  const int n_pix = 6 * C.pixel_face * C.pixel_face;
  const double golden = 0.6180339887498949;
  const double two_pi = 2.0 * kPi;
  const int lane = threadIdx.x & 31;
  const int64_t n_pad = (n_subseg + 31) & ~(int64_t)31;  // warps never straddle node blocks
  const int n_blocks = (C.ring_nodes + kO1RingBlock - 1) / kO1RingBlock;
  const int64_t total = n_pad * n_blocks;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  __shared__ double s_stage[kO1RingThreads / 32][32 * kO1Moments];
  double* stage = s_stage[threadIdx.x >> 5];
  double step_s, step_c;
  sincos(two_pi / C.ring_nodes, &step_s, &step_c);
  const double guess = (double)E.n_el / (double)n_subseg;
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < total; k += stride) {
    const int64_t sub = k % n_pad;
    const int q_begin = (int)(k / n_pad) * kO1RingBlock;
    const int q_end = min(q_begin + kO1RingBlock, C.ring_nodes);
    const bool live = sub < n_subseg;
    double ux = 0, uy = 0, uz = 1, e1x = 1, e1y = 0, e1z = 0, e2x = 0, e2y = 1, e2z = 0;
    double cc = 0, cs = 0, arc2 = 0, sub2 = 0, w0 = 0, w2 = 0, offset = 0;
    O1Subseg P{};
    long long cell = 0;
    if (live) {
      // element of this sub-segment: last i with subseg_offset[i] <= sub. Short
      // elements hold one each, so the proportional guess is mostly right.
      int64_t lo = min((int64_t)((double)sub * guess), (int64_t)E.n_el - 1);
      if (!(subseg_offset[lo] <= sub && sub < subseg_offset[lo + 1])) {
        int64_t hi = E.n_el;
        lo = 0;
        while (hi - lo > 1) {
          int64_t mid = (lo + hi) >> 1;
          if (subseg_offset[mid] <= sub) lo = mid; else hi = mid;
        }
      }
      const int64_t i = lo;
      const int64_t ia = sub - subseg_offset[i];
      const int64_t n_a = subseg_offset[i + 1] - subseg_offset[i];
      ux = E.direction[3 * i]; uy = E.direction[3 * i + 1]; uz = E.direction[3 * i + 2];
      double hx, hy, hz;
      if (fabs(uz) < 0.9) { hx = 0.0; hy = 0.0; hz = 1.0; } else { hx = 1.0; hy = 0.0; hz = 0.0; }
      e1x = uy * hz - uz * hy; e1y = uz * hx - ux * hz; e1z = ux * hy - uy * hx;
      const double inv_norm = rsqrt(e1x * e1x + e1y * e1y + e1z * e1z);
      e1x *= inv_norm; e1y *= inv_norm; e1z *= inv_norm;
      e2x = uy * e1z - uz * e1y; e2y = uz * e1x - ux * e1z; e2z = ux * e1y - uy * e1x;
      cc = E.cone_cos[i];
      cs = sqrt(fmax(1.0 - cc * cc, 0.0));
      const double share = 1.0 / ((double)n_a * C.ring_nodes);
      const double arc = two_pi * cs / C.ring_nodes;
      arc2 = arc * arc / 12.0;
      const double sl = E.length[i] / n_a;
      sub2 = sl * sl / 12.0;
      w0 = E.c0[i] * share;
      w2 = E.c2[i] * share;
      const double ig = (double)i * golden;
      offset = (ig - floor(ig)) * two_pi / C.ring_nodes;
      P = o1_subseg(E, i, ia, n_a);
      const long long cx = min(max((long long)floor((P.px - E.grid_origin[0]) / C.cell_m), 0ll), (long long)E.grid_dims[0] - 1);
      const long long cy = min(max((long long)floor((P.py - E.grid_origin[1]) / C.cell_m), 0ll), (long long)E.grid_dims[1] - 1);
      const long long cz = min(max((long long)floor((P.pz - E.grid_origin[2]) / C.cell_m), 0ll), (long long)E.grid_dims[2] - 1);
      cell = (cx * E.grid_dims[1] + cy) * E.grid_dims[2] + cz;
    }
    const double px = P.px, py = P.py, pz = P.pz, t = P.t;
    double sp, cp;
    sincos(offset + two_pi * q_begin / C.ring_nodes, &sp, &cp);
    for (int q = q_begin; q < q_end; ++q) {
      if (q > q_begin) {  // the next node: one step of the ring
        const double turned = cp * step_c - sp * step_s;
        sp = sp * step_c + cp * step_s;
        cp = turned;
      }
      const double sx = cc * ux + cs * (cp * e1x + sp * e2x);
      const double sy = cc * uy + cs * (cp * e1y + sp * e2y);
      const double sz = cc * uz + cs * (cp * e1z + sp * e2z);
      const long long key = live ? cell * n_pix + o1_pixel(sx, sy, sz, C.pixel_face) : -1ll;
      const unsigned group = __match_any_sync(0xffffffffu, key);
      const bool leader = live && lane == __ffs(group) - 1;
      double* row = nullptr;
      if (leader) {
        bool fresh;
        // slots in key order (keys of one cell are contiguous) so that the
        // compacted pencils come out spatially ordered
        const int64_t slot = o1_insert(keys, capacity, key, rows, kO1Moments, fresh, status, true);
        if (slot >= 0) row = rows + slot * kO1Moments;
      }
      const double tx = -sp * e1x + cp * e2x, ty = -sp * e1y + cp * e2y, tz = -sp * e1z + cp * e2z;
      const double m[kO1Moments] = {
          w0, w2, w0 * px, w0 * py, w0 * pz, w0 * t, w0 * sx, w0 * sy, w0 * sz,
          w0 * (px * px + py * py + pz * pz + sub2), w0 * t * t,
          w0 * (sx * sx + arc2 * tx * tx), w0 * (sy * sy + arc2 * ty * ty),
          w0 * (sz * sz + arc2 * tz * tz), w0 * (sx * sy + arc2 * tx * ty),
          w0 * (sx * sz + arc2 * tx * tz), w0 * (sy * sz + arc2 * ty * tz),
          w0 * (px * px + sub2 * ux * ux), w0 * (py * py + sub2 * uy * uy),
          w0 * (pz * pz + sub2 * uz * uz), w0 * (px * py + sub2 * ux * uy),
          w0 * (px * pz + sub2 * ux * uz), w0 * (py * pz + sub2 * uy * uz)};
      double* mine = stage + lane * kO1Moments;
#pragma unroll
      for (int k = 0; k < kO1Moments; ++k) mine[k] = m[k];
      o1_warp_group_add(stage, kO1Moments, group, leader, row);
    }
  }
}

// Ring-table slots per compaction CTA. The fullest tile decides when the finish ends:
// 35.3 us for the screen's passes with 4096, 24.6 with 2048 and with 1024, whose counts
// of 16.8M slots take longer (8 showers: 0.25, 0.18 and 0.28 ms).
constexpr int kO1Tile = 2048;
constexpr int kO1FinishThreads = 256;  // slots t, t + 256, ... of the tile for thread t

LH_DEVICE bool o1_slot_used(const long long* keys, const double* rows, int64_t slot) {
  return keys[slot] != -1ll && rows[slot * kO1Moments] > 0.0;
}

// Exclusive prefix sum of `v` over the CTA (blockDim a multiple of 32, at most
// 1024); `total` receives the CTA's sum.
LH_DEVICE int o1_block_exclusive_scan(int v, int& total) {
  __shared__ int warp_sums[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n_warps = blockDim.x >> 5;
  int inclusive = v;
  for (int off = 1; off < 32; off <<= 1) {
    const int up = __shfl_up_sync(0xffffffffu, inclusive, off);
    if (lane >= off) inclusive += up;
  }
  __syncthreads();  // warp_sums may still be read by a previous call
  if (lane == 31) warp_sums[warp] = inclusive;
  __syncthreads();
  if (warp == 0) {
    int w = lane < n_warps ? warp_sums[lane] : 0;
    for (int off = 1; off < 32; off <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, w, off);
      if (lane >= off) w += up;
    }
    warp_sums[lane] = w;  // inclusive over warps
  }
  __syncthreads();
  total = warp_sums[n_warps - 1];
  return inclusive - v + (warp ? warp_sums[warp - 1] : 0);
}

// The slot of `key` in an ordered-start table, or -1 when absent.
LH_DEVICE int64_t o1_find(const long long* keys, int64_t capacity, long long key) {
  const uint64_t mask = (uint64_t)capacity - 1;
  uint64_t slot = (uint64_t)key & mask;
  for (int64_t probe = 0; probe < capacity; ++probe) {
    const long long k = keys[slot];
    if (k == key) return (int64_t)slot;
    if (k == -1ll) return -1;
    slot = (slot + 1) & mask;
  }
  return -1;
}

// parent_keys (_prompt_screen.py:44-54): the pixel of the nested parent face
// in the same position cell.
LH_DEVICE long long o1_parent_key(long long key, int face, int parent_face) {
  const long long per_cell = 6ll * face * face;
  const long long cell = key / per_cell, pixel = key % per_cell;
  const long long cube = pixel / ((long long)face * face), ij = pixel % ((long long)face * face);
  const long long i = ij / face, j = ij % face, factor = face / parent_face;
  return cell * (6ll * parent_face * parent_face) + (cube * parent_face + i / factor) * parent_face +
         j / factor;
}

// compress_screen's parents (_prompt_screen.py:56-85): every occupied child
// slot adds its moments to its parent pixel's slot (the parents of one cell
// are the sums of its children, as finish_pencils sums them).
__global__ void __launch_bounds__(kO1FinishThreads)
o1_parent_kernel(const long long* keys, const double* rows, int64_t capacity, int face,
                 int parent_face, long long* parent_keys, double* parent_rows,
                 int64_t parent_capacity, int32_t* status) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t slot = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; slot < capacity;
       slot += stride) {
    const long long key = keys[slot];
    if (key == -1ll) continue;
    bool fresh;
    const int64_t ps = o1_insert(parent_keys, parent_capacity,
                                 o1_parent_key(key, face, parent_face), parent_rows, kO1Moments,
                                 fresh, status, true);
    if (ps < 0) continue;
    for (int k = 0; k < kO1Moments; ++k)
      atomicAdd(parent_rows + ps * kO1Moments + k, rows[slot * kO1Moments + k]);
  }
}

// Pencils of a screen table: parents plus children.
__global__ void o1_total_kernel(const int32_t* children, const int32_t* parents, int32_t* total) {
  if (threadIdx.x == 0 && blockIdx.x == 0) *total = *children + *parents;
}

// Used slots per tile of the ring table. Thread t takes slots t, t + 256, ...
// of its tile, so that a warp's key loads are contiguous.
__global__ void __launch_bounds__(kO1FinishThreads)
o1_tile_count_kernel(const long long* keys, const double* rows, int64_t capacity,
                     int32_t* tile_count) {
  constexpr int per = kO1Tile / kO1FinishThreads;
  const int64_t tile0 = blockIdx.x * (int64_t)kO1Tile + threadIdx.x;
  int mine = 0;
#pragma unroll
  for (int j = 0; j < per; ++j) {
    const int64_t slot = tile0 + (int64_t)j * kO1FinishThreads;
    if (slot < capacity && o1_slot_used(keys, rows, slot)) ++mine;
  }
  int total;
  o1_block_exclusive_scan(mine, total);
  if (threadIdx.x == 0) tile_count[blockIdx.x] = total;
}

// Exclusive tile offsets (in place) and the pencil count, in one CTA.
__global__ void __launch_bounds__(1024)
o1_tile_scan_kernel(int32_t* tile, int64_t n_tiles, int32_t* count) {
  int carry = 0;
  for (int64_t base = 0; base < n_tiles; base += blockDim.x) {
    const int64_t i = base + threadIdx.x;
    const int v = i < n_tiles ? tile[i] : 0;
    int total;
    const int before = o1_block_exclusive_scan(v, total);
    if (i < n_tiles) tile[i] = carry + before;
    carry += total;
  }
  if (threadIdx.x == 0) *count = carry;
}

LH_DEVICE void o1_write_pencil(const double* a, lh_order1_pencil_table& Pn, int q);

// finish_pencils (_prompt_numba.py:2247-2354) for slots with a positive weight,
// compacted into the pencil table in slot order: one CTA per tile ranks its used
// slots (a CTA scan plus the tile's offset), lists them, and takes one per thread.
// Slot order follows the keys, so pencils of a cell are neighbours in the table.
// What bounds it is the float64 chain of a pencil (an eigenbasis with sincos and
// atan2). Used slots are few in a hundred: with each thread finishing its own slots,
// round by round, a warp ran that chain 16 times for a lane or two each (82.7 us for
// 94509 pencils in 2.1M slots, 44.4 from the list).
// Screen tables (the coarse charge screen) take their parents first: parent
// rows [0, n_parents) record their row per slot in `slot_row`; child rows
// follow from `base_count` and look up their parent's row by its key.
__global__ void __launch_bounds__(kO1FinishThreads)
o1_finish_kernel(const long long* keys, int64_t capacity, const double* rows,
                 lh_order1_pencil_table Pn, const int32_t* tile_offset, const int32_t* count,
                 const int32_t* base_count, int32_t* slot_row, const long long* parent_keys,
                 int64_t parent_capacity, const int32_t* parent_row, int face, int parent_face,
                 int32_t* status) {
  constexpr int per = kO1Tile / kO1FinishThreads;  // rounds of 256 consecutive slots
  constexpr int warps = kO1FinishThreads / 32;
  constexpr int counts = per * warps / 32;  // (round, warp) counts per lane of the scan
  static_assert(per <= 32 && per * warps % 32 == 0, "one 32-bit mask per thread");
  __shared__ int before[per * warps];  // used slots ahead of each (round, warp) in the tile
  __shared__ uint16_t list[kO1Tile];   // the used slots in slot order
  __shared__ int in_tile;
  const int64_t n = *count;
  const int64_t base = base_count ? *base_count : 0;
  if (base + n > Pn.capacity) {  // the caller redoes the stage with a larger table
    if (blockIdx.x == 0 && threadIdx.x == 0)
      atomicOr(reinterpret_cast<unsigned*>(status), LH_STATUS_OVERFLOW);
    return;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t tile0 = blockIdx.x * (int64_t)kO1Tile + threadIdx.x;
  unsigned used = 0;  // bit j: this thread's slot of round j holds a pencil
#pragma unroll
  for (int j = 0; j < per; ++j) {
    const int64_t slot = tile0 + (int64_t)j * kO1FinishThreads;
    if (slot < capacity && o1_slot_used(keys, rows, slot)) used |= 1u << j;
  }
#pragma unroll
  for (int j = 0; j < per; ++j) {
    const unsigned b = __ballot_sync(0xffffffffu, (used >> j) & 1u);
    if (lane == 0) before[j * warps + warp] = __popc(b);
  }
  __syncthreads();
  if (warp == 0) {  // exclusive scan of the (round, warp) counts in slot order
    int v[counts], sum = 0;
    for (int i = 0; i < counts; ++i) {
      v[i] = before[counts * lane + i];
      sum += v[i];
    }
    int inclusive = sum;
    for (int off = 1; off < 32; off <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, inclusive, off);
      if (lane >= off) inclusive += up;
    }
    int running = inclusive - sum;
    if (lane == 31) in_tile = inclusive;
    for (int i = 0; i < counts; ++i) {
      before[counts * lane + i] = running;
      running += v[i];
    }
  }
  __syncthreads();
  const unsigned lower = (1u << lane) - 1u;
#pragma unroll
  for (int j = 0; j < per; ++j) {
    const unsigned b = __ballot_sync(0xffffffffu, (used >> j) & 1u);
    if ((used >> j) & 1u)
      list[before[j * warps + warp] + __popc(b & lower)] =
          (uint16_t)(j * kO1FinishThreads + threadIdx.x);
  }
  __syncthreads();
  // rank order = slot order: a cell's pencils are neighbours in the table, so that
  // the 32 pencils of a stage-B warp share their groups (about four items per group
  // against one for a random order) and the warp sums them before the atomics
  const int64_t tile = blockIdx.x * (int64_t)kO1Tile;
  const int64_t row0 = base + tile_offset[blockIdx.x];
  for (int i = threadIdx.x; i < in_tile; i += kO1FinishThreads) {
    const int64_t slot = tile + list[i];
    const int row = (int)(row0 + i);
    o1_write_pencil(rows + slot * kO1Moments, Pn, row);
    if (slot_row) slot_row[slot] = row;
    if (Pn.parent) {
      int32_t parent = -1;
      if (parent_keys) {
        const int64_t ps = o1_find(parent_keys, parent_capacity,
                                   o1_parent_key(keys[slot], face, parent_face));
        if (ps < 0) atomicOr(reinterpret_cast<unsigned*>(status), LH_STATUS_OVERFLOW);
        else parent = parent_row[ps];
      }
      Pn.parent[row] = parent;
    }
  }
}

LH_DEVICE void o1_write_pencil(const double* a, lh_order1_pencil_table& Pn, int q) {
  {
    const double w = a[0];
    const double mx = a[2] / w, my = a[3] / w, mz = a[4] / w;
    Pn.position[3 * q] = mx; Pn.position[3 * q + 1] = my; Pn.position[3 * q + 2] = mz;
    Pn.time[q] = a[5] / w;
    Pn.w0[q] = w;
    Pn.w2[q] = a[1];
    const double rx = a[6] / w, ry = a[7] / w, rz = a[8] / w;
    const double norm = sqrt(rx * rx + ry * ry + rz * rz);
    const double dx = rx / norm, dy = ry / norm, dz = rz / norm;
    Pn.direction[3 * q] = dx; Pn.direction[3 * q + 1] = dy; Pn.direction[3 * q + 2] = dz;
    const double cxx = a[11] / w - rx * rx, cyy = a[12] / w - ry * ry, czz = a[13] / w - rz * rz;
    const double cxy = a[14] / w - rx * ry, cxz = a[15] / w - rx * rz, cyz = a[16] / w - ry * rz;
    double hx, hy, hz;
    if (fabs(dz) < 0.9) { hx = 0.0; hy = 0.0; hz = 1.0; } else { hx = 1.0; hy = 0.0; hz = 0.0; }
    double e1x = dy * hz - dz * hy, e1y = dz * hx - dx * hz, e1z = dx * hy - dy * hx;
    const double nn = sqrt(e1x * e1x + e1y * e1y + e1z * e1z);
    e1x /= nn; e1y /= nn; e1z /= nn;
    const double e2x = dy * e1z - dz * e1y, e2y = dz * e1x - dx * e1z, e2z = dx * e1y - dy * e1x;
    const double c11 = e1x * (cxx * e1x + cxy * e1y + cxz * e1z) + e1y * (cxy * e1x + cyy * e1y + cyz * e1z) +
                       e1z * (cxz * e1x + cyz * e1y + czz * e1z);
    const double c22 = e2x * (cxx * e2x + cxy * e2y + cxz * e2z) + e2y * (cxy * e2x + cyy * e2y + cyz * e2z) +
                       e2z * (cxz * e2x + cyz * e2y + czz * e2z);
    const double c12 = e1x * (cxx * e2x + cxy * e2y + cxz * e2z) + e1y * (cxy * e2x + cyy * e2y + cyz * e2z) +
                       e1z * (cxz * e2x + cyz * e2y + czz * e2z);
    const double half = 0.5 * (c11 + c22);
    const double disc = sqrt(fmax(0.25 * (c11 - c22) * (c11 - c22) + c12 * c12, 0.0));
    Pn.var_major[q] = fmax(half + disc, 0.0);
    Pn.var_minor[q] = fmax(half - disc, 0.0);
    double sa, ca;
    sincos(0.5 * atan2(2.0 * c12, c11 - c22), &sa, &ca);
    Pn.major[3 * q] = ca * e1x + sa * e2x;
    Pn.major[3 * q + 1] = ca * e1y + sa * e2y;
    Pn.major[3 * q + 2] = ca * e1z + sa * e2z;
    Pn.pos_cov[6 * q] = fmax(a[17] / w - mx * mx, 0.0);
    Pn.pos_cov[6 * q + 1] = fmax(a[18] / w - my * my, 0.0);
    Pn.pos_cov[6 * q + 2] = fmax(a[19] / w - mz * mz, 0.0);
    Pn.pos_cov[6 * q + 3] = a[20] / w - mx * my;
    Pn.pos_cov[6 * q + 4] = a[21] / w - mx * mz;
    Pn.pos_cov[6 * q + 5] = a[22] / w - my * mz;
  }
}

// ------------------------------------------------------------------ stage B

// Node sums of the Gaussian inverse-radius measure shared by
// gauss_inverse_mean_prepared (_prompt_numba.py:115-129) and
// inverse_radius_rule (_prompt_screen.py:101-140), for every lane of `need`
// (arguments u, v, var_u, var_v): the warp evaluates one lane's nodes at a
// time, lane j taking nodes j, j + 32, ..., and a butterfly reduction adds
// them, so a lane that needs the 48-node sum does not run it alone while the
// rest of its warp waits. Each lane of `need` receives s0 = 1 / sqrt(scale),
// scale = 2 (var_u + var_v) + u^2 + v^2 (its sums stay 0 when scale <= 0),
// the sum of the node masses and of mass x the radial second moment. Call
// with the whole warp; the second moment only with kRadial.
template <bool kRadial>
LH_DEVICE void o1_node_sums(unsigned need, double u, double v, double var_u, double var_v,
                            const double* tangent, const double* wsec2, int n, double& s0_out,
                            double& mass_out, double& radial_out) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  s0_out = mass_out = radial_out = 0.0;
  while (need) {
    const int src = __ffs(need) - 1;
    need &= need - 1;
    const double bu = __shfl_sync(full, u, src), bv = __shfl_sync(full, v, src);
    const double bvu = __shfl_sync(full, var_u, src), bvv = __shfl_sync(full, var_v, src);
    const double scale = 2.0 * (bvu + bvv) + bu * bu + bv * bv;
    if (scale <= 0.0) continue;  // the same for the whole warp
    const double s0 = rsqrt(scale);
    const double uu = bu * bu, vv = bv * bv;
    double mass = 0.0, radial = 0.0;
    for (int k = lane; k < n; k += 32) {
      // a = 1 + 2 t^2 var_u, b likewise; their inverses from one reciprocal root
      const double t = s0 * tangent[k], t2 = t * t;
      const double a = fma(2.0 * t2, bvu, 1.0), b = fma(2.0 * t2, bvv, 1.0);
      const double root = rsqrt(a * b), inv = root * root;  // 1 / sqrt(a b), 1 / (a b)
      const double ia = b * inv, ib = a * inv;
      const double m = wsec2[k] * exp(-t2 * (uu * ia + vv * ib)) * root;
      mass += m;
      if (kRadial) radial += m * (ia * (bvu + uu * ia) + ib * (bvv + vv * ib));
    }
    for (int off = 16; off; off >>= 1) {
      mass += __shfl_xor_sync(full, mass, off);
      if (kRadial) radial += __shfl_xor_sync(full, radial, off);
    }
    if (lane == src) {
      s0_out = s0;
      mass_out = mass;
      radial_out = radial;
    }
  }
}

// gauss_inverse_mean_prepared from its node sums.
LH_DEVICE double o1_gauss_inverse_mean(double u, double v, double var_u, double var_v, double s0,
                                       double mass) {
  if (2.0 * (var_u + var_v) + u * u + v * v <= 0.0) return 1e300;
  return 2.0 / sqrt(kPi) * s0 * mass;
}

// inverse_radius_rule from its node sums: a positive two-node rule for the
// Gaussian measure over the radius (w0, t0, w1, t1).
LH_DEVICE void o1_inverse_radius_rule(double u, double v, double var_u, double var_v, double s0,
                                      double mass, double radial, double& w0, double& t0,
                                      double& w1, double& t1) {
  w0 = t0 = w1 = t1 = 0.0;
  if (2.0 * (var_u + var_v) + u * u + v * v <= 0.0) return;
  const double multiplier = 2.0 / sqrt(kPi) * s0;
  const double inverse = mass * multiplier;
  radial *= multiplier;
  if (inverse <= 0.0) return;
  const double mean = 1.0 / inverse, second = radial / inverse;
  const double variance = second - mean * mean;
  if (variance <= 0.0) {
    w0 = inverse; t0 = mean; t1 = mean;
    return;
  }
  const double third = (u * u + v * v + var_u + var_v) / inverse;
  const double other = (third - 2.0 * mean * second + mean * mean * mean) / variance;
  const double disc = sqrt((mean - other) * (mean - other) + 4.0 * variance);
  const double low = 0.5 * (mean + other - disc), high = 0.5 * (mean + other + disc);
  const double low_weight = inverse * (high - mean) / (high - low);
  w0 = low_weight; t0 = low; w1 = inverse - low_weight; t1 = high;
}

// The coarse screen's refinement test (_prompt_screen.py:233-240): the OM
// looks into pencil x's angular extent (forward, theta^2 < s^2 extent^2).
LH_DEVICE bool o1_refined(const lh_order1_config& C, const lh_order1_pencil_table& Pn, int x,
                          double rx, double ry, double rz) {
  const double dx = rx - Pn.position[3 * x], dy = ry - Pn.position[3 * x + 1],
               dz = rz - Pn.position[3 * x + 2];
  const double inv_r = rsqrt(dx * dx + dy * dy + dz * dz);
  const double hx = dx * inv_r, hy = dy * inv_r, hz = dz * inv_r;
  const double sx = Pn.direction[3 * x], sy = Pn.direction[3 * x + 1], sz = Pn.direction[3 * x + 2];
  const double cosine = hx * sx + hy * sy + hz * sz;
  const double qx = hx - cosine * sx, qy = hy - cosine * sy, qz = hz - cosine * sz;
  const double* cov = Pn.pos_cov + 6 * x;
  const double extent2 = Pn.var_major[x] + (cov[0] + cov[1] + cov[2]) * (inv_r * inv_r);
  const double sf = C.smoothing_factor;
  // theta >= sin(theta): most pencils are decided without the angle
  const double s2 = qx * qx + qy * qy + qz * qz;
  if (!(s2 < sf * sf * extent2 * (1.0 + 1e-12))) return false;
  const double theta = atan2(sqrt(s2), cosine);
  return theta < 0.5 * kPi && theta * theta < sf * sf * extent2;
}

// floor(log(x) * scale + shift) of a positive normal x: the hardware's float32
// logarithm decides it wherever its value is further than 2e-3 from a whole number
// (its error is below 1.8e-3 for |scale| <= 64 and |value| < 1024: three ulp of a
// logarithm below 70), the float64 logarithm elsewhere, so the result is the
// float64 one.
LH_DEVICE int o1_log_floor(double x, double scale, double shift) {
  const float xf = (float)x;
  if (xf > 1e-30f && xf < 1e30f && fabs(scale) <= 64.0) {
    const float lf = __logf(xf);
    const float v = fmaf(lf, (float)scale, (float)shift);
    const float f = floorf(v), part = v - f;
    if (part > 2e-3f && part < 1.0f - 2e-3f && fabsf(v) < 1024.0f) return (int)f;
  }
  return (int)floor(fma(log(x), scale, shift));
}

constexpr int kO1GroupOms = 8;       // work OMs per warp chunk of the group stage
constexpr int kO1PencilFields = 20;  // float64 fields of a pencil read by the group stage

// The monomials of a quadratic acceptance in their usual order.
LH_DEVICE bool o1_quadratic(const lh_order1_config& C, const int* ipow, const int* jpow) {
  return C.n_mono == 6 && ipow[0] == 0 && jpow[0] == 0 && ipow[1] == 0 && jpow[1] == 1 &&
         ipow[2] == 1 && jpow[2] == 0 && ipow[3] == 0 && jpow[3] == 2 && ipow[4] == 1 &&
         jpow[4] == 1 && ipow[5] == 2 && jpow[5] == 0;
}

struct O1GroupShared {
  double tangent[kO1MaxGauss], wsec2[kO1MaxGauss];
  double coef[kO1MaxMono];
  int ipow[kO1MaxMono], jpow[kO1MaxMono];
};

// One thread per (work OM, pencil): _grouped_pencils_order1_block's pencil
// loop (_prompt_numba.py:1827-1921) with the generic moment layout. kScreen
// (kScreen): the coarse screen's instance; the fine instance carries none of
// the screen's code (a smaller loop for the instruction cache).
template <bool kScreen>
__global__ void __launch_bounds__(256, 2)
o1_group_kernel(const lh_order1_config C, const lh_order1_pencil_table Pn,
                                int32_t n_pencils_bound, const int32_t* n_pencils_device,
                                const int32_t* work, int32_t n_work,
                                const double* origins, long long* gkeys, double* grows,
                                int32_t* gcount, int32_t* status, unsigned long long* units) {
  __shared__ O1GroupShared S;
  for (int k = threadIdx.x; k < C.n_gauss; k += blockDim.x) {
    const double t = tan(C.gauss_tau[k]);
    S.tangent[k] = t;
    S.wsec2[k] = C.gauss_w[k] * (1.0 + t * t);
  }
  for (int k = threadIdx.x; k < C.n_mono; k += blockDim.x) {
    S.coef[k] = C.coef[k];
    S.ipow[k] = C.ipow[k];
    S.jpow[k] = C.jpow[k];
  }
  __syncthreads();
  const int n_values = 2 * C.n_mono + 6;
  // the monomials of a quadratic acceptance in their usual order: their powers in
  // registers instead of arrays indexed at run time
  const bool quadratic = o1_quadratic(C, S.ipow, S.jpow);
  const double theta_scale = 1.0 / log(1.0 + C.theta_ratio);
  const double theta_shift = -log(C.theta_lo) * theta_scale;
  const double log_r_scale = 0.5 / C.log_r_step;  // of log(r^2)
  const double tau_scale = 1.0 / C.tau_step, inv_speed = 1.0 / C.speed_ref;
  const int theta_bins = C.theta_bins;
  const int64_t cap = C.group_capacity;
  // the pencil count is read on the device when given (no host round trip)
  const int32_t n_pencils =
      n_pencils_device ? min(*n_pencils_device, n_pencils_bound) : n_pencils_bound;
  const int64_t total = (int64_t)n_work * n_pencils;
  if (units && blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(units, (unsigned long long)total);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // [warp][32][n_values] group staging, then [warp][field][32] pencil fields
  extern __shared__ double o1g_stage[];
  double* stage = o1g_stage + warp * 32 * n_values;
  double* pen = o1g_stage + (blockDim.x >> 5) * 32 * n_values + warp * 32 * kO1PencilFields + lane;
  // A warp takes 32 consecutive pencils (neighbours in space) and kO1GroupOms
  // consecutive work OMs: each lane reads its pencil once (into shared memory)
  // and evaluates it against every OM of the chunk in turn. Chunks take the OM
  // blocks fastest and the pencil blocks in a fixed permutation
  // ((q (2^31 - 1)) mod blocks, 2^31 - 1 prime), so that the warps running at
  // once work on different OMs and distant parts of the shower rather than
  // competing for the same group rows. Lanes past the last pencil compute on
  // pencil 0 and take no part in any group.
  const int64_t pblocks = ((int64_t)n_pencils + 31) / 32;
  const int64_t oblocks = (n_work + kO1GroupOms - 1) / kO1GroupOms;
  const int64_t chunks = pblocks * oblocks;
  const int64_t warps_total = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t chunk = blockIdx.x * (int64_t)(blockDim.x >> 5) + warp; chunk < chunks;
       chunk += warps_total) {
    const int64_t p_raw = (((chunk / oblocks) * 2147483647ll) % pblocks) * 32 + lane;
    const int w_first = (int)(chunk % oblocks) * kO1GroupOms;
    const bool p_ok = p_raw < n_pencils;
    const int p = p_ok ? (int)p_raw : 0;
    pen[0] = Pn.position[3 * p]; pen[32] = Pn.position[3 * p + 1]; pen[64] = Pn.position[3 * p + 2];
    pen[96] = Pn.time[p];
    pen[128] = Pn.direction[3 * p]; pen[160] = Pn.direction[3 * p + 1];
    pen[192] = Pn.direction[3 * p + 2];
    pen[224] = Pn.major[3 * p]; pen[256] = Pn.major[3 * p + 1]; pen[288] = Pn.major[3 * p + 2];
    pen[320] = Pn.var_major[p]; pen[352] = Pn.var_minor[p];
    for (int f = 0; f < 6; ++f) pen[(12 + f) * 32] = Pn.pos_cov[6 * p + f];
    pen[576] = Pn.w0[p]; pen[608] = Pn.w2[p];
    const int parent = kScreen ? Pn.parent[p] : -1;
    for (int k = 0; k < kO1GroupOms; ++k) {
    const int w = w_first + k;
    if (w >= n_work) break;  // the same for the whole warp
    bool live = p_ok;
    const int d = work[w];
    const double rx = C.om_pos[3 * d], ry = C.om_pos[3 * d + 1], rz = C.om_pos[3 * d + 2];
    const double nx = C.om_look[3 * d], ny = C.om_look[3 * d + 1], nz = C.om_look[3 * d + 2];
    // _prepare_receiver_geometry (_prompt_numba.py:1590-1612)
    const double dx = rx - pen[0], dy = ry - pen[32], dz = rz - pen[64];
    const double r2 = dx * dx + dy * dy + dz * dz;
    const double inv_r = rsqrt(r2), r = r2 * inv_r;
    const double hx = dx * inv_r, hy = dy * inv_r, hz = dz * inv_r;
    // the screen's charge batches ignore emission time (_prompt_screen.py:220-229)
    const double t_emit = kScreen ? 0.0 : pen[96] - origins[d];
    const double tau = kScreen ? 0.0 : fma(r, inv_speed, t_emit);
    const long long key0 = (long long)o1_log_floor(r2, log_r_scale, 0.0) + (1ll << 20);
    long long base = key0 * 2 * theta_bins;
    if (!kScreen) {
      const int tau_bin = __double2int_rd(tau * tau_scale);  // saturates
      const long long key1 =
          (long long)(min(max(tau_bin, -(1 << 20)), (1 << 20) - 1) + (1 << 20));
      base = ((key1 << 21) + key0) * 2 * theta_bins;
    }
    if (kScreen && live) {  // a parent unless the OM looks into it, else its children
      // rows of a table whose stage A overflowed are not written (the caller
      // redoes it): an index outside the table is never followed
      if (parent >= n_pencils || parent < -1) live = false;
      else live = parent < 0 ? !o1_refined(C, Pn, p, rx, ry, rz)
                             : o1_refined(C, Pn, parent, rx, ry, rz);
    }
    // children stand in for their parent only where the OM looks into it, so
    // most screen warps over children have nothing to add
    if (kScreen && !__any_sync(0xffffffffu, live)) continue;
    // _pencil_frame_from_ray_cached_look (_prompt_numba.py:594-606)
    const double sx = pen[128], sy = pen[160], sz = pen[192];
    const double c1 = sx * nx + sy * ny + sz * nz;
    const double cosine = hx * sx + hy * sy + hz * sz;
    const double qx = hx - cosine * sx, qy = hy - cosine * sy, qz = hz - cosine * sz;
    const double s2 = qx * qx + qy * qy + qz * qz;
    const bool off_axis = s2 > 0.0;
    const double inv_sine = off_axis ? rsqrt(s2) : 0.0, sine = s2 * inv_sine;
    const double c3 = (qx * nx + qy * ny + qz * nz) * inv_sine;
    double theta = atan2(sine, cosine);
    const bool backward = theta > 0.5 * kPi;
    double weight = 0.0, weight2 = 0.0, theta2 = theta;
    bool averaged = false;
    const double ax = pen[224], ay = pen[256], az = pen[288];
    const double cov[6] = {pen[384], pen[416], pen[448], pen[480], pen[512], pen[544]};
    // _prepare_pencil_shape (_prompt_numba.py:1347-1370)
    const double bx = sy * az - sz * ay, by = sz * ax - sx * az, bz = sx * ay - sy * ax;
    const double trace = cov[0] + cov[1] + cov[2];
    const double sf = C.smoothing_factor;
    // How this lane's weight is formed: 0 done; 1 the screen's two-node radial
    // rule; 2 the Gauss inverse mean; 3 the far-field expansion. Modes 1 and 2
    // need a 48-node sum, which the whole warp evaluates for each such lane.
    int mode = 0;
    bool far = true;
    double m11 = 0.0, m22 = 0.0, m12 = 0.0, mu1 = 0.0, mu2 = 0.0, extent = 0.0;
    double u_ = 0.0, v_ = 0.0, r_extent = 0.0;
    double arg_u = 0.0, arg_v = 0.0, arg_var_u = 0.0, arg_var_v = 0.0;  // of the node sums
    if (backward) {
      weight = inv_r;
    } else {
      const double inv_r2 = inv_r * inv_r;
      const double bound = pen[320] + pen[352] + trace * inv_r2;
      if (off_axis && bound < 1e-4 * s2) {
        weight = inv_sine * inv_r;
      } else {
        // _pencil_shape_factor_from_ray (_prompt_numba.py:1389-1436)
        const double caa = ax * (cov[0] * ax + cov[3] * ay + cov[4] * az) +
                           ay * (cov[3] * ax + cov[1] * ay + cov[5] * az) +
                           az * (cov[4] * ax + cov[5] * ay + cov[2] * az);
        const double cbb = bx * (cov[0] * bx + cov[3] * by + cov[4] * bz) +
                           by * (cov[3] * bx + cov[1] * by + cov[5] * bz) +
                           bz * (cov[4] * bx + cov[5] * by + cov[2] * bz);
        const double cab = ax * (cov[0] * bx + cov[3] * by + cov[4] * bz) +
                           ay * (cov[3] * bx + cov[1] * by + cov[5] * bz) +
                           az * (cov[4] * bx + cov[5] * by + cov[2] * bz);
        m11 = pen[320] + caa * inv_r2;
        m22 = pen[352] + cbb * inv_r2;
        m12 = cab * inv_r2;
        const double upper = fmax(m11, m22) + fabs(m12);
        far = fmax(fmax(fabs(m11), fabs(m22)), fabs(m12)) < 1e150 &&
              theta * theta > sf * sf * fmax(upper, 0.0) * (1.0 + 1e-12);
        if (!far) {
          const double half_tr = 0.5 * (m11 + m22);
          const double disc = sqrt(fmax(0.25 * (m11 - m22) * (m11 - m22) + m12 * m12, 0.0));
          mu1 = half_tr + disc;
          mu2 = fmax(half_tr - disc, 1e-16 * mu1 + 1e-300);
          extent = sqrt(fmax(mu1, 0.0));
        }
        u_ = hx * ax + hy * ay + hz * az;
        v_ = hx * bx + hy * by + hz * bz;
        mode = (!far && extent > 0.0 && theta < sf * extent) ? 2 : 3;
        if (kScreen) {
          // pencil_radial_rule (_prompt_screen.py:143-169): two radial nodes where the
          // OM lies within the pencil's angular smoothing extent
          const double half_tr = 0.5 * (m11 + m22);
          const double disc = sqrt(fmax(0.25 * (m11 - m22) * (m11 - m22) + m12 * m12, 0.0));
          const double r_mu1 = half_tr + disc;
          const double r_mu2 = fmax(half_tr - disc, 1e-16 * r_mu1 + 1e-300);
          r_extent = sqrt(fmax(r_mu1, 0.0));
          if (r_extent > 0.0 && theta < sf * r_extent) {
            const double st = off_axis ? theta * inv_sine : 1.0;
            const double uu = u_ * st, vv = v_ * st;
            double sa, ca;
            sincos(0.5 * atan2(2.0 * m12, m11 - m22), &sa, &ca);
            arg_u = ca * uu + sa * vv;
            arg_v = -sa * uu + ca * vv;
            arg_var_u = r_mu1;
            arg_var_v = r_mu2;
            mode = 1;
          }
        }
      }
    }
    if (!live) mode = 0;  // nothing of this lane is added
    const unsigned full = 0xffffffffu;
    double s0n, mass, radial;
    const unsigned need_rule = __ballot_sync(full, mode == 1);
    if (need_rule) {
      o1_node_sums<true>(need_rule, arg_u, arg_v, arg_var_u, arg_var_v, S.tangent, S.wsec2, C.n_gauss,
                   s0n, mass, radial);
      if (mode == 1) {
        double w0r, t0r, w1r, t1r;
        o1_inverse_radius_rule(arg_u, arg_v, arg_var_u, arg_var_v, s0n, mass, radial, w0r, t0r,
                               w1r, t1r);
        if (t0r > 0.0 && t1r < 0.5 * kPi && w0r > 0.0 && w1r >= 0.0) {
          averaged = theta < r_extent;
          weight = (w0r * t0r / sin(t0r)) * inv_r;
          weight2 = (w1r * t1r / sin(t1r)) * inv_r;
          theta = t0r;
          theta2 = t1r;
          mode = 0;
        } else {
          mode = (!far && extent > 0.0 && theta < sf * extent) ? 2 : 3;
        }
      }
    }
    if (mode == 2) {
      double sa, ca;
      sincos(0.5 * atan2(2.0 * m12, m11 - m22), &sa, &ca);
      arg_u = ca * u_ + sa * v_;
      arg_v = -sa * u_ + ca * v_;
      arg_var_u = mu1;
      arg_var_v = mu2;
    }
    const unsigned need_mean = __ballot_sync(full, mode == 2);
    if (need_mean) {
      o1_node_sums<false>(need_mean, arg_u, arg_v, arg_var_u, arg_var_v, S.tangent, S.wsec2, C.n_gauss,
                   s0n, mass, radial);
      if (mode == 2) {
        const double mean = o1_gauss_inverse_mean(arg_u, arg_v, arg_var_u, arg_var_v, s0n, mass);
        const double factor = mean * (off_axis ? theta * inv_sine : 1.0);
        averaged = theta < extent;
        theta = factor > 1.0 ? asin(fmin(1.0, 1.0 / factor)) : theta;
        weight = factor * inv_r;
      }
    }
    if (mode == 3) {
      if (!off_axis) live = false;
      const double d2 = u_ * u_ + v_ * v_;
      double factor = inv_sine;
      if (d2 > 0.0) {
        const double qf = m11 * u_ * u_ + 2.0 * m12 * u_ * v_ + m22 * v_ * v_;
        const double inv_d2 = 1.0 / d2;
        factor *= 1.0 + 0.5 * (3.0 * qf * inv_d2 - (m11 + m22)) * inv_d2;
      }
      weight = factor * inv_r;
    }
    const double perp2 = fmax(1.0 - c1 * c1, 0.0);
    const int nm = C.n_mono;
    // one group entry per radial node: the screen's two-node rule adds a second
    // (_prompt_screen.py:281-336); every lane of the warp takes both rounds
    const int nodes = kScreen ? 2 : 1;
    for (int node = 0; node < nodes; ++node) {
      const bool live_n = live && (node == 0 || weight2 > 0.0);
      const double wn = node == 0 ? weight : weight2;
      const double th = node == 0 ? theta : theta2;
      // theta index (scalar_theta_index, _prompt_numba.py:1628-1631)
      int i_theta = 0;
      if (th >= C.theta_lo)
        i_theta = min(1 + max(o1_log_floor(th, theta_scale, theta_shift), 0), theta_bins - 1);
      const long long key = base + (backward ? theta_bins : 0) + i_theta;
      // lanes with the same group key (the OM is the warp's) sum their moments; the
      // group's lowest lane inserts the key and adds the sums
      const unsigned group = __match_any_sync(0xffffffffu, live_n ? key : -1ll);
      const bool leader = live_n && lane == __ffs(group) - 1;
      double* row = nullptr;
      if (leader) {
        bool fresh;
        long long* keys = gkeys + (int64_t)w * cap;
        const int64_t slot = o1_insert(keys, cap, key, grows + (int64_t)w * cap * kO1MaxValues,
                                       kO1MaxValues, fresh, status);
        if (slot >= 0) {
          if (fresh) atomicAdd(gcount + w, 1);
          row = grows + ((int64_t)w * cap + slot) * kO1MaxValues;
        }
      }
      const double field0 = wn * pen[576], field2 = wn * pen[608];
      // the angular powers (_fill_moments_averaged_pair, _prompt_numba.py:1260-1277)
      double omega;
      double* mine = stage + lane * n_values;
      if (quadratic) {
        const double p1 = averaged ? 0.0 : c3, p2 = averaged ? 0.5 * perp2 : c3 * c3;
        const double basis[6] = {1.0, p1, c1, p2, c1 * p1, c1 * c1};
#pragma unroll
        for (int m = 0; m < 6; ++m) {
          mine[m] = field0 * basis[m];
          mine[6 + m] = field2 * basis[m];
        }
        omega = fabs(field0);
      } else {
        double cpw[5], spw[5];
        cpw[0] = 1.0;
        spw[0] = 1.0;
        for (int q = 1; q <= C.max_power; ++q) {
          cpw[q] = cpw[q - 1] * c1;
          if (averaged) spw[q] = (q & 1) ? 0.0 : spw[q - 2] * perp2 * (q - 1.0) / q;
          else spw[q] = spw[q - 1] * c3;
        }
        omega = 0.0;
        for (int m = 0; m < nm; ++m) {
          const double basis = cpw[S.ipow[m]] * spw[S.jpow[m]];
          const double v0 = field0 * basis;
          if (m == 0) omega = fabs(v0);
          mine[m] = v0;
          mine[nm + m] = field2 * basis;
        }
      }
      mine[2 * nm] = omega;
      mine[2 * nm + 1] = omega * th;
      mine[2 * nm + 2] = omega * r;
      mine[2 * nm + 3] = omega * t_emit;
      mine[2 * nm + 4] = omega * tau;
      mine[2 * nm + 5] = omega * tau * tau;
      o1_warp_group_add(stage, n_values, group, leader, row);
    }
    }  // OMs of the chunk
  }
}

// One CTA per work OM: sort the OM's group keys and list its (tau, r) batches.
__global__ void __launch_bounds__(1024)
o1_batches_kernel(const lh_order1_config C, int32_t n_work, const long long* gkeys,
                  int32_t* sorted_slots, int32_t* batch_list, int32_t* batch_total,
                  unsigned long long* sort_keys, int32_t* sort_slots, int32_t* status) {
  // Tables up to kO1SmemSort slots sort (key << 14 | slot) in shared memory;
  // larger ones (steps whose pencils mix times, e.g. delayed light) sort keys
  // and slots side by side in the workspace.
  extern __shared__ __align__(16) unsigned char o1b_smem[];
  __shared__ int n_used;
  const int w = blockIdx.x;
  const int64_t cap = C.group_capacity;
  const bool packed = cap <= kO1SmemSort;
  unsigned long long* v =
      packed ? reinterpret_cast<unsigned long long*>(o1b_smem) : sort_keys + (int64_t)w * cap;
  int32_t* vs = packed ? nullptr : sort_slots + (int64_t)w * cap;
  const long long* keys = gkeys + (int64_t)w * cap;
  if (threadIdx.x == 0) n_used = 0;
  __syncthreads();
  for (int64_t slot = threadIdx.x; slot < cap; slot += blockDim.x) {
    const long long key = keys[slot];
    if (key == -1ll) continue;
    const int k = atomicAdd(&n_used, 1);
    if (packed) {
      v[k] = ((unsigned long long)key << 14) | (unsigned long long)slot;
    } else {
      v[k] = (unsigned long long)key;
      vs[k] = (int32_t)slot;
    }
  }
  __syncthreads();
  const int used = n_used;
  int n = 1;
  while (n < used) n <<= 1;
  for (int k = used + threadIdx.x; k < n; k += blockDim.x) {
    v[k] = ~0ull;
    if (!packed) vs[k] = -1;
  }
  __syncthreads();
  // bitonic sort, ascending (shared or, for large tables, global memory: the
  // barrier makes the block's global writes visible to the block)
  for (int size = 2; size <= n; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int k = threadIdx.x; k < n; k += blockDim.x) {
        const int partner = k ^ stride;
        if (partner > k) {
          const bool up = (k & size) == 0;
          const unsigned long long a = v[k], b = v[partner];
          if ((a > b) == up) {
            v[k] = b;
            v[partner] = a;
            if (!packed) {
              const int32_t t = vs[k];
              vs[k] = vs[partner];
              vs[partner] = t;
            }
          }
        }
      }
      __syncthreads();
    }
  }
  int32_t* out = sorted_slots + (int64_t)w * cap;
  const long long tb = C.theta_bins;
  auto key_of = [&](int k) { return packed ? (long long)(v[k] >> 14) : (long long)v[k]; };
  for (int k = threadIdx.x; k < used; k += blockDim.x) {
    out[k] = packed ? (int32_t)(v[k] & 0x3fffull) : vs[k];
    const long long bk = key_of(k) / tb;
    if (k == 0 || key_of(k - 1) / tb != bk) {
      int stop = k + 1;
      while (stop < used && key_of(stop) / tb == bk) ++stop;
      const int b = atomicAdd(batch_total, 1);
      batch_list[3 * b] = w;
      batch_list[3 * b + 1] = k;
      batch_list[3 * b + 2] = stop;
    }
  }
  (void)status;
}

// _ifuncs (_prompt_numba.py:139-154): I_k(z) = int_0^1 x^k e^{z x} dx, k = 0, 1, 2,
// with ez = e^z. Below |z| = 1 the series of I_2 (sum z^n / (n! (n + 3)); 19 terms
// reach 1e-18), then I_1 and I_0 by parts, I_{k-1} = (e^z - z I_k) / k. They carry the
// rounding of e^z, as a panel's two ends do: its integral is no further off than with a
// series each (bins against the oracle 2e-14 in the median either way), which took 9 %
// longer (o1_batch_warp_kernel 0.229 against 0.210 ms for 6637 elements, 64 OMs).
LH_DEVICE void o1_ifuncs(double z, double ez, double& i0, double& i1, double& i2) {
  if (fabs(z) < 1.0) {
    constexpr int kTerms = 19;
    double f = 1.0, c[kTerms];
#pragma unroll
    for (int n = 0; n < kTerms; ++n) {
      if (n > 0) f /= n;
      c[n] = f / (n + 3.0);
    }
    i2 = c[kTerms - 1];
#pragma unroll
    for (int n = kTerms - 2; n >= 0; --n) i2 = fma(i2, z, c[n]);
    i1 = 0.5 * fma(-z, i2, ez);
    i0 = fma(-z, i1, ez);
    return;
  }
  const double inv = 1.0 / z;
  i0 = (ez - 1.0) * inv;
  i1 = (ez - i0) * inv;
  i2 = (ez - 2.0 * i1) * inv;
}

// _quad_integral (_prompt_numba.py:158-163)
__device__ __noinline__ double o1_quad(double e_start, double alpha, double beta, double gamma, double width,
                         double kappa, double e_end) {
  const double z = kappa * width;
  const double ez = e_start > 0.0 ? e_end / e_start : exp(z);
  double i0, i1, i2;
  o1_ifuncs(z, ez, i0, i1, i2);
  return e_start * width * (alpha * i0 + width * (beta * i1 + width * gamma * i2));
}

// _find_bin (_prompt_numba.py:167-182)
LH_DEVICE int o1_find_bin(const double* edges, int nb, double t) {
  if (t < edges[0]) return -1;
  if (t >= edges[nb]) return nb;
  int low = 0, high = nb;
  while (high - low > 1) {
    const int middle = (low + high) / 2;
    if (t < edges[middle]) high = middle; else low = middle;
  }
  return low;
}

// _deposit_panel (_prompt_numba.py:186-254) into the OM's accumulators
// pre[3] and acc[nb][4] of one band.
__device__ __noinline__ void o1_deposit_panel(double t_a, double t_b, double e_a, double e_b, double alpha,
                                double beta, double gamma, double kappa, const double* edges,
                                const double* eedge, int nb, double* pre, double* acc,
                                int direct_bins) {
  const double lo = t_a > edges[0] ? t_a : edges[0];
  const double hi = t_b < edges[nb] ? t_b : edges[nb];
  if (hi <= lo) return;
  const int k_lo = o1_find_bin(edges, nb, lo);
  int k_hi = o1_find_bin(edges, nb, hi);
  if (k_hi >= nb || (k_hi > k_lo && hi <= edges[k_hi])) k_hi -= 1;
  if (k_hi - k_lo + 1 <= direct_bins) {
    for (int k = k_lo; k <= k_hi; ++k) {
      const double s_lo = lo > edges[k] ? lo : edges[k];
      const double s_hi = hi < edges[k + 1] ? hi : edges[k + 1];
      if (s_hi <= s_lo) continue;
      double e_lo = s_lo == t_a ? e_a : eedge[k];
      if (s_lo != t_a && s_lo != edges[k]) e_lo = exp(kappa * s_lo);
      double e_hi = s_hi == t_b ? e_b : eedge[k + 1];
      if (s_hi != t_b && s_hi != edges[k + 1]) e_hi = exp(kappa * s_hi);
      const double shift = s_lo - t_a;
      const double a_loc = alpha + shift * (beta + shift * gamma);
      const double b_loc = beta + 2.0 * gamma * shift;
      atomicAdd(acc + 4 * k + 3, o1_quad(e_lo, a_loc, b_loc, gamma, s_hi - s_lo, kappa, e_hi));
    }
    return;
  }
  const double big_a = alpha - t_a * (beta - gamma * t_a);
  const double big_b = beta - 2.0 * gamma * t_a;
  const double big_c = gamma;
  if (t_a < edges[0]) {
    atomicAdd(pre + 0, big_a);
    atomicAdd(pre + 1, big_b);
    atomicAdd(pre + 2, big_c);
  } else {
    const int k = k_lo;
    atomicAdd(acc + 4 * k + 0, big_a);
    atomicAdd(acc + 4 * k + 1, big_b);
    atomicAdd(acc + 4 * k + 2, big_c);
    atomicAdd(acc + 4 * k + 3, o1_quad(e_a, alpha, beta, gamma, edges[k + 1] - t_a, kappa, eedge[k + 1]));
  }
  if (t_b < edges[nb]) {
    const int k = o1_find_bin(edges, nb, t_b);
    atomicAdd(acc + 4 * k + 0, -big_a);
    atomicAdd(acc + 4 * k + 1, -big_b);
    atomicAdd(acc + 4 * k + 2, -big_c);
    const double shift = t_b - t_a;
    const double a_loc = alpha + shift * (beta + shift * gamma);
    const double b_loc = beta + 2.0 * gamma * shift;
    atomicAdd(acc + 4 * k + 3,
              -o1_quad(e_b, a_loc, b_loc, gamma, edges[k + 1] - t_b, kappa, eedge[k + 1]));
  }
}

struct O1BandDeposit {
  double v, kappa, spread, t_base, e_emit, w0, w2, h_front;
  int last, pairs, panels;
  bool outside;
};

// What the batch's path grid and deposit need: mean radius and emission time,
// front width, grid scale, its two ends and node counts.
struct O1BatchGrid {
  double r_b, t_b, front_extra, sigma, u_win, u_end;
  int n_in, n_out, n;  // n = n_in + n_out + 1 nodes, 0: nothing to deposit
  bool backward;
};

// The batch's grid from its groups' sums (_batch_sigma, _batch_grid:
// _prompt_numba.py:258-292).
LH_DEVICE O1BatchGrid o1_batch_grid(const lh_order1_config& C, bool backward, double omega_sum,
                                    double r_sum, double t_sum, double tau_sum, double tau2_sum,
                                    double theta_small, double mut_min, double speed_max,
                                    int32_t* status) {
  O1BatchGrid G{};
  G.backward = backward;
  if (!(omega_sum > 0.0)) return G;
  const int nb = C.n_edges - 1;
  const double inv = 1.0 / omega_sum;
  const double r_b = r_sum * inv, t_b = t_sum * inv, tau_mean = tau_sum * inv;
  const double tau_var = fmax(tau2_sum * inv - tau_mean * tau_mean, 0.0);
  const double g = C.g;
  const double y_g = g != 0.0 ? (1.0 - fabs(g)) / (1.0 + fabs(g)) : 1.0;
  theta_small = fmax(theta_small, 1e-9);
  double sin_t, cos_t;
  sincos(theta_small, &sin_t, &cos_t);
  double sigma;
  if (backward)
    sigma = fmax(0.5 * r_b * sin_t * y_g, 0.25 * r_b * (1.0 - cos_t));
  else
    sigma = fmax(0.5 * r_b * sin_t * fmax(y_g, 0.5 * tan(0.5 * theta_small)), 1e-9 * r_b);
  const double ext_end = C.tail_exponent / mut_min;
  // the screen's grids run to the tail without a window edge
  // (_prompt_screen.py:413: edge_end = inf)
  double ext_win = C.screen ? ext_end : speed_max * (C.edges[nb] - t_b) - r_b;
  ext_win = fmin(fmax(ext_win, 0.0), ext_end);
  double u_end = 0.0, u_win = 0.0;
#pragma unroll 1
  for (int i = 0; i < 2; ++i) {  // one copy of asinh
    u_end = u_win;
    u_win = asinh((i ? ext_win : ext_end) / sigma);
  }
  if (!(u_win >= 0.0) || !(u_end >= u_win) || !(u_end < 1e6)) {
    atomicOr(reinterpret_cast<unsigned*>(status), LH_STATUS_OVERFLOW);
    return G;
  }
  long long n_in = u_win > 0.0 ? (long long)ceil(u_win / C.path_step) : 0;
  long long n_out = u_end > u_win ? (long long)ceil((u_end - u_win) / C.path_step_tail) : 0;
  const int capacity = C.max_path_nodes;
  if (n_in + n_out + 1 > capacity) {
    const double scale = (capacity - 1.0) / (double)(n_in + n_out);
    n_in = (long long)(n_in * scale);
    n_out = capacity - 1 - n_in;
  }
  G.r_b = r_b; G.t_b = t_b; G.front_extra = sqrt(12.0 * tau_var);
  G.sigma = sigma; G.u_win = u_win; G.u_end = u_end;
  G.n_in = (int)n_in; G.n_out = (int)n_out;
  G.n = (int)(n_in + n_out + 1);
  return G;
}

LH_DEVICE double o1_batch_node(const O1BatchGrid& G, int k) {
  if (k == 0) return G.r_b;
  const double u = k <= G.n_in ? G.u_win * k / G.n_in
                               : G.u_win + (G.u_end - G.u_win) * (k - G.n_in) / G.n_out;
  return G.r_b + G.sigma * sinh(u);
}

// Profile at path s of the groups [q0, q1): _batch_add_moments
// (_prompt_numba.py:394-447), generic monomials. `mom` holds rows of nv values.
LH_DEVICE void o1_batch_profile(const lh_order1_config& C, const O1BatchGrid& G, double s,
                                const double* mom, int nv, const double* sin_q,
                                const double* cos_q, const double* coef, const int* ipow,
                                const int* jpow, bool quadratic, int q0, int q1, double& out0,
                                double& out2) {
  const int nm = C.n_mono;
  const double g = C.g, g1 = 1.0 + g * g, gg = 2.0 * g, norm = (1.0 - g * g) / (4.0 * kPi);
  double a0s = 0.0, a2s = 0.0;
  for (int q = q0; q < q1; ++q) {
    const double* row = mom + q * nv;
    if (row[2 * nm] <= 0.0) continue;
    const double sin_t = sin_q[q], cos_t = cos_q[q];
    const double rs = G.r_b * sin_t;
    double c, sn, path_jacobian;
    if (G.backward) {
      const double shift = s - G.r_b * cos_t;
      const double inv = 1.0 / (rs * rs + shift * shift);
      c = (rs * rs - shift * shift) * inv;
      sn = 2.0 * rs * shift * inv;
      path_jacobian = 2.0 * G.r_b * inv;
    } else {
      const double inv_rs = 1.0 / rs;
      const double y = (s - G.r_b) * inv_rs + sin_t / (1.0 + cos_t);
      const double inv = 1.0 / (1.0 + y * y);
      c = (1.0 - y * y) * inv;
      sn = 2.0 * y * inv;
      path_jacobian = 2.0 * inv_rs * inv;
    }
    double a0 = 0.0, a2 = 0.0;
    if (quadratic) {
      const double basis[6] = {coef[0], coef[1] * sn, coef[2] * c, coef[3] * (sn * sn),
                               coef[4] * (c * sn), coef[5] * (c * c)};
#pragma unroll
      for (int m = 0; m < 6; ++m) {
        a0 += basis[m] * row[m];
        a2 += basis[m] * row[6 + m];
      }
    } else {
      double cpw[5], spw[5];
      cpw[0] = 1.0;
      spw[0] = 1.0;
      for (int pw = 1; pw <= C.max_power; ++pw) {
        cpw[pw] = cpw[pw - 1] * c;
        spw[pw] = spw[pw - 1] * sn;
      }
      for (int m = 0; m < nm; ++m) {
        const double basis = coef[m] * cpw[ipow[m]] * spw[jpow[m]];
        a0 += basis * row[m];
        a2 += basis * row[nm + m];
      }
    }
    const double root = rsqrt(g1 - gg * c);
    const double value = path_jacobian * norm * (root * root * root);
    a0s += a0 * value;
    a2s += a2 * value;
  }
  out0 = a0s;
  out2 = a2s;
}

// A band's deposit constants (_batch_deposit, _prompt_numba.py:451-551).
LH_DEVICE void o1_band_setup(const lh_order1_config& C, const O1BatchGrid& G, int lam,
                             const double* s, const double* g0, const double* g2,
                             O1BandDeposit& B) {
  const int nb = C.n_edges - 1;
  B.panels = 0;
  B.pairs = 0;
  if (C.mus[lam] == 0.0) return;
  const double v = C.speed[lam];
  int last = G.n - 1;
  const double limit = G.r_b + C.tail_exponent / C.mut[lam];
  while (last > 2 && s[last - 1] > limit) last -= 1;
  if (last < 2) return;
  B.v = v;
  B.kappa = -C.mut[lam] * v;
  B.last = last;
  B.spread = fmin(G.front_extra, (s[last] - G.r_b) / v);
  const double front_time = G.t_b + G.r_b / v;
  const double end_time = G.t_b + s[last] / v;
  B.outside = front_time - 0.5 * B.spread >= C.edges[nb] ||
              end_time + 0.5 * B.spread <= C.edges[0];
  B.t_base = B.outside ? 0.0 : G.t_b;
  B.e_emit = exp(B.kappa * B.t_base);
  const double h_scale = C.mus[lam] * v / B.e_emit;
  B.w0 = C.s0w[lam] * h_scale;
  B.w2 = C.s2w[lam] * h_scale;
  B.h_front = B.w0 * g0[0] + B.w2 * g2[0];
  // panels start at even nodes with step 2; an odd `last` ends with one step
  B.pairs = last / 2;
  B.panels = B.pairs + (last & 1);
}

// Panel pi of band lam: its integral (returned) and its deposit into the bins.
LH_DEVICE double o1_panel(const lh_order1_config& C, const O1BandDeposit& B, int lam, int pi,
                          const double* s, const double* g0, const double* g2, double* pre) {
  const int nb = C.n_edges - 1;
  const double inv_v = 1.0 / B.v, mut = C.mut[lam];
  auto node_t = [&](int j) { return B.t_base + s[j] * inv_v; };
  auto node_h = [&](int j) { return (B.w0 * g0[j] + B.w2 * g2[j]) - B.h_front; };
  // the parabola through nodes j, j + 1, j + 2: a panel spans both steps, the
  // single last step of an odd grid only the second
  const bool tail = pi >= B.pairs;
  const int j = tail ? B.last - 2 : 2 * pi;
  const double t0 = node_t(j), t1 = node_t(j + 1), t_b2 = node_t(j + 2);
  const double h0 = node_h(j), h1 = node_h(j + 1), h2 = node_h(j + 2);
  const double u_m = t1 - t0;
  const double d1 = (h1 - h0) / u_m;
  const double gamma = ((h2 - h1) / (t_b2 - t1) - d1) / (t_b2 - t0);
  const double t_a = tail ? t1 : t0, alpha = tail ? h1 : h0;
  const double beta = tail ? d1 - gamma * u_m + 2.0 * gamma * u_m : d1 - gamma * u_m;
  const double e_a = B.e_emit * exp(-mut * s[tail ? j + 1 : j]);
  const double e_b = B.e_emit * exp(-mut * s[j + 2]);
  if (pre)
    o1_deposit_panel(t_a, t_b2, e_a, e_b, alpha, beta, gamma, B.kappa, C.edges,
                     C.eedge + (int64_t)lam * C.n_edges, nb, pre, pre + 3, C.direct_bins);
  return o1_quad(e_a, alpha, beta, gamma, t_b2 - t_a, B.kappa, e_b);
}

// The front step of band lam as a mass-normalised ramp of width `spread`; adds
// the band's charge (`total`: its panels') and deposits the ramp.
LH_DEVICE void o1_front(const lh_order1_config& C, const O1BandDeposit& B, int lam,
                        const double* s, double total, double* pre, double* chg) {
  const int nb = C.n_edges - 1;
  const double* eedge = C.eedge + (int64_t)lam * C.n_edges;
  const double e_first = B.e_emit * exp(-C.mut[lam] * s[0]);
  const double e_last = B.e_emit * exp(-C.mut[lam] * s[B.last]);
  const double t_f = B.t_base + s[0] / B.v, t_end = B.t_base + s[B.last] / B.v;
  const double spread = B.spread, kappa = B.kappa;
  const double exact = o1_quad(e_first, B.h_front, 0.0, 0.0, t_end - t_f, kappa, e_last);
  atomicAdd(chg, total + exact);
  if (!pre) return;
  // the step's part behind the ramp: from t_2 at `height` to the end
  double t_2 = t_f, e_2 = e_first, height = B.h_front;
  if (spread > 0.0) {
    const double t_1 = t_f - 0.5 * spread;
    t_2 = t_f + 0.5 * spread;
    const double e_1 = exp(kappa * t_1);
    e_2 = exp(kappa * t_2);
    const double ramp = o1_quad(e_1, 0.0, 1.0 / spread, 0.0, spread, kappa, e_2);
    const double flat = t_end > t_2 ? o1_quad(e_2, 1.0, 0.0, 0.0, t_end - t_2, kappa, e_last) : 0.0;
    height = ramp + flat != 0.0 ? exact / (ramp + flat) : 0.0;
    o1_deposit_panel(t_1, t_2, e_1, e_2, 0.0, height / spread, 0.0, kappa, C.edges, eedge,
                     nb, pre, pre + 3, C.direct_bins);
  }
  if (t_end > t_2)
    o1_deposit_panel(t_2, t_end, e_2, e_last, height, 0.0, 0.0, kappa, C.edges, eedge, nb,
                     pre, pre + 3, C.direct_bins);
}

LH_DEVICE void o1_band_extremes(const lh_order1_config& C, double& mut_min, double& speed_max) {
  mut_min = C.mut[0];
  speed_max = C.speed[0];
  for (int l = 1; l < C.n_bands; ++l) {
    mut_min = fmin(mut_min, C.mut[l]);
    speed_max = fmax(speed_max, C.speed[l]);
  }
}

// _grouped_pencils_order1_block's batch loop (_prompt_numba.py:1934-1993) with
// _batch_grid, _batch_add_moments and _batch_deposit (_prompt_numba.py:258-551),
// one warp per batch. A batch is small (typically 7 groups, 33 path nodes and 51
// (band, panel) items), so its steps are chains of short loops: with a CTA of four
// warps per batch they waited on one another (barrier 13 of 25 stall cycles per
// issue, 0.61 ms for 8400 batches); a warp needs no barrier and 20 of them per SM
// work on batches of their own (0.22 ms, and 0.035 ms for the deferred ones; 3, 4
// or 6 CTAs per SM are 1-3 % slower). What is left is the latency of one batch's
// float64 chain, ~40 us, and its instruction fetch. Batches with more than
// kO1WarpNodes nodes or kO1WarpGroups groups go to `deferred`.
constexpr int kO1WarpNodes = 128;
constexpr int kO1WarpGroups = 32;
constexpr int kO1WarpSums = 256;  // (node, part) sums of the profile
constexpr int kO1BatchWarps = 4;  // per CTA

struct O1WarpBatch {
  double s[kO1WarpNodes];
  double g0[kO1WarpSums], g2[kO1WarpSums];
  double sin_q[kO1WarpGroups], cos_q[kO1WarpGroups];
  O1BandDeposit band[kO1MaxBands];
};

static size_t o1_warp_batch_bytes(const lh_order1_config& C) {
  return kO1BatchWarps *
         (sizeof(O1WarpBatch) + sizeof(double) * kO1WarpGroups * (size_t)(2 * C.n_mono + 6));
}

LH_DEVICE double o1_warp_sum(double v) {
  for (int off = 16; off; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}

__global__ void __launch_bounds__(32 * kO1BatchWarps, 5)
o1_batch_warp_kernel(const lh_order1_config C, const long long* gkeys, const double* grows,
                     const int32_t* sorted_slots, const int32_t* batch_list,
                     const int32_t* batch_total, int32_t* deferred, int32_t* n_deferred,
                     double* accum, int32_t* status) {
  extern __shared__ __align__(16) unsigned char o1w_smem[];
  __shared__ double s_coef[kO1MaxMono];
  __shared__ int s_ipow[kO1MaxMono], s_jpow[kO1MaxMono];
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nm = C.n_mono, nv = 2 * nm + 6, nb = C.n_edges - 1, NL = C.n_bands;
  O1WarpBatch& S = reinterpret_cast<O1WarpBatch*>(o1w_smem)[warp];
  double* mom = reinterpret_cast<double*>(o1w_smem + kO1BatchWarps * sizeof(O1WarpBatch)) +
                warp * kO1WarpGroups * nv;
  for (int k = threadIdx.x; k < nm; k += blockDim.x) {
    s_coef[k] = C.coef[k];
    s_ipow[k] = C.ipow[k];
    s_jpow[k] = C.jpow[k];
  }
  __syncthreads();
  const bool quadratic = o1_quadratic(C, s_ipow, s_jpow);
  double mut_min, speed_max;
  o1_band_extremes(C, mut_min, speed_max);
  const int64_t cap = C.group_capacity;
  const int64_t per_om = (int64_t)NL * (3 + 4 * nb + 1);
  const int total = *batch_total;
  const int warps = gridDim.x * kO1BatchWarps;
  for (int b = blockIdx.x * kO1BatchWarps + warp; b < total; b += warps) {
    const int w = batch_list[3 * b], start = batch_list[3 * b + 1],
              count = batch_list[3 * b + 2] - start;
    if (count > kO1WarpGroups) {
      if (lane == 0) deferred[atomicAdd(n_deferred, 1)] = b;
      continue;
    }
    const double* rows = grows + (int64_t)w * cap * kO1MaxValues;
    const int slot = lane < count ? sorted_slots[(int64_t)w * cap + start + lane] : 0;
    for (int q0 = 0; q0 < count; q0 += 8) {  // eight rows on their way at a time
      double value[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int from = __shfl_sync(full, slot, min(q0 + j, count - 1));
        value[j] = lane < nv ? rows[(int64_t)from * kO1MaxValues + lane] : 0.0;
      }
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (q0 + j < count && lane < nv) mom[(q0 + j) * nv + lane] = value[j];
    }
    const bool backward =
        ((gkeys[(int64_t)w * cap + __shfl_sync(full, slot, 0)] / C.theta_bins) & 1) == 1;
    __syncwarp();
    // the groups' sums and mean angles, one lane per group
    const double* row = mom + lane * nv + 2 * nm;
    const double omega = lane < count ? row[0] : 0.0;
    const bool some = omega > 0.0;
    const double angle = some ? row[1] / omega : kPi;
    double small = angle;
    for (int off = 16; off; off >>= 1) small = fmin(small, __shfl_xor_sync(full, small, off));
    const double omega_sum = o1_warp_sum(some ? omega : 0.0);
    const double r_sum = o1_warp_sum(some ? row[2] : 0.0);
    const double t_sum = o1_warp_sum(some ? row[3] : 0.0);
    const double tau_sum = o1_warp_sum(some ? row[4] : 0.0);
    const double tau2_sum = o1_warp_sum(some ? row[5] : 0.0);
    double sin_t = 0.0, cos_t = 0.0;
    if (some) sincos(fmax(angle, 1e-9), &sin_t, &cos_t);
    S.sin_q[lane] = sin_t;
    S.cos_q[lane] = cos_t;
    const O1BatchGrid G = o1_batch_grid(C, backward, omega_sum, r_sum, t_sum, tau_sum, tau2_sum,
                                        small, mut_min, speed_max, status);
    const int n = G.n;
    if (n > kO1WarpNodes) {
      if (lane == 0) deferred[atomicAdd(n_deferred, 1)] = b;
      __syncwarp();
      continue;
    }
    if (n == 0) {
      __syncwarp();
      continue;
    }
    for (int k = lane; k < n; k += 32) S.s[k] = o1_batch_node(G, k);
    __syncwarp();
    // the profile: the groups in `parts` ranges, as many as keep the warp's rounds
    // over (node, part) shortest (33 nodes with one part idle 31 lanes in two)
    int parts = 1, best = ((n + 31) >> 5) * count;
    for (int p = 2; p <= 4 && p <= count && n * p <= kO1WarpSums; ++p) {
      const int cost = ((n * p + 31) >> 5) * ((count + p - 1) / p);
      if (cost < best) {
        best = cost;
        parts = p;
      }
    }
    for (int it = lane; it < n * parts; it += 32) {
      const int part = it / n, k = it - part * n;
      o1_batch_profile(C, G, S.s[k], mom, nv, S.sin_q, S.cos_q, s_coef, s_ipow, s_jpow, quadratic,
                       part * count / parts, (part + 1) * count / parts, S.g0[it], S.g2[it]);
    }
    __syncwarp();
    if (parts > 1) {
      for (int k = lane; k < n; k += 32)
        for (int p = 1; p < parts; ++p) {
          S.g0[k] += S.g0[p * n + k];
          S.g2[k] += S.g2[p * n + k];
        }
      __syncwarp();
    }
    if (lane < NL) o1_band_setup(C, G, lane, S.s, S.g0, S.g2, S.band[lane]);
    __syncwarp();
    double* accw = accum + (int64_t)w * per_om;
    int n_panels = 0;
    for (int lam = 0; lam < NL; ++lam) n_panels += S.band[lam].panels;
    double band_total = 0.0;  // lane lam: the charge of band lam's panels
    for (int first = 0; first < n_panels; first += 32) {
      int lam = 0, pi = first + lane;
      while (lam < NL && pi >= S.band[lam].panels) pi -= S.band[lam].panels, ++lam;
      double value = 0.0;
      if (lam < NL)
        value = o1_panel(C, S.band[lam], lam, pi, S.s, S.g0, S.g2,
                         C.compute_bins && !S.band[lam].outside
                             ? accw + (int64_t)lam * (3 + 4 * nb + 1) : nullptr);
      for (int l = 0; l < NL; ++l) {
        const double sum = o1_warp_sum(lam == l ? value : 0.0);
        if (lane == l) band_total += sum;
      }
    }
    if (lane < NL && S.band[lane].panels > 0) {
      double* pre = accw + (int64_t)lane * (3 + 4 * nb + 1);
      o1_front(C, S.band[lane], lane, S.s, band_total,
               C.compute_bins && !S.band[lane].outside ? pre : nullptr, pre + 3 + 4 * nb);
    }
    __syncwarp();
  }
}

// The deferred batches: one CTA per batch, up to kO1MaxNodes nodes and 128 groups.
struct O1BatchShared {
  double s[kO1MaxNodes];
  double g0[kO1MaxNodes];
  double g2[kO1MaxNodes];
  double mom[kO1MaxValues * 128];  // moments of the batch's theta groups (<= 128)
  double sin_q[128], cos_q[128];   // per group: sin, cos of its mean angle (0, 0: empty)
  double coef[kO1MaxMono];
  double total[kO1MaxBands];
  int ipow[kO1MaxMono], jpow[kO1MaxMono];
  O1BandDeposit band[kO1MaxBands];
  O1BatchGrid grid;
};

__global__ void __launch_bounds__(kO1BatchThreads)
o1_batch_kernel(const lh_order1_config C, const long long* gkeys, const double* grows,
                const int32_t* sorted_slots, const int32_t* batch_list, const int32_t* deferred,
                const int32_t* n_deferred, double* accum, int32_t* status) {
  extern __shared__ __align__(16) unsigned char o1_smem[];
  O1BatchShared& S = *reinterpret_cast<O1BatchShared*>(o1_smem);
  const int tid = threadIdx.x;
  const int nm = C.n_mono, nv = 2 * nm + 6, nb = C.n_edges - 1, NL = C.n_bands;
  const int64_t cap = C.group_capacity;
  const int total = *n_deferred;
  if ((int)blockIdx.x >= total) return;
  for (int k = tid; k < nm; k += blockDim.x) {
    S.coef[k] = C.coef[k];
    S.ipow[k] = C.ipow[k];
    S.jpow[k] = C.jpow[k];
  }
  __syncthreads();
  const bool quadratic = o1_quadratic(C, S.ipow, S.jpow);
  double mut_min, speed_max;
  o1_band_extremes(C, mut_min, speed_max);
  const int64_t per_om = (int64_t)NL * (3 + 4 * nb + 1);
  for (int i = blockIdx.x; i < total; i += gridDim.x) {
    const int b = deferred[i];
    __syncthreads();
    const int w = batch_list[3 * b], start = batch_list[3 * b + 1], stop = batch_list[3 * b + 2];
    const int count = stop - start;
    const int32_t* slots = sorted_slots + (int64_t)w * cap + start;
    const double* rows = grows + (int64_t)w * cap * kO1MaxValues;
    if (count > 128) {
      if (tid == 0) atomicOr(reinterpret_cast<unsigned*>(status), LH_STATUS_OVERFLOW);
      continue;
    }
    for (int k = tid; k < count * nv; k += blockDim.x) {
      const int q = k / nv, c = k - q * nv;
      S.mom[k] = rows[(int64_t)slots[q] * kO1MaxValues + c];
    }
    const bool backward = ((gkeys[(int64_t)w * cap + slots[0]] / C.theta_bins) & 1) == 1;
    if (tid < NL) S.total[tid] = 0.0;
    __syncthreads();
    if (tid == 0) {
      double omega_sum = 0, r_sum = 0, t_sum = 0, tau_sum = 0, tau2_sum = 0, theta_small = kPi;
      for (int q = 0; q < count; ++q) {
        const double* row = S.mom + q * nv;
        const double omega = row[2 * nm];
        if (omega > 0.0) {
          omega_sum += omega;
          r_sum += row[2 * nm + 2];
          t_sum += row[2 * nm + 3];
          tau_sum += row[2 * nm + 4];
          tau2_sum += row[2 * nm + 5];
          theta_small = fmin(theta_small, row[2 * nm + 1] / omega);
        }
      }
      S.grid = o1_batch_grid(C, backward, omega_sum, r_sum, t_sum, tau_sum, tau2_sum, theta_small,
                             mut_min, speed_max, status);
    }
    for (int q = tid; q < count; q += blockDim.x) {
      const double* row = S.mom + q * nv;
      const double omega = row[2 * nm];
      double sin_t = 0.0, cos_t = 0.0;
      if (omega > 0.0) sincos(fmax(row[2 * nm + 1] / omega, 1e-9), &sin_t, &cos_t);
      S.sin_q[q] = sin_t;
      S.cos_q[q] = cos_t;
    }
    __syncthreads();
    const int n = S.grid.n;
    if (n == 0) continue;
    for (int k = tid; k < n; k += blockDim.x) {
      const double s = o1_batch_node(S.grid, k);
      S.s[k] = s;
      o1_batch_profile(C, S.grid, s, S.mom, nv, S.sin_q, S.cos_q, S.coef, S.ipow, S.jpow,
                       quadratic, 0, count, S.g0[k], S.g2[k]);
    }
    __syncthreads();
    if (tid < NL) o1_band_setup(C, S.grid, tid, S.s, S.g0, S.g2, S.band[tid]);
    __syncthreads();
    double* accw = accum + (int64_t)w * per_om;
    int n_panels = 0;
    for (int lam = 0; lam < NL; ++lam) n_panels += S.band[lam].panels;
    for (int item = tid; item < n_panels; item += blockDim.x) {
      int lam = 0, pi = item;
      while (pi >= S.band[lam].panels) pi -= S.band[lam].panels, ++lam;
      const double value = o1_panel(C, S.band[lam], lam, pi, S.s, S.g0, S.g2,
                                    C.compute_bins && !S.band[lam].outside
                                        ? accw + (int64_t)lam * (3 + 4 * nb + 1) : nullptr);
      atomicAdd(&S.total[lam], value);
    }
    __syncthreads();
    if (tid < NL && S.band[tid].panels > 0) {
      double* pre = accw + (int64_t)tid * (3 + 4 * nb + 1);
      o1_front(C, S.band[tid], tid, S.s, S.total[tid],
               C.compute_bins && !S.band[tid].outside ? pre : nullptr, pre + 3 + 4 * nb);
    }
  }
}

// _finalize (_prompt_numba.py:610-632): one CTA per work OM, one warp per band.
// The running coefficients of the bins are prefix sums over 32 bins at a time
// (one thread per band walked the 160 bins in 61 us, each bin's loads behind the
// last's).
constexpr int kO1FinalWarps = 4;

__global__ void __launch_bounds__(32 * kO1FinalWarps)
o1_finalize_kernel(const lh_order1_config C, const int32_t* work, int32_t n_work,
                   const double* accum, double* charge, double* bins) {
  const int w = blockIdx.x;
  const int d = work[w];
  const int nb = C.n_edges - 1;
  const int NL = C.n_bands;
  const int64_t per_om = (int64_t)NL * (3 + 4 * nb + 1);
  const double* accw = accum + (int64_t)w * per_om;
  const double area = C.om_area[d];
  if (threadIdx.x == 0) {
    double total = 0.0;
    for (int lam = 0; lam < NL; ++lam) total += accw[(int64_t)lam * (3 + 4 * nb + 1) + 3 + 4 * nb];
    charge[d] = area * total;
  }
  if (!C.compute_bins || !bins) return;
  extern __shared__ __align__(16) unsigned char o1f_smem[];
  double* band_bins = reinterpret_cast<double*>(o1f_smem);
  const int lane = threadIdx.x & 31;
  for (int lam = threadIdx.x >> 5; lam < NL; lam += kO1FinalWarps) {
    const double* pre = accw + (int64_t)lam * (3 + 4 * nb + 1);
    const double* acc = pre + 3;
    const double* eedge = C.eedge + (int64_t)lam * C.n_edges;
    const double* itab = C.itab + (int64_t)lam * nb * 3;
    double carry[3] = {pre[0], pre[1], pre[2]};
    for (int first = 0; first < nb; first += 32) {
      const int k = first + lane;
      // up to each bin, and what the bins before it deposited: the lane below's sum (this
      // one's less its own would lose what its own dwarfs)
      double run[3], before[3];
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        run[j] = k < nb ? acc[4 * k + j] : 0.0;
        for (int off = 1; off < 32; off <<= 1) {
          const double up = __shfl_up_sync(0xffffffffu, run[j], off);
          if (lane >= off) run[j] += up;
        }
        before[j] = __shfl_up_sync(0xffffffffu, run[j], 1);
        if (lane == 0) before[j] = 0.0;
      }
      if (k < nb) {
        const double a = carry[0] + before[0], b = carry[1] + before[1], c = carry[2] + before[2];
        const double e_k = C.edges[k];
        const double width = C.edges[k + 1] - e_k;
        const double a_loc = a + e_k * (b + c * e_k);
        const double b_loc = b + 2.0 * c * e_k;
        const double value = eedge[k] * width *
                             (a_loc * itab[3 * k] + width * (b_loc * itab[3 * k + 1] + width * c * itab[3 * k + 2]));
        band_bins[(int64_t)lam * nb + k] = area * (value + acc[4 * k + 3]);
      }
#pragma unroll
      for (int j = 0; j < 3; ++j) carry[j] += __shfl_sync(0xffffffffu, run[j], 31);
    }
  }
  __syncthreads();
  for (int k = threadIdx.x; k < nb; k += blockDim.x) {
    double sum = 0.0;
    for (int lam = 0; lam < NL; ++lam) sum += band_bins[(int64_t)lam * nb + k];
    bins[(int64_t)d * nb + k] = sum;
  }
}

// ------------------------------------------------------------------ host side

struct O1Workspace {
  long long* pkeys;
  double* prows;
  int32_t* pcount;
  int32_t* tiles;
  long long* parent_keys;  // screen tables: parent pixels (same capacity as pkeys)
  double* parent_rows;
  int32_t* parent_tiles;
  int32_t* parent_row;     // row of each parent slot in the pencil table
  long long* gkeys;
  double* grows;
  int32_t* gcount;
  int32_t* sorted;
  int32_t* batch_list;
  int32_t* batch_total;  // [4]: batches, then batches deferred to the full-size grid
  int32_t* deferred;     // batches too large for one warp
  double* accum;
  unsigned long long* sort_keys;  // tables above kO1SmemSort only
  int32_t* sort_slots;
  size_t bytes;
};

static size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

static O1Workspace o1_layout(const lh_order1_config& C, int64_t pencil_capacity, int64_t ring_capacity,
                             int32_t n_work, unsigned char* base) {
  O1Workspace W{};
  size_t off = 0;
  auto take = [&](size_t bytes) {
    unsigned char* p = base ? base + off : nullptr;
    off += align256(bytes);
    return p;
  };
  const int nb = C.n_edges - 1;
  W.pkeys = reinterpret_cast<long long*>(take(sizeof(long long) * ring_capacity));
  W.prows = reinterpret_cast<double*>(take(sizeof(double) * kO1Moments * ring_capacity));
  W.pcount = reinterpret_cast<int32_t*>(take(sizeof(int32_t) * 4));
  W.tiles = reinterpret_cast<int32_t*>(take(sizeof(int32_t) * (ring_capacity / kO1Tile + 1)));
  const int64_t parent_cap = C.screen ? ring_capacity : 0;
  W.parent_keys = reinterpret_cast<long long*>(take(sizeof(long long) * parent_cap));
  W.parent_rows = reinterpret_cast<double*>(take(sizeof(double) * kO1Moments * parent_cap));
  W.parent_tiles = reinterpret_cast<int32_t*>(take(sizeof(int32_t) * (parent_cap / kO1Tile + 1)));
  W.parent_row = reinterpret_cast<int32_t*>(take(sizeof(int32_t) * parent_cap));
  W.gkeys = reinterpret_cast<long long*>(take(sizeof(long long) * (size_t)n_work * C.group_capacity));
  W.grows = reinterpret_cast<double*>(
      take(sizeof(double) * kO1MaxValues * (size_t)n_work * C.group_capacity));
  W.gcount = reinterpret_cast<int32_t*>(take(sizeof(int32_t) * (size_t)n_work));
  W.sorted = reinterpret_cast<int32_t*>(take(sizeof(int32_t) * (size_t)n_work * C.group_capacity));
  W.batch_list =
      reinterpret_cast<int32_t*>(take(sizeof(int32_t) * 3 * (size_t)n_work * C.group_capacity));
  W.batch_total = reinterpret_cast<int32_t*>(take(sizeof(int32_t) * 4));
  W.deferred = reinterpret_cast<int32_t*>(take(sizeof(int32_t) * (size_t)n_work * C.group_capacity));
  W.accum = reinterpret_cast<double*>(take(sizeof(double) * (size_t)n_work * C.n_bands * (3 + 4 * nb + 1)));
  const size_t sort_n = C.group_capacity > kO1SmemSort ? (size_t)n_work * C.group_capacity : 0;
  W.sort_keys = reinterpret_cast<unsigned long long*>(take(sizeof(unsigned long long) * sort_n));
  W.sort_slots = reinterpret_cast<int32_t*>(take(sizeof(int32_t) * sort_n));
  (void)pencil_capacity;
  W.bytes = off;
  return W;
}

static int64_t next_pow2(int64_t x) {
  int64_t p = 1;
  while (p < x) p <<= 1;
  return p;
}

int64_t o1_ring_capacity(int64_t n_subseg, int32_t ring_nodes) {
  return next_pow2(std::max<int64_t>(4096, n_subseg * ring_nodes));
}

static int grid_for(int64_t items, int threads) {
  int64_t blocks = (items + threads - 1) / threads;
  if (blocks < 1) blocks = 1;
  if (blocks > 148 * 64) blocks = 148 * 64;
  return (int)blocks;
}

}  // namespace lh

namespace {
bool o1_config_valid(const lh_order1_config* C) {
  if (!C) return false;
  if (C->n_om < 1 || !C->om_pos || !C->om_look || !C->om_area) return false;
  if (C->n_bands < 1 || C->n_bands > lh::kO1MaxBands || !C->mus || !C->mut || !C->speed ||
      !C->s0w || !C->s2w)
    return false;
  if (C->n_mono < 1 || C->n_mono > lh::kO1MaxMono || C->max_power < 0 || C->max_power > 4 ||
      !C->coef || !C->ipow || !C->jpow)
    return false;
  if (C->n_edges < 2 || !C->edges || !C->eedge || !C->itab) return false;
  if (C->max_path_nodes < 4 || C->max_path_nodes > lh::kO1MaxNodes) return false;
  if (C->n_gauss < 1 || C->n_gauss > lh::kO1MaxGauss || !C->gauss_tau || !C->gauss_w) return false;
  if (C->group_capacity < 1024 || C->group_capacity > (1 << 20) ||
      (C->group_capacity & (C->group_capacity - 1)))
    return false;
  if (C->theta_bins < 2 || C->theta_bins > 128 || !(C->theta_lo > 0) || !(C->theta_ratio > 0) ||
      !(C->tau_step > 0) || !(C->log_r_step > 0))
    return false;
  if (C->pixel_face < 1 || C->ring_nodes < 1 || !(C->cell_m > 0)) return false;
  if (C->screen && (C->parent_face < 1 || C->pixel_face % C->parent_face || C->compute_bins))
    return false;
  return true;
}
}  // namespace

extern "C" size_t lh_order1_workspace_bytes(const lh_order1_config* C, int64_t n_subseg,
                                            int32_t n_work) {
  if (!o1_config_valid(C) || n_subseg < 0 || n_work < 0) return 0;
  const int64_t ring_cap = lh::o1_ring_capacity(n_subseg, C->ring_nodes);
  return lh::o1_layout(*C, 0, ring_cap, n_work, nullptr).bytes;
}

extern "C" int lh_order1_pencils(const lh_order1_config* C, const lh_order1_elements* E,
                                 const lh_order1_pencil_table* P, int32_t* n_pencils_device,
                                 void* workspace, size_t workspace_bytes, int32_t* status,
                                 void* stream) {
  if (!o1_config_valid(C) || !E || !P || !n_pencils_device || !status) return LH_EINVAL;
  if (C->screen && !P->parent) return LH_EINVAL;
  if (E->n_el < 0 || E->n_subseg < 0 || (E->n_el && (!E->subseg_offset || !E->start ||
                                                     !E->direction || !E->length || !E->c0 ||
                                                     !E->c2 || !E->cone_cos || !E->t0 || !E->t1)))
    return LH_EINVAL;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int64_t ring_cap = lh::o1_ring_capacity(E->n_subseg, C->ring_nodes);
  lh::O1Workspace W = lh::o1_layout(*C, 0, ring_cap, 0, static_cast<unsigned char*>(workspace));
  if (!workspace || workspace_bytes < W.bytes) return LH_ENOMEM;
  cudaMemsetAsync(n_pencils_device, 0, sizeof(int32_t), s);
  if (E->n_el == 0 || E->n_subseg == 0) return cudaGetLastError() == cudaSuccess ? LH_OK : LH_ECUDA;
  cudaMemsetAsync(W.pkeys, 0xff, sizeof(long long) * ring_cap, s);  // rows: zeroed on claim
  const int64_t ring_threads = ((E->n_subseg + 31) / 32) * 32 *
                               ((C->ring_nodes + lh::kO1RingBlock - 1) / lh::kO1RingBlock);
  {
    lh::TimedLaunch timed_launch(LH_KT_O1_RING, s);
    lh::o1_ring_kernel<<<lh::grid_for(ring_threads, lh::kO1RingThreads), lh::kO1RingThreads, 0, s>>>(
        *C, *E, E->subseg_offset, E->n_subseg, W.pkeys, ring_cap, W.prows, status);
  }
  const int64_t n_tiles = (ring_cap + lh::kO1Tile - 1) / lh::kO1Tile;
  if (!C->screen) {
    lh::o1_tile_count_kernel<<<(unsigned)n_tiles, lh::kO1FinishThreads, 0, s>>>(
        W.pkeys, W.prows, ring_cap, W.tiles);
    lh::o1_tile_scan_kernel<<<1, 1024, 0, s>>>(W.tiles, n_tiles, n_pencils_device);
    lh::o1_finish_kernel<<<(unsigned)n_tiles, lh::kO1FinishThreads, 0, s>>>(
        W.pkeys, ring_cap, W.prows, *P, W.tiles, n_pencils_device, nullptr, nullptr, nullptr, 0,
        nullptr, 0, 0, status);
    return cudaGetLastError() == cudaSuccess ? LH_OK : LH_ECUDA;
  }
  // the coarse screen: parents (sums of their children) take rows [0, n_parents),
  // children follow with their parent's row
  cudaMemsetAsync(W.parent_keys, 0xff, sizeof(long long) * ring_cap, s);
  cudaMemsetAsync(W.parent_row, 0xff, sizeof(int32_t) * ring_cap, s);
  lh::o1_parent_kernel<<<lh::grid_for(ring_cap, lh::kO1FinishThreads), lh::kO1FinishThreads, 0, s>>>(
      W.pkeys, W.prows, ring_cap, C->pixel_face, C->parent_face, W.parent_keys, W.parent_rows,
      ring_cap, status);
  lh::o1_tile_count_kernel<<<(unsigned)n_tiles, lh::kO1FinishThreads, 0, s>>>(
      W.parent_keys, W.parent_rows, ring_cap, W.parent_tiles);
  lh::o1_tile_scan_kernel<<<1, 1024, 0, s>>>(W.parent_tiles, n_tiles, W.pcount + 1);
  lh::o1_finish_kernel<<<(unsigned)n_tiles, lh::kO1FinishThreads, 0, s>>>(
      W.parent_keys, ring_cap, W.parent_rows, *P, W.parent_tiles, W.pcount + 1, nullptr,
      W.parent_row, nullptr, 0, nullptr, 0, 0, status);
  lh::o1_tile_count_kernel<<<(unsigned)n_tiles, lh::kO1FinishThreads, 0, s>>>(
      W.pkeys, W.prows, ring_cap, W.tiles);
  lh::o1_tile_scan_kernel<<<1, 1024, 0, s>>>(W.tiles, n_tiles, W.pcount);
  lh::o1_finish_kernel<<<(unsigned)n_tiles, lh::kO1FinishThreads, 0, s>>>(
      W.pkeys, ring_cap, W.prows, *P, W.tiles, W.pcount, W.pcount + 1, nullptr, W.parent_keys,
      ring_cap, W.parent_row, C->pixel_face, C->parent_face, status);
  lh::o1_total_kernel<<<1, 32, 0, s>>>(W.pcount, W.pcount + 1, n_pencils_device);
  return cudaGetLastError() == cudaSuccess ? LH_OK : LH_ECUDA;
}

extern "C" int lh_order1_grouped(const lh_order1_config* C, const lh_order1_pencil_table* P,
                                 int32_t n_pencils, const int32_t* n_pencils_device,
                                 const int32_t* work, int32_t n_work,
                                 const double* origins, double* charge, double* bins,
                                 void* workspace, size_t workspace_bytes, int32_t* status,
                                 void* stream) {
  if (!o1_config_valid(C) || !P || n_pencils < 0 || n_work < 0 || !status || !charge) return LH_EINVAL;
  if (C->screen && !P->parent) return LH_EINVAL;
  if (n_work && (!work || !origins)) return LH_EINVAL;
  if (C->compute_bins && !bins) return LH_EINVAL;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // the grouped stage reuses the workspace from its start (pencils live elsewhere)
  lh::O1Workspace W = lh::o1_layout(*C, 0, 0, n_work, static_cast<unsigned char*>(workspace));
  if (!workspace || workspace_bytes < W.bytes) return LH_ENOMEM;
  const int nb = C->n_edges - 1;
  cudaMemsetAsync(charge, 0, sizeof(double) * C->n_om, s);
  if (C->compute_bins) cudaMemsetAsync(bins, 0, sizeof(double) * (size_t)C->n_om * nb, s);
  if (n_work == 0 || n_pencils == 0) return cudaGetLastError() == cudaSuccess ? LH_OK : LH_ECUDA;
  const int64_t cap = C->group_capacity;
  cudaMemsetAsync(W.gkeys, 0xff, sizeof(long long) * (size_t)n_work * cap, s);  // rows: zeroed on claim
  cudaMemsetAsync(W.gcount, 0, sizeof(int32_t) * (size_t)n_work, s);
  cudaMemsetAsync(W.batch_total, 0, sizeof(int32_t) * 4, s);
  cudaMemsetAsync(W.accum, 0, sizeof(double) * (size_t)n_work * C->n_bands * (3 + 4 * nb + 1), s);
  const size_t group_smem =
      sizeof(double) * 32 * (256 / 32) * (2 * C->n_mono + 6 + lh::kO1PencilFields);
  if (group_smem > 48 * 1024 &&
      cudaFuncSetAttribute(C->screen ? lh::o1_group_kernel<true> : lh::o1_group_kernel<false>,
                           cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)group_smem) != cudaSuccess)
    return LH_ECUDA;
  {
    lh::TimedLaunch timed_launch(LH_KT_O1_GROUP, s);
    // persistent: two resident CTAs per SM take the warp chunks in turn (the
    // host's pencil count is the table's capacity, far above the pencils a
    // shower makes, so a grid sized from it would mostly launch idle CTAs)
    const int group_grid = std::min(lh::grid_for((int64_t)n_work * n_pencils, 256), 148 * 2);
    unsigned long long* units = lh::kernel_units() ? lh::kernel_units() + LH_KT_O1_GROUP : nullptr;
    if (C->screen)
      lh::o1_group_kernel<true><<<group_grid, 256, group_smem, s>>>(
          *C, *P, n_pencils, n_pencils_device, work, n_work, origins, W.gkeys, W.grows,
          W.gcount, status, units);
    else
      lh::o1_group_kernel<false><<<group_grid, 256, group_smem, s>>>(
          *C, *P, n_pencils, n_pencils_device, work, n_work, origins, W.gkeys, W.grows,
          W.gcount, status, units);
  }
  const size_t sort_smem =
      cap <= lh::kO1SmemSort ? sizeof(unsigned long long) * (size_t)cap : 0;
  if (sort_smem > 48 * 1024 &&
      cudaFuncSetAttribute(lh::o1_batches_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)sort_smem) != cudaSuccess)
    return LH_ECUDA;
  lh::o1_batches_kernel<<<n_work, 1024, sort_smem, s>>>(*C, n_work, W.gkeys, W.sorted, W.batch_list,
                                                        W.batch_total, W.sort_keys, W.sort_slots,
                                                        status);
  const size_t warp_smem = lh::o1_warp_batch_bytes(*C);
  const size_t full_smem = sizeof(lh::O1BatchShared);
  if (cudaFuncSetAttribute(lh::o1_batch_warp_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)warp_smem) != cudaSuccess ||
      cudaFuncSetAttribute(lh::o1_batch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)full_smem) != cudaSuccess)
    return LH_ECUDA;
  {
    lh::TimedLaunch timed_launch(LH_KT_O1_BATCH, s);
    lh::o1_batch_warp_kernel<<<148 * 5, 32 * lh::kO1BatchWarps, warp_smem, s>>>(
        *C, W.gkeys, W.grows, W.sorted, W.batch_list, W.batch_total, W.deferred,
        W.batch_total + 1, W.accum, status);
    lh::o1_batch_kernel<<<148 * 2, lh::kO1BatchThreads, full_smem, s>>>(
        *C, W.gkeys, W.grows, W.sorted, W.batch_list, W.deferred, W.batch_total + 1, W.accum,
        status);
  }
  const size_t fin_smem = sizeof(double) * C->n_bands * nb;
  if (fin_smem > 200 * 1024) return LH_EUNSUPPORTED;
  if (cudaFuncSetAttribute(lh::o1_finalize_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)fin_smem) != cudaSuccess)
    return LH_ECUDA;
  lh::o1_finalize_kernel<<<n_work, 32 * lh::kO1FinalWarps, fin_smem, s>>>(*C, work, n_work, W.accum, charge, bins);
  return cudaGetLastError() == cudaSuccess ? LH_OK : LH_ECUDA;
}
