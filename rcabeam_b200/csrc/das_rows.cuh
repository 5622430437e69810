// Frame-batched RCA delay-and-sum on the CUDA cores (float32 arithmetic, exact
// geometry): OPW, XDoppler, separate apertures, RC-FMAS, DMAS-CCF-ACF and the
// subset statistics of St-SW from one staged pipeline (the last three from a few
// thousand voxels on: das_generic.cuh).  The reference does the same arithmetic per
// sample from a per-call geometry table (ensemble.cu:143-454).
//
// Work: an item is a tile of 128 voxels (consecutive in a spatially compact
// order) x a chunk of up to 104 frames; a CTA runs one.  Its steps are the
// (aperture, channel, angle) triples; for each, the tile's interpolation taps fall
// in a short window of consecutive sample rows.
//   * Builder warps (3 as a rule, steps dealt round robin) form a step's taps --
//     receive delays once per channel, transmit delays from a per-tile table, both
//     as fixed-point sample positions that are simply added -- and start the
//     window's copy into a ring stage: TMA boxes of 8 rows, or bulk copies of the
//     rows where odd frame counts or unaligned buffers rule a tensor map out.
//     Only the rows that taps need are copied.
//   * Where the walk changes channel with every step, a helper warp per builder
//     forms its receive delays one step ahead (48 x 96 x 48 voxels, 384 x 128 x 7 x
//     64, RC-FMAS: 37.6 ms without, 30.7 with).
//   * Consumer warps own 32 voxels x up to 26 frames each: a lane one voxel, its
//     frames' sums in registers.  Per step a lane reads its tap once and then both
//     rows of each frame pair with 16-byte shared-memory loads at immediate
//     offsets; rows lie 16 bytes beyond a multiple of 128 apart, so eight lanes on
//     neighbouring rows hit distinct banks.
//
// What bounds it: those loads.  16 bytes per interpolated sample against 128
// bytes per clock and SM allow 8 samples per clock; ncu shows the shared-memory
// pipe 90 % busy with 0.8 % bank conflicts, the issue slots 64 %.  Lanes hold
// voxels rather than frames because taps, row addresses and loop control then
// cost one register each for 26 frames; a form with lanes over frames and each
// row kept in registers for the voxels that share it loaded less but spent its
// issue slots on selecting rows (5.5 samples per clock against 6.6).  One producer
// warp per 64 voxels, which formed every tap in float64 and with it set the pace
// of short ensembles and of odd frame counts, was what this form replaced.
//
// Measured on one B200 (median of runs, DAS alone): 64 x 96 x 64 voxels, 512 x 128
// x 11 x 200 channels 185.5 -> 118.4 ms (6.65 samples per clock and SM); 64 x 64 x
// 64, 100 frames 86.1 -> 44.0 ms; 64 x 128 x 64, 384 x 128 x 7 x 32 41.5 -> 21.8 ms;
// 32 x 64 x 32, 256 x 64 x 5 x 16 2.16 -> 1.00 ms; 40 x 70 x 36, 300 x 96 x 9 x 75
// (odd frames, no tensor map) 182 -> 12.1 ms.
#pragma once

#include <climits>
#include <type_traits>

#include "common.cuh"

namespace rcb {
namespace das {

constexpr int kTileVoxels = 128;
constexpr int kBlocks = kTileVoxels / 32;  // consumer warps per frame group
constexpr int kMaxBuilders = 4;
constexpr int kMaxGroups = 4;              // frame groups of an item (plan_items: 104 frames in 26s, 64 in 16s)
constexpr int kBoxRows = 8;                // sample rows of one TMA box
constexpr int kMaxBoxes = 32;              // boxes of one window: each lane issues at most one

// St-SW (method 4) with K angle subsets is kStsw + K.
enum Mode : int { kOpw = 0, kXdoppler = 1, kFmas = 2, kDmas = 3, kApertures = 5, kStsw = 8 };
template <int MODE>
constexpr int kSubsets = MODE > kStsw ? MODE - kStsw : 0;
// Stage tags: the run a step belongs to and whether another window of the same
// step follows; or the end of an item.
constexpr int kTagEnd = -1, kTagMore = 1 << 30, kTagMask = kTagMore - 1;

struct Args {
  const void* rc;
  const void* cr;
  const float* scan;
  const float* xe;
  const float* ye;
  const float* angles;
  const float* starts;
  const unsigned* order;  // traversal order (nullptr = identity)
  float* pd;
  float2* signal;
  int ns, nc, na, nt, nv;
  double c, fs, fd, fn;
  int* err;
  const double* offsets;  // [2][nc] receive-delay offsets in seconds (RC, CR), or nullptr
  float2* series;         // St-SW: (nv, K^2, nt) correlation series
};

// Packed (slab, sample, frame) channels of both apertures as TMA tensors.
struct Maps {
  CUtensorMap map[2];
};

// How one ensemble is split into items (host, plan_rows()).
struct Shape {
  int frames;      // frames per item (2 pairs groups)
  int groups;      // frame groups: consumer warps of one voxel block
  int pairs;       // frame pairs per thread
  int chunks;      // items per tile
  int rows;        // sample rows a stage holds with half as many stages
  int rows_deep;   // and with all of them
  int pitch;       // bytes between staged rows
  int boxes;       // 1: TMA boxes of 8 rows; 0: bulk copies of rows
  int contiguous;  // bulk copies: an item spans all frames, so a window is one copy
  int tx_table;    // 1: transmit delays of one aperture are tabulated per tile
};

// Shared memory and warps of one launch.
struct Layout {
  int builders;     // builder warps
  int helpers;      // warps that form receive delays for them: one each, or none
  int stages;       // ring stages: two per builder
  int stage_bytes;  // taps and rows of one of them
  int zero_bytes;   // a row of zeros: what voxels outside a step read
  int stash_bytes;  // partial results of the methods that fold sums
  int angles;       // angle table entries
  int table_bytes;  // transmit delay table
  int threads;
  int smem;
};

// ------------------------------------------------------------ shared memory --
constexpr int kTapBytes = kTileVoxels * 16;  // per voxel: weight, phase, offset of its row
constexpr int kMaxStages = 16;

struct Shared {
  unsigned char* base;    // stages
  unsigned char* zero;
  float* stash;
  uint64_t* full;
  uint64_t* empty;
  uint64_t* rx_full;      // [2][kMaxBuilders] helpers' receive delays ready, taken
  uint64_t* rx_empty;
  int2* tag;              // run of the stage's step; voxel blocks with a tap in it (bit per block)
  unsigned* vox;          // voxel ids of the tile
  float* pos;             // [3][128] x, z, y
  double* power;          // [2][groups][128] sums over a group's frames
  float* active;          // [128] channels inside the aperture (DMAS)
  float* bounds;          // tile minimum and maximum of x and of y, maximum of z, rows a step can span
  double* angle;          // [na][3] cos, sin, start
  double* limit;          // [128] f-number half aperture at the voxel's depth
  long long* rx;          // [2][kMaxBuilders][128] receive delays: two blocks of channels, or two steps per builder
  unsigned* rxc;
  long long* tx;          // [na][128] transmit delay minus start, 2^-32 samples
  unsigned* txc;          // [na][128] transmit phase, 2^-32 cycles
};

__host__ __device__ inline int align16(int x) { return (x + 15) & ~15; }

// The ring of one item: tiles that are compact in space run two stages per
// builder, others one of twice the size, so that a step's window still fits one.
struct Ring {
  int stages, bytes, rows;
};
constexpr int kRxEntries = 2 * kMaxBuilders * kTileVoxels;
constexpr int kFixedBytes = kMaxStages * 24 + 4 * kMaxBuilders * 8 + kTileVoxels * (4 * (1 + 3 + 1) + 8 * 2 * kMaxGroups) + 64 + kTileVoxels * 8 + kRxEntries * 12;

__device__ __forceinline__ Shared carve(unsigned char* smem, const Layout& l) {
  Shared s;
  s.base = smem;
  unsigned char* q = smem + l.stages * l.stage_bytes;
  s.zero = q;
  q += l.zero_bytes;
  s.stash = reinterpret_cast<float*>(q);
  q += l.stash_bytes;
  s.tx = reinterpret_cast<long long*>(q);
  s.txc = reinterpret_cast<unsigned*>(q + l.table_bytes / 3 * 2);
  q += l.table_bytes;
  s.angle = reinterpret_cast<double*>(q);
  s.limit = s.angle + 3 * l.angles;
  s.rx = reinterpret_cast<long long*>(s.limit + kTileVoxels);
  s.full = reinterpret_cast<uint64_t*>(s.rx + kRxEntries);
  s.empty = s.full + kMaxStages;
  s.rx_full = s.empty + kMaxStages;
  s.rx_empty = s.rx_full + 2 * kMaxBuilders;
  s.tag = reinterpret_cast<int2*>(s.rx_empty + 2 * kMaxBuilders);
  s.vox = reinterpret_cast<unsigned*>(s.tag + kMaxStages);
  s.pos = reinterpret_cast<float*>(s.vox + kTileVoxels);
  s.power = reinterpret_cast<double*>(s.pos + 3 * kTileVoxels);
  s.active = reinterpret_cast<float*>(s.power + 2 * kMaxGroups * kTileVoxels);
  s.bounds = s.active + kTileVoxels;
  s.rxc = reinterpret_cast<unsigned*>(s.bounds + 16);
  return s;
}

// ------------------------------------------------------------------ delays --
// Sample positions and demodulation cycles are summed as fixed-point numbers of
// 2^-32: a step's tap then costs a 64-bit and a 32-bit integer addition per voxel, and
// the cycles wrap by themselves.  The position's rounding is below that of the float32
// weight formed from it for weights from 2^-8 on; smaller weights are off by up to
// 2.3e-10 of a sample interval, against sums whose float32 rounding is 1e-7.
constexpr long long kNever = -(1ll << 62);      // a delay outside every window
constexpr double kFixedLimit = 536870912.0;     // |delay| < 2^29 samples

__device__ __forceinline__ long long fixed32(double x) {
  // Adding 1.5 x 2^20 leaves 32 fraction bits in the mantissa, rounded to nearest.
  if (fabs(x) < 524288.0) return __double_as_longlong(x + 1572864.0) - 0x4138000000000000ll;
  return fabs(x) < kFixedLimit ? __double2ll_rn(x * 4294967296.0) : kNever;
}
__device__ __forceinline__ unsigned cycles32(double cyc) {
  if (fabs(cyc) < 524288.0) return unsigned(__double_as_longlong(cyc + 1572864.0));
  cyc -= rint(cyc);
  return unsigned(__double2ll_rn(cyc * 4294967296.0));
}

// sqrt(m) to about 2^-43: the float32 reciprocal root and one Newton step in
// float64 (a path of 1000 samples keeps 1e-10 of a sample).
__device__ __forceinline__ double path_root(double m) {
  if (!(m > 1e-30 && m < 1e30)) return __dsqrt_rn(m);
  const double y = double(rsqrtf(float(m)));
  return m * (y * fma(-0.5 * m * y, y, 1.5));
}

// ------------------------------------------------------------------ copies --
__device__ __forceinline__ void bulk_copy(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}

// A copy of [start, start + len) of the buffer [lo, hi) puts byte `start` at
// dst + (start & 15).  widen() gives the 16-byte bounds [a, b) of the bulk copy,
// which stay inside the buffer; what they leave out (an unaligned first sample of the
// whole ensemble, or last one of a slab) stage_copy() stores by hand, E bytes at a time.
__device__ __forceinline__ uint32_t widen(uintptr_t start, uintptr_t len, uintptr_t lo, uintptr_t hi, uintptr_t* a,
                                          uintptr_t* b) {
  *a = start & ~uintptr_t(15);
  *b = (start + len + 15) & ~uintptr_t(15);
  if (*a < lo) *a += 16;
  if (*b > hi) *b -= 16;
  if (*b < *a) *b = *a;
  return uint32_t(*b - *a);
}
template <int E>
__device__ __forceinline__ void stage_copy(unsigned char* dst, uintptr_t start, uintptr_t len, uintptr_t a,
                                           uintptr_t b, uint64_t* bar) {
  unsigned char* origin = dst - ptrdiff_t(start & ~uintptr_t(15));  // dst address of global address 0
  if (b > a) bulk_copy(origin + a, reinterpret_cast<const void*>(a), uint32_t(b - a), bar);
  using W = typename std::conditional<E == 8, unsigned long long, unsigned>::type;
  for (uintptr_t q = start; q < start + len && q < a; q += E)
    *reinterpret_cast<W*>(origin + q) = *reinterpret_cast<const W*>(q);
  for (uintptr_t q = b > start ? b : start; q < start + len; q += E)
    if (q >= a) *reinterpret_cast<W*>(origin + q) = *reinterpret_cast<const W*>(q);
  if (start < a || b < start + len) fence_async_smem();  // a later window's copy may cover these bytes
}

// Sample position in float64, in the operation order of the float64 oracle:
// decides taps next to the ends of the recorded window.  Returns the tap row
// (-1: outside) and its weight.
__device__ __noinline__ int edge_tap(double v, double u, double z, double e, double extra, double cs, double sn,
                                     double start, double c, double fs, int ns, float* w) {
  bool active;
  const double trx = __dadd_rn(receive_delay(v, z, e, c, -1.0, &active), extra);
  const double ttx = transmit_delay(u, z, cs, sn, c);
  const double sample = __dmul_rn(__dadd_rn(__dadd_rn(ttx, trx), -start), fs);
  if (!(sample >= 0.0 && sample <= double(ns - 1))) return -1;
  const double fl = floor(sample);
  *w = float(sample - fl);
  return int(fl);
}

// ---------------------------------------------------------------- builders --
template <bool HALF, bool BOXES>
struct Builder {
  static constexpr int E = HALF ? 4 : 8;
  const Args& p;
  const Shape& sp;
  const Layout& lt;
  const Shared& sh;
  const Ring ring;
  const CUtensorMap* maps;  // RC, CR (boxes)
  int frame0, warp, lane;
  int stage;        // this builder's next stage
  int turn;         // steps until this builder's next one
  uint32_t phase;   // parity of each stage's next use
  bool ok;
  double ks, kc;    // samples and demodulation cycles per metre

  __device__ __forceinline__ Builder(const Args& p_, const Shape& sp_, const Layout& lt_, const Shared& sh_,
                                     const Ring& ring_, const CUtensorMap* maps_, int f0, int warp_, uint32_t phase_)
      : p(p_), sp(sp_), lt(lt_), sh(sh_), ring(ring_), maps(maps_), frame0(f0), warp(warp_),
        lane(threadIdx.x & 31), phase(phase_), ok(true), ks(p_.fs / p_.c), kc(p_.fd / p_.c) {
    turn = stage = warp;  // every item starts at stage 0
  }

  __device__ __forceinline__ void sync_builders() const {
    asm volatile("bar.sync 1, %0;" ::"r"(lt.builders * 32) : "memory");
  }

  // Receive delays and phases of this lane's voxels for one channel.
  __device__ __forceinline__ void receive(int cfg, int ch, long long (&rx)[4], unsigned (&rxc)[4]) const {
    const double e = double((cfg ? p.ye : p.xe)[ch]), extra = p.offsets ? p.offsets[cfg * p.nc + ch] : 0.0;
    double s[4], cyc[4], most = 0.0;
    bool out[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int i = lane + 32 * j;
      const double z = double(sh.pos[kTileVoxels + i]);
      const double d = __dadd_rn(double(sh.pos[(cfg ? 2 : 0) * kTileVoxels + i]), -e);
      const double r = path_root(fma(d, d, z * z));
      out[j] = sh.vox[i] == UINT_MAX || (p.fn > 0.0 && !(fabs(d) <= sh.limit[i]));
      s[j] = fma(r, ks, extra * p.fs);
      cyc[j] = fma(r, kc, extra * p.fd);
      most = fmax(most, fabs(s[j]) + fabs(cyc[j]));
      if (isnan(r)) most = INFINITY;
    }
    // One range check for all (fixed32, cycles32).
    if (__all_sync(0xffffffffu, most < 524288.0)) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        rx[j] = __double_as_longlong(s[j] + 1572864.0) - 0x4138000000000000ll;
        rxc[j] = unsigned(__double_as_longlong(cyc[j] + 1572864.0));
      }
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        rx[j] = fixed32(s[j]);
        rxc[j] = cycles32(cyc[j]);
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (out[j]) rx[j] = kNever;
  }

  // The two slots of receive delays between a helper and its builder.
  __device__ __forceinline__ int rx_at(int s) const { return (s * kMaxBuilders + warp) * kTileVoxels + lane; }
  __device__ __forceinline__ bool rx_wait(uint64_t* bars, int s, uint32_t flip, int code) {
    ok = ok && __all_sync(0xffffffffu, mbar_wait_fast(&bars[s * kMaxBuilders + warp], ((phase >> (30 + s)) & 1) ^ flip,
                                                      p.err, code));
    phase ^= 1u << (30 + s);
    return ok;
  }
  __device__ __forceinline__ void rx_arrive(uint64_t* bars, int s) const {
    __syncwarp();
    if (lane == 0) mbar_arrive(&bars[s * kMaxBuilders + warp]);
  }

  // Transmit delay (minus the angle's start) and phase of tile slot i.
  __device__ __forceinline__ void transmit(int cfg, int a, int i, long long* delay, unsigned* cyc) const {
    const double u = double(sh.pos[(cfg ? 0 : 2) * kTileVoxels + i]), z = double(sh.pos[kTileVoxels + i]);
    const double path = fma(z, sh.angle[3 * a], u * sh.angle[3 * a + 1]);
    *delay = fixed32(fma(path, ks, -sh.angle[3 * a + 2] * p.fs));
    *cyc = cycles32(path * kc);
  }

  // Fills the transmit table of one aperture (all builder warps together).
  __device__ __forceinline__ void fill_table(int cfg) const {
    if (!sp.tx_table) return;
    sync_builders();  // the previous aperture's reads are done
    for (int e = warp * 32 + lane; e < p.na * kTileVoxels; e += lt.builders * 32)
      transmit(cfg, e / kTileVoxels, e % kTileVoxels, sh.tx + e, sh.txc + e);
    sync_builders();
  }

  // False when no voxel of the tile can lie in the channel's f-number aperture
  // (same answer in every builder; a superset of the per-voxel test).
  __device__ __forceinline__ bool reachable(int cfg, int ch) const {
    if (p.fn <= 0.0) return true;
    const double e = double((cfg ? p.ye : p.xe)[ch]);
    const double lo = double(sh.bounds[cfg ? 2 : 0]), hi = double(sh.bounds[cfg ? 3 : 1]);
    const double gap = fmax(fmax(__dadd_rn(lo, -e), __dadd_rn(e, -hi)), 0.0);
    return !(gap > __ddiv_rn(double(sh.bounds[4]), __dmul_rn(2.0, p.fn)));
  }

  __device__ __forceinline__ bool claim() {
    ok = ok && __all_sync(0xffffffffu,
                          mbar_wait_fast(&sh.empty[stage], ((phase >> stage) & 1) ^ 1, p.err, kErrWaitEmpty));
    return ok;
  }
  __device__ __forceinline__ void publish(int tag, unsigned blocks) {
    if (lane == 0) sh.tag[stage] = make_int2(tag, int(blocks));
    __syncwarp();
    if (lane == 0) mbar_arrive(&sh.full[stage]);
    phase ^= 1u << stage;
  }
  __device__ __forceinline__ void next_stage() {
    stage += lt.builders;
    if (stage >= ring.stages) stage -= ring.stages;
  }

  // Starts the copy of the `count` rows from address row0 (slab row `base`) of
  // the buffer [lo, hi).
  __device__ __forceinline__ void copy_rows(unsigned char* data, int cfg, int slab, int base, int count,
                                            uintptr_t row0, uintptr_t lo, uintptr_t hi) const {
    uint64_t* bar = &sh.full[stage];
    if constexpr (BOXES) {
      const int n = (count + kBoxRows - 1) / kBoxRows;
      if (lane == 0) expect_tx(bar, uint32_t(n * kBoxRows * sp.pitch));
      __syncwarp();
      if (lane < n)
        tma_load_3d(data + lane * kBoxRows * sp.pitch, maps + cfg, bar, frame0, base + lane * kBoxRows, slab);
    } else {
      const uintptr_t stride = uintptr_t(p.nt) * E;
      const bool past_end = count > p.ns - base;
      if (past_end) count = p.ns - base;
      uintptr_t a, b;
      if (sp.contiguous) {
        // Not a byte of the next slab: its place is the row of zeros stored below.
        if (past_end) hi = row0 + uintptr_t(count) * stride;
        if (lane == 0) {
          expect_tx(bar, widen(row0, count * stride, lo, hi, &a, &b));
          stage_copy<E>(data, row0, count * stride, a, b, bar);
        }
      } else {
        const uint32_t len = uint32_t(min(sp.frames, p.nt - frame0)) * E;
        uint32_t bytes = 0;
        for (int r = lane; r < count; r += 32) bytes += widen(row0 + r * stride, len, lo, hi, &a, &b);
        bytes = __reduce_add_sync(0xffffffffu, bytes);
        if (lane == 0) expect_tx(bar, bytes);
        __syncwarp();
        // Row r's samples start at data + (row0 & 15) + r pitch: the pitch equals
        // the row stride modulo 16, so that the copies' 16-byte bounds agree.
        for (int r = lane; r < count; r += 32) {
          const unsigned at = unsigned(row0 & 15) + unsigned(r * sp.pitch);
          widen(row0 + r * stride, len, lo, hi, &a, &b);
          stage_copy<E>(data + (at & ~15u), row0 + r * stride, len, a, b, bar);
        }
      }
      // The row after the last sample, which a tap on the last sample weighs by zero.
      if (past_end) {
        unsigned char* past = data + unsigned(row0 & 15) + count * sp.pitch;
        const int words = (sp.contiguous ? p.nt : sp.frames) * (E / 4);
        for (int i = lane; i < words; i += 32) reinterpret_cast<unsigned*>(past)[i] = 0u;
        fence_async_smem();  // a later window's copy covers these bytes
      }
    }
  }

  // One (aperture, channel, angle) step: its taps and its sample window, in as
  // many visits to the step's stage as the window needs (kTagMore: another
  // visit follows).  rx, rxc: receive delays of this lane's voxels.
  __device__ __forceinline__ void emit(int cfg, int ch, int a, int tag, const long long (&rx)[4],
                                       const unsigned (&rxc)[4]) {
    int i0[4];
    float w[4];
    unsigned cyc[4];
    int lo = INT_MAX, hi = -1;
    const unsigned inner = unsigned(max(p.ns - 3, 0));
    unsigned edges = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int i = lane + 32 * j;
      long long t;
      unsigned tc;
      if (sp.tx_table) {
        t = sh.tx[a * kTileVoxels + i];
        tc = sh.txc[a * kTileVoxels + i];
      } else {
        transmit(cfg, a, i, &t, &tc);
      }
      const long long s = t + rx[j];
      i0[j] = int(s >> 32);
      w[j] = float(unsigned(s)) * 0x1p-32f;
      cyc[j] = tc + rxc[j];
      // Rows 1 ... ns - 3 are inside; the rows at the window's ends are decided in float64.
      if (unsigned(i0[j] - 1) >= inner) {
        if (s < (-1ll << 32) || s >= (long long)(p.ns) << 32) i0[j] = -1;
        else edges |= 1u << j;
      }
    }
    if (__any_sync(0xffffffffu, edges != 0)) {
      const double* an = sh.angle + 3 * a;
      const double e = double((cfg ? p.ye : p.xe)[ch]), extra = p.offsets ? p.offsets[cfg * p.nc + ch] : 0.0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (!(edges >> j & 1)) continue;
        const int i = lane + 32 * j;
        float edge_w = 0.f;
        i0[j] = edge_tap(double(sh.pos[(cfg ? 2 : 0) * kTileVoxels + i]),
                         double(sh.pos[(cfg ? 0 : 2) * kTileVoxels + i]), double(sh.pos[kTileVoxels + i]), e, extra,
                         an[0], an[1], an[2], p.c, p.fs, p.ns, &edge_w);
        w[j] = edge_w;
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (i0[j] >= 0) {
        lo = min(lo, i0[j]);
        hi = max(hi, i0[j]);
      }
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if (lo == INT_MAX) {  // no voxel of the tile sees this step
      if (claim()) publish(tag, 0);
      next_stage();
      return;
    }
    const uintptr_t buf = reinterpret_cast<uintptr_t>(cfg ? p.cr : p.rc);
    const uintptr_t stride = uintptr_t(p.nt) * E;
    const uintptr_t slab = buf + uintptr_t(ch * p.na + a) * uintptr_t(p.ns) * stride + uintptr_t(frame0) * E;
    const uintptr_t end = buf + uintptr_t(p.nc) * p.na * uintptr_t(p.ns) * stride;
    unsigned char* block = sh.base + stage * ring.bytes;
    float4* taps = reinterpret_cast<float4*>(block);
    unsigned char* data = block + kTapBytes;
    const unsigned zero_off = unsigned(sh.zero - sh.base);
    for (int base = lo; base <= hi;) {
      const int last = min(hi, base + ring.rows - 2);  // last tap row of this visit
      const uintptr_t row0 = slab + uintptr_t(base) * stride;
      if (!claim()) return;
      copy_rows(data, cfg, ch * p.na + a, base, last + 2 - base, row0, buf, end);
      const unsigned data_off = unsigned(data - sh.base) + (BOXES ? 0u : unsigned(row0 & 15));
      unsigned blocks = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const bool in = i0[j] >= base && i0[j] <= last;
        blocks |= __any_sync(0xffffffffu, in) ? 1u << j : 0u;
        float pr, pi;
        sincospif(float(int(cyc[j])) * 0x1p-31f, &pi, &pr);
        const unsigned off = in ? data_off + unsigned((i0[j] - base) * sp.pitch) : zero_off;
        taps[lane + 32 * j] = make_float4(in ? w[j] : 0.f, in ? pr : 0.f, in ? pi : 0.f, __uint_as_float(off));
      }
      // The next row a tap needs (tiles may fall into far-apart parts).
      int next = INT_MAX;
      if (last < hi) {
#pragma unroll
        for (int j = 0; j < 4; ++j) next = i0[j] > last ? min(next, i0[j]) : next;
        next = __reduce_min_sync(0xffffffffu, next);
      }
      base = next;
      publish(base <= hi ? tag | kTagMore : tag, blocks);
    }
    next_stage();
  }

  __device__ __forceinline__ void finish() {
    if (turn == 0) {
      if (claim()) publish(kTagEnd, 0);
      next_stage();
      turn = lt.builders;
    }
    --turn;
    // Copies under way land before the CTA may leave, also where consumers gave up waiting.
    for (int st = warp; st < ring.stages; st += lt.builders)
      mbar_wait(&sh.full[st], ((phase >> st) & 1) ^ 1, p.err, kErrWaitDrain);
  }

  // Both apertures, channel by channel; tag = first + aperture * nc + channel.
  // Each builder forms the receive delays of one channel of a block for all, in one of
  // two slots in turn (over both apertures: the barrier of the block between two uses of
  // a slot is what ends its reads).
  __device__ __forceinline__ void walk_channels(int first) {
    int half = 0;
    for (int cfg = 0; cfg < 2; ++cfg) {
      fill_table(cfg);
      for (int c0 = 0; c0 < p.nc; c0 += lt.builders, half ^= 1) {
        if (c0 + warp < p.nc) {
          long long rx[4];
          unsigned rxc[4];
          receive(cfg, c0 + warp, rx, rxc);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            sh.rx[rx_at(half) + 32 * j] = rx[j];
            sh.rxc[rx_at(half) + 32 * j] = rxc[j];
          }
        }
        sync_builders();
        for (int ch = c0; ch < min(c0 + lt.builders, p.nc); ++ch) {
          if (!reachable(cfg, ch)) continue;
          if (turn >= p.na) {
            turn -= p.na;
            continue;
          }
          long long rx[4];
          unsigned rxc[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int at = (half * kMaxBuilders + ch - c0) * kTileVoxels + lane + 32 * j;
            rx[j] = sh.rx[at];
            rxc[j] = sh.rxc[at];
          }
          int a = turn;
          for (; a < p.na && ok; a += lt.builders) emit(cfg, ch, a, first + cfg * p.nc + ch, rx, rxc);
          turn = a - p.na;
        }
      }
    }
  }

  // Both apertures, angle by angle (subset by subset: angles s, s + subsets, ...);
  // tag = aperture * na + angle.  The channel changes with every step, so a helper
  // warp forms the receive delays of its builder's next step meanwhile.
  template <bool HELPER>
  __device__ __forceinline__ void walk_angles(int subsets) {
    int s = 0;
    for (int cfg = 0; cfg < 2; ++cfg) {
      if constexpr (!HELPER) fill_table(cfg);
      for (int i = 0, a = 0; i < p.na; ++i) {
        for (int ch = 0; ch < p.nc && ok; ++ch) {
          if (!reachable(cfg, ch)) continue;
          if (turn-- > 0) continue;
          turn = lt.builders - 1;
          long long rx[4];
          unsigned rxc[4];
          if constexpr (HELPER) {
            if (!rx_wait(sh.rx_empty, s, 1, kErrWaitEmpty)) continue;
            receive(cfg, ch, rx, rxc);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              sh.rx[rx_at(s) + 32 * j] = rx[j];
              sh.rxc[rx_at(s) + 32 * j] = rxc[j];
            }
            rx_arrive(sh.rx_full, s);
          } else {
            if (!rx_wait(sh.rx_full, s, 0, kErrWaitFull)) continue;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              rx[j] = sh.rx[rx_at(s) + 32 * j];
              rxc[j] = sh.rxc[rx_at(s) + 32 * j];
            }
            rx_arrive(sh.rx_empty, s);
            emit(cfg, ch, a, cfg * p.na + a, rx, rxc);
          }
          s ^= 1;
        }
        a += subsets;
        if (a >= p.na) a = a % subsets + 1;  // the next subset's first angle
      }
    }
  }

  template <int MODE>
  __device__ __forceinline__ void walk() {
    if constexpr (MODE == kFmas) {
      walk_angles<false>(1);
    } else if constexpr (kSubsets<MODE> > 0) {
      walk_angles<false>(kSubsets<MODE>);
    } else if constexpr (MODE == kDmas) {
      walk_angles<false>(1);
      walk_channels(2 * p.na);
    } else {
      walk_channels(0);
    }
    finish();
  }
};

// Voxel ids, positions and bounds of one tile.
template <int MODE>
__device__ __forceinline__ void load_tile(const Args& p, const Shared& sh, size_t tile0) {
  const int t = threadIdx.x;
  for (int i = t; i < kTileVoxels; i += blockDim.x) {
    const size_t q = tile0 + i;
    const unsigned v = q < size_t(p.nv) ? (p.order ? p.order[q] : unsigned(q)) : UINT_MAX;
    float pos[3];
    for (int d = 0; d < 3; ++d) {
      pos[d] = v != UINT_MAX ? p.scan[3 * size_t(v) + d] : 0.f;
      sh.pos[d * kTileVoxels + i] = pos[d];
    }
    sh.vox[i] = v;
    const double limit = __ddiv_rn(double(pos[1]), __dmul_rn(2.0, p.fn));
    sh.limit[i] = limit;
    if constexpr (MODE == kDmas) {  // channels of both apertures inside the f-number aperture
      float count = 0.f;
      for (int ch = 0; ch < p.nc; ++ch) {
        count += p.fn <= 0.0 || fabs(__dadd_rn(double(pos[0]), -double(p.xe[ch]))) <= limit ? 1.f : 0.f;
        count += p.fn <= 0.0 || fabs(__dadd_rn(double(pos[2]), -double(p.ye[ch]))) <= limit ? 1.f : 0.f;
      }
      sh.active[i] = count;
    }
  }
  for (int a = t; a < p.na; a += blockDim.x) {
    const double th = double(p.angles[a]);
    sh.angle[3 * a] = cos(th);
    sh.angle[3 * a + 1] = sin(th);
    sh.angle[3 * a + 2] = double(p.starts[a]);
  }
  __syncthreads();
  if (t < 32) {
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY}, steer = 0.f;
    for (int i = t; i < kTileVoxels; i += 32) {
      if (sh.vox[i] == UINT_MAX) continue;
      for (int d = 0; d < 3; ++d) {
        lo[d] = fminf(lo[d], sh.pos[d * kTileVoxels + i]);
        hi[d] = fmaxf(hi[d], sh.pos[d * kTileVoxels + i]);
      }
    }
    for (int a = t; a < p.na; a += 32) steer = fmaxf(steer, fabsf(float(sh.angle[3 * a + 1])));
    for (int off = 16; off > 0; off >>= 1) {
      for (int d = 0; d < 3; ++d) {
        lo[d] = fminf(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], off));
        hi[d] = fmaxf(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], off));
      }
      steer = fmaxf(steer, __shfl_xor_sync(0xffffffffu, steer, off));
    }
    if (t == 0) {
      sh.bounds[0] = lo[0];
      sh.bounds[1] = hi[0];
      sh.bounds[2] = lo[2];
      sh.bounds[3] = hi[2];
      sh.bounds[4] = hi[1];
      // Rows a step of the tile can span: the receive path moves by at most the
      // distance, the transmit path by depth and steering.
      const float dz = hi[1] - lo[1], lateral = fmaxf(hi[0] - lo[0], hi[2] - lo[2]);
      sh.bounds[5] = (sqrtf(dz * dz + lateral * lateral) + dz + lateral * steer) * float(p.fs / p.c);
    }
  }
  __syncthreads();
}

// --------------------------------------------------------------- consumers --
// Two neighbouring frames of a staged row.  BOXES: rows are 16-byte aligned.
template <bool HALF, bool BOXES>
__device__ __forceinline__ float4 load_frames(const unsigned char* q) {
  if constexpr (HALF) {
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(q));
    const float2 b = __half22float2(*reinterpret_cast<const __half2*>(q + 4));
    return make_float4(a.x, a.y, b.x, b.y);
  } else if constexpr (BOXES) {
    return *reinterpret_cast<const float4*>(q);
  } else {
    const float2 a = *reinterpret_cast<const float2*>(q), b = *reinterpret_cast<const float2*>(q + 8);
    return make_float4(a.x, a.y, b.x, b.y);
  }
}

// Adds one staged step to a thread's voxel: its frames of the two rows of its
// tap, interpolated, rotated and accumulated.  WHOLE: all PAIRS are live, so the
// loads of later pairs can be started early.
template <int PAIRS, bool HALF, bool BOXES, bool WHOLE>
__device__ __forceinline__ void add_step(float4 (&acc)[PAIRS], const float4& tap, const unsigned char* row, int pitch,
                                         int pairs) {
  constexpr int E = HALF ? 4 : 8;
  const unsigned char* next = row + pitch;
  const float2 ph = make_float2(tap.y, tap.z);
#pragma unroll
  for (int k = 0; k < PAIRS; ++k) {
    if (!WHOLE && k >= pairs) break;
    const float4 a = load_frames<HALF, BOXES>(row + 2 * E * k), b = load_frames<HALF, BOXES>(next + 2 * E * k);
    const float2 v0 = make_float2(fmaf(tap.x, b.x - a.x, a.x), fmaf(tap.x, b.y - a.y, a.y));
    const float2 v1 = make_float2(fmaf(tap.x, b.z - a.z, a.z), fmaf(tap.x, b.w - a.w, a.w));
    const float2 s0 = cmac(ph, v0, make_float2(acc[k].x, acc[k].y));
    const float2 s1 = cmac(ph, v1, make_float2(acc[k].z, acc[k].w));
    acc[k] = make_float4(s0.x, s0.y, s1.x, s1.y);
  }
}

// Methods that walk their angles one after another.
template <int MODE>
constexpr bool kAngleMajor = MODE == kFmas || MODE == kDmas || MODE > kStsw;

// Floats per voxel and frame that a thread keeps in shared memory (its own).
template <int MODE>
constexpr int kStash = MODE == kOpw ? 0 : MODE == kFmas || MODE > kStsw ? 4 : MODE == kDmas ? 5 : 2;

// Methods whose power is the mean of a complex product.
template <int MODE>
constexpr bool kCross = MODE == kXdoppler || MODE > kStsw;

// Threads of a CTA: 16 consumer warps and 3 builders at 96 registers fill an SM;
// OPW of few frames takes 80 registers and shares the SM with other CTAs.
template <int MODE>
__host__ __device__ constexpr int max_threads(int pairs) {
  return MODE == kDmas ? 512 : MODE == kOpw && pairs <= 8 ? 384 : 608;
}
template <int MODE>
__host__ __device__ constexpr int min_ctas(int pairs) {
  return MODE == kOpw && pairs <= 8 ? 2 : 1;
}

// |x|^2 in float64.
__device__ __forceinline__ double power_of(float2 x) {
  return fma(double(x.x), double(x.x), double(x.y) * double(x.y));
}

// Correlation of two subsets from their means and mean squared deviations (reference
// stsw.py:45-66); zero where it has no value.
__device__ __forceinline__ float2 correlation(float2 r, float spread_r, float2 q, float spread_q) {
  const float2 num = cmul(r, cconj(q));
  const float den = cabs2(r) + cabs2(q) + (spread_r + spread_q) * 0.5f - hypotf(num.x, num.y);
  const float2 value = den > 0.f ? make_float2(num.x / den, num.y / den) : make_float2(0.f, 0.f);
  return isfinite(value.x) && isfinite(value.y) ? value : make_float2(0.f, 0.f);
}

// A consumer thread owns one voxel (a warp 32 of them) and one group of frames.
template <int MODE, int PAIRS, bool HALF, bool BOXES>
struct Consumer {
  static constexpr int E = HALF ? 4 : 8;
  static constexpr int kFrames = 2 * PAIRS;
  const Args& p;
  const Shape& sp;
  const Layout& lt;
  const Shared& sh;
  const Ring ring;
  int first, slot, group, thread, count;
  int state;  // DMAS: 0 RC angles, 1 CR angles, 2 channels; St-SW: aperture * K + subset
  float4 acc[PAIRS];

  __device__ __forceinline__ Consumer(const Args& p_, const Shape& sp_, const Layout& lt_, const Shared& sh_,
                                      const Ring& ring_, int f0)
      : p(p_), sp(sp_), lt(lt_), sh(sh_), ring(ring_), thread(int(threadIdx.x) - 32 * (lt_.builders + lt_.helpers)),
        count(lt_.threads - 32 * (lt_.builders + lt_.helpers)), state(0) {
    slot = thread % kTileVoxels;
    group = thread / kTileVoxels;
    first = f0 + 2 * sp.pairs * group;
    clear();
    if constexpr (kStash<MODE> > 0)
      for (int i = 0; i < kStash<MODE> * 2 * sp.pairs; ++i) sh.stash[i * count + thread] = 0.f;
  }

  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int k = 0; k < PAIRS; ++k) acc[k] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  __device__ __forceinline__ float2 value(int k) const {
    const float4& q = acc[k / 2];
    return k & 1 ? make_float2(q.z, q.w) : make_float2(q.x, q.y);
  }
  __device__ __forceinline__ float& stash(int s, int k) const { return sh.stash[(s * 2 * sp.pairs + k) * count + thread]; }
  __device__ __forceinline__ float2 load(int s, int k) const { return make_float2(stash(s, k), stash(s + 1, k)); }
  __device__ __forceinline__ void store(int s, int k, float2 v) const {
    stash(s, k) = v.x;
    stash(s + 1, k) = v.y;
  }

  // What ends a run of steps is called, not inlined: in the step loop its addresses
  // and temporaries spilled the loop's state, a local store per step that every
  // release of a stage then waited for (37 x 51 x 35 voxels, 400 x 96 x 9 x 90: St-SW, k = 3, 36.4 ms
  // inlined, 18.2 called; 48 x 96 x 48, 384 x 128 x 7 x 64: RC-FMAS 30.7 -> 24.5,
  // DMAS 83 -> 68).  `q` is the thread's first float
  // of slot 0, its frames `step` and slots `slots` floats apart.
  struct Sums {
    float4 q[PAIRS];
    __device__ __forceinline__ float2 value(int k) const {
      return k & 1 ? make_float2(q[k / 2].z, q[k / 2].w) : make_float2(q[k / 2].x, q[k / 2].y);
    }
  };
  __device__ __forceinline__ Sums sums() const {
    Sums s;
#pragma unroll
    for (int k = 0; k < PAIRS; ++k) s.q[k] = acc[k];
    return s;
  }

  // XDoppler, apertures: the first aperture's sums, kept in slots 0 and 1.
  static __device__ __noinline__ void keep(const Sums sums, float* q, int step, int slots, int frames) {
#pragma unroll
    for (int k = 0; k < kFrames; ++k, q += step) {
      if (k >= frames) return;
      const float2 v = sums.value(k);
      q[0] = v.x;
      q[slots] = v.y;
    }
  }

  // RC-FMAS, one angle: the signed square root.
  static __device__ __noinline__ void add_root(const Sums sums, float* q, int step, int slots, int frames) {
#pragma unroll
    for (int k = 0; k < kFrames; ++k, q += step) {
      if (k >= frames) return;
      const float2 r = csroot(sums.value(k));
      q[0] += r.x;
      q[slots] += r.y;
    }
  }
  // DMAS, one angle: sum and energy.
  static __device__ __noinline__ void add_moments(const Sums sums, float* q, int step, int slots, int frames) {
#pragma unroll
    for (int k = 0; k < kFrames; ++k, q += step) {
      if (k >= frames) return;
      const float2 v = sums.value(k);
      q[0] += v.x;
      q[slots] += v.y;
      q[2 * slots] += cabs2(v);
    }
  }
  // DMAS, one channel: signed square root (slots 1, 2) and magnitude (slot 3).
  static __device__ __noinline__ void add_roots(const Sums sums, float* q, int step, int slots, int frames) {
#pragma unroll
    for (int k = 0; k < kFrames; ++k, q += step) {
      if (k >= frames) return;
      const float2 v = sums.value(k), r = csroot(v);
      q[slots] += r.x;
      q[2 * slots] += r.y;
      q[3 * slots] += hypotf(v.x, v.y);
    }
  }
  // DMAS: closes the sums of state 0 (slots 0, 1: r; 2: energy) into |mean|^2
  // and variance, those of state 1 (slots 2, 3: q; 4: energy) with them into
  // the angular coherence (slot 0), and clears the next state's slots.
  static __device__ __noinline__ void close_state(float* q, int step, int slots, int frames, int state, float inv) {
    for (int k = 0; k < frames; ++k, q += step) {
      const float* from = q + (state == 0 ? 0 : 2 * slots);
      const float n = cabs2(make_float2(from[0], from[slots])) * inv * inv;
      const float v = fmaxf(from[2 * slots] * inv - n, 0.f);
      if (state == 0) {
        q[0] = n;
        q[slots] = v;
        q[2 * slots] = 0.f;
      } else {
        const float rn = q[0], rv = q[slots];
        const float num = sqrtf(rn) * sqrtf(n), den = rn + n + (rv + v) / 2 - num;
        q[0] = den > 0.f ? num / den : 0.f;
        q[slots] = q[2 * slots] = q[3 * slots] = 0.f;
      }
    }
  }
  __device__ __forceinline__ void advance(int to) {
    for (; state < to; ++state)
      close_state(sh.stash + thread, count, 2 * sp.pairs * count, 2 * sp.pairs, state, 1.0f / float(p.na));
  }

  // St-SW: a voxel-frame's subset statistics (aperture, subset: mean, mean squared
  // deviation), floats 3 index + (0, 1, 2), are kept in pairs where its correlation
  // series goes later, in the caller's workspace of K^2 float2; K = 2, which has 12
  // floats, leaves the last subset in slots 0-2 and the deviation before it in slot
  // 3.  The deviation of an even subset waits in slot 3 for its pair: each 32-byte
  // sector is then written once and in full.
  static constexpr int K = kSubsets<MODE>;
  __device__ __forceinline__ float2& statistics(unsigned v, int pair, int k) const {
    return p.series[(size_t(v) * (K * K) + size_t(pair)) * size_t(p.nt) + size_t(first + k)];
  }
  __device__ __forceinline__ float statistic(unsigned v, int f, int k) const {
    if (K == 2 && f >= 8) return stash(f == 8 ? 3 : f - 9, k);
    const float2 q = statistics(v, f / 2, k);
    return f & 1 ? q.y : q.x;
  }

  // One angle: Welford's update of slots 0-2 (no E|x|^2 - |E x|^2 cancellation).
  static __device__ __noinline__ void add_angle(const Sums sums, float* q, int step, int slots, int frames,
                                                float inv) {
#pragma unroll
    for (int k = 0; k < kFrames; ++k, q += step) {
      if (k >= frames) return;
      const float2 v = sums.value(k);
      const float2 m = make_float2(q[0], q[slots]), d = make_float2(v.x - m.x, v.y - m.y);
      const float2 now = make_float2(fmaf(d.x, inv, m.x), fmaf(d.y, inv, m.y));
      q[0] = now.x;
      q[slots] = now.y;
      q[2 * slots] += d.x * (v.x - now.x) + d.y * (v.y - now.y);
    }
  }
  // Ends subset `index` (slots 0-2) of `angles` angles; `to` is the voxel's first
  // series value of the thread's frames, of which `live` exist.
  static __device__ __noinline__ void end_subset(float* q, int step, int slots, int frames, int index, int angles,
                                                 float2* to, int nt, int live) {
    for (int k = 0; k < frames; ++k, q += step) {
      const float2 mean = make_float2(q[0], q[slots]);
      const float spread = q[2 * slots] / float(angles);
      if (K == 2 && index == 2 * K - 1) {
        q[2 * slots] = spread;
        continue;
      }
      if (index % 2 == 0) {
        if (k < live) to[size_t(3 * index / 2) * nt + k] = mean;
        q[3 * slots] = spread;
      } else if (k < live) {
        to[size_t((3 * index - 1) / 2) * nt + k] = make_float2(q[3 * slots], mean.x);
        to[size_t((3 * index + 1) / 2) * nt + k] = make_float2(mean.y, spread);
      }
      q[0] = q[slots] = q[2 * slots] = 0.f;
    }
  }
  __device__ __forceinline__ void close_subset(int index, int angles) const {
    const unsigned v = sh.vox[slot];
    const int live = v == UINT_MAX || group >= sp.groups ? 0 : min(2 * sp.pairs, p.nt - first);
    end_subset(sh.stash + thread, count, 2 * sp.pairs * count, 2 * sp.pairs, index, angles,
               live > 0 ? &statistics(v, 0, 0) : nullptr, p.nt, live);
  }

  // Angles of subset i: i, i + K, ... < na.
  __device__ __forceinline__ int subset_angles(int i) const { return (p.na - 1 - i) / K + 1; }

  // Ends a run of steps of one tag.
  __device__ __forceinline__ void fold(int tag) {
    // Keeps the products below out of the step loop's registers.
    if constexpr (MODE == kDmas || K > 0) asm volatile("" : "+r"(count), "+r"(thread));
    float* q = sh.stash + thread;
    const int frames = 2 * sp.pairs, slots = frames * count;
    if constexpr (MODE == kXdoppler || MODE == kApertures) {
      if (tag != 0) return;
      keep(sums(), q, count, slots, frames);
    } else if constexpr (MODE == kFmas) {
      add_root(sums(), q + (tag < p.na ? 0 : 2 * slots), count, slots, frames);
    } else if constexpr (MODE == kDmas) {
      advance(tag < p.na ? 0 : tag < 2 * p.na ? 1 : 2);
      if (state == 2)
        add_roots(sums(), q, count, slots, frames);
      else
        add_moments(sums(), q + (state == 0 ? 0 : 2 * slots), count, slots, frames);
    } else if constexpr (K > 0) {
      const int a = tag % p.na, index = tag / p.na * K + a % K;
      for (; state < index; ++state) close_subset(state, subset_angles(state % K));
      // The angle's place in its subset; angles that no voxel of the tile sees are
      // zero sums that still count.
      add_angle(sums(), q, count, slots, frames, 1.0f / float(a / K + 1));
    }
    clear();
  }

  // Accumulates one item's steps; false when a wait gave up.
  __device__ __forceinline__ bool accumulate(uint32_t& phase) {
    uint32_t stage = 0;
    const unsigned char* mine = sh.base + 2 * E * sp.pairs * group;
    const bool whole = sp.pairs == PAIRS, work = group < sp.groups;
    const int block = slot / 32;
    int open = -1;
    bool ready = mbar_test(&sh.full[stage], (phase >> stage) & 1);
    for (;;) {
      const uint32_t st = stage;
      if (!__all_sync(0xffffffffu, ready || mbar_wait(&sh.full[st], (phase >> st) & 1, p.err, kErrWaitFull)))
        return false;
      phase ^= 1u << st;
      const int2 meta = sh.tag[st];
      const int tag = meta.x;
      const float4 tap = reinterpret_cast<const float4*>(sh.base + st * ring.bytes)[slot];
      if (tag == kTagEnd || !(tag & kTagMore)) stage = st + 1 == uint32_t(ring.stages) ? 0 : st + 1;
      // The next stage's state, asked for ahead of this stage's arithmetic.
      ready = tag != kTagEnd && mbar_test(&sh.full[stage], (phase >> stage) & 1);
      if constexpr (MODE != kOpw) {
        if (tag != kTagEnd) {
          int t = tag & kTagMask;
          // The two-aperture methods fold once, between the apertures.
          if constexpr (MODE == kXdoppler || MODE == kApertures) t = t >= p.nc ? 1 : 0;
          if (t != open) {
            if (open >= 0) fold(open);
            open = t;
          }
        }
      }
      if (work && (meta.y >> block & 1)) {
        const unsigned char* row = mine + __float_as_uint(tap.w);
        if (whole)
          add_step<PAIRS, HALF, BOXES, true>(acc, tap, row, sp.pitch, PAIRS);
        else
          add_step<PAIRS, HALF, BOXES, false>(acc, tap, row, sp.pitch, sp.pairs);
      }
      __syncwarp();
      if ((threadIdx.x & 31) == 0) mbar_arrive(&sh.empty[st]);
      if (tag == kTagEnd) break;
    }
    if constexpr (MODE != kOpw)
      if (open >= 0) fold(open);
    if constexpr (MODE == kDmas) advance(2);
    if constexpr (K > 0)
      for (; state < 2 * K; ++state) close_subset(state, subset_angles(state % K));
    return true;
  }

  // The frames' values and, in float64, their power.  A thread adds up to 26 frames
  // one after another: in float32 that showed in the power maps (48 x 96 x 48 voxels,
  // 384 x 128 x 7 x 64, RC-FMAS: 1.4e-7 from float64, 5.9e-8 with these sums; 40 x 70 x
  // 36, 300 x 96 x 9 x 75, OPW of filtered channels: 1.69e-7 and 1.3e-7).
  __device__ __forceinline__ void write() {
    if (group >= sp.groups) return;
    const unsigned v = sh.vox[slot];
    const int frames = v == UINT_MAX ? 0 : min(2 * sp.pairs, p.nt - first);
    double pr = 0.0, pi = 0.0;
#pragma unroll
    for (int k = 0; k < kFrames; ++k) {
      if (k >= frames) continue;
      const float2 x = value(k);
      const size_t at = size_t(v) * p.nt + first + k;
      if constexpr (MODE == kOpw) {
        if (p.signal) p.signal[at] = x;
        pr += power_of(x);
      } else if constexpr (MODE == kApertures) {
        p.signal[at + size_t(v) * p.nt] = load(0, k);
        p.signal[at + size_t(v) * p.nt + p.nt] = x;
      } else if constexpr (MODE == kXdoppler) {
        const float2 val = cmul(load(0, k), cconj(x));
        if (p.signal) p.signal[at] = val;
        pr += double(val.x);
        pi += double(val.y);
      } else if constexpr (MODE == kFmas) {
        const float2 val = cmul(load(0, k), load(2, k));
        if (p.signal) p.signal[at] = val;
        pr += power_of(val);
      } else if constexpr (K > 0) {
        const float2 val = write_series(v, k);
        pr += double(val.x);
        pi += double(val.y);
      } else {
        const float mag = stash(3, k), act = sh.active[slot];
        const float dm = cabs2(load(1, k)) - mag;
        const float wc = (act > 0.f && mag > 0.f) ? fmaxf(dm, 0.f) / act / mag : 0.f;
        float pw = dm * wc * stash(0, k);
        if (!isfinite(pw)) pw = 0.f;
        if (p.signal) p.signal[at] = make_float2(pw, 0.f);
        pr += double(pw);
      }
    }
    sh.power[group * kTileVoxels + slot] = pr;
    if constexpr (kCross<MODE>) sh.power[(kMaxGroups + group) * kTileVoxels + slot] = pi;
  }

  // St-SW: the K x K correlation series of one frame from its subset statistics
  // (reference stsw.py:45-66); returns r conj(q) of the aperture sums.
  __device__ __forceinline__ float2 write_series(unsigned v, int k) {
    float2 mean[2][K > 0 ? K : 1], sum[2];
    float spread[2][K > 0 ? K : 1];
#pragma unroll
    for (int ap = 0; ap < 2; ++ap) {
      sum[ap] = make_float2(0.f, 0.f);
#pragma unroll
      for (int i = 0; i < K; ++i) {
        const int index = ap * K + i;
        mean[ap][i] = make_float2(statistic(v, 3 * index, k), statistic(v, 3 * index + 1, k));
        spread[ap][i] = statistic(v, 3 * index + 2, k);
        const float n = float(subset_angles(i));
        sum[ap] = make_float2(fmaf(n, mean[ap][i].x, sum[ap].x), fmaf(n, mean[ap][i].y, sum[ap].y));
      }
    }
#pragma unroll
    for (int i = 0; i < K; ++i) {
#pragma unroll
      for (int j = 0; j < K; ++j) {
        const float2 value = correlation(mean[0][i], spread[0][i], mean[1][j], spread[1][j]);
        p.series[(size_t(v) * (K * K) + size_t(i * K + j)) * size_t(p.nt) + size_t(first + k)] = value;
      }
    }
    return cmul(sum[0], cconj(sum[1]));
  }
};

__device__ __forceinline__ void init_shared(const Shared& sh, const Layout& lt) {
  if (threadIdx.x == 0) {
    for (int s = 0; s < lt.stages; ++s) {
      mbar_init(&sh.full[s], 1);
      mbar_init(&sh.empty[s], lt.threads / 32 - lt.builders - lt.helpers);
    }
    for (int s = 0; s < 2 * kMaxBuilders; ++s) {
      mbar_init(&sh.rx_full[s], 1);
      mbar_init(&sh.rx_empty[s], 1);
    }
    fence_mbar_init();
  }
  for (int i = threadIdx.x; i < lt.zero_bytes / 4; i += blockDim.x) reinterpret_cast<unsigned*>(sh.zero)[i] = 0u;
}

// One item: tile `tile`, frames from chunk * frames.  phase carries the stages'
// parities from item to item.  All threads take part; false when a wait gave up.
template <int MODE, int PAIRS, bool HALF, bool BOXES>
__device__ __forceinline__ bool run_item(const Args& p, const Shape& sp, const Layout& lt, const Shared& sh,
                                         const CUtensorMap* maps, int tile, int chunk, uint32_t& phase) {
  load_tile<MODE>(p, sh, size_t(tile) * kTileVoxels);
  const bool deep = sh.bounds[5] + 2.f <= float(sp.rows_deep);
  const Ring ring{deep ? lt.stages : lt.stages / 2, deep ? lt.stage_bytes : 2 * lt.stage_bytes,
                  deep ? sp.rows_deep : sp.rows};
  const int frame0 = chunk * sp.frames, warp = threadIdx.x >> 5;
  bool ok;
  if (warp < lt.builders + lt.helpers) {
    const bool helper = kAngleMajor<MODE> && warp >= lt.builders;
    fence_async_smem();  // with another ring, copies fall where the item before kept taps
    Builder<HALF, BOXES> b(p, sp, lt, sh, ring, maps, frame0, helper ? warp - lt.builders : warp, phase);
    if constexpr (kAngleMajor<MODE>) {
      if (helper)
        b.template walk_angles<true>(kSubsets<MODE> > 0 ? kSubsets<MODE> : 1);
      else
        b.template walk<MODE>();
    } else {
      b.template walk<MODE>();
    }
    phase = b.phase;
    ok = b.ok;
  } else {
    Consumer<MODE, PAIRS, HALF, BOXES> c(p, sp, lt, sh, ring, frame0);
    ok = c.accumulate(phase);
    if (ok) c.write();
  }
  ok = __syncthreads_and(ok);
  if constexpr (MODE != kApertures) {
    for (int i = threadIdx.x; ok && i < kTileVoxels; i += blockDim.x) {
      const unsigned v = sh.vox[i];
      if (v == UINT_MAX) continue;
      double re = 0.0, im = 0.0;
      for (int g = 0; g < sp.groups; ++g) {
        re += sh.power[g * kTileVoxels + i];
        if constexpr (kCross<MODE>) im += sh.power[(kMaxGroups + g) * kTileVoxels + i];
      }
      atomicAdd(p.pd + 2 * size_t(v), float(re / double(p.nt)));
      if constexpr (kCross<MODE>) atomicAdd(p.pd + 2 * size_t(v) + 1, float(im / double(p.nt)));
    }
  }
  return ok;
}

template <int MODE, int PAIRS, bool HALF, bool BOXES>
__global__ void __launch_bounds__(max_threads<MODE>(PAIRS), min_ctas<MODE>(PAIRS))
    das_rows(const __grid_constant__ Maps maps, const __grid_constant__ Args p, const __grid_constant__ Shape sp,
             const __grid_constant__ Layout lt) {
  extern __shared__ __align__(1024) unsigned char smem[];
  const Shared sh = carve(smem, lt);
  init_shared(sh, lt);
  uint32_t phase = 0;
  run_item<MODE, PAIRS, HALF, BOXES>(p, sp, lt, sh, maps.map, int(blockIdx.x) / sp.chunks,
                                     int(blockIdx.x) % sp.chunks, phase);
}

// pd[2v] = |pd[2v] + j pd[2v + 1]| (XDoppler magnitude of the mean cross product).
__global__ void finish_magnitude(float* pd, size_t nv) {
  size_t v = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (v < nv) pd[2 * v] = hypotf(pd[2 * v], pd[2 * v + 1]);
}

}  // namespace das
}  // namespace rcb
