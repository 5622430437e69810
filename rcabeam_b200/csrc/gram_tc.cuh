// Tensor-core (tcgen05) temporal Gram matrix of a complex64 Casorati matrix.
//
// The complex64 rows x T matrix X is read as a real rows x 2T float32 matrix Y
// (real and imaginary parts interleaved, no copy).  D = Y^T Y holds the complex
// Gram G = X^H X as
//     G[m][n] = (D[2m][2n] + D[2m+1][2n+1]) + j (D[2m][2n+1] - D[2m+1][2n]),
// so the whole product is one real symmetric GEMM with K = rows.  Only the
// upper triangle of 128 x 128 blocks of D is formed (block b of D is the
// 64-frame tile b of G, the tiling the float64 Gram and its finish kernel use).
//
// Work: the upper blocks (b <= c) are packed into units of up to four output
// blocks that stage at most three 128-column blocks (plan_units: triangles
// {a, b, c} first); every unit runs on `slices` CTAs, each over
// one contiguous range of rows, so the CTAs of one slice read the same rows at
// the same time (one HBM read, the rest from L2).  TMEM holds the unit's four
// 128 x 128 float32 accumulators (512 columns); every kFlushRows rows (and at
// the end of the slice) the epilogue adds them, in float64, to the upper
// triangle with atomics, which bounds the float32 accumulation length.  The
// accumulators pass through shared memory first, so that a warp's atomics fall on
// two runs of 128 bytes; with accumulator rows on the lanes every one was a sector
// of its own, and the MMAs stood still for a quarter of the kernel.
//
// Precision (both with float32 accumulation):
//   tf32   : operands rounded to nearest TF32 (cvt.rna) -- one MMA per K=8;
//   bf16x3 : operands split into BF16 hi + lo, three MMAs per K=16
//            (Ahi Bhi + Alo Bhi + Ahi Blo).
// Before rounding or splitting every element is multiplied by 2^-e, where 2^e
// bounds the Casorati scale s (max |component|), which keeps the products in
// range exactly as the scaled float64 Gram does; the epilogue applies (2^e/s)^2.
//
// Roles (448 threads, one CTA per SM):
//   warp 0       TMA producer: raw float32 boxes (32 columns x 16 rows;
//                SWIZZLE_128B_ATOM_32B for TF32, SWIZZLE_128B for 3xBF16) of
//                the unit's staged blocks into the staging ring;
//   warp 1       TMEM allocator; lane 0 issues tcgen05.mma and commits;
//   warps 2-13   converters: TF32 rounds the staged floats in place (the
//                layouts coincide), so the staging ring is the operand ring
//                (2 x ring stages, eight with three staged blocks); 3xBF16
//                writes hi/lo operands in the UMMA MN-major SWIZZLE_128B
//                layout (ring staging stages and ring operand stages in the
//                same shared memory; ring = 4 with three staged blocks);
//                they are also the epilogue at every flush, three warps per
//                TMEM lane quarter.
//
// What bounds it: the hand-over of 16-row stages between the roles.  Per stage the
// MMA thread issues up to 12 MMAs and has to find the stage converted, so its
// descriptors are held in registers and the converters (twelve warps, all their
// loads in flight; eight or sixteen were slower) work a stage ahead; every flush
// stops it, so flushes write whole sectors; pairs of outputs share MMAs of 256
// columns, which read less shared memory.  Each of these alone gave little, since
// the next one bound (4194304 x 400 3xBF16, one B200): 16.9 ms before, 14.8 to
// 18.9 with some, 11.6 with all of them; TF32 14.0 -> 8.6 ms; 4194304 x 200 3xBF16
// 7.3 -> 4.65, TF32 6.0 -> 3.6 ms; 1000000 x 16 TF32 0.27 -> 0.20 ms.  The MMAs
// themselves take about 7 ms at 400 frames in 3xBF16.
#pragma once

#include <cuda_bf16.h>

#include "common.cuh"
#include "das_tc.cuh"

namespace rcb {
namespace gramtc {

constexpr int kBlock = 128;        // real columns per Gram block (64 complex frames)
constexpr int kRows = 16;          // rows per stage
constexpr int kMaxLoads = 6;       // staged column blocks per unit
constexpr int kMaxTasks = 4;       // output blocks per unit (4 x 128 TMEM columns)
constexpr int kMaxUnits = 48;      // nb <= 16 blocks (T <= 1024): 136 upper blocks -> 43 units
constexpr int kMaxBlocks = 16;
constexpr int kMaxRing = 4;        // deepest 3xBF16 staging and operand rings (TF32: one ring of 2 x ring)
constexpr int kConvWarps = 12;
constexpr int kConverters = kConvWarps * 32;
constexpr int kThreads = 64 + kConverters;
constexpr int kSlotBytes = kBlock * kRows * 4;  // 8192: one staged block per stage (f32 or bf16 hi+lo)
// The tensor core rounds each float32 accumulation toward zero (a shrink of
// ~1.3e-8 per update); flushing to float64 every 2048 rows (256 TF32 or 384
// BF16 updates) keeps that bias near 3e-6 of a Gram entry.
constexpr int kFlushRows = 2048;
constexpr int kTmemCols = 512;
constexpr int kControlBytes = 1024;  // barriers and the TMEM slot
constexpr int kTilePitch = 17;       // floats between rows of an epilogue warp's transposition tile
constexpr int kFlushTile = 32 * kTilePitch;
// MN-major TF32 operands take the 128-byte swizzle with 32-byte granules (the
// TMA's SWIZZLE_128B_ATOM_32B): 4-row K atoms, so SBO = 512 B; BF16 operands
// take the plain 128-byte swizzle (8-row atoms, SBO = 1024 B).
constexpr uint32_t kLayoutSw128Base32 = 1;

struct Unit {
  int nload;
  int load[kMaxLoads];  // staged block per slot
  int ntask;
  int a_slot[kMaxTasks], b_slot[kMaxTasks];  // of the output blocks, in TMEM order
  int a_blk[kMaxTasks], b_blk[kMaxTasks];
  int nop;
  int op_task[kMaxTasks];  // first output of each MMA
  int op_n[kMaxTasks];     // its columns: 256 when it covers two outputs, else 128
};

struct Params {
  int nunits, slices, nload_max, nt;
  int ring;  // 3xBF16 staging and operand ring depth; TF32 converts in place in one ring of 2 x ring
  long long rows, slice_rows;
  const double* scale;
  double* upper;
  int* err;
  Unit units[kMaxUnits];
};

__host__ __device__ inline size_t smem_bytes(int nload_max, int ring) {
  return size_t(2 * ring) * nload_max * kSlotBytes + 1024 + kControlBytes + kConvWarps * kFlushTile * sizeof(float);
}

// kind::tf32 / kind::f16(BF16) instruction descriptor: F32 accumulate, A and B MN-major.
__host__ __device__ constexpr uint32_t idesc_mn(bool tf32, int m, int n) {
  return (1u << 4) | ((tf32 ? 2u : 1u) << 7) | ((tf32 ? 2u : 1u) << 10) | (1u << 15) | (1u << 16) |
         (uint32_t(n >> 3) << 17) | (uint32_t(m >> 4) << 24);
}

__device__ __forceinline__ void mma_tf32(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}

__device__ __forceinline__ float round_tf32(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return __uint_as_float(r);
}

__device__ __forceinline__ uint32_t pack_bf16(float lo_elem, float hi_elem) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo_elem, hi_elem);
  return *reinterpret_cast<uint32_t*>(&v);
}

// Split 8 scaled floats into BF16 hi and lo 16-byte chunks.
__device__ __forceinline__ void split8(const float (&v)[8], uint4& hi, uint4& lo) {
  uint32_t h[4], l[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __nv_bfloat162 b = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
    h[i] = *reinterpret_cast<const uint32_t*>(&b);
    l[i] = pack_bf16(v[2 * i] - __low2float(b), v[2 * i + 1] - __high2float(b));
  }
  hi = make_uint4(h[0], h[1], h[2], h[3]);
  lo = make_uint4(l[0], l[1], l[2], l[3]);
}

// 32 lanes x 16 consecutive 32-bit columns.
__device__ __forceinline__ void tmem_ld16(uint32_t addr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(addr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

template <bool TF32>
__global__ void __launch_bounds__(kThreads, 1) gram_tc(const __grid_constant__ CUtensorMap map, const Params p) {
  using namespace rcb::tc;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const Unit& u = p.units[blockIdx.x % p.nunits];
  const int slice = blockIdx.x / p.nunits;
  // TF32: one ring of 2 x ring stages converted in place; 3xBF16: ring staging + ring operand stages.
  const int R = TF32 ? 2 * p.ring : p.ring;
  const size_t stage_bytes = size_t(p.nload_max) * kSlotBytes;
  unsigned char* staging = smem;
  unsigned char* operands = TF32 ? smem : smem + p.ring * stage_bytes;
  uint64_t* stg_full = reinterpret_cast<uint64_t*>(smem + 2 * p.ring * stage_bytes);
  uint64_t* stg_empty = stg_full + R;
  uint64_t* op_full = stg_empty + R;
  uint64_t* op_empty = op_full + R;
  uint64_t* acc_full = op_empty + R;
  uint64_t* acc_empty = acc_full + 1;
  uint64_t* drain = acc_empty + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
  float* flush_tiles = reinterpret_cast<float*>(smem + 2 * p.ring * stage_bytes + kControlBytes);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long r0 = (long long)slice * p.slice_rows;
  const long long r1 = r0 + p.slice_rows < p.rows ? r0 + p.slice_rows : p.rows;
  const int nstages = r1 > r0 ? int((r1 - r0 + kRows - 1) / kRows) : 0;
  constexpr int kStagesPerFlush = kFlushRows / kRows;

  if (threadIdx.x == 0) {
    for (int s = 0; s < R; ++s) {
      mbar_init(&stg_full[s], 1);
      mbar_init(&stg_empty[s], TF32 ? 1 : kConvWarps);  // TF32: freed by the MMA commit
      mbar_init(&op_full[s], kConvWarps);
      mbar_init(&op_empty[s], 1);
    }
    mbar_init(acc_full, 1);
    mbar_init(acc_empty, kConvWarps);
    mbar_init(drain, 1);
    fence_mbar_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  // Exact power-of-two prescale 2^-e with s = f 2^e, f in [0.5, 1).
  const double s = *p.scale;
  int e = 0;
  if (s > 0.0 && s <= 1.79e308) frexp(s, &e);
  const float prescale = s > 0.0 ? float(ldexp(1.0, -e)) : 1.0f;
  const double factor = s > 0.0 ? (ldexp(1.0, e) / s) * (ldexp(1.0, e) / s) : 1.0;

  if (warp == 0) {
    // ------------------------------------------------------------- producer --
    if (lane == 0) prefetch_tensormap(&map);
    int k = 0, s_ = 0;
    uint32_t parity = 1;  // of the phase that frees the stage: the first round finds it free
    const int nload = u.nload;
    const int box_col = lane < 4 * nload ? u.load[lane >> 2] * kBlock + 32 * (lane & 3) : 0;
    for (; k < nstages; ++k) {
      if (!__all_sync(0xffffffffu, mbar_wait_fast(&stg_empty[s_], parity, p.err, kErrWaitEmpty))) break;
      const int row = int(r0 + (long long)k * kRows);
      if (lane == 0) mbar_arrive_expect_tx(&stg_full[s_], uint32_t(nload * kSlotBytes));
      __syncwarp();
      // 4 boxes (32 columns) per staged block, one box per lane.
      if (lane < 4 * nload)
        tma_load_2d(staging + s_ * stage_bytes + lane * 2048, &map, &stg_full[s_], box_col, row);
      if (++s_ == R) {
        s_ = 0;
        parity ^= 1;
      }
    }
    // Drain: the last issued stages' copies have landed before the CTA exits.
    if (lane == 0) {
      for (int d = k - R < 0 ? 0 : k - R; d < k; ++d)
        mbar_wait(&stg_full[d % R], (d / R) & 1, p.err, kErrWaitDrain);
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA --
    if (lane == 0) {
      // Everything about the unit's MMAs that does not change from stage to stage is
      // held in registers: this one thread's time per stage sets the kernel's pace
      // as soon as the converters keep up.
      constexpr uint32_t kAHalf = TF32 ? kSlotBytes : kSlotBytes / 2;  // bytes of one staged operand
      const int nop = u.nop;
      uint32_t a_at[kMaxTasks], b_at[kMaxTasks], d_at[kMaxTasks], idesc[kMaxTasks];
#pragma unroll
      for (int i = 0; i < kMaxTasks; ++i) {
        const int t = i < nop ? u.op_task[i] : 0;
        a_at[i] = uint32_t(u.a_slot[t]) * kAHalf >> 4;
        b_at[i] = uint32_t(u.b_slot[t]) * kAHalf >> 4;
        d_at[i] = tmem + uint32_t(kBlock * t);
        idesc[i] = idesc_mn(TF32, 128, i < nop ? u.op_n[i] : kBlock);
      }
      const uint64_t fixed = TF32 ? smem_desc(0, 2048, 512, kLayoutSw128Base32) : smem_desc(0, 2048, 1024, kLayoutSw128);
      const uint32_t lo = uint32_t(p.nload_max) * (kSlotBytes / 2) >> 4;
      const uint32_t first = smem_u32(operands) >> 4, step = uint32_t(stage_bytes) >> 4;
      int flushes = 0, s_ = 0, in_seg = 0;
      uint32_t parity = 0;
      for (int k = 0; k < nstages; ++k) {
        if (in_seg == 0 && flushes > 0 && !mbar_wait_fast(acc_empty, (flushes - 1) & 1, p.err, kErrWaitEmpty)) break;
        if (!mbar_wait_fast(&op_full[s_], parity, p.err, kErrWaitFull)) break;
        tc_fence_after();
        const uint64_t op = fixed + (first + uint32_t(s_) * step);
        const uint32_t more = in_seg > 0 ? 1u : 0u;
#pragma unroll
        for (int i = 0; i < kMaxTasks; ++i) {
          if (i >= nop) break;
          const uint64_t a = op + a_at[i], b = op + b_at[i];
          if constexpr (TF32) {
            mma_tf32(d_at[i], a, b, idesc[i], more);
            mma_tf32(d_at[i], a + 64, b + 64, idesc[i], 1u);  // rows 8-15: 1024 bytes on
          } else {
            mma_f16(d_at[i], a, b, idesc[i], more);
            mma_f16(d_at[i], a + lo, b, idesc[i], 1u);
            mma_f16(d_at[i], a, b + lo, idesc[i], 1u);
          }
        }
        mma_commit(TF32 ? &stg_empty[s_] : &op_empty[s_]);
        if (++in_seg == kStagesPerFlush || k == nstages - 1) {
          mma_commit(acc_full);
          ++flushes;
          in_seg = 0;
        }
        if (++s_ == R) {
          s_ = 0;
          parity ^= 1;
        }
      }
      mma_commit(drain);
      mbar_wait(drain, 0, p.err, kErrWaitDrain);
    }
    __syncwarp();
  } else {
    // ------------------------------------------------ converters / epilogue --
    const int ct = threadIdx.x - 64;  // 0 .. kConverters - 1
    const int quarter = warp & 3, part = (warp - 2) >> 2;  // TMEM lanes, share of a quarter's columns
    const int nload = u.nload;
    int flushes = 0, s_ = 0, in_seg = 0;
    uint32_t parity = 0;
    for (int k = 0; k < nstages; ++k) {
      if (!__all_sync(0xffffffffu, mbar_wait_fast(&stg_full[s_], parity, p.err, kErrWaitFull))) break;
      if (!TF32 && !__all_sync(0xffffffffu, mbar_wait_fast(&op_empty[s_], parity ^ 1, p.err, kErrWaitEmpty))) break;
      const unsigned char* src = staging + s_ * stage_bytes;
      unsigned char* dst = operands + s_ * stage_bytes;
      if constexpr (TF32) {
        // In place (dst == src): an elementwise map over the staged bytes, four
        // loads in flight per thread.
        const int chunks = nload * (kSlotBytes / 16);
        for (int i0 = ct; i0 < chunks; i0 += 4 * kConverters) {
          float4 v[4];
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (i0 + j * kConverters < chunks) v[j] = reinterpret_cast<const float4*>(src)[i0 + j * kConverters];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            v[j].x = round_tf32(v[j].x * prescale);
            v[j].y = round_tf32(v[j].y * prescale);
            v[j].z = round_tf32(v[j].z * prescale);
            v[j].w = round_tf32(v[j].w * prescale);
            if (i0 + j * kConverters < chunks) reinterpret_cast<float4*>(dst)[i0 + j * kConverters] = v[j];
          }
        }
      } else {
        // Item = (slot, row, 64-column atom, 16-byte output chunk of 8 BF16); both of
        // a thread's items are loaded before either is converted.
        unsigned char* hi = dst;
        unsigned char* lo = dst + size_t(p.nload_max) * (kSlotBytes / 2);
        const int items = nload * kRows * 16;
        for (int i0 = ct; i0 < items; i0 += 2 * kConverters) {
          float4 x[2][2];
          int off[2];
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const int i = min(i0 + j * kConverters, items - 1);
            const int slot = i >> 8, rem = i & 255;
            const int row = rem >> 4, atom = (rem >> 3) & 1, c = rem & 7;
            const int sw = row & 7;
            const int box = 2 * atom + (c >> 2);
            const int c0 = 2 * (c & 3);
            const unsigned char* rbase = src + slot * kSlotBytes + box * 2048 + (row >> 3) * 1024 + sw * 128;
            x[j][0] = *reinterpret_cast<const float4*>(rbase + ((c0 ^ sw) << 4));
            x[j][1] = *reinterpret_cast<const float4*>(rbase + (((c0 + 1) ^ sw) << 4));
            off[j] = slot * (kSlotBytes / 2) + atom * 2048 + (row >> 3) * 1024 + sw * 128 + ((c ^ sw) << 4);
          }
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const float v[8] = {x[j][0].x * prescale, x[j][0].y * prescale, x[j][0].z * prescale, x[j][0].w * prescale,
                                x[j][1].x * prescale, x[j][1].y * prescale, x[j][1].z * prescale, x[j][1].w * prescale};
            uint4 h, l;
            split8(v, h, l);
            if (i0 + j * kConverters < items) {
              *reinterpret_cast<uint4*>(hi + off[j]) = h;
              *reinterpret_cast<uint4*>(lo + off[j]) = l;
            }
          }
        }
      }
      fence_async_smem();  // generic-proxy writes -> visible to the tensor core
      __syncwarp();
      if (lane == 0) {
        if (!TF32) mbar_arrive(&stg_empty[s_]);
        mbar_arrive(&op_full[s_]);
      }
      if (++s_ == R) {
        s_ = 0;
        parity ^= 1;
      }
      if (++in_seg == kStagesPerFlush || k == nstages - 1) {
        in_seg = 0;
        if (!__all_sync(0xffffffffu, mbar_wait(acc_full, flushes & 1, p.err, kErrWaitFull))) break;
        tc_fence_after();
        float* tile = flush_tiles + (warp - 2) * kFlushTile;
        const int col = lane & 15;
        for (int t = 0; t < u.ntask; ++t) {
          // A block below the diagonal is stored as its conjugate transpose.
          const bool lower = u.a_blk[t] > u.b_blk[t];
          for (int c0 = 0; c0 < kBlock; c0 += 16) {
            if ((t * (kBlock / 16) + c0 / 16) % (kConvWarps / 4) != part) continue;
            float val[16];
            tmem_ld16(tmem + (uint32_t(32 * quarter) << 16) + uint32_t(kBlock * t + c0), val);
#pragma unroll
            for (int i = 0; i < 16; ++i) tile[lane * kTilePitch + i] = val[i];
            __syncwarp();
            // Sixteen lanes take the components of eight frame pairs (m, n), n along
            // the lanes: re = D[2m][2n] + D[2m+1][2n+1], im = D[2m][2n+1] - D[2m+1][2n].
            const int n = (u.b_blk[t] * kBlock + c0 + col) / 2;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const int row = 2 * (2 * i + (lane >> 4));
              const int m = (u.a_blk[t] * kBlock + 32 * quarter + row) / 2;
              const double x = double(tile[row * kTilePitch + col]), y = double(tile[(row + 1) * kTilePitch + (col ^ 1)]);
              const double v = col & 1 ? (lower ? y - x : x - y) : x + y;
              if (m < p.nt && n < p.nt)
                atomicAdd(p.upper + 2 * (lower ? size_t(n) * p.nt + m : size_t(m) * p.nt + n) + (col & 1), v * factor);
            }
            __syncwarp();  // the tile is read before the next columns overwrite it
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(acc_empty);
        ++flushes;
      }
    }
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
  }
}

inline int unit_slot(const Unit& un, int blk) {
  for (int j = 0; j < un.nload; ++j)
    if (un.load[j] == blk) return j;
  return -1;
}

// Output (a, b) of a unit, staging blocks a and b if it does not yet.
inline void unit_add(Unit& un, int a, int b) {
  if (unit_slot(un, a) < 0) un.load[un.nload++] = a;
  if (unit_slot(un, b) < 0) un.load[un.nload++] = b;
  un.a_slot[un.ntask] = unit_slot(un, a);
  un.b_slot[un.ntask] = unit_slot(un, b);
  un.a_blk[un.ntask] = a;
  un.b_blk[un.ntask] = b;
  ++un.ntask;
}

// Augmenting path for diagonal block d: a unit among the first n that stages d
// and has a free output slot, possibly after moving a diagonal it holds on.
inline bool diagonal_path(int d, int nb, int n, const Unit* units, int* owner, bool* seen) {
  for (int u = 0; u < n; ++u) {
    if (seen[u] || unit_slot(units[u], d) < 0) continue;
    seen[u] = true;
    int held = 0;
    for (int e = 0; e < nb; ++e) held += owner[e] == u;
    if (units[u].ntask + held < kMaxTasks) {
      owner[d] = u;
      return true;
    }
    for (int e = 0; e < nb; ++e)
      if (owner[e] == u && diagonal_path(e, nb, n, units, owner, seen)) {
        owner[d] = u;
        return true;
      }
  }
  return false;
}

// Orders a unit's staged blocks so that as many pairs of outputs as possible share
// one MMA of 256 columns, (a, b) and (a, c) with b and c staged side by side, and
// lists its outputs (either triangle) and MMAs in that order.  An MMA of 128
// columns reads its two operands for half the work of one with 256: the MMAs'
// operand reads are most of the kernel's shared-memory traffic, which bounds it.
inline void merge_outputs(Unit& un) {
  bool need[kMaxBlocks][kMaxBlocks] = {};
  for (int t = 0; t < un.ntask; ++t)
    need[un.a_blk[t]][un.b_blk[t]] = need[un.b_blk[t]][un.a_blk[t]] = true;
  static const int kOrders[6][3] = {{0, 1, 2}, {0, 2, 1}, {1, 0, 2}, {1, 2, 0}, {2, 0, 1}, {2, 1, 0}};
  Unit best{};
  for (const auto& order : kOrders) {
    Unit c{};
    c.nload = un.nload;
    bool valid = true;
    for (int j = 0; j < un.nload; ++j) {
      valid = valid && order[j] < un.nload;
      c.load[j] = un.load[order[j] < un.nload ? order[j] : 0];
    }
    if (!valid) continue;
    bool open[kMaxBlocks][kMaxBlocks];
    for (int a = 0; a < kMaxBlocks; ++a)
      for (int b = 0; b < kMaxBlocks; ++b) open[a][b] = need[a][b];
    auto add = [&](int i, int j, int outputs) {
      c.op_task[c.nop] = c.ntask;
      c.op_n[c.nop++] = outputs * kBlock;
      for (int k = j; k < j + outputs; ++k) {
        const int a = c.load[i], b = c.load[k];
        c.a_slot[c.ntask] = i;
        c.b_slot[c.ntask] = k;
        c.a_blk[c.ntask] = a;
        c.b_blk[c.ntask++] = b;
        open[a][b] = open[b][a] = false;
      }
    };
    for (int i = 0; i < c.nload; ++i)
      for (int j = 0; j + 1 < c.nload; ++j)
        if (open[c.load[i]][c.load[j]] && open[c.load[i]][c.load[j + 1]]) add(i, j, 2);
    for (int i = 0; i < c.nload; ++i)
      for (int j = 0; j < c.nload; ++j)
        if (open[c.load[i]][c.load[j]]) add(i, j, 1);
    if (!best.nop || c.nop < best.nop) best = c;
  }
  un = best;
}

// Pack the upper 128-column blocks (b <= c) of an nb-block Gram into units of
// at most four output blocks (the 512 TMEM columns).  A CTA stages its unit's
// blocks for every row, so units are built to stage few blocks for their
// outputs: first edge-disjoint triangles {a, b, c} (three staged blocks for the
// off-diagonal outputs (a,b), (a,c), (b,c); a Steiner triple system where nb
// allows, e.g. nb = 7), then the remaining off-diagonal outputs in units of at
// most three blocks, then each diagonal output (b,b) in a unit that already
// stages b and has room (augmenting-path matching), the rest in units of up to
// three diagonals.  At most three staged blocks per unit (T = 400: 7 units of
// 4 outputs and 21 staged blocks, against 27 when rows b and nb-1-b were
// paired).  Returns the unit count, or 0.
inline int plan_units(int nb, Unit* units, int* nload_max) {
  if (nb < 1 || nb > kMaxBlocks) return 0;
  bool open[kMaxBlocks][kMaxBlocks] = {};  // off-diagonal outputs (a < b) not yet in a unit
  for (int a = 0; a < nb; ++a)
    for (int b = a + 1; b < nb; ++b) open[a][b] = true;
  int count = 0;
  auto fresh = [&]() -> Unit* {
    if (count == kMaxUnits) return nullptr;
    Unit* un = &units[count++];
    un->nload = 0;
    un->ntask = 0;
    return un;
  };
  // 1. Triangles.
  for (int a = 0; a < nb; ++a)
    for (int b = a + 1; b < nb; ++b)
      for (int c = b + 1; c < nb; ++c) {
        if (!(open[a][b] && open[a][c] && open[b][c])) continue;
        Unit* un = fresh();
        if (!un) return 0;
        unit_add(*un, a, b);
        unit_add(*un, a, c);
        unit_add(*un, b, c);
        open[a][b] = open[a][c] = open[b][c] = false;
      }
  // 2. Remaining off-diagonal outputs, up to three per unit of <= three blocks.
  for (int a = 0; a < nb; ++a)
    for (int b = a + 1; b < nb; ++b) {
      if (!open[a][b]) continue;
      Unit* un = fresh();
      if (!un) return 0;
      unit_add(*un, a, b);
      open[a][b] = false;
      for (int c = 0; c < nb && un->ntask < 3; ++c)
        for (int d = c + 1; d < nb && un->ntask < 3; ++d) {
          if (!open[c][d] || un->nload + (unit_slot(*un, c) < 0) + (unit_slot(*un, d) < 0) > 3) continue;
          unit_add(*un, c, d);
          open[c][d] = false;
        }
    }
  // 3. Diagonal outputs into units that stage their block.
  const int paired = count;
  int owner[kMaxBlocks];
  bool seen[kMaxUnits];
  for (int d = 0; d < nb; ++d) {
    owner[d] = -1;
    for (int u = 0; u < paired; ++u) seen[u] = false;
    diagonal_path(d, nb, paired, units, owner, seen);
  }
  for (int d = 0; d < nb; ++d)
    if (owner[d] >= 0) unit_add(units[owner[d]], d, d);
  // 4. Diagonal outputs left over: up to three per unit.
  Unit* rest = nullptr;
  for (int d = 0; d < nb; ++d) {
    if (owner[d] >= 0) continue;
    if (!rest || rest->ntask == 3) rest = fresh();
    if (!rest) return 0;
    unit_add(*rest, d, d);
  }
  for (int u = 0; u < count; ++u) merge_outputs(units[u]);
  *nload_max = 0;
  for (int u = 0; u < count; ++u)
    if (units[u].nload > *nload_max) *nload_max = units[u].nload;
  return count;
}

}  // namespace gramtc
}  // namespace rcb
