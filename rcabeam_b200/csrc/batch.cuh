// Batching form: one persistent kernel over a queue of uneven ensembles.
//
// The queue is a device table of ensembles (packed RC/CR channels, geometry,
// power output, method, item split).  Its work is flattened into (voxel tile,
// frame chunk) items in queue order, each run by the device functions of the
// single-ensemble kernel (das_rows.cuh); DMAS-CCF-ACF items make both of their
// passes.  Persistent CTAs take items from a global counter, so small and large
// ensembles share the GPU without launch gaps or tails.  XDoppler magnitudes are
// finished per tile by the CTA that completes the tile's last frame chunk, and
// the CTA that completes an ensemble's last item stamps its completion time.
// A persistent launch serves one method (its kernel is compiled for it); a queue of
// several methods is grouped by method, one launch after another.
#pragma once

#include "common.cuh"
#include "das_rows.cuh"

namespace rcb {
namespace batch {

constexpr int kMaxAngles = 64;

struct alignas(64) Ensemble {
  das::Maps maps;          // TMA tensors of the channels (shape.boxes)
  das::Args args;          // pointers, sizes and constants (signal unused)
  das::Shape shape;        // item split
  int method;              // 0 OPW, 1 XDoppler, 3 DMAS-CCF-ACF
  int width;               // frame pairs the kernel variant is compiled for
  int tiles;               // voxel tiles; items = tiles x shape.chunks
  int index;               // position in the queue
  long long first_item;    // items before this ensemble in its launch
  long long tile_base;     // first per-tile counter of this ensemble (XDoppler)
};

struct Queue {
  const Ensemble* ens;
  das::Layout layout;            // of the launch: every ensemble fits it
  int n;
  long long total_items;
  unsigned long long* next;      // work counter
  unsigned* done;                // [n] completed items
  unsigned* tile_done;           // per (ensemble, tile) completed chunks (XDoppler)
  unsigned long long* times;     // [queue + 1]: kernel start, completion per ensemble (globaltimer ns)
};

template <int MODE>
__device__ __forceinline__ bool item_of(const Ensemble& e, const das::Args& args, const das::Shape& sp,
                                        const Queue& q, const das::Shared& sh, int tile, int chunk, uint32_t& phase) {
  const CUtensorMap* maps = e.maps.map;
  if constexpr (MODE != das::kDmas) {
    if (e.width > 8)
      return sp.boxes ? das::run_item<MODE, 13, false, true>(args, sp, q.layout, sh, maps, tile, chunk, phase)
                      : das::run_item<MODE, 13, false, false>(args, sp, q.layout, sh, maps, tile, chunk, phase);
  }
  return sp.boxes ? das::run_item<MODE, 8, false, true>(args, sp, q.layout, sh, maps, tile, chunk, phase)
                  : das::run_item<MODE, 8, false, false>(args, sp, q.layout, sh, maps, tile, chunk, phase);
}

template <int MODE>
__global__ void __launch_bounds__(das::max_threads<MODE>(13), 1) run(const __grid_constant__ Queue q) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ long long item_slot;
  __shared__ int ens_slot, fail, last_chunk;
  const das::Shared sh = das::carve(smem, q.layout);
  das::init_shared(sh, q.layout);
  if (threadIdx.x == 0) {
    fail = 0;
    if (blockIdx.x == 0) atomicMin(q.times, static_cast<unsigned long long>(global_ns()));
  }
  uint32_t phase = 0;  // the stages' parities, carried from item to item
  for (;;) {
    __syncthreads();  // the previous item's tables and slots are no longer read
    if (threadIdx.x == 0) {
      const long long item = fail ? q.total_items : static_cast<long long>(atomicAdd(q.next, 1ull));
      int lo = 0, hi = q.n - 1;
      if (item < q.total_items) {
        while (lo < hi) {  // last ensemble whose first item <= item
          const int mid = (lo + hi + 1) / 2;
          if (q.ens[mid].first_item <= item) lo = mid;
          else hi = mid - 1;
        }
      }
      item_slot = item;
      ens_slot = lo;
      last_chunk = 0;
    }
    __syncthreads();
    const long long item = item_slot;
    if (item >= q.total_items) break;
    const int ei = ens_slot;
    const Ensemble& e = q.ens[ei];
    // Private copies: the table in global memory could alias the item's stores,
    // so its fields would be reloaded inside the hot loops.
    const das::Args args = e.args;
    const das::Shape sp = e.shape;
    const long long local = item - e.first_item;
    const int tile = int(local / sp.chunks), chunk = int(local % sp.chunks);
    const bool ok = item_of<MODE>(e, args, sp, q, sh, tile, chunk, phase);
    if (!ok) atomicExch(&fail, 1);
    __syncthreads();  // every warp's results of this item are issued
    if (threadIdx.x == 0) {
      __threadfence();
      if constexpr (MODE == das::kXdoppler)  // last chunk of this tile: the voxels' magnitudes are due
        last_chunk = atomicAdd(q.tile_done + e.tile_base + tile, 1u) + 1 == unsigned(sp.chunks);
      const unsigned d = atomicAdd(q.done + ei, 1u) + 1;
      if (d == unsigned(e.tiles) * unsigned(sp.chunks)) q.times[1 + e.index] = global_ns();
    }
    if constexpr (MODE == das::kXdoppler) {
      __syncthreads();
      if (last_chunk) {
        __threadfence();
        for (int i = threadIdx.x; i < das::kTileVoxels; i += blockDim.x) {
          const unsigned v = sh.vox[i];
          if (v != UINT_MAX) {
            float* pd = args.pd + 2 * size_t(v);
            pd[0] = hypotf(__ldcg(pd), __ldcg(pd + 1));
          }
        }
      }
    }
  }
}

// Per-ensemble grid mode of the queue: a global-timer stamp after each
// ensemble's launches (start = 1: the queue's start, kept as a minimum).
__global__ void stamp(unsigned long long* t, int start) {
  if (start) atomicMin(t, static_cast<unsigned long long>(global_ns()));
  else *t = global_ns();
}

}  // namespace batch
}  // namespace rcb
