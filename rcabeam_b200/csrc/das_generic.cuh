// RC-FMAS, DMAS-CCF-ACF and St-SW of few voxels with one warp per voxel, the pair
// sums of St-SW (method 4) and the per-frame entry points of the reference's
// single-frame API (core.cu).
#pragma once

#include "common.cuh"
#include "das_rows.cuh"

namespace rcb {
namespace generic {

constexpr int kWarps = 4;

struct Voxel {
  double x, z, y;
};

__device__ __forceinline__ Voxel load_voxel(const float* scan, size_t v) {
  return Voxel{double(scan[3 * v]), double(scan[3 * v + 1]), double(scan[3 * v + 2])};
}

// Tap of (voxel, aperture config, channel, angle) from raw float inputs.
__device__ __forceinline__ Tap tap_of(const Voxel& q, int config, const float* el, int ch, const float* angles,
                                      const float* starts, int a, double c, double fs, double fd, double fn, int ns) {
  bool act;
  double trx = receive_delay(config ? q.y : q.x, q.z, double(el[ch]), c, fn, &act);
  double th = double(angles[a]);
  double ttx = transmit_delay(config ? q.x : q.y, q.z, cos(th), sin(th), c);
  return make_tap(__dadd_rn(ttx, trx), double(starts[a]), fs, fd, ns, act);
}

// ---------------------------------------------------- one warp per voxel --
// The nonlinear methods of few voxels: a warp owns one voxel, a lane one frame (grid.y
// counts blocks of 32).  The staged kernel (das_rows.cuh) walks all channels and angles
// of 128 voxels in one CTA; with few tiles most SMs have none, and the walk's latency is
// the call's time.  Here the same steps run on as many warps as there are voxels, bound
// by the latency of the per-frame gathers until the SMs are full (about 4000 warps):
// 128 channels, 11 angles, 64 frames, 1000 voxels over 10 mm: RC-FMAS 4.84 -> 1.08 ms,
// DMAS 37.6 -> 2.3, St-SW (k = 3) 5.27 -> 1.06; within 2 mm, where a tile's windows are
// short, 1.35 -> 1.05, 3.37 -> 1.95 and 1.51 -> 1.07.  rcabeam.cu (few_voxels) draws the line.
struct WarpTaps {
  Tap rc[32], cr[32];
};

// Interpolated, rotated sample of a packed (c, a, s, t) complex64 ensemble.
__device__ __forceinline__ float2 packed_sample(const void* iq, const Tap& t, int ch, int a, int frame,
                                                const das::Args& p) {
  if (t.i0 < 0 || frame >= p.nt) return make_float2(0.f, 0.f);
  const float2* at =
      static_cast<const float2*>(iq) + ((size_t(ch) * p.na + a) * p.ns + size_t(t.i0)) * p.nt + frame;
  const float2 va = at[0], vb = at[t.i0 == p.ns - 1 ? 0 : p.nt];
  return cmul(make_float2(fmaf(t.w, vb.x - va.x, va.x), fmaf(t.w, vb.y - va.y, va.y)), t.phase);
}

// Sums of both apertures over the channels of angle a.  A lane forms one channel's
// taps, which the warp then reads back from shared memory.
__device__ __forceinline__ void angle_sums(const das::Args& p, const Voxel& q, int a, int frame, WarpTaps& taps,
                                           float2& r, float2& s) {
  const int lane = threadIdx.x & 31;
  const double th = double(p.angles[a]), cs = cos(th), sn = sin(th), start = double(p.starts[a]);
  const double tx_rc = transmit_delay(q.y, q.z, cs, sn, p.c), tx_cr = transmit_delay(q.x, q.z, cs, sn, p.c);
  r = s = make_float2(0.f, 0.f);
  for (int c0 = 0; c0 < p.nc; c0 += 32) {
    const int count = min(32, p.nc - c0);
    __syncwarp();  // the previous taps have been read
    if (lane < count) {
      bool active;
      const double rx_rc = receive_delay(q.x, q.z, double(p.xe[c0 + lane]), p.c, p.fn, &active);
      taps.rc[lane] = make_tap(__dadd_rn(tx_rc, rx_rc), start, p.fs, p.fd, p.ns, active);
      const double rx_cr = receive_delay(q.y, q.z, double(p.ye[c0 + lane]), p.c, p.fn, &active);
      taps.cr[lane] = make_tap(__dadd_rn(tx_cr, rx_cr), start, p.fs, p.fd, p.ns, active);
    }
    __syncwarp();
    for (int j = 0; j < count; ++j) {
      r = cadd(r, packed_sample(p.rc, taps.rc[j], c0 + j, a, frame, p));
      s = cadd(s, packed_sample(p.cr, taps.cr[j], c0 + j, a, frame, p));
    }
  }
}

// Sums of both apertures over the angles of channel ch.
__device__ __forceinline__ void channel_sums(const das::Args& p, const Voxel& q, int ch, int frame, WarpTaps& taps,
                                             float2& r, float2& s) {
  const int lane = threadIdx.x & 31;
  r = s = make_float2(0.f, 0.f);
  for (int a0 = 0; a0 < p.na; a0 += 32) {
    const int count = min(32, p.na - a0);
    __syncwarp();
    if (lane < count) {
      taps.rc[lane] = tap_of(q, 0, p.xe, ch, p.angles, p.starts, a0 + lane, p.c, p.fs, p.fd, p.fn, p.ns);
      taps.cr[lane] = tap_of(q, 1, p.ye, ch, p.angles, p.starts, a0 + lane, p.c, p.fs, p.fd, p.fn, p.ns);
    }
    __syncwarp();
    for (int j = 0; j < count; ++j) {
      r = cadd(r, packed_sample(p.rc, taps.rc[j], ch, a0 + j, frame, p));
      s = cadd(s, packed_sample(p.cr, taps.cr[j], ch, a0 + j, frame, p));
    }
  }
}

// Power of one frame by RC-FMAS: signed square roots of the channel sums, added over angles.
__device__ __forceinline__ double fmas_frame(const das::Args& p, const Voxel& q, size_t v, int frame, WarpTaps& taps) {
  float2 r = make_float2(0.f, 0.f), s = r;
  for (int a = 0; a < p.na; ++a) {
    float2 ar, as;
    angle_sums(p, q, a, frame, taps, ar, as);
    r = cadd(r, csroot(ar));
    s = cadd(s, csroot(as));
  }
  const float2 value = cmul(r, s);
  if (p.signal && frame < p.nt) p.signal[v * p.nt + frame] = value;
  return das::power_of(value);
}

// Power of one frame by DMAS-CCF-ACF (reference ensemble.cu:143-232): channel sums
// for the DMAS and coherence terms, then angle sums for the angular coherence.
__device__ __forceinline__ double dmas_frame(const das::Args& p, const Voxel& q, size_t v, int frame, WarpTaps& taps) {
  float2 root = make_float2(0.f, 0.f), r = root, s = root;
  float magnitude = 0.f, active = 0.f, er = 0.f, es = 0.f;
  for (int ch = 0; ch < p.nc; ++ch) {
    float2 cr, cs;
    channel_sums(p, q, ch, frame, taps, cr, cs);
    root = cadd(root, cadd(csroot(cr), csroot(cs)));
    magnitude += hypotf(cr.x, cr.y) + hypotf(cs.x, cs.y);
    bool act_r, act_s;
    receive_delay(q.x, q.z, double(p.xe[ch]), p.c, p.fn, &act_r);
    receive_delay(q.y, q.z, double(p.ye[ch]), p.c, p.fn, &act_s);
    active += float(act_r) + float(act_s);
  }
  for (int a = 0; a < p.na; ++a) {
    float2 ar, as;
    angle_sums(p, q, a, frame, taps, ar, as);
    r = cadd(r, ar);
    s = cadd(s, as);
    er += cabs2(ar);
    es += cabs2(as);
  }
  const float inv = 1.0f / float(p.na);
  const float dm = cabs2(root) - magnitude;
  const float wc = (active > 0.f && magnitude > 0.f) ? fmaxf(dm, 0.f) / active / magnitude : 0.f;
  const float nr = cabs2(r) * inv * inv, ns = cabs2(s) * inv * inv;
  const float var = fmaxf(er * inv - nr, 0.f) + fmaxf(es * inv - ns, 0.f);
  const float num = sqrtf(nr) * sqrtf(ns), den = nr + ns + var / 2 - num;
  float power = den > 0.f ? dm * wc * (num / den) : 0.f;
  if (!isfinite(power)) power = 0.f;
  if (p.signal && frame < p.nt) p.signal[v * p.nt + frame] = make_float2(power, 0.f);
  return double(power);
}

// St-SW, one frame: the K x K correlation series (below) and r conj(q) of the aperture sums.
template <int K>
__device__ __forceinline__ float2 stsw_frame(const das::Args& p, const Voxel& q, size_t v, int frame, WarpTaps& taps) {
  float2 r = make_float2(0.f, 0.f), s = r, mr[K] = {}, ms[K] = {};
  float vr[K] = {}, vs[K] = {};
  for (int a = 0; a < p.na; ++a) {
    float2 ar, as;
    angle_sums(p, q, a, frame, taps, ar, as);
    r = cadd(r, ar);
    s = cadd(s, as);
    // Welford update of subset a % K, whose (a / K + 1)-th angle this is.
    const float inv = 1.0f / float(a / K + 1);
#pragma unroll
    for (int i = 0; i < K; ++i) {
      if (i != a % K) continue;
      const float2 dr = make_float2(ar.x - mr[i].x, ar.y - mr[i].y), ds = make_float2(as.x - ms[i].x, as.y - ms[i].y);
      mr[i] = make_float2(fmaf(dr.x, inv, mr[i].x), fmaf(dr.y, inv, mr[i].y));
      ms[i] = make_float2(fmaf(ds.x, inv, ms[i].x), fmaf(ds.y, inv, ms[i].y));
      vr[i] += dr.x * (ar.x - mr[i].x) + dr.y * (ar.y - mr[i].y);
      vs[i] += ds.x * (as.x - ms[i].x) + ds.y * (as.y - ms[i].y);
    }
  }
#pragma unroll
  for (int i = 0; i < K; ++i) {
    const float ni = float((p.na - 1 - i) / K + 1);  // angles i, i + K, ... < na
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const float nj = float((p.na - 1 - j) / K + 1);
      const float2 value = das::correlation(mr[i], vr[i] / ni, ms[j], vs[j] / nj);
      if (frame < p.nt) p.series[(v * (K * K) + size_t(i * K + j)) * size_t(p.nt) + size_t(frame)] = value;
    }
  }
  return cmul(r, cconj(s));
}

__device__ __forceinline__ double warp_sum(double x) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
  return x;
}

// MODE as in das_rows.cuh: kFmas, kDmas or kStsw + K.  Ten CTAs of St-SW per SM (48
// registers) hide more of the gathers than nine (8192 voxels, 64 frames, 128 channels, 11
// angles: 4.41 -> 3.33 ms; twelve, with spills, 3.55).
template <int MODE>
__global__ void __launch_bounds__(kWarps * 32, MODE > das::kStsw ? 10 : 1) ensemble_warps(const __grid_constant__ das::Args p) {
  __shared__ __align__(16) WarpTaps all[kWarps];
  const size_t v = size_t(blockIdx.x) * kWarps + (threadIdx.x >> 5);
  if (v >= size_t(p.nv)) return;
  WarpTaps& taps = all[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31, frame = int(blockIdx.y) * 32 + lane;
  const Voxel q = load_voxel(p.scan, v);
  double re = 0.0, im = 0.0;
  if constexpr (MODE == das::kFmas) {
    re = fmas_frame(p, q, v, frame, taps);
  } else if constexpr (MODE == das::kDmas) {
    re = dmas_frame(p, q, v, frame, taps);
  } else {
    const float2 cross = stsw_frame<das::kSubsets<MODE>>(p, q, v, frame, taps);
    re = double(cross.x);
    im = double(cross.y);
  }
  // Frames past the end are sums of nothing: zeros.
  re = warp_sum(re);
  if constexpr (das::kCross<MODE>) im = warp_sum(im);
  if (lane == 0) {
    atomicAdd(p.pd + 2 * v, float(re / double(p.nt)));
    if constexpr (das::kCross<MODE>) atomicAdd(p.pd + 2 * v + 1, float(im / double(p.nt)));
  }
}

// ------------------------------------------------------------ St-SW --
// St-SW (method 4; reference stsw.py:10-107, ensemble.cu:457-627).  Angles of
// each aperture fall into K interleaved subsets (a % K).  Per frame: the
// subset means m and mean squared deviations v of the per-angle sums, the
// K x K series c[i][j] = m_rc[i] conj(m_cr[j]) / (|m_rc[i]|^2 + |m_cr[j]|^2 +
// (v_rc[i] + v_cr[j]) / 2 - |m_rc[i] conj(m_cr[j])|); over frames the raw
// weight |sum over (i1 < i2, j1 != j2) of sum_t c1 conj(c2) / sqrt(E1 E2)| with
// E the series energies; the power is the XDoppler |mean_t r conj(q)|.
//
// The series come from the staged kernel (das_rows.cuh), whose angles run subset by
// subset, or from ensemble_warps; both also sum r conj(q) into pd[2v], pd[2v + 1].
//
// stsw_finish (one warp per voxel): series energies over frames, then the pair sum
// with running row / column sums of the normalized series (for row i, the
// earlier rows' total minus their column j pairs with c[i][j]), the raw weight
// |acc| and the XDoppler magnitude in pd[2v].
template <int K>
__global__ void __launch_bounds__(kWarps * 32) stsw_finish(float* pd, float* weights, const float2* series,
                                                           size_t nv, int nt) {
  const size_t v = size_t(blockIdx.x) * kWarps + (threadIdx.x >> 5);
  if (v >= nv) return;
  const int lane = threadIdx.x & 31;
  const float2* base = series + v * (K * K) * size_t(nt);
  float scale[K * K];
#pragma unroll
  for (int e = 0; e < K * K; ++e) {
    float energy = 0.f;
    for (int t = lane; t < nt; t += 32) energy += cabs2(base[size_t(e) * nt + t]);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) energy += __shfl_xor_sync(0xffffffffu, energy, off);
    scale[e] = energy > 0.f ? 1.0f / sqrtf(energy) : 0.f;
  }
  float2 acc = make_float2(0.f, 0.f);
  for (int t = lane; t < nt; t += 32) {
    float2 total = make_float2(0.f, 0.f), column[K] = {};
#pragma unroll
    for (int i = 0; i < K; ++i) {
      float2 row = make_float2(0.f, 0.f);
#pragma unroll
      for (int j = 0; j < K; ++j) {
        const float2 raw = base[size_t(i * K + j) * nt + t];
        const float2 value = make_float2(raw.x * scale[i * K + j], raw.y * scale[i * K + j]);
        const float2 earlier = make_float2(total.x - column[j].x, total.y - column[j].y);
        acc = cadd(acc, cmul(earlier, cconj(value)));
        column[j] = cadd(column[j], value);
        row = cadd(row, value);
      }
      total = cadd(total, row);
    }
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    acc.x += __shfl_xor_sync(0xffffffffu, acc.x, off);
    acc.y += __shfl_xor_sync(0xffffffffu, acc.y, off);
  }
  if (lane == 0) {
    weights[v] = hypotf(acc.x, acc.y);
    pd[2 * v] = hypotf(pd[2 * v], pd[2 * v + 1]);
  }
}

// --------------------------------------------- single-frame API (core.cu) --
// Channel layout (samples, channels, angles); one frame.
__device__ __forceinline__ float2 frame_sample(const float2* iq, const Voxel& q, const float* el, const float* angles,
                                               const float* starts, int ns, int nc, int na, int ch, int a, int config,
                                               double c, double fs, double fd, double fn) {
  Tap t = tap_of(q, config, el, ch, angles, starts, a, c, fs, fd, fn, ns);
  if (t.i0 < 0) return make_float2(0.f, 0.f);
  size_t i0 = (size_t(t.i0) * nc + ch) * na + a;
  size_t i1 = (size_t(t.i0 == ns - 1 ? t.i0 : t.i0 + 1) * nc + ch) * na + a;
  float2 va = iq[i0], vb = iq[i1];
  float2 val = make_float2(fmaf(t.w, vb.x - va.x, va.x), fmaf(t.w, vb.y - va.y, va.y));
  return cmul(val, t.phase);
}

struct FrameArgs {
  const float2* rc;
  const float2* cr;
  const float* scan;
  const float* xe;
  const float* ye;
  const float* angles;
  const float* starts;
  int ns, nc, na;
  size_t nv;
  double c, fs, fd, fn;
};

// out[v, a] = sum over channels (one aperture).
__global__ void frame_angle_sums(FrameArgs p, int config, float2* out) {
  size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= p.nv * p.na) return;
  size_t v = i / p.na;
  int a = int(i % p.na);
  Voxel q = load_voxel(p.scan, v);
  float2 acc = make_float2(0.f, 0.f);
  for (int ch = 0; ch < p.nc; ++ch)
    acc = cadd(acc, frame_sample(p.rc, q, p.xe, p.angles, p.starts, p.ns, p.nc, p.na, ch, a, config, p.c, p.fs, p.fd,
                                 p.fn));
  out[i] = acc;
}

// channel_sum[v, c] = sum over angles; n_active[v] = active channel count.
__global__ void frame_channel_sums(FrameArgs p, int config, float2* channel_sum, float* n_active) {
  size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= p.nv * p.nc) return;
  size_t v = i / p.nc;
  int ch = int(i % p.nc);
  Voxel q = load_voxel(p.scan, v);
  float2 acc = make_float2(0.f, 0.f);
  for (int a = 0; a < p.na; ++a)
    acc = cadd(acc, frame_sample(p.rc, q, p.xe, p.angles, p.starts, p.ns, p.nc, p.na, ch, a, config, p.c, p.fs, p.fd,
                                 p.fn));
  channel_sum[i] = acc;
  if (ch == 0) {
    float count = 0.f;
    for (int e = 0; e < p.nc; ++e) {
      bool act;
      receive_delay(config ? q.y : q.x, q.z, double(p.xe[e]), p.c, p.fn, &act);
      count += act ? 1.f : 0.f;
    }
    n_active[v] = count;
  }
}

enum FrameOut : int { kFrameOpw = 1, kFrameXd = 2, kFrameFmas = 4, kFrameDmas = 8 };

// Per-voxel single-frame reductions of both apertures.
__global__ void frame_reduce(FrameArgs p, int which, float* opw_out, float* xd_out, float* fmas_out,
                             float* dmas_out) {
  size_t v = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (v >= p.nv) return;
  Voxel q = load_voxel(p.scan, v);
  float2 opw = {}, rsum = {}, qsum = {}, fr = {}, fq = {};
  float er = 0.f, eq = 0.f;
  for (int a = 0; a < p.na; ++a) {
    float2 ra = {}, qa = {};
    for (int ch = 0; ch < p.nc; ++ch) {
      ra = cadd(ra, frame_sample(p.rc, q, p.xe, p.angles, p.starts, p.ns, p.nc, p.na, ch, a, 0, p.c, p.fs, p.fd, p.fn));
      qa = cadd(qa, frame_sample(p.cr, q, p.ye, p.angles, p.starts, p.ns, p.nc, p.na, ch, a, 1, p.c, p.fs, p.fd, p.fn));
    }
    opw = cadd(opw, cadd(ra, qa));
    rsum = cadd(rsum, ra);
    qsum = cadd(qsum, qa);
    fr = cadd(fr, csroot(ra));
    fq = cadd(fq, csroot(qa));
    er += cabs2(ra);
    eq += cabs2(qa);
  }
  if (which & kFrameOpw) opw_out[v] = cabs2(opw);
  if (which & kFrameXd) {
    float2 x = cmul(rsum, cconj(qsum));
    xd_out[v] = hypotf(x.x, x.y);
  }
  if (which & kFrameFmas) fmas_out[v] = cabs2(cmul(fr, fq));
  if (which & kFrameDmas) {
    float2 sqrt_sum = {};
    float abs_sum = 0.f, active = 0.f;
    for (int ch = 0; ch < p.nc; ++ch) {
      float2 sr = {}, sq = {};
      for (int a = 0; a < p.na; ++a) {
        sr = cadd(sr, frame_sample(p.rc, q, p.xe, p.angles, p.starts, p.ns, p.nc, p.na, ch, a, 0, p.c, p.fs, p.fd, p.fn));
        sq = cadd(sq, frame_sample(p.cr, q, p.ye, p.angles, p.starts, p.ns, p.nc, p.na, ch, a, 1, p.c, p.fs, p.fd, p.fn));
      }
      sqrt_sum = cadd(sqrt_sum, cadd(csroot(sr), csroot(sq)));
      abs_sum += hypotf(sr.x, sr.y) + hypotf(sq.x, sq.y);
      bool ar, aq;
      receive_delay(q.x, q.z, double(p.xe[ch]), p.c, p.fn, &ar);
      receive_delay(q.y, q.z, double(p.ye[ch]), p.c, p.fn, &aq);
      active += float(ar) + float(aq);
    }
    float dm = cabs2(sqrt_sum) - abs_sum;
    float wc = (abs_sum > 0.f && active > 0.f) ? fmaxf(dm, 0.f) / active / abs_sum : 0.f;
    float inv = 1.0f / float(p.na);
    float2 mr = make_float2(rsum.x * inv, rsum.y * inv), mq = make_float2(qsum.x * inv, qsum.y * inv);
    float nr = cabs2(mr), nq = cabs2(mq);
    float var = fmaxf(er * inv - nr, 0.f) + fmaxf(eq * inv - nq, 0.f);
    float2 cx = cmul(mr, cconj(mq));
    float num = hypotf(cx.x, cx.y);
    float den = nr + nq + 0.5f * var - num;
    float wa = den > 0.f ? num / den : 0.f;
    float res = dm * wc * wa;
    dmas_out[v] = isfinite(res) ? res : 0.f;
  }
}

// Per-angle IQ (voxels, angles, frames) reductions of the single-frame API.
__global__ void angles_opw(const float2* iq, float2* out, size_t nv, size_t na, size_t nt) {
  size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= nv * nt) return;
  size_t v = i / nt, t = i % nt;
  float2 acc = {};
  for (size_t a = 0; a < na; ++a) acc = cadd(acc, iq[(v * na + a) * nt + t]);
  out[i] = acc;
}

__global__ void angles_pd(const float2* iq, float* out, size_t nv, size_t na, size_t nt, size_t rs, size_t rn,
                          size_t cs, size_t cn, int fmas) {
  size_t v = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (v >= nv) return;
  float2 mean = {};
  float power = 0.f;
  for (size_t t = 0; t < nt; ++t) {
    float2 r = {}, q = {};
    for (size_t a = 0; a < rn; ++a) {
      float2 x = iq[(v * na + rs + a) * nt + t];
      r = cadd(r, fmas ? csroot(x) : x);
    }
    for (size_t a = 0; a < cn; ++a) {
      float2 x = iq[(v * na + cs + a) * nt + t];
      q = cadd(q, fmas ? csroot(x) : x);
    }
    if (fmas)
      power += cabs2(cmul(r, q));
    else
      mean = cadd(mean, cmul(r, cconj(q)));
  }
  out[v] = fmas ? power / float(nt) : hypotf(mean.x / float(nt), mean.y / float(nt));
}

}  // namespace generic
}  // namespace rcb
