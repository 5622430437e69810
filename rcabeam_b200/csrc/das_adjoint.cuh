// Differentiable OPW delay-and-sum: forward with per-element delay offsets and
// a sound speed parameter, and its hand-written adjoint.
//
// Model (both apertures A = RC, CR; receive element e_c; offset d[A][c]):
//   tau   = (z cos th_a + u sin th_a) / c_s + sqrt(z^2 + (w - e_c)^2) / c_s + d[A][c]
//   s     = (tau - start_a) fs, valid iff 0 <= s <= ns - 1 and inside the f-number aperture
//   y     = ((1 - f) X[i0] + f X[i1]) exp(+j 2 pi fd tau),  i0 = floor(s), f = s - i0, i1 = min(i0 + 1, ns - 1)
//   IQ    = sum over A, c, a of y;  PD = mean_t |IQ|^2
// Adjoint, for the upstream gradient G = dL/dIQ (dL/dRe + j dL/dIm):
//   dX[i0] += (1 - f) conj(phase) G,  dX[i1] += f conj(phase) G          (scatter, atomics)
//   dL/dtau = Re sum_t conj(G) (fs (X[i1] - X[i0]) phase + j 2 pi fd y)
//   d offsets[A][c] += dL/dtau,  d c_s += dL/dtau * (-(tau - d[A][c]) / c_s)
// (reference model: src/rcabeam/sim.py:344-393 and opw.py:8-21; offsets and c_s
// are the parameters of the differentiation form).
//
// Both kernels work on a list of voxels and a chunk of at most kChunk frames,
// so the autograd layer recomputes IQ chunk by chunk in the backward pass
// instead of keeping the ensemble.  REAL = float reads complex64 channels and
// accumulates in float32 (phases from a float64-reduced cycle count, as the
// main path); REAL = double reads complex128 and is float64 throughout (the
// finite-difference checker).  Geometry is float64 in both.
#pragma once

#include "common.cuh"

namespace rcb {
namespace adj {

constexpr int kChunk = 8;  // frames per launch (registers per thread)

template <typename R>
struct Cx;
template <>
struct Cx<float> {
  using type = float2;
};
template <>
struct Cx<double> {
  using type = double2;
};

struct Geometry {
  const float* scan;
  const unsigned* voxels;  // list of voxel indices into scan, or null (identity)
  const float* xe;
  const float* ye;
  const float* angles;
  const float* starts;
  const double* offsets;  // [2][nc]
  double c, fs, fd, fn;
  int nvl, ns, nc, na, nt, f0, frames;
};

struct Tap64 {
  bool ok;
  int i0, i1;
  double tau, f;
};

// cos, sin and start of the first kTable angles, formed once per CTA.
constexpr int kTable = 128;
struct Angles {
  double cs[kTable], sn[kTable], start[kTable];
};
__device__ __forceinline__ void fill_angles(const Geometry& g, Angles& t) {
  for (int a = threadIdx.x; a < min(g.na, kTable); a += blockDim.x) {
    sincos(double(g.angles[a]), &t.sn[a], &t.cs[a]);
    t.start[a] = double(g.starts[a]);
  }
  __syncthreads();
}

// Receive delay of a voxel (w along the receive elements) and channel.
struct Receive {
  double delay, offset;
  bool active;
};
__device__ __forceinline__ Receive receive_of(const Geometry& g, double w, double z, int ap, int ch) {
  Receive r;
  r.active = true;
  r.delay = receive_delay(w, z, double(ap ? g.ye[ch] : g.xe[ch]), g.c, g.fn, &r.active);
  r.offset = g.offsets[ap * g.nc + ch];
  return r;
}

__device__ __forceinline__ Tap64 tap(const Geometry& g, const Angles& t, const Receive& rx, double u, double z,
                                     int a) {
  Tap64 q;
  double cs, sn, start;
  if (a < kTable) {
    cs = t.cs[a];
    sn = t.sn[a];
    start = t.start[a];
  } else {
    sincos(double(g.angles[a]), &sn, &cs);
    start = double(g.starts[a]);
  }
  q.tau = __dadd_rn(__dadd_rn(transmit_delay(u, z, cs, sn, g.c), rx.delay), rx.offset);
  const double s = __dmul_rn(__dadd_rn(q.tau, -start), g.fs);
  q.ok = rx.active && s >= 0.0 && s <= double(g.ns - 1);
  const double fl = floor(s);
  q.i0 = q.ok ? int(fl) : 0;
  q.i1 = min(q.i0 + 1, g.ns - 1);
  q.f = s - fl;
  return q;
}

template <typename R>
__device__ __forceinline__ typename Cx<R>::type phase_of(double fd, double tau) {
  double cyc = fd * tau;
  cyc -= rint(cyc);
  if constexpr (sizeof(R) == 4) {
    float sn, cs;
    sincospif(2.0f * float(cyc), &sn, &cs);
    return make_float2(cs, sn);
  } else {
    double sn, cs;
    sincospi(2.0 * cyc, &sn, &cs);
    return make_double2(cs, sn);
  }
}

__device__ __forceinline__ void voxel_pos(const Geometry& g, int l, double& x, double& z, double& y) {
  const size_t v = g.voxels ? size_t(g.voxels[l]) : size_t(l);
  x = double(g.scan[3 * v]);
  z = double(g.scan[3 * v + 1]);
  y = double(g.scan[3 * v + 2]);
}

// IQ of frames [f0, f0 + frames) and/or its power sum, a warp per listed voxel:
// each lane sums every 32nd (aperture, channel) pair, then the warp adds
// up.  A region of interest lists far fewer voxels than the GPU has threads (1332
// for a 1 mm sphere): one thread each left eleven CTAs walking all channels one
// after another (3.35 ms per 8-frame chunk at 2 x 128 channels and 7 angles, angles'
// sines formed per tap); with a warp each the same chunk takes 0.19 ms, and 100000
// voxels 10.1 ms against 11.5 (complex128 10.3 against 11.8).  A channel's
// angles are summed in R, the channels in float64: the delay and sound-speed
// gradients are float64 sums over all of a region's samples, and what they lose is
// mostly the rounding of the IQ formed here.
template <typename R>
__global__ void __launch_bounds__(128) forward(Geometry g, const typename Cx<R>::type* __restrict__ rc,
                                               const typename Cx<R>::type* __restrict__ cr,
                                               typename Cx<R>::type* __restrict__ iq, double* __restrict__ power) {
  using C = typename Cx<R>::type;
  __shared__ Angles table;
  fill_angles(g, table);
  const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int sub = int(id % 32);
  if (id / 32 >= g.nvl) return;
  const int l = int(id / 32);
  double x, z, y;
  voxel_pos(g, l, x, z, y);
  double re[kChunk], im[kChunk];
#pragma unroll
  for (int t = 0; t < kChunk; ++t) re[t] = im[t] = 0.0;
  for (int pair = sub; pair < 2 * g.nc; pair += 32) {
    const int ap = pair >= g.nc, ch = pair - ap * g.nc;
    const C* X = ap ? cr : rc;
    const double u = ap ? x : y;
    const Receive rx = receive_of(g, ap ? y : x, z, ap, ch);
    if (!rx.active) continue;
    R sr[kChunk], si[kChunk];
#pragma unroll
    for (int k = 0; k < kChunk; ++k) sr[k] = si[k] = R(0);
    for (int a = 0; a < g.na; ++a) {
      const Tap64 t = tap(g, table, rx, u, z, a);
      if (!t.ok) continue;
      const C ph = phase_of<R>(g.fd, t.tau);
      const R f = R(t.f), f0w = R(1) - f;
      const size_t b0 = ((size_t(t.i0) * g.nc + ch) * g.na + a) * g.nt + g.f0;
      const size_t b1 = ((size_t(t.i1) * g.nc + ch) * g.na + a) * g.nt + g.f0;
#pragma unroll
      for (int k = 0; k < kChunk; ++k) {
        if (k < g.frames) {
          const C x0 = X[b0 + k], x1 = X[b1 + k];
          const R vr = f0w * x0.x + f * x1.x, vi = f0w * x0.y + f * x1.y;
          sr[k] += vr * ph.x - vi * ph.y;
          si[k] += vr * ph.y + vi * ph.x;
        }
      }
    }
#pragma unroll
    for (int k = 0; k < kChunk; ++k) {
      re[k] += double(sr[k]);
      im[k] += double(si[k]);
    }
  }
#pragma unroll
  for (int k = 0; k < kChunk; ++k) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      re[k] += __shfl_xor_sync(0xffffffffu, re[k], off);
      im[k] += __shfl_xor_sync(0xffffffffu, im[k], off);
    }
  }
  if (sub != 0) return;
  double p = 0.0;
#pragma unroll
  for (int k = 0; k < kChunk; ++k) {
    if (k < g.frames) {
      if (iq) iq[size_t(l) * g.frames + k] = C{R(re[k]), R(im[k])};
      p += re[k] * re[k] + im[k] * im[k];
    }
  }
  if (power) power[l] += p / double(g.nt);
}

__device__ __forceinline__ void atomic_add_c(float2* p, float2 v) {
  atomicAdd(p, v);  // one 8-byte vector reduction
}
__device__ __forceinline__ void atomic_add_c(double2* p, double2 v) {
  atomicAdd(&p->x, v.x);
  atomicAdd(&p->y, v.y);
}

// Adds w0 v[k] and w1 v[k] of the chunk's frames to rows b0 and b1 of the channel
// gradients: 16-byte vector reductions where the rows allow them (two frames per
// reduction instead of one component).
template <typename R>
__device__ __forceinline__ void scatter(typename Cx<R>::type* GX, size_t b0, size_t b1, R w0, R w1,
                                        const typename Cx<R>::type (&v)[kChunk], int frames, bool paired) {
  using C = typename Cx<R>::type;
  if constexpr (sizeof(R) == 4) {
    if (paired) {
#pragma unroll
      for (int k = 0; k < kChunk; k += 2) {
        if (k >= frames) break;
        // frames is even here, so both frames of the pair are live.
        atomicAdd(reinterpret_cast<float4*>(GX + b0 + k),
                  make_float4(w0 * v[k].x, w0 * v[k].y, w0 * v[k + 1].x, w0 * v[k + 1].y));
        atomicAdd(reinterpret_cast<float4*>(GX + b1 + k),
                  make_float4(w1 * v[k].x, w1 * v[k].y, w1 * v[k + 1].x, w1 * v[k + 1].y));
      }
      return;
    }
  }
#pragma unroll
  for (int k = 0; k < kChunk; ++k) {
    if (k < frames) {
      atomic_add_c(GX + b0 + k, C{w0 * v[k].x, w0 * v[k].y});
      atomic_add_c(GX + b1 + k, C{w1 * v[k].x, w1 * v[k].y});
    }
  }
}

// One thread per (listed voxel, aperture, channel): scatter of G into the
// channel gradients and the delay / sound-speed gradient sums.
template <typename R>
__global__ void __launch_bounds__(128) adjoint(Geometry g, const typename Cx<R>::type* __restrict__ rc,
                                               const typename Cx<R>::type* __restrict__ cr,
                                               const typename Cx<R>::type* __restrict__ grad_iq,
                                               typename Cx<R>::type* grad_rc, typename Cx<R>::type* grad_cr,
                                               double* grad_offsets, double* grad_c) {
  using C = typename Cx<R>::type;
  __shared__ Angles table;
  fill_angles(g, table);
  const size_t id = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  const size_t total = size_t(g.nvl) * 2 * g.nc;
  double d_tau_sum = 0.0, d_c = 0.0;
  int ap = 0, ch = 0;
  if (id < total) {
    const int l = int(id / (2 * g.nc));
    ap = int((id / g.nc) % 2);
    ch = int(id % g.nc);
    double x, z, y;
    voxel_pos(g, l, x, z, y);
    const C* X = ap ? cr : rc;
    C* GX = ap ? grad_cr : grad_rc;
    const double u = ap ? x : y, w = ap ? y : x;
    C G[kChunk];
#pragma unroll
    for (int k = 0; k < kChunk; ++k) G[k] = k < g.frames ? grad_iq[size_t(l) * g.frames + k] : C{R(0), R(0)};
    const double two_pi_fd = 2.0 * 3.141592653589793 * g.fd;
    const Receive rx = receive_of(g, w, z, ap, ch);
    const bool paired = sizeof(R) == 4 && g.nt % 2 == 0 && g.f0 % 2 == 0 && g.frames % 2 == 0 &&
                        reinterpret_cast<uintptr_t>(GX) % 16 == 0;
    for (int a = 0; rx.active && a < g.na; ++a) {
      const Tap64 t = tap(g, table, rx, u, z, a);
      if (!t.ok) continue;
      const C ph = phase_of<R>(g.fd, t.tau);
      const R f = R(t.f), f0w = R(1) - f;
      const size_t b0 = ((size_t(t.i0) * g.nc + ch) * g.na + a) * g.nt + g.f0;
      const size_t b1 = ((size_t(t.i1) * g.nc + ch) * g.na + a) * g.nt + g.f0;
      double dtau = 0.0;
      C back[kChunk];  // conj(phase) G
#pragma unroll
      for (int k = 0; k < kChunk; ++k) {
        back[k] = C{ph.x * G[k].x + ph.y * G[k].y, ph.x * G[k].y - ph.y * G[k].x};
        if (k < g.frames) {
          const C x0 = X[b0 + k], x1 = X[b1 + k];
          // y and its tau derivative.
          const double vr = double(f0w) * x0.x + double(f) * x1.x, vi = double(f0w) * x0.y + double(f) * x1.y;
          const double yr = vr * ph.x - vi * ph.y, yi = vr * ph.y + vi * ph.x;
          const double sr = g.fs * (double(x1.x) - x0.x), si = g.fs * (double(x1.y) - x0.y);
          const double dr = sr * ph.x - si * ph.y - two_pi_fd * yi;
          const double di = sr * ph.y + si * ph.x + two_pi_fd * yr;
          dtau += double(G[k].x) * dr + double(G[k].y) * di;  // Re(conj(G) dy)
        }
      }
      scatter<R>(GX, b0, b1, f0w, f, back, g.frames, paired);
      d_tau_sum += dtau;
      d_c += dtau * (-(t.tau - g.offsets[ap * g.nc + ch]) / g.c);
    }
    if (d_tau_sum != 0.0) atomicAdd(grad_offsets + ap * g.nc + ch, d_tau_sum);
  }
  for (int off = 16; off > 0; off >>= 1) d_c += __shfl_xor_sync(0xffffffffu, d_c, off);
  if ((threadIdx.x & 31) == 0 && d_c != 0.0) atomicAdd(grad_c, d_c);
}

}  // namespace adj
}  // namespace rcb
