// The position model under Patch sampling (physwkim/ptyrs engine/features.rs:337-527,
// engine/lsqml.rs:237-270): each frame's probe moved by its sub-pixel offset on the periodic
// grid, the adjoint move of the probe directions, the Fourier derivative of the object window,
// pty-chi's gradient position sums and its clipped SGD step (in double).
#pragma once
#include "frame.cuh"

namespace ptyb {

enum MoveMode : int {
  kMoveBack = 1,      // planes[slot][m] = conj(q)·T_{−d}(q·planes)  (the adjoint move, in place)
  kDerivWindow = 2,   // planes[slot][a] = ∂_a O_window (periodic Fourier derivative), a = y, x
  kSpectrum = 4,      // planes[m] = DFT(q·P_m), unnormalised, [ky][kx] (one slot)
  kFromSpectrum = 5,  // planes[slot][m] = conj(q)·T_d(q·P_m), probe of frame f moved by d_f,
                      // from the spectrum `spec`
  kDerivSums = 6,     // per frame and axis, the position sums of AP, DM and ML from ∂T_d(q·P)
  kBackSpectrum = 7,  // planes[slot][m] = DFT(conj(O_win)·c_m)·exp(+2πi f·d)/N², [ky][kx]: one
                      // frame's term of the probe back-projection through the move's adjoint
  kPlainInverse = 8,  // planes[m] = conj(q)·IDFT(spec_m), unnormalised (one slot)
  kMoveOwn = 9,       // planes[slot][m] = conj(q)·T_d(q·planes), in place: each frame's own
                      // probe planes (the probe variation's) moved by its offset
  kDerivMove = 10     // planes[slot][m] = conj(q)·∂T_d(q·P_m) from the spectrum `spec`: the
                      // first (deriv 1 y, 2 x) or second (3 yy, 4 yx, 5 xx) derivative over
                      // the offset of kFromSpectrum's moved probe (BH's position terms)
};

struct MoveArgs {
  const float2* probe;    // [K][N][N] shared probe (kSpectrum)
  const float2* quad;     // [N][N]
  const float2* tw;       // [N]
  const float2* object;   // [nyo][nxo] (kDerivWindow, kDerivSums, kBackSpectrum)
  const int* frames;
  const int2* corners;
  const double* offsets;  // [nframe][2] (dy, dx) in object pixels
  float2* planes;         // [slot][K][N][N]
  int nxo, K;
  const float2* spec;     // [K][N][N] a spectrum, [ky][kx] (kFromSpectrum, kDerivSums,
                          // kPlainInverse)
  const float2* c;        // [slot][K][N][N] natural: the change of the exit wave (kDerivSums),
                          // the exit-plane gradient (kBackSpectrum)
  double* sums;           // [nframe][4] num_y, num_x, den_y, den_x (kDerivSums)
  int deriv;              // kDerivMove: 1 ∂y, 2 ∂x, 3 ∂y∂y, 4 ∂y∂x, 5 ∂x∂x
  // Optional, [slot][K][N][N] natural: each frame's moved probes W; kDerivSums and
  // kBackSpectrum then take c − W·O·q, the carried waves' residual against the model
  // (AP / DM / RAAR, engine/features.rs:653-725, 992-1025).
  const float2* minus;
};

// numpy fftfreq of index k of n points (engine/features.rs:337-344).
PTYB_D float fft_freq(int k, int n) { return (float)(k < (n + 1) / 2 ? k : k - n) / (float)n; }

// Shared memory of K planes: frame_smem_bytes and the translation phase's N row factors.
template <int N, int C>
__host__ __device__ constexpr size_t move_smem_bytes(int K) {
  return frame_smem_bytes<N, C>(K) + N * sizeof(float2);
}

// One frame per cluster, planes through plane.cuh's line transforms: forward from natural rows
// (or a spectrum read in the columns), the phase in the columns, inverse to natural rows. As the
// frame kernel, bound by latency (its exchanges and cluster barriers); per frame on one B200 at
// 256² x 2 modes: moves from the spectrum 1.42 -> 0.79 us, probe gradient spectra 1.57 -> 0.90,
// position sums 3.21 -> 2.03 (four inverse transforms; 2.15 on clusters of 8), one plane's spectrum
// 27 -> 17 us a call.
template <int N, int C, int MODE>
__global__ void __launch_bounds__(PlaneShape<N, C>::T,
                                  plane_min_blocks<N, C>(MODE != kDerivSums &&
                                                         MODE != kDerivWindow))
    move_kernel(MoveArgs a) {
  using L = Lines<N, C>;
  constexpr int H = L::H, T = L::T, E = L::N1, N2 = L::N2;
  extern __shared__ __align__(128) unsigned char plane_smem[];
  const int K = MODE == kDerivWindow ? 2 : a.K;
  // planes held in shared memory: the position sums hold the two axes of one mode at a time
  const int KP = MODE == kDerivSums ? max(K, 2) : K;
  float2* S = reinterpret_cast<float2*>(plane_smem);
  float2* table = S + (size_t)KP * H * N;
  float2* ey = table + N;
  double* red = reinterpret_cast<double*>(ey + N);
  cg::cluster_group cluster = cg::this_cluster();
  const int r = C > 1 ? (int)cluster.block_rank() : 0;
  const int slot = blockIdx.x / C;
  constexpr bool one = MODE == kSpectrum || MODE == kPlainInverse;  // not per frame
  const int f = one ? 0 : a.frames[slot];
  const int2 corner = one ? make_int2(0, 0) : a.corners[f];
  const int tid = threadIdx.x;
  const L ln(S, table, r);
  L::fill_table(table, a.tw);
  constexpr size_t plane = (size_t)N * N;
  constexpr float inv_n2 = 1.0f / ((float)N * (float)N);
  constexpr float two_pi = 2.f * 3.14159265358979f;
  constexpr bool from_spec = MODE == kFromSpectrum || MODE == kDerivSums ||
                             MODE == kPlainInverse || MODE == kDerivMove;
  constexpr bool in_place = MODE == kMoveBack || MODE == kMoveOwn;
  constexpr bool moves = in_place || MODE == kFromSpectrum || MODE == kDerivSums ||
                         MODE == kDerivMove || MODE == kBackSpectrum;
  constexpr int kRow = N2 * N;  // pixels between a thread's elements of a column
  // Row-mapped: natural row y, first element's pixel; column-mapped: column kx, its first ky's.
  const int y = r * H + ln.y, rpix = y * N + ln.rt;
  const int kx = r * H + ln.c, cpix = ln.t * N + kx;
  float2* out = a.planes + (size_t)slot * K * plane;
  const float2* obj = a.object + (size_t)(corner.x + y) * a.nxo + corner.y + ln.rt;
  const float2* quad = a.quad + rpix;

  // The translation phase exp(−2πi f·d) = exp(−2πi fy·dy)·exp(−2πi fx·dx), over N²: the row
  // factor of every ky in shared memory, the column factor of this thread's one column.
  float2 ex = make_float2(1.f, 0.f);
  if (moves) {
    const float sgn = MODE == kMoveBack || MODE == kBackSpectrum ? -1.f : 1.f;
    const float dy = sgn * (float)a.offsets[2 * f], dx = sgn * (float)a.offsets[2 * f + 1];
    float sn, cs;
    for (int k = tid; k < N; k += T) {
      sincospif(-2.f * fft_freq(k, N) * dy, &sn, &cs);
      ey[k] = make_float2(cs * inv_n2, sn * inv_n2);
    }
    sincospif(-2.f * fft_freq(kx, N) * dx, &sn, &cs);
    ex = make_float2(cs, sn);
  }
  // The phase at element i of this thread's column (fy of it beside).
  auto phase = [&](int i) { return moves ? cmul(ey[N2 * i + ln.t], ex) : make_float2(1.f, 0.f); };
  auto freq_y = [&](int i) { return two_pi * fft_freq(N2 * i + ln.t, N); };
  const float freq_x = two_pi * fft_freq(kx, N);

  float2 v[E];
  if (!from_spec) {
    // Natural-layout rows, times q or the window's conjugate, through the row transforms; the
    // window derivatives transform their one plane once for both axes.
    float2 w[E];
    if (MODE != kDerivWindow) {
      const float2* src = MODE == kBackSpectrum ? obj : quad;
#pragma unroll
      for (int i = 0; i < E; ++i) w[i] = src[N2 * i];
    }
    const int kin = MODE == kDerivWindow ? 1 : K;
#pragma unroll 1
    for (int m = 0; m < kin; ++m) {
      const float2* src = MODE == kDerivWindow    ? obj
                          : MODE == kSpectrum     ? a.probe + m * plane + rpix
                          : MODE == kBackSpectrum ? a.c + ((size_t)slot * K + m) * plane + rpix
                                                  : out + m * plane + rpix;
#pragma unroll
      for (int i = 0; i < E; ++i) v[i] = src[N2 * i];
      if (MODE == kBackSpectrum) {
        if (a.minus) {
          const float2* wave = a.minus + ((size_t)slot * K + m) * plane + rpix;
#pragma unroll
          for (int i = 0; i < E; ++i)
            v[i] = csub(v[i], cmul(cmul(wave[N2 * i], w[i]), quad[N2 * i]));
        }
#pragma unroll
        for (int i = 0; i < E; ++i) v[i] = cmulc(w[i], v[i]);
      } else if (MODE != kDerivWindow) {
#pragma unroll
        for (int i = 0; i < E; ++i) v[i] = cmul(w[i], v[i]);
      }
      if (m == 0) __syncthreads();  // the twiddle table, the row factors
      ln.rows_forward(v, m);
    }
    L::publish();
  }

  if (MODE == kDerivSums) {
    // Both axes of one mode at a time, the planes holding ∂_y and ∂_x of mode m's moved probe;
    // the field plane and the window are read per axis, the second time from the caches. Held in
    // registers over the second axis' transform they took 2.17 us per frame of 256² x 2 instead of
    // 2.03, with 268 bytes of spills instead of 80.
    const float2* cf = a.c + (size_t)slot * K * plane + rpix;
    double v4[4] = {0.0, 0.0, 0.0, 0.0};  // num_y, num_x, den_y, den_x
#pragma unroll 1
    for (int m = 0; m < K; ++m) {
      float2 s[E];
      const float2* spec = a.spec + m * plane + cpix;
#pragma unroll
      for (int i = 0; i < E; ++i) s[i] = spec[i * kRow];
      if (m == 0) __syncthreads();  // the twiddle table, the row factors
#pragma unroll
      for (int i = 0; i < E; ++i) s[i] = cmul(s[i], phase(i));
      // × (−2πi·f_axis): the derivative of the translation phase (engine/features.rs:372-387)
#pragma unroll
      for (int i = 0; i < E; ++i) {
        const float w = freq_y(i);
        v[i] = make_float2(w * s[i].y, -w * s[i].x);
      }
      ln.columns_inverse(v, 0);
#pragma unroll
      for (int i = 0; i < E; ++i) v[i] = make_float2(freq_x * s[i].y, -freq_x * s[i].x);
      ln.columns_inverse(v, 1);
      L::publish();
      // dψ = O·∂W on natural rows; num = Σ Re(conj(c)·dψ), den = Σ |dψ|² over modes and
      // pixels (engine/features.rs:992-1025)
#pragma unroll
      for (int ax = 0; ax < 2; ++ax) {
        ln.rows_inverse(v, ax);
        float2 cv[E];
#pragma unroll
        for (int i = 0; i < E; ++i) cv[i] = cf[m * plane + N2 * i];
        if (a.minus) {
          const float2* wave = a.minus + ((size_t)slot * K + m) * plane + rpix;
#pragma unroll
          for (int i = 0; i < E; ++i)
            cv[i] = csub(cv[i], cmul(cmul(wave[N2 * i], obj[N2 * i]), quad[N2 * i]));
        }
#pragma unroll
        for (int i = 0; i < E; ++i) {
          const float2 d = cmul(obj[N2 * i], v[i]);
          v4[ax] += (double)cv[i].x * d.x + (double)cv[i].y * d.y;
          v4[2 + ax] += (double)d.x * d.x + (double)d.y * d.y;
        }
      }
    }
    cluster_sum4<T, C>(v4, red, cluster);
    if (r == 0 && tid == 0)
#pragma unroll
      for (int k = 0; k < 4; ++k) a.sums[(size_t)f * 4 + k] = v4[k];
    return;
  }

  if (MODE == kDerivWindow) {
    // × 2πi·f_axis / N² for both axes
    ln.columns_forward(v, 0);
    float2 u[E];
#pragma unroll
    for (int ax = 0; ax < 2; ++ax) {
#pragma unroll
      for (int i = 0; i < E; ++i) {
        const float w = (ax == 0 ? freq_y(i) : freq_x) * inv_n2;
        u[i] = make_float2(-w * v[i].y, w * v[i].x);
      }
      ln.columns_inverse(u, ax);
    }
  } else {
#pragma unroll 1
    for (int m = 0; m < K; ++m) {
      if (from_spec) {
        const float2* spec = a.spec + m * plane + cpix;
#pragma unroll
        for (int i = 0; i < E; ++i) v[i] = spec[i * kRow];
        if (m == 0) __syncthreads();  // the twiddle table, the row factors
      } else {
        ln.columns_forward(v, m);
      }
      if (MODE == kDerivMove) {
        // × (−2πi·f_a) or × (−2πi·f_a)(−2πi·f_b) = −4π²·f_a·f_b
#pragma unroll
        for (int i = 0; i < E; ++i) {
          float2 e = phase(i);
          const float wy = freq_y(i), wx = freq_x;
          if (a.deriv <= 2) {
            const float w = a.deriv == 1 ? wy : wx;
            e = make_float2(w * e.y, -w * e.x);
          } else {
            const float w = a.deriv == 3 ? -wy * wy : a.deriv == 4 ? -wy * wx : -wx * wx;
            e = make_float2(w * e.x, w * e.y);
          }
          v[i] = cmul(v[i], e);
        }
      } else if (moves) {
#pragma unroll
        for (int i = 0; i < E; ++i) v[i] = cmul(v[i], phase(i));
      }
      if (MODE == kSpectrum || MODE == kBackSpectrum) {
        // the spectrum's columns to [slot][m][ky][kx]
        float2* dst = out + m * plane + cpix;
#pragma unroll
        for (int i = 0; i < E; ++i) dst[i * kRow] = v[i];
      } else {
        ln.columns_inverse(v, m);
      }
    }
  }
  if (MODE == kSpectrum || MODE == kBackSpectrum) return;
  L::publish();

  float2 w[E];
  if (MODE != kDerivWindow) {
#pragma unroll
    for (int i = 0; i < E; ++i) w[i] = quad[N2 * i];
  }
#pragma unroll 1
  for (int m = 0; m < K; ++m) {
    ln.rows_inverse(v, m);
    float2* dst = out + m * plane + rpix;
#pragma unroll
    for (int i = 0; i < E; ++i) dst[N2 * i] = MODE == kDerivWindow ? v[i] : cmulc(w[i], v[i]);
  }
}

// planes[slot][m] = w·χ_m per natural pixel: each frame's probe direction before its adjoint
// move, w = conj(q·O_window) (LSQML, engine/lsqml.rs:200-207) or, with `omax`, rPIE's weight
// conj(q·O)/((1 − α)|O|² + α·max|O|²) (engine/ptycho.rs:1007-1026).
static __global__ void probe_terms_kernel(const float2* object, const float2* quad, const float2* chi,
                                   const int* frames, const int2* corners, int nxo, int K, int N,
                                   float2* planes, const float* omax = nullptr,
                                   float alpha = 0.f) {
  const int slot = blockIdx.y;
  const size_t plane = (size_t)N * N;
  const int2 c = corners[frames[slot]];
  for (int pix = blockIdx.x * blockDim.x + threadIdx.x; pix < N * N;
       pix += gridDim.x * blockDim.x) {
    const int y = pix / N, x = pix % N;
    const float2 o = object[(size_t)(c.x + y) * nxo + c.y + x];
    float2 w = cconj(cmul(quad[pix], o));
    if (omax) w = cscale(w, 1.f / ((1.f - alpha) * cnorm2(o) + alpha * omax[slot]));
    for (int m = 0; m < K; ++m) {
      const size_t i = ((size_t)slot * K + m) * plane + pix;
      planes[i] = cmul(w, chi[i]);
    }
  }
}

// Per slot, pty-chi's position sums on mode 0 (engine/features.rs:459-492): with w the
// frame's moved probe times q, per axis num = Σ Re(conj(∂O·w)·χ), den = Σ |∂O·w|²;
// sums[slot] = (num_y, num_x, den_y, den_x) in double.
static __global__ void __launch_bounds__(256) position_sums_kernel(const float2* dwin,
                                                           const float2* wave, int wave_stride,
                                                           const float2* quad,
                                                           const float2* chi, int K, int N,
                                                           double* sums) {
  __shared__ double sh[8];
  const int slot = blockIdx.x;
  const size_t plane = (size_t)N * N;
  double s[4] = {0, 0, 0, 0};
  for (int pix = threadIdx.x; pix < N * N; pix += 256) {
    const float2 w = cmul(wave[(size_t)slot * wave_stride + pix], quad[pix]);
    const float2 c = chi[(size_t)slot * K * plane + pix];
    for (int a = 0; a < 2; ++a) {
      const float2 u = cmul(dwin[((size_t)slot * 2 + a) * plane + pix], w);
      s[a] += (double)u.x * c.x + (double)u.y * c.y;
      s[2 + a] += (double)u.x * u.x + (double)u.y * u.y;
    }
  }
  for (int k = 0; k < 4; ++k) {
    double v = warp_sum(s[k]);
    if (threadIdx.x % 32 == 0) sh[threadIdx.x / 32] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
      double t = 0.0;
      for (int w = 0; w < 8; ++w) t += sh[w];
      sums[(size_t)slot * 4 + k] = t;
    }
    __syncthreads();
  }
}

// pty-chi's gradient position step on the batch (engine/features.rs:496-521) in double, one
// block: delta = num/(den + max(max_batch den, eps)), dx = 0.3·delta at the batch's frames
// (0 elsewhere), each axis clipped to min(10·mean|dx − mean dx|, 0.1) over every frame. The
// sums run in slot order, one warp per axis, over terms every thread forms (by one thread alone,
// its divisions took 113 us a batch of 150).
static __global__ void __launch_bounds__(1024) position_step_kernel(const double* sums, int nslot,
                                                                    int nframe, double eps,
                                                                    const int* frames,
                                                                    double* offsets) {
  __shared__ double term[2][1024], red[2][32], mx[2], acc[2];
  const int t = threadIdx.x;
  double m0 = eps, m1 = eps;
  for (int s = t; s < nslot; s += 1024) {
    m0 = fmax(m0, sums[s * 4 + 2]);
    m1 = fmax(m1, sums[s * 4 + 3]);
  }
  for (int o = 16; o > 0; o >>= 1) {
    m0 = fmax(m0, __shfl_xor_sync(0xffffffffu, m0, o));
    m1 = fmax(m1, __shfl_xor_sync(0xffffffffu, m1, o));
  }
  if (t % 32 == 0) {
    red[0][t / 32] = m0;
    red[1][t / 32] = m1;
  }
  __syncthreads();
  if (t < 2) {
    double m = eps;
    for (int w = 0; w < 32; ++w) m = fmax(m, red[t][w]);
    mx[t] = m;
  }
  __syncthreads();
  auto dx = [&](int s, int a) { return 0.3 * (sums[s * 4 + a] / (sums[s * 4 + 2 + a] + mx[a])); };
  // Σ f(dx) over the slots in order, per axis, into acc[axis]
  auto sum = [&](auto f) {
    if (t < 2) acc[t] = 0.0;
    for (int s0 = 0; s0 < nslot; s0 += 1024) {
      const int n = min(1024, nslot - s0);
      if (t < n) {
        term[0][t] = f(dx(s0 + t, 0), 0);
        term[1][t] = f(dx(s0 + t, 1), 1);
      }
      __syncthreads();
      if (t == 0 || t == 32) acc[t / 32] += ordered_sum(term[t / 32], 0, n);
      __syncthreads();
    }
  };
  sum([](double x, int) { return x; });
  const double mean[2] = {acc[0] / nframe, acc[1] / nframe};
  __syncthreads();
  sum([&](double x, int a) { return fabs(x - mean[a]); });
  double limit[2];
  for (int a = 0; a < 2; ++a)
    limit[a] = fmin(10.0 * (((double)(nframe - nslot) * fabs(mean[a]) + acc[a]) / nframe), 0.1);
  for (int s = t; s < nslot; s += 1024)
    for (int a = 0; a < 2; ++a)
      offsets[2 * frames[s] + a] += fmin(fmax(dx(s, a), -limit[a]), limit[a]);
}

// Block sum of one double per thread in a fixed order (lane trees, then warps in order).
template <int T>
PTYB_D double fixed_block_sum(double v, double* sh) {
  v = warp_sum(v);
  __syncthreads();
  if (threadIdx.x % 32 == 0) sh[threadIdx.x / 32] = v;
  __syncthreads();
  double s = 0.0;
  for (int w = 0; w < T / 32; ++w) s += sh[w];
  return s;
}

// The position step of AP, DM and ML on every frame (engine/features.rs:1028-1047), one block:
// per axis, with max the largest den, step = clip(0.3·num / (den + max), ±0.1) (0 where that
// denominator is not positive) and d += step − mean(step) over every frame.
static __global__ void __launch_bounds__(1024) ml_position_step_kernel(const double* sums, int nframe,
                                                               double* offsets) {
  __shared__ double sh[32];
  const int t = threadIdx.x;
  for (int a = 0; a < 2; ++a) {
    double mx = 0.0;
    for (int f = t; f < nframe; f += 1024) mx = fmax(mx, sums[(size_t)f * 4 + 2 + a]);
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    __syncthreads();
    if (t % 32 == 0) sh[t / 32] = mx;
    __syncthreads();
    mx = 0.0;
    for (int w = 0; w < 32; ++w) mx = fmax(mx, sh[w]);
    auto step = [&](int f) {
      const double den = sums[(size_t)f * 4 + 2 + a] + mx;
      return den > 0.0 ? fmin(fmax(0.3 * sums[(size_t)f * 4 + a] / den, -0.1), 0.1) : 0.0;
    };
    double part = 0.0;
    for (int f = t; f < nframe; f += 1024) part += step(f);
    const double mean = fixed_block_sum<1024>(part, sh) / nframe;
    for (int f = t; f < nframe; f += 1024) offsets[2 * f + a] += step(f) - mean;
    __syncthreads();
  }
}

}  // namespace ptyb
