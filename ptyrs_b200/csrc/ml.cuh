// Poisson maximum-likelihood conjugate gradient on the device (physwkim/ptyrs
// engine/ptycho.rs:775-842): the line-search numerator and denominator of
// `cg_poisson_gamma` (engine/ops.rs:206-253) per frame, and the array reductions of the
// Polak–Ribière β and of `scale_obj_probe` (engine/ptycho.rs:577-591).
#pragma once
#include "frame.cuh"

namespace ptyb {

// Per frame: with po = F(P·O·q) the gradient pass kept, a = F(P·dO·q + dP·O·q) and
// b = F(dP·dO·q) mode by mode, per-pixel accumulators calc = Σ|po|², r = Σ Re(p̄o·a),
// s = Σ |a|² + 2·Re(p̄o·b); then over unmasked pixels, d = 1 − I/max(calc, 1e-32):
// num = −Σ 2·r·d, den = Σ 2·s·d + I·(2r/calc)². The b-term of den is linear in b, so it is
// taken in the exit plane against the gradient pass's field (no transform of b). Shared memory
// holds the K planes of a; the accumulators are each thread's pixels, in registers. Bound by the
// latency of its loads (six arrays in the rows: 4.0 of 10.4 stalled warps per issue) at 14 warps
// per SM: 3.4 -> 2.39 us per frame of 256² x 2, 1.47 -> 0.935 at 192², against one plane at a time
// with the accumulators in shared memory.
struct GammaArgs {
  const float2* object;
  const float2* d_obj;
  const float2* probe;
  const float2* d_probe;
  const float2* quad;
  const float2* tw;
  const float* iobs;
  const int* frames;
  const int2* corners;
  double* out;  // [slot][2]: num, den
  int nyo, nxo, nprobe, nobj;
  // Elements between consecutive slots' probe and probe direction: 0 for the shared ones,
  // K·N·N for the per-frame moved ones of the position model.
  int probe_stride;
  // po = DFT(P·O·q) of every slot and mode as the gradient pass kept it, [slot][K][ky][kx],
  // and its exit-plane gradient field g = IDFT(2(1 − I/Ĩ)·po)/N² (masked 0), [slot][K][N][N].
  const float2* psi;
  const float2* g;
};

template <int N, int C>
__global__ void __launch_bounds__(PlaneShape<N, C>::T, plane_min_blocks<N, C>())
    gamma_kernel(GammaArgs a) {
  using L = Lines<N, C>;
  constexpr int H = L::H, T = L::T, E = L::N1, N2 = L::N2;
  extern __shared__ __align__(128) unsigned char plane_smem[];
  const int K = a.nprobe * a.nobj;
  float2* S = reinterpret_cast<float2*>(plane_smem);
  float2* table = S + (size_t)K * H * N;
  double* red = reinterpret_cast<double*>(table + N);
  cg::cluster_group cluster = cg::this_cluster();
  const int r = C > 1 ? (int)cluster.block_rank() : 0;
  const int slot = blockIdx.x / C;
  const int f = a.frames[slot];
  const int2 corner = a.corners[f];
  const int tid = threadIdx.x;
  const L ln(S, table, r);
  L::fill_table(table, a.tw);
  constexpr size_t plane = (size_t)N * N;
  constexpr float inv_n2 = 1.0f / ((float)N * (float)N);
  const int ny = (r * H + ln.y + N / 2) % N, rpix = ny * N + ln.rt;

  // What the cluster reads after the first mode's rows, fetched into L2 now (192² 1.060 -> 0.936 us
  // per frame, 256² x 2 2.466 -> 2.406).
  for (int m = 0; m < K; ++m) {
    const size_t m0 = ((size_t)slot * K + m) * plane;
    if (m > 0) {
      const size_t row = m0 + (size_t)ny * N;
      ln.prefetch_row(a.g + row);
      if (a.probe_stride) {
        ln.prefetch_row(a.probe + row);
        ln.prefetch_row(a.d_probe + row);
      }
    }
    L::prefetch_columns(a.psi + m0 + r * H);
  }
  L::prefetch_columns(a.iobs + (size_t)f * plane + r * H);

  // The b-term of den, Σ_pix 2·d·2·Re(p̄o·B)/N², by Parseval in the exit plane:
  // 2·Re Σ_x conj(g)·b with g = IDFT(2d·po)/N² the gradient pass's field (0 where masked).
  double gb = 0.0;
  float2 v[E];
#pragma unroll 1
  for (int m = 0, om = 0, pm = 0; m < K; ++m) {
    // Exit-plane rows of a; b and its product with g on the way.
    const size_t pi = (size_t)slot * a.probe_stride + pm * plane + rpix;
    const size_t oi = ((size_t)om * a.nyo + corner.x + ny) * a.nxo + corner.y + ln.rt;
    const float2 *p = a.probe + pi, *dp = a.d_probe + pi, *o = a.object + oi, *dob = a.d_obj + oi;
    const float2 *q = a.quad + rpix, *g = a.g + ((size_t)slot * K + m) * plane + rpix;
#pragma unroll
    for (int i = 0; i < E; ++i) {
      const int x = N2 * ((i + E / 2) % E);
      const float2 dpv = dp[x], dov = dob[x], qv = q[x];
      v[i] = cmul(cadd(cmul(p[x], dov), cmul(dpv, o[x])), qv);
      const float2 b = cmul(cmul(dpv, dov), qv), gv = g[x];
      gb += (double)gv.x * b.x + (double)gv.y * b.y;
    }
    if (m == 0) __syncthreads();  // the twiddle table
    ln.rows_forward(v, m);
    if (++pm == a.nprobe) {
      pm = 0;
      ++om;
    }
  }
  L::publish();
  // Columns kx = r·H + c, elements ky = N2·i + t; po as the gradient pass kept it.
  const int cpix = ln.t * N + r * H + ln.c;
  float calc[E], rr[E], ss[E];
#pragma unroll
  for (int i = 0; i < E; ++i) calc[i] = rr[i] = ss[i] = 0.f;
#pragma unroll 1
  for (int m = 0; m < K; ++m) {
    ln.columns_forward(v, m);
    const float2* po = a.psi + ((size_t)slot * K + m) * plane + cpix;
#pragma unroll
    for (int i = 0; i < E; ++i) {
      const float2 w = po[i * N2 * N];
      calc[i] += cnorm2(w) * inv_n2;
      rr[i] += (w.x * v[i].x + w.y * v[i].y) * inv_n2;
      ss[i] += cnorm2(v[i]) * inv_n2;
    }
  }
  const float* iobs = a.iobs + (size_t)f * plane + cpix;
  double s4[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
  for (int i = 0; i < E; ++i) {
    const float yo = iobs[i * N2 * N];
    if (yo < 0.f) continue;
    const double c = fmax((double)calc[i], 1e-32);
    const double d = 1.0 - (double)yo / c;
    s4[0] -= 2.0 * rr[i] * d;
    const double t = 2.0 * rr[i] / c;
    s4[1] += 2.0 * ss[i] * d + (double)yo * t * t;
  }
  s4[1] += 2.0 * gb;
  block_sum<T>(s4, 2, red);
  csync<C>(cluster);
  if (r == 0 && tid == 0) {
    double num = 0.0, den = 0.0;
    for (int q = 0; q < C; ++q) {
      const double* rq = C > 1 ? cluster.map_shared_rank(red, q) : red;
      num += rq[0];
      den += rq[1];
    }
    a.out[slot * 2] = num;
    a.out[slot * 2 + 1] = den;
  }
  csync<C>(cluster);
}

// Per block, in double: mode 0 Σ Re(conj(g)·(g − h)) and Σ |h|² (Polak–Ribière);
// mode 1 Σ |g| (the modulus sum of scale_obj_probe); mode 2 Σ Re(conj(g)·h) (BH's ⟨g, D⟩).
// Partial sums [block][2].
static __global__ void __launch_bounds__(256) array_sums_kernel(const float2* g, const float2* h,
                                                         size_t n, int mode, double* partial) {
  __shared__ double sh[16];
  double s0 = 0.0, s1 = 0.0;
  for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (size_t)gridDim.x * 256) {
    const float2 a = g[i];
    if (mode == 0) {
      const float2 b = h[i];
      s0 += (double)a.x * ((double)a.x - b.x) + (double)a.y * ((double)a.y - b.y);
      s1 += (double)b.x * b.x + (double)b.y * b.y;
    } else if (mode == 2) {
      const float2 b = h[i];
      s0 += (double)a.x * b.x + (double)a.y * b.y;
    } else {
      s0 += sqrt((double)a.x * a.x + (double)a.y * a.y);
    }
  }
  s0 = warp_sum(s0);
  s1 = warp_sum(s1);
  if (threadIdx.x % 32 == 0) {
    sh[threadIdx.x / 32] = s0;
    sh[8 + threadIdx.x / 32] = s1;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a0 = 0.0, a1 = 0.0;
    for (int w = 0; w < 8; ++w) {
      a0 += sh[w];
      a1 += sh[8 + w];
    }
    partial[blockIdx.x * 2] = a0;
    partial[blockIdx.x * 2 + 1] = a1;
  }
}

// d = beta·d − g.
static __global__ void cg_direction_kernel(float2* d, const float2* g, float beta, size_t n) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float2 a = d[i], b = g[i];
  d[i] = make_float2(a.x * beta - b.x, a.y * beta - b.y);
}

// x += gamma·d (gamma in double, applied in float).
static __global__ void axpy_kernel(float2* x, const float2* d, float gamma, size_t n) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  x[i] = cadd(x[i], cscale(d[i], gamma));
}

// x *= s.
static __global__ void scale_kernel(float2* x, float s, size_t n) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  x[i] = cscale(x[i], s);
}

// The centroid of the probe's far field for `zero_phase_ramp` (engine/ptycho.rs:1134-1152), in
// double: one block per line, thread k taking X[k] = Σ_j x[j]·e^{−2πi·jk/N} as the direct sum
// over a table of N twiddles in shared memory. K·N² outputs of N terms (33.5 M complex FMAs per
// direction at 256² x 2) take about 20 µs a direction, so no fast transform in double is worth
// its code here. The plane is not shifted before the transform: a shift changes
// the spectrum's phases and not its modulus.
PTYB_D double2 dft_line_term(const double2* x, const double2* w, int N) {
  double2 s = make_double2(0.0, 0.0);
  int i = 0;
  const int k = threadIdx.x;
#pragma unroll 4
  for (int j = 0; j < N; ++j) {
    const double2 a = x[j], b = w[i];
    s.x += a.x * b.x - a.y * b.y;
    s.y += a.x * b.y + a.y * b.x;
    i += k;
    if (i >= N) i -= N;
  }
  return s;
}

PTYB_D void dft_line_twiddles(double2* w, int N) {
  double sn, cs;
  sincospi(-2.0 * threadIdx.x / N, &sn, &cs);
  w[threadIdx.x] = make_double2(cs, sn);
}

// Block (y, m), N threads: rows[m][y][k].
static __global__ void __launch_bounds__(256) ramp_rows_kernel(const float2* probe, int N,
                                                               double2* rows) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* x = reinterpret_cast<double2*>(smem_raw);
  const size_t line = ((size_t)blockIdx.y * N + blockIdx.x) * N;
  const float2 v = probe[line + threadIdx.x];
  x[threadIdx.x] = make_double2(v.x, v.y);
  dft_line_twiddles(x + N, N);
  __syncthreads();
  rows[line + threadIdx.x] = dft_line_term(x, x + N, N);
}

// Block (kx, m), N threads: with v(ky) = |F(ky, kx)|², Σ v, Σ v·iy and Σ v·ix over the column at
// the natural indices iy = (ky + N/2) % N, ix, into sums[m·N + kx][3].
static __global__ void __launch_bounds__(256) ramp_columns_kernel(const double2* rows, int N,
                                                                  double* sums) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double red[2][8];
  double2* x = reinterpret_cast<double2*>(smem_raw);
  const int kx = blockIdx.x, t = threadIdx.x;
  x[t] = rows[((size_t)blockIdx.y * N + t) * N + kx];
  dft_line_twiddles(x + N, N);
  __syncthreads();
  const double2 f = dft_line_term(x, x + N, N);
  const double v = f.x * f.x + f.y * f.y;
  const double s0 = warp_sum(v), s1 = warp_sum(v * (double)((t + N / 2) % N));
  if (t % 32 == 0) {
    red[0][t / 32] = s0;
    red[1][t / 32] = s1;
  }
  __syncthreads();
  if (t == 0) {
    double a = 0.0, b = 0.0;
    for (int w = 0; w < N / 32; ++w) {
      a += red[0][w];
      b += red[1][w];
    }
    double* out = sums + ((size_t)blockIdx.y * N + kx) * 3;
    out[0] = a;
    out[1] = b;
    out[2] = a * (double)((kx + N / 2) % N);
  }
}

// shift = centroid − N/2 along y and x from the columns' sums, one warp, fixed order.
static __global__ void __launch_bounds__(32) ramp_centroid_kernel(const double* sums, int n,
                                                                  int N, double* shift) {
  double s[3] = {0.0, 0.0, 0.0};
  for (int i = threadIdx.x; i < n; i += 32)
    for (int k = 0; k < 3; ++k) s[k] += sums[(size_t)i * 3 + k];
  for (int k = 0; k < 3; ++k) s[k] = warp_sum(s[k]);
  if (threadIdx.x == 0) {
    shift[0] = s[1] / s[0] - (double)(N / 2);
    shift[1] = s[2] / s[0] - (double)(N / 2);
  }
}

// x[k][y][x] *= exp(i·2π·sign·(dy·(y − hy)/sy + dx·(x − hx)/sx)) for every plane k
// (the ramps of `zero_phase_ramp`, engine/ptycho.rs:1153-1170) with (dy, dx) = shift, phase in
// double.
static __global__ void ramp_kernel(float2* x, int nplanes, int ny, int nx, const double* shift,
                                   double sy, double sx, double sign) {
  const double dy = shift[0], dx = shift[1];
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t n = (size_t)nplanes * ny * nx;
  if (i >= n) return;
  const int yy = (int)((i / nx) % ny), xx = (int)(i % nx);
  const double ph = sign * 2.0 * 3.14159265358979323846 *
                    (dy * (yy - ny / 2) / sy + dx * (xx - nx / 2) / sx);
  double sn, cs;
  sincos(ph, &sn, &cs);
  const float2 v = x[i];
  x[i] = make_float2((float)(v.x * cs - v.y * sn), (float)(v.x * sn + v.y * cs));
}

}  // namespace ptyb
