// The per-frame pass of the reconstruction: exit waves → 2-D FFT → detector-plane residual →
// inverse 2-D FFT → exit-wave update, for every probe mode of one diffraction frame, on one
// thread-block cluster whose distributed shared memory holds the frame's K planes.
//
// Cluster of C CTAs, CTA rank r owning H = N/C rows, then columns (plane.cuh): each thread loads
// its elements of a row into registers and forms the exit wave there, the row FFTs leave their
// spectra in shared memory, the transpose reads them from the other CTAs' shared memory straight
// into the column FFTs' registers, and the per-pixel projection (which needs every mode at a
// pixel: the modes but the last wait in shared memory) runs on the column in registers between
// the forward and the inverse FFT; the way back is the same. Nothing but the object window, the
// probes, the counts and the output touches global memory.
//
// What bounds it: latency. The exit waves' loads, the exchanges and the cluster barriers around
// the transposes leave 34 % of the issue slots busy in the 256² x 2 gradient (24 warps per SM
// allowed, 20 resident on average) and 35 % in the carry pass (16 and 14); DRAM moves 1.8 and 1.0
// TB/s. Against the form it replaces (planes in shared memory for every step: 13 reads and 12
// writes of each element per pass instead of 6.5 and 6.5, four global loads in flight instead of
// 16) the passes take, per frame on one B200: gradient 256² x 2 3.53 -> 1.86 us, carry 4.17 ->
// 2.19, LSQML 128² x 3 forward 0.77 -> 0.48 and backward 1.06 -> 0.62, amplitude 96² x 2 0.83 ->
// 0.48, gradient 192² 1.53 -> 0.61, rPIE 64² 36 -> 12.8 us per batch of 100.
//
// Reference operators followed (physwkim/ptyrs): exit wave `obj_probe_to_psi`
// (engine/ops.rs:47-71), unitary FFT (engine/fft.rs:155-234), the rPIE modulus
// (engine/ptycho.rs:928-945), the Poisson gradient (engine/ops.rs:161-195), the LSQML residual
// (engine/lsqml.rs:155-170), the LLK sums (engine/ops.rs:119-154) and PyNX's AP, DM and RAAR
// mixes of carried exit waves around the magnitude projection (engine/ptycho.rs:609-730).
#pragma once
#include <cooperative_groups.h>

#include "common.cuh"
#include "fft.cuh"
#include "plane.cuh"

namespace cg = cooperative_groups;

namespace ptyb {

enum FrameMode : int {
  kRpie = 0,       // rPIE modulus; out = Δ = ψ' − ψ
  kLsqmlFused = 1, // LSQML residual from a per-frame a_far; out = χ = ψ' − ψ
  kMlGrad = 2,     // Poisson gradient 2(1 − I/Ĩ), masked 0; out = ψ'
  kLlk = 3,        // forward only; per-frame LLK sums
  kStore = 4,      // forward only; detector field and Σ_modes |Ψ|² to global
  kFromStore = 5,  // detector field from global; LSQML residual; out = χ
  kProject = 6,    // magnitude projection √I/max(√Ĩ, 1e-12), masked kept; out = ψ' − ψ
  kProjectKept = 7,// from the detector field a kMlGrad pass kept (psi_out): out = ψ' − ψ as
                   // the inverse of Ψ' − Ψ
  kCarry = 8,      // AP / DM / RAAR: projection of a mix of P·O·q and the carried waves
  kBhGrad = 9,     // BH's amplitude gradient 2(1 − √I/A), A = √Ĩ + 1e-8, masked 0; out = ψ'
                   // (kMlGrad's pass otherwise: the detector field kept in psi_out)
};

// kCostBh: BH's amplitude gradient 2(1 − √I/A), A = √Ĩ + 1e-8 (the multislice gradient pass)
enum Cost : int { kCostPoisson = 0, kCostAmplitude = 1, kCostBh = 2 };

struct FrameArgs {
  const float2* object;  // [nobj][nyo][nxo]
  const float2* probe;   // [nprobe][N][N] natural layout
  const float2* quad;    // [N][N] natural: the plane phase the exit transform starts with
  const float2* tw;      // [N]: e^{-2πi·t/N}
  const float* iobs;     // [nframe][N][N] FFT-shifted layout; < 0 masked
  const int* frames;     // frame of each slot of the launch
  const int2* corners;   // [nframe] window corner (x = oy, y = ox)
  float2* out;           // [slot][K][N][N] natural layout
  float2* field;         // [slot][C][K][E][T] detector field, thread by thread: written by the
                         // pass before and read back by the same threads
  float* icalc;          // [slot][N][N] Σ_modes |Ψ|², detector layout
  float* omax;           // [slot] max |O|² over the window (object mode 0)
  double* llk;           // [slot][4] Poisson, Gaussian, Euclidian, photons
  const float* a_far;    // [slot] LSQML far-field step (kLsqmlFused)
  // LSQML Poisson far-field step, PtychoShelves' xi solver in two passes
  // (engine/lsqml.rs:133-150): kStore runs pass 1 from `a_prev` (by frame when
  // `a_prev_by_frame`), kFromStore pass 2 from `a_mid`; each writes its result to `a_out`.
  const float* a_prev;
  const float* a_mid;
  float* a_out;
  int a_prev_by_frame, nslot;
  int nyo, nxo, nprobe, nobj, cost;
  // Elements between consecutive slots' probes: 0 for the shared probe, K·N·N for the
  // per-frame (moved) probes of the position model.
  int probe_stride;
  // kMlGrad, optional: the detector field Ψ = DFT(P·O·q) of every mode kept for the line
  // search and the magnitude projection, [slot][K][ky][kx]; kProjectKept reads it back.
  float2* psi_out;
  // kCarry (AP, DM, RAAR; engine/ptycho.rs:609-730): the carried exit waves `carry` and RAAR's
  // iterate `iter` of the launch's frames, [slot][K][N][N] natural layout. The projection's
  // input is S = c_po·PO + c_psi·carry + c_it·iter (iter ← S when `iter` is set); the carried
  // waves become Π(S) + c_refl·(PO − S). Terms whose coefficient is 0 are not read. With `llk`
  // set, the pass also writes the per-frame LLK sums of the field it projects.
  float2* carry;
  float2* iter;
  float c_po, c_psi, c_it, c_refl;
};

template <int N, int C>
struct FrameShape {
  static constexpr int H = N / C;           // rows (then columns) per CTA
  static constexpr int T = H * N / 16;      // threads: 16 transposed values each per mode
  static constexpr int L = N;               // line stride in float2 (lines are swizzled)
  static constexpr int G = LineShape<N>::N2; // threads per line FFT
  static constexpr int E = H * N / T;       // = 16
};

template <int N, int C>
__host__ __device__ constexpr size_t frame_smem_bytes(int K) {
  return (size_t)K * FrameShape<N, C>::H * FrameShape<N, C>::L * sizeof(float2) +
         N * sizeof(float2) + 160 * sizeof(double);
}

// Barrier over the cluster (a plain block barrier when the cluster is one CTA).
template <int C>
PTYB_D void csync(cg::cluster_group& cluster) {
  if (C > 1)
    cluster.sync();
  else
    __syncthreads();
}

// Every local line through a forward (DIR = -1) or inverse (+1) line FFT; the block barrier at
// the end publishes every line to every thread of the CTA.
template <int N, int C, int DIR>
PTYB_D void all_lines(float2* S, int nlines, const LineTwiddles<N>& tw) {
  using F = FrameShape<N, C>;
  const int g = threadIdx.x / F::G, t = threadIdx.x % F::G;
  for (int line = g; line < nlines; line += F::T / F::G)
    line_fft<N, DIR>(S + line * F::L, t, tw, swz(line));
  __syncthreads();
}

// Cluster-wide transpose of the K planes: rows → columns or back (the same map). Value
// (line m·H + c, element j) of CTA r comes from CTA j/H, line m·H + j%H, element r·H + c.
template <int N, int C>
PTYB_D void transpose(float2* S, int K, cg::cluster_group& cluster) {
  using F = FrameShape<N, C>;
  const int r = C > 1 ? (int)cluster.block_rank() : 0;
  csync<C>(cluster);
  for (int m = 0; m < K; ++m) {
    float2 v[F::E];
#pragma unroll
    for (int i = 0; i < F::E; ++i) {
      const int e = threadIdx.x + i * F::T;
      const int c = e % F::H, j = e / F::H;
      const float2* src = C > 1 ? cluster.map_shared_rank(S, j / F::H) : S;
      const int sl = m * F::H + j % F::H;
      v[i] = src[sl * F::L + ((r * F::H + c) ^ swz(sl))];
    }
    csync<C>(cluster);
#pragma unroll
    for (int i = 0; i < F::E; ++i) {
      const int e = threadIdx.x + i * F::T;
      const int c = e % F::H, j = e / F::H;
      const int dl = m * F::H + c;
      S[dl * F::L + (j ^ swz(dl))] = v[i];
    }
  }
  __syncthreads();
}

// Block-wide sums of n ≤ 4 doubles into red[0..n) of thread 0 (others undefined).
template <int T>
PTYB_D void block_sum(double (&v)[4], int n, double* red) {
  for (int k = 0; k < n; ++k) v[k] = warp_sum(v[k]);
  __syncthreads();
  const int w = threadIdx.x / 32, lane = threadIdx.x % 32;
  double* part = red + 8;  // [T/32][4]
  if (lane == 0)
    for (int k = 0; k < n; ++k) part[w * 4 + k] = v[k];
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 0; k < n; ++k) {
      double s = 0.0;
      for (int q = 0; q < T / 32; ++q) s += part[q * 4 + k];
      red[k] = s;
    }
  }
  __syncthreads();
}

// Mean of the launch's far-field steps, summed by warp 0 in a fixed order (lane-strided
// partial sums, then a fixed butterfly), so every CTA gets the same value; broadcast through
// `slot` in shared memory (block barrier inside).
PTYB_D double batch_mean(const float* v, const int* frames, int by_frame, int nslot,
                         double* slot) {
  if (threadIdx.x < 32) {
    double s = 0.0;
    for (int i = threadIdx.x; i < nslot; i += 32) s += v[by_frame ? frames[i] : i];
    s = warp_sum(s);
    if (threadIdx.x == 0) *slot = s / nslot;
  }
  __syncthreads();
  return *slot;
}

// Cluster-wide sums of two doubles over CTAs of T threads (every CTA gets the totals, added in
// rank order).
template <int T, int C>
PTYB_D void cluster_sum2(double& x, double& y, double* red, cg::cluster_group& cluster) {
  double v[4] = {x, y, 0.0, 0.0};
  block_sum<T>(v, 2, red);
  csync<C>(cluster);
  double sx = 0.0, sy = 0.0;
  for (int q = 0; q < C; ++q) {
    const double* rq = C > 1 ? cluster.map_shared_rank(red, q) : red;
    sx += rq[0];
    sy += rq[1];
  }
  csync<C>(cluster);
  x = sx;
  y = sy;
}

// Cluster-wide sums of four doubles, every thread getting them (rank order, as cluster_sum2).
template <int T, int C>
PTYB_D void cluster_sum4(double (&v)[4], double* red, cg::cluster_group& cluster) {
  block_sum<T>(v, 4, red);
  csync<C>(cluster);
  double t[4] = {0.0, 0.0, 0.0, 0.0};
  for (int q = 0; q < C; ++q) {
    const double* rq = C > 1 ? cluster.map_shared_rank(red, q) : red;
#pragma unroll
    for (int k = 0; k < 4; ++k) t[k] += rq[k];
  }
  csync<C>(cluster);
#pragma unroll
  for (int k = 0; k < 4; ++k) v[k] = t[k];
}

// The projection's input S = c_po·po + c_psi·carry + c_it·iter (kCarry) in place of po at a
// thread's row-mapped elements, `base` the offset of the first one in the carried planes; the
// prologue (`store`) also writes it to RAAR's iterate.
template <int N, int C>
PTYB_D void carry_mix(const FrameArgs& a, float2 (&v)[PlaneShape<N, C>::E], size_t base,
                      bool store) {
  using F = PlaneShape<N, C>;
  auto xof = [](int i) { return F::G * ((i + F::E / 2) % F::E); };
#pragma unroll
  for (int i = 0; i < F::E; ++i) v[i] = cscale(v[i], a.c_po);
  if (a.c_psi != 0.f) {
    const float2* src = a.carry + base;
#pragma unroll
    for (int i = 0; i < F::E; ++i) v[i] = cadd(v[i], cscale(src[xof(i)], a.c_psi));
  }
  if (a.c_it != 0.f) {
    const float2* src = a.iter + base;
#pragma unroll
    for (int i = 0; i < F::E; ++i) v[i] = cadd(v[i], cscale(src[xof(i)], a.c_it));
  }
  if (store && a.iter) {
    float2* dst = a.iter + base;
#pragma unroll
    for (int i = 0; i < F::E; ++i) dst[xof(i)] = v[i];
  }
}

template <int N, int C, int MODE>
__global__ void __launch_bounds__(PlaneShape<N, C>::T,
                                  plane_min_blocks<N, C>(MODE == kMlGrad || MODE == kBhGrad ||
                                                         MODE == kProjectKept))
    frame_kernel(FrameArgs a) {
  using L = Lines<N, C>;
  constexpr int H = L::H, T = L::T, E = L::N1, N2 = L::N2;
  extern __shared__ __align__(128) unsigned char plane_smem[];
  const int K = a.nprobe * a.nobj;
  float2* S = reinterpret_cast<float2*>(plane_smem);
  float2* table = S + (size_t)K * H * N;
  double* red = reinterpret_cast<double*>(table + N);  // 8 results + [T/32 ≤ 32][4] partials
  cg::cluster_group cluster = cg::this_cluster();
  const int r = C > 1 ? (int)cluster.block_rank() : 0;
  const int slot = blockIdx.x / C;
  const int f = a.frames[slot];
  const int2 corner = a.corners[f];
  const int tid = threadIdx.x;
  const L ln(S, table, r);
  L::fill_table(table, a.tw);
  constexpr size_t plane = (size_t)N * N;
  constexpr bool from_field = MODE == kFromStore || MODE == kProjectKept;

  // Row-mapped: the row's natural index and its first element; element i of the thread is the
  // shifted column N2·i + rt, natural column N2·((i + E/2) % E) + rt.
  const int ny = (r * H + ln.y + N / 2) % N;
  const int rpix = ny * N + ln.rt;
  auto xof = [](int i) { return N2 * ((i + E / 2) % E); };
  // O·q of the row under object mode om; `omax` takes the largest |O|².
  auto window = [&](float2 (&oq)[E], int om, float& omax) {
    const float2* o = a.object + ((size_t)om * a.nyo + corner.x + ny) * a.nxo + corner.y + ln.rt;
    const float2* q = a.quad + rpix;
#pragma unroll
    for (int i = 0; i < E; ++i) oq[i] = o[xof(i)];
#pragma unroll
    for (int i = 0; i < E; ++i) {
      if (MODE == kRpie) omax = fmaxf(omax, cnorm2(oq[i]));
      oq[i] = cmul_rn(oq[i], q[xof(i)]);
    }
  };

  // What the cluster reads after the first row transforms, fetched into L2 now (256² x 2 gradient
  // 1.883 -> 1.854 us per frame, carry 2.214 -> 2.192, rPIE 128² x 2 0.545 -> 0.518; at 64² the
  // addresses cost more than the loads' latency).
  if (!from_field && N > 64) {
    L::prefetch_columns(a.iobs + (size_t)f * plane + r * H);
    for (int m = 1; m < K; ++m) {
      const size_t row = ((size_t)slot * K + m) * plane + (size_t)ny * N;
      if (a.probe_stride) ln.prefetch_row(a.probe + row);
      if (MODE == kCarry && a.c_psi != 0.f) ln.prefetch_row(a.carry + row);
      if (MODE == kCarry && a.c_it != 0.f) ln.prefetch_row(a.iter + row);
    }
  }
  float2 v[E];
  if (!from_field) {
    // Exit waves ψ = P·O·q of the rows, mode by mode; (P·O)·q as P·(O·q): the reference's
    // product up to rounding.
    float2 oq[E];
    float omax = 0.f;
#pragma unroll 1
    for (int m = 0, om = 0, pm = 0; m < K; ++m) {
      if (pm == 0) window(oq, om, omax);
      const float2* p = a.probe + (size_t)slot * a.probe_stride + pm * plane + rpix;
#pragma unroll
      for (int i = 0; i < E; ++i) v[i] = p[xof(i)];
#pragma unroll
      for (int i = 0; i < E; ++i) v[i] = cmul_rn(v[i], oq[i]);
      if (MODE == kCarry)
        carry_mix<N, C>(a, v, ((size_t)slot * K + m) * plane + rpix, true);
      if (m == 0) __syncthreads();  // the twiddle table
      ln.rows_forward(v, m);
      if (++pm == a.nprobe) {
        pm = 0;
        ++om;
      }
    }
    if (MODE == kRpie) {
      // max |O|² over the window: block max, then across the cluster in rank order.
      omax = warp_max(omax);
      float* fred = reinterpret_cast<float*>(red + 8);
      if (tid % 32 == 0) fred[tid / 32] = omax;
      __syncthreads();
      if (tid == 0) {
        float mx = 0.f;
        for (int q = 0; q < T / 32; ++q) mx = fmaxf(mx, fred[q]);
        reinterpret_cast<float*>(red)[0] = mx;
      }
    }
    L::publish();
    if (MODE == kRpie && r == 0 && tid == 0) {
      float mx = 0.f;
      for (int q = 0; q < C; ++q)
        mx = fmaxf(mx, *reinterpret_cast<float*>(C > 1 ? cluster.map_shared_rank(red, q) : red));
      a.omax[slot] = mx;
    }
  }

  // Detector plane, column-mapped: element i is the pixel (ky, kx) = (N2·i + t, r·H + c).
  // Unnormalised transforms: Ψ_ortho = Ψ/N, and the inverse of the update takes a 1/N more.
  constexpr float inv_n2 = 1.0f / ((float)N * (float)N);
  const int kx = r * H + ln.c, dpix = ln.t * N + kx;
  constexpr int kRow = N2 * N;  // pixels between a thread's elements
  float yo[E], ic[E];
  {
    const float* iobs = a.iobs + (size_t)f * plane + dpix;
#pragma unroll
    for (int i = 0; i < E; ++i) {
      yo[i] = iobs[i * kRow];
      ic[i] = 0.f;
    }
  }
  // The field of a kStore pass, by the thread that reads it back.
  float2* field = a.field + ((size_t)slot * C + r) * K * H * N + tid;
#pragma unroll 1
  for (int m = 0; m < K; ++m) {
    if (MODE == kFromStore) {
#pragma unroll
      for (int i = 0; i < E; ++i) v[i] = field[(size_t)m * H * N + i * T];
    } else if (MODE == kProjectKept) {
      const float2* src = a.psi_out + ((size_t)slot * K + m) * plane + dpix;
#pragma unroll
      for (int i = 0; i < E; ++i) v[i] = src[i * kRow];
    } else {
      ln.columns_forward(v, m);
    }
    if ((MODE == kMlGrad || MODE == kBhGrad) && a.psi_out) {
      float2* dst = a.psi_out + ((size_t)slot * K + m) * plane + dpix;
#pragma unroll
      for (int i = 0; i < E; ++i) dst[i * kRow] = v[i];
    }
    if (MODE == kStore) {
#pragma unroll
      for (int i = 0; i < E; ++i) field[(size_t)m * H * N + i * T] = v[i];
    }
#pragma unroll
    for (int i = 0; i < E; ++i) ic[i] += fmaf(v[i].x, v[i].x, v[i].y * v[i].y);
    // the last mode stays in registers
    if (MODE != kStore && MODE != kLlk && m + 1 < K) ln.stash(v, m);
  }
  if (from_field) __syncthreads();  // the twiddle table
#pragma unroll
  for (int i = 0; i < E; ++i) ic[i] *= inv_n2;
  float afar = MODE == kLsqmlFused ? a.a_far[slot] : 0.f;
  if ((MODE == kStore || MODE == kFromStore) && a.cost == kCostPoisson && a.a_out) {
    // One pass of the Poisson xi solver over this frame: with prev the batch mean of the
    // previous pass, a = clip(prev/2 + Σ xi·(Ĩ − I/(1 − prev·xi)) / Σ xi²·Ĩ / 2, 0, 1).
    const double prev = MODE == kStore
                            ? batch_mean(a.a_prev, a.frames, a.a_prev_by_frame, a.nslot, red + 7)
                            : batch_mean(a.a_mid, a.frames, 0, a.nslot, red + 7);
    double num = 0.0, den = 0.0;
#pragma unroll
    for (int i = 0; i < E; ++i) {
      if (yo[i] < 0.f) continue;
      const double yp = (double)ic[i], yt = yo[i];
      const double xi = 1.0 - yt / (yp + 1e-5);
      num += xi * (yp - yt / (1.0 - prev * xi));
      den += xi * xi * yp;
    }
    cluster_sum2<T, C>(num, den, red, cluster);
    const double ratio = den > 0.0 ? num / den : 0.0;
    afar = (float)fmin(fmax(0.5 * prev + 0.5 * ratio, 0.0), 1.0);
    if (r == 0 && tid == 0) a.a_out[slot] = afar;
  }
  if (MODE == kStore) {
    if (a.icalc) {
#pragma unroll
      for (int i = 0; i < E; ++i) a.icalc[(size_t)slot * plane + dpix + i * kRow] = ic[i];
    }
    return;
  }
  if (MODE == kLlk || (MODE == kCarry && a.llk)) {
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int i = 0; i < E; ++i) {
      if (yo[i] < 0.f) continue;
      const double y = yo[i], c = ic[i];
      acc[0] += yo[i] > 0.f ? c - y + y * log(y / c) : c;
      const double dg = y - c;
      acc[1] += dg * dg / (y + 1.0);
      const double de = sqrt(y) - sqrt(c);
      acc[2] += 4.0 * de * de;
      acc[3] += c;
    }
    block_sum<T>(acc, 4, red);
    csync<C>(cluster);
    if (r == 0 && tid == 0) {
      for (int k = 0; k < 4; ++k) {
        double s = 0.0;
        for (int q = 0; q < C; ++q) s += (C > 1 ? cluster.map_shared_rank(red, q) : red)[k];
        a.llk[(size_t)slot * 4 + k] = s;
      }
    }
    csync<C>(cluster);
    if (MODE == kLlk) return;
  }
  // The factor of every mode at the pixel, into ic.
#pragma unroll
  for (int i = 0; i < E; ++i) {
    const float y = yo[i], c = ic[i];
    const bool masked = y < 0.f;
    float fac;
    if (MODE == kRpie) {
      fac = masked ? 1.f : sqrtf(y + 1e-7f) / (sqrtf(c) + 1e-7f);
    } else if (MODE == kProjectKept) {
      // ApplyAmplitude (engine/ops.rs:83-107) minus the identity: the kept field Ψ = DFT(ψ)
      // goes to ΔΨ = Ψ' − Ψ, whose inverse is the change ψ' − ψ itself (no model re-read)
      fac = masked ? 0.f : sqrtf(y) / fmaxf(sqrtf(c), 1e-12f) - 1.f;
    } else if (MODE == kProject || MODE == kCarry) {
      // ApplyAmplitude (engine/ops.rs:83-107)
      fac = masked ? 1.f : sqrtf(y) / fmaxf(sqrtf(c), 1e-12f);
    } else if (MODE == kMlGrad) {
      fac = masked ? 0.f : 2.f * (1.f - y / fmaxf(c, 1e-12f));
    } else if (MODE == kBhGrad) {
      // BH's residual (engine/bh.rs:255-265)
      fac = masked ? 0.f : 2.f * (1.f - sqrtf(y) / (sqrtf(c) + 1e-8f));
    } else {
      float cres = 0.f;
      if (!masked)
        cres = a.cost == kCostPoisson ? 1.f - y / (c + 1e-6f)
                                      : 2.f * (1.f - sqrtf(fmaxf(y, 0.f)) / (sqrtf(c) + 1e-9f));
      fac = 1.f - afar * cres;
    }
    ic[i] = fac * inv_n2;
  }
#pragma unroll 1
  for (int m = K - 1; m >= 0; --m) {
    if (m + 1 < K) ln.unstash(v, m);
#pragma unroll
    for (int i = 0; i < E; ++i) v[i] = cscale_rn(v[i], ic[i]);
    ln.columns_inverse(v, m);
  }
  L::publish();

  // Rows again, row-mapped: ψ' − ψ (or ψ'), natural layout.
  constexpr bool subtract = MODE != kMlGrad && MODE != kBhGrad && MODE != kProjectKept;
  float2 oq[E];
  float unused = 0.f;
#pragma unroll 1
  for (int m = 0, om = 0, pm = 0; m < K; ++m) {
    const size_t gi = ((size_t)slot * K + m) * plane + rpix;
    ln.rows_inverse(v, m);
    if (MODE == kCarry) {
      // carried waves ← Π(S) + c_refl·(PO − S), in place (this thread read these pixels above)
      if (a.c_refl != 0.f) {
        if (pm == 0) window(oq, om, unused);
        const float2* p = a.probe + (size_t)slot * a.probe_stride + pm * plane + rpix;
        float2 po[E], x[E];
#pragma unroll
        for (int i = 0; i < E; ++i) x[i] = po[i] = cmul_rn(p[xof(i)], oq[i]);
        carry_mix<N, C>(a, x, gi, false);
#pragma unroll
        for (int i = 0; i < E; ++i) v[i] = cadd(v[i], cscale(csub(po[i], x[i]), a.c_refl));
      }
      float2* dst = a.carry + gi;
#pragma unroll
      for (int i = 0; i < E; ++i) dst[xof(i)] = v[i];
    } else {
      if (subtract) {
        if (pm == 0) window(oq, om, unused);
        const float2* p = a.probe + (size_t)slot * a.probe_stride + pm * plane + rpix;
#pragma unroll
        for (int i = 0; i < E; ++i) v[i] = csub(v[i], cmul_rn(p[xof(i)], oq[i]));
      }
      float2* dst = a.out + gi;
#pragma unroll
      for (int i = 0; i < E; ++i) dst[xof(i)] = v[i];
    }
    if (++pm == a.nprobe) {
      pm = 0;
      ++om;
    }
  }
}

}  // namespace ptyb
