// 2-D transforms of planes that one thread-block cluster holds in shared memory, with the line
// in registers between the memory steps.
//
// A cluster of C CTAs, CTA r owning H = N/C lines of every plane: rows r·H .. r·H+H-1, then
// columns r·H .. r·H+H-1. A line of N = N1·N2 elements belongs to N2 threads; thread t holds the
// N1 elements N2·i + t in registers before a line FFT and after it, so what happens between two
// FFTs (loading, the detector step, storing) is register work, and a line FFT touches shared
// memory once, for the exchange between its N1-point and N2-point stages.
//
// Threads map to lines in two ways. Row-mapped, t runs fastest: N2 neighbouring threads hold one
// row, so global accesses along rows coalesce and the row FFT's exchange stays in a warp.
// Column-mapped, the line runs fastest: the threads of a warp hold neighbouring columns of the
// same rows, so the transpose reads 8·H contiguous bytes of another CTA's row through
// distributed shared memory, and the columns' global accesses ([ky][kx]) coalesce; the exchange
// then crosses warps, behind block barriers. A row inverse FFT pulls its lines column-mapped and
// leaves them row-mapped: the exchange changes the map.
//
// A plane's element e of line l sits at l·N + (e ^ swz(l)); with N2·i and t on disjoint bits
// every access is one base register XOR a constant plus a constant, and the half-warps' accesses
// hit 16 distinct 8-byte banks in both maps (the exchange's rotation by k1 does it where the map
// changes).
#pragma once
#include "common.cuh"
#include "fft.cuh"

namespace ptyb {

template <int N, int C>
struct PlaneShape {
  static constexpr int H = N / C;             // rows (then columns) per CTA
  static constexpr int E = LineShape<N>::N1;  // elements of a line per thread
  static constexpr int G = LineShape<N>::N2;  // threads per line
  static constexpr int T = H * G;             // threads per CTA: one line each group
};

// CTAs per SM the plane kernels are compiled for: 512 threads (128 registers each) where a
// thread holds 16 elements, 1024 at side 64 (8 elements), two CTAs of 192 at 24 elements. A
// kernel that holds little beside its line (`light`) takes 768 threads of 80 registers at side
// 256: moves 0.906 -> 0.797 us per frame of 256² x 2, their spectra 0.998 -> 0.896, projection
// 1.211 -> 1.055, gradient 1.941 -> 1.871. Some spill a little there and gain all the same (bytes
// stored: gradient 76, own moves and moves back 60, spectra 40 and 56, projection 4, the other
// moves none). What holds more loses: line search 2.46 -> 3.25, carry pass 2.21 -> 2.69, at side
// 128 the LSQML passes 0.618 -> 0.757; at 128 registers they spill 20, 104 and 0 bytes.
template <int N, int C>
__host__ __device__ constexpr int plane_min_blocks(bool light = false) {
  return N == 64 ? 2
         : LineShape<N>::N1 == 24 ? 2
         : (light && N == 256 && PlaneShape<N, C>::T == 256 ? 768 : 512) / PlaneShape<N, C>::T;
}

PTYB_D float2 lds2(unsigned a) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a));
  return v;
}
PTYB_D void sts2(unsigned a, float2 v) {
  asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(v.x), "f"(v.y) : "memory");
}
// The same location in the shared memory of the cluster's CTA q, and a load from there.
PTYB_D unsigned at_rank(unsigned a, int q) {
  unsigned d;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(q));
  return d;
}
PTYB_D float2 ldc2(unsigned a) {
  float2 v;
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a));
  return v;
}
PTYB_D void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
PTYB_D void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// One thread's place in the CTA's planes and the line transforms from it.
template <int N, int C>
struct Lines {
  using F = PlaneShape<N, C>;
  static constexpr int N1 = LineShape<N>::N1, N2 = LineShape<N>::N2, P = N1 / N2;
  static constexpr int H = F::H, T = F::T;
  static constexpr unsigned kPlane = H * N * sizeof(float2);
  int t, c;    // column-mapped: offset in the line, line
  int rt, y;   // row-mapped
  unsigned own, xch;       // column-mapped: own elements, the exchange's reads
  unsigned row, rxch;      // row-mapped
  unsigned from;           // column-mapped: the transpose's source lines
  unsigned tw, rtw;        // twiddle table entries of t and rt

  // The constant parts of an element index e0 (a multiple of N2): low four bits XORed, rest added.
  static PTYB_HD constexpr unsigned lo(int e0) { return (unsigned)(e0 & 15) * 8u; }
  static PTYB_HD constexpr unsigned hi(int e0) { return (unsigned)(e0 & ~15) * 8u; }
  static PTYB_HD constexpr int bank(int l) { return ((l & 1) << 3) | ((l >> 1) & 7); }  // swz

  // `planes` (128-byte aligned) and the table of N twiddles in shared memory; rank r.
  PTYB_D Lines(const float2* planes, const float2* table, int r) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(planes);
    const unsigned w = (unsigned)__cvta_generic_to_shared(table);
    c = threadIdx.x % H;
    t = threadIdx.x / H;
    rt = threadIdx.x % N2;
    y = threadIdx.x / N2;
    own = s + c * (N * 8) + (unsigned)(t ^ swz(c)) * 8u;
    xch = s + c * (N * 8) + (unsigned)((N2 * t) ^ swz(c)) * 8u;
    row = s + y * (N * 8) + (unsigned)(rt ^ swz(y)) * 8u;
    rxch = s + y * (N * 8) + (unsigned)((N2 * rt + rt) ^ swz(y)) * 8u;
    from = s + t * (N * 8) + (unsigned)((r * H + c) ^ swz(t)) * 8u;
    tw = w + t * 8;
    rtw = w + rt * 8;
  }

  // The twiddles ω_N^{t·k1} as [k1][t]; a block barrier must follow before the first FFT.
  static PTYB_D void fill_table(float2* table, const float2* tw_global) {
    for (int i = threadIdx.x; i < N; i += T) table[i] = tw_global[((i / N2) * (i % N2)) % N];
  }

  // Own elements to and from plane m (column-mapped); only this thread touches them.
  PTYB_D void stash(const float2 (&v)[N1], int m) const {
    const unsigned b = own + m * kPlane;
#pragma unroll
    for (int i = 0; i < N1; ++i) sts2((b ^ lo(N2 * i)) + hi(N2 * i), v[i]);
  }
  PTYB_D void unstash(float2 (&v)[N1], int m) const {
    const unsigned b = own + m * kPlane;
#pragma unroll
    for (int i = 0; i < N1; ++i) v[i] = lds2((b ^ lo(N2 * i)) + hi(N2 * i));
  }

  // First stage: the N1-point DFT over i and the twiddles of offset t.
  template <int DIR>
  static PTYB_D void stage1(float2 (&v)[N1], unsigned tw) {
    dft<N1, DIR>(v);
#pragma unroll
    for (int k1 = 1; k1 < N1; ++k1) {
      const float2 w = lds2(tw + k1 * N2 * 8);
      v[k1] = cmul_rn(DIR < 0 ? w : cconj(w), v[k1]);
    }
  }
  // Second stage on the exchanged values u[p·N2 + n2]: the natural elements N2·i + t.
  template <int DIR>
  static PTYB_D void stage2(float2 (&v)[N1]) {
    float2 o[N1];
#pragma unroll
    for (int p = 0; p < P; ++p) {
      float2 u[N2];
#pragma unroll
      for (int n2 = 0; n2 < N2; ++n2) u[n2] = v[p * N2 + n2];
      dft<N2, DIR>(u);
#pragma unroll
      for (int k2 = 0; k2 < N2; ++k2) o[p + P * k2] = u[k2];
    }
#pragma unroll
    for (int i = 0; i < N1; ++i) v[i] = o[i];
  }
  // The exchange's reads from `base` (xch or rxch of a plane).
  static PTYB_D void gather(float2 (&v)[N1], unsigned base) {
#pragma unroll
    for (int p = 0; p < P; ++p)
#pragma unroll
      for (int n2 = 0; n2 < N2; ++n2) v[p * N2 + n2] = lds2((base ^ (n2 * 8u)) + p * (N2 * N2 * 8));
  }
  // The exchange's writes rotated by k1, from `base` (own or row of a plane).
  static PTYB_D void scatter_rotated(const float2 (&v)[N1], unsigned base) {
#pragma unroll
    for (int k1 = 0; k1 < N1; ++k1)
      sts2((base ^ (lo(N2 * k1) ^ (unsigned)((k1 & (N2 - 1)) * 8))) + hi(N2 * k1), v[k1]);
  }

  // This thread's elements of line r·H + c across the other map's lines of plane m: element
  // N2·i + t from CTA (N2·i + t)/H.
  PTYB_D void pull(float2 (&v)[N1], int m) const {
    const unsigned b = from + m * kPlane;
#pragma unroll
    for (int i = 0; i < N1; ++i) {
      const int q = (N2 * i) / H, l = (N2 * i) % H;
      const unsigned a = b ^ (unsigned)(bank(l & 15) * 8);
      v[i] = C > 1 ? ldc2(at_rank(a, q) + l * (N * 8)) : lds2(a + l * (N * 8));
    }
  }

  // Fetches this CTA's part of a global plane [N][N] into L2 ahead of its use: the row of this
  // row-mapped thread (`row0` its first element), or the CTA's columns r·H .. of every ky
  // (`col0` the first of them), for elements of B bytes.
  template <typename V>
  PTYB_D void prefetch_row(const V* row0) const {
    constexpr int kLines = N * (int)sizeof(V) / 128;
    for (int l = rt; l < kLines; l += N2) prefetch(reinterpret_cast<const char*>(row0) + l * 128);
  }
  template <typename V>
  static PTYB_D void prefetch_columns(const V* col0) {
    constexpr int kSpan = H * (int)sizeof(V), kLines = (kSpan + 127) / 128;
    for (int i = threadIdx.x; i < N * kLines; i += T)
      prefetch(reinterpret_cast<const char*>(col0 + (size_t)(i / kLines) * N) + (i % kLines) * 128);
  }

  // Every CTA's lines visible to the cluster.
  static PTYB_D void publish() {
    if (C > 1) {
      cluster_arrive();
      cluster_wait();
    } else {
      __syncthreads();
    }
  }

  // Forward FFT of this thread's row (row-mapped) into plane m.
  PTYB_D void rows_forward(float2 (&v)[N1], int m) const {
    stage1<-1>(v, rtw);
    scatter_rotated(v, row + m * kPlane);
    __syncwarp();
    gather(v, rxch + m * kPlane);
    __syncwarp();
    stage2<-1>(v);
    const unsigned b = row + m * kPlane;
#pragma unroll
    for (int i = 0; i < N1; ++i) sts2((b ^ lo(N2 * i)) + hi(N2 * i), v[i]);
  }
  // Forward FFT of column r·H + c of plane m (published rows) into registers; the plane is free
  // for this thread's own elements afterwards.
  PTYB_D void columns_forward(float2 (&v)[N1], int m) const {
    pull(v, m);
    if (C > 1) cluster_arrive();
    stage1<-1>(v, tw);
    if (C > 1)
      cluster_wait();
    else
      __syncthreads();
    exchange(v, m);
    stage2<-1>(v);
  }
  // Inverse FFT of the column in registers into plane m.
  PTYB_D void columns_inverse(float2 (&v)[N1], int m) const {
    stage1<+1>(v, tw);
    exchange(v, m);
    stage2<+1>(v);
    stash(v, m);
  }
  // Inverse FFT of a row of plane m (published columns) into registers, row-mapped.
  PTYB_D void rows_inverse(float2 (&v)[N1], int m) const {
    pull(v, m);
    if (C > 1) cluster_arrive();
    stage1<+1>(v, tw);
    if (C > 1)
      cluster_wait();
    else
      __syncthreads();
    scatter_rotated(v, own + m * kPlane);
    __syncthreads();
    gather(v, rxch + m * kPlane);
    __syncwarp();  // the row is free for rows_forward
    stage2<+1>(v);
  }

 private:
  static PTYB_D void prefetch(const void* a) {
    asm volatile("prefetch.global.L2 [%0];" ::"l"(a));
  }
  PTYB_D void exchange(float2 (&v)[N1], int m) const {
    stash(v, m);
    __syncthreads();
    gather(v, xch + m * kPlane);
    __syncthreads();
  }
};

}  // namespace ptyb
