// Deterministic scatter-adds of the per-view updates onto the object and the probe.
//
// Object: one CTA owns half of a 16×16 square of the object and lists the launch's views that
// overlap the square in ascending slot order (the reference's view order); four thread groups
// per pixel take every fourth view of that list, each with Kahan-compensated float sums, and the
// groups' sums are added in group order. No atomics touch the object and the result does not
// depend on scheduling (the reference's tile-owned gather, ptyrs-kernels/src/lib.rs:388-437;
// operator engine/ops.rs:282-310). Probe: the slots are cut into chunks, each CTA sums one chunk
// in slot order for 512 probe pixels, and a second pass adds the chunk sums in chunk order
// (engine/ops.rs:315-345).
#pragma once
#include "common.cuh"

namespace ptyb {

constexpr int kTile = 16;      // object tile width
constexpr int kTileThreads = 512;                    // threads of a tile's CTA
constexpr int kTileRows = kTileThreads / 4 / kTile;  // object tile height (kGroups threads a pixel)
constexpr int kGroups = 4;     // view groups per pixel
constexpr int kMaxModes = 4;

enum GatherMode : int {
  kGatherRpie = 0,   // rPIE's sums: out = num_m, pre = D_m (−1 where no view covers the pixel),
                     // pmax = max over pixels of Σ_m D_m
  kGatherLsqml = 1,  // d_obj = Σ conj(q·P)·χ / √(pre² + floor²)
  kGatherMl = 2,     // grad += Σ conj(q·P)·g (compensated across launches)
  kGatherIllum = 4,    // pre = (pre + I)/2 with I = Σ|P|² over every view
  kGatherBlend = 5,    // the object blend's sums: out = num, pre = norm, pmax = max norm
};

struct GatherArgs {
  const float2* probe;     // [nprobe][N][N]
  const float2* quad;      // [N][N]
  const float2* upd;       // [slot][K][N][N] natural: Δ, χ or g
  const int* frames;       // [nslot]
  const int2* corners;     // [nframe]
  float* pmax;             // rPIE overlap max (device scalar)
  float* pre;              // LSQML preconditioner [nyo][nxo], rPIE [K][nyo][nxo]
  const float* pre_max;    // LSQML: max of pre (device scalar)
  float2* out;             // LSQML d_obj / ML gradient sum [nyo][nxo], rPIE [K][nyo][nxo]
  float2* comp;            // ML gradient compensation [nyo][nxo]
  float pre_scale;
  int nslot, nyo, nxo, nprobe, N;
  int probe_stride;        // elements between slots' probes (0: the shared probe)
};

// The launch's slots in [s0, s1) (at most kTileThreads) whose window overlaps the square
// [ty0, ty0 + kTile) × [tx0, tx0 + kTile), in ascending order with their corners: an ordered
// compaction by the whole CTA (warp ballots, then a prefix over the warps).
PTYB_D int tile_list(const GatherArgs& a, int s0, int s1, int ty0, int tx0, int* list,
                     int2* corner) {
  __shared__ int wbase[32];
  __shared__ int total;
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const int s = s0 + t;
  bool hit = false;
  int2 c = make_int2(0, 0);
  if (s < s1) {
    c = a.corners[a.frames[s]];
    hit = c.x < ty0 + kTile && c.x + a.N > ty0 && c.y < tx0 + kTile && c.y + a.N > tx0;
  }
  const unsigned m = __ballot_sync(0xffffffffu, hit);
  if (lane == 0) wbase[w] = __popc(m);
  __syncthreads();
  if (w == 0) {
    const int v = lane < kTileThreads / 32 ? wbase[lane] : 0;
    int incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += u;
    }
    wbase[lane] = incl - v;
    if (lane == 31) total = incl;
  }
  __syncthreads();
  if (hit) {
    const int pos = wbase[w] + __popc(m & ((1u << lane) - 1u));
    list[pos] = s;
    corner[pos] = c;
  }
  __syncthreads();
  const int n = total;
  __syncthreads();
  return n;
}

// One tile of the object for a launch of K probe modes: every group of threads walks its
// views in order, `kAhead` of them at a time: their loads are all issued before the first is
// added. K is a template parameter so that a view costs the registers its modes need.
template <int MODE, int K>
PTYB_D void object_tile(const GatherArgs& a) {
  constexpr int kChunk = kTileThreads;
  constexpr int kPix = kTile * kTileRows;  // pixels, kGroups threads each
  constexpr int kAhead = K <= 2 ? 2 : 1;
  constexpr bool kNum = MODE != kGatherIllum;
  constexpr bool kDen = MODE == kGatherIllum || MODE == kGatherRpie || MODE == kGatherBlend;
  constexpr int NM = MODE == kGatherRpie ? K : 1;  // numerators kept apart
  constexpr int DM = kDen ? K : 1;
  // The view list (during the walk), then the groups' partial sums (after it).
  constexpr int kListBytes = kChunk * (sizeof(int) + sizeof(int2));
  constexpr int kNumBytes = (kGroups - 1) * NM * kPix * sizeof(float2);
  constexpr int kDenBytes = (kGroups - 1) * DM * kPix * sizeof(float);
  constexpr int kPartBytes = kNumBytes + kDenBytes + (kGroups - 1) * kPix * sizeof(int);
  __shared__ __align__(16) unsigned char sm[kListBytes > kPartBytes ? kListBytes : kPartBytes];
  __shared__ float red[32];
  int* list = reinterpret_cast<int*>(sm);
  int2* lcorner = reinterpret_cast<int2*>(sm + kChunk * sizeof(int));
  float2(*part_num)[NM][kPix] = reinterpret_cast<float2(*)[NM][kPix]>(sm);
  float(*part_den)[DM][kPix] = reinterpret_cast<float(*)[DM][kPix]>(sm + kNumBytes);
  int(*part_cov)[kPix] = reinterpret_cast<int(*)[kPix]>(sm + kNumBytes + kDenBytes);
  const int tiles_x = (a.nxo + kTile - 1) / kTile;
  const int tx0 = (blockIdx.x % tiles_x) * kTile, ty0 = (blockIdx.x / tiles_x) * kTileRows;
  const int px = threadIdx.x % kPix, grp = threadIdx.x / kPix;
  const int x = tx0 + px % kTile, y = ty0 + px / kTile;
  const bool inside = x < a.nxo && y < a.nyo;
  const int N = a.N;
  const size_t plane = (size_t)N * N;
  KahanC num[NM];
  Kahan den[DM];
#pragma unroll
  for (int m = 0; m < NM; ++m) num[m].init();
#pragma unroll
  for (int m = 0; m < DM; ++m) den[m].init();
  bool covered = false, any = false;
  for (int s0 = 0; s0 < a.nslot; s0 += kChunk) {
    const int s1 = min(a.nslot, s0 + kChunk);
    const int n = tile_list(a, s0, s1, ty0 & ~(kTile - 1), tx0, list, lcorner);
    any |= n > 0;
    for (int i0 = grp; i0 < n; i0 += kGroups * kAhead) {
      bool ok[kAhead];
      float2 q[kAhead], u[kAhead][K], p[kAhead][K];
#pragma unroll
      for (int j = 0; j < kAhead; ++j) {
        const int i = i0 + j * kGroups;
        ok[j] = false;
        if (i >= n) continue;
        const int s = list[i];
        const int2 c = lcorner[i];
        const int yy = y - c.x, xx = x - c.y;
        ok[j] = inside && yy >= 0 && yy < N && xx >= 0 && xx < N;
        if (!ok[j]) continue;
        const int pix = yy * N + xx;
        if (kNum) q[j] = a.quad[pix];
#pragma unroll
        for (int m = 0; m < K; ++m) {
          if (kNum) u[j][m] = a.upd[((size_t)s * K + m) * plane + pix];
          p[j][m] = a.probe[(size_t)s * a.probe_stride + m * plane + pix];
        }
      }
#pragma unroll
      for (int j = 0; j < kAhead; ++j) {
        if (!ok[j]) continue;
        covered = true;
#pragma unroll
        for (int m = 0; m < K; ++m) {
          if (kDen) den[m].add(cnorm2(p[j][m]));
          // conj(P·q)·u
          if (kNum) num[NM == 1 ? 0 : m].add(cmulc_rn(cmul_rn(p[j][m], q[j]), u[j][m]));
        }
      }
    }
  }
  // Groups 1..3 hand their compensated sums to group 0, which adds them in group order.
  __syncthreads();  // the list's space becomes the partial sums'
  if (grp > 0) {
#pragma unroll
    for (int m = 0; m < NM; ++m)
      part_num[grp - 1][m][px] = make_float2(num[m].re.s - num[m].re.c, num[m].im.s - num[m].im.c);
#pragma unroll
    for (int m = 0; m < DM; ++m) part_den[grp - 1][m][px] = den[m].s - den[m].c;
    part_cov[grp - 1][px] = covered;
  }
  __syncthreads();
  if (grp == 0) {
#pragma unroll
    for (int g = 0; g < kGroups - 1; ++g) {
#pragma unroll
      for (int m = 0; m < NM; ++m) num[m].add(part_num[g][m][px]);
#pragma unroll
      for (int m = 0; m < DM; ++m) den[m].add(part_den[g][m][px]);
      covered |= part_cov[g][px] != 0;
    }
  }
  const size_t o = (size_t)y * a.nxo + x;
  if (MODE == kGatherRpie || MODE == kGatherBlend) {
    float d = 0.f;
#pragma unroll
    for (int m = 0; m < DM; ++m) d += den[m].s;
    if (MODE == kGatherBlend && inside && grp == 0) {
      // psi_to_obj_probe's object sums (engine/ops.rs:352-369), every pixel, covered or not
      a.out[o] = num[0].value();
      a.pre[o] = d;
    }
    if (MODE == kGatherRpie && inside && grp == 0) {
      const size_t no = (size_t)a.nyo * a.nxo;
#pragma unroll
      for (int m = 0; m < NM; ++m) {
        a.out[m * no + o] = num[m].value();
        a.pre[m * no + o] = covered ? den[m].s : -1.f;
      }
    }
    d = warp_max(inside && grp == 0 ? d : 0.f);
    if (threadIdx.x % 32 == 0) red[threadIdx.x / 32] = d;
    __syncthreads();
    if (threadIdx.x == 0) {
      float mx = 0.f;
      for (int w = 0; w < kTileThreads / 32; ++w) mx = fmaxf(mx, red[w]);
      atomic_max_nonneg(a.pmax, mx);
    }
    return;
  }
  if (!inside || grp != 0) return;
  if (MODE == kGatherLsqml) {
    const float p = a.pre[o];
    const float fl = 0.1f * (*a.pre_max);
    a.out[o] = cscale(num[0].value(), rsqrtf(p * p + fl * fl));
  } else if (MODE == kGatherMl) {
    if (!any) return;
    // out += num with the running compensation in comp.
    const float2 v = num[0].value();
    float2 g = a.out[o], cc = a.comp[o];
    const float yr = v.x - cc.x, yi = v.y - cc.y;
    const float tr = g.x + yr, ti = g.y + yi;
    cc = make_float2((tr - g.x) - yr, (ti - g.y) - yi);
    a.out[o] = make_float2(tr, ti);
    a.comp[o] = cc;
  } else if (MODE == kGatherIllum) {
    float d = 0.f;
#pragma unroll
    for (int m = 0; m < DM; ++m) d += den[m].s;
    // pty-chi's schedule: (pre + I)/2, the first from pre = I·pre_scale.
    a.pre[o] = a.pre_scale >= 0.f ? 0.5f * (d * a.pre_scale + d) : 0.5f * (a.pre[o] + d);
  }
}

// CTAs of 512 threads per SM a tile kernel is compiled for, by what a thread holds, in us per frame
// on one B200:
// - three (40 registers) for two views of up to two modes: ML 256² x 2 0.462, blend 0.378, LSQML
//   96² x 2 0.290, blend 128² x 1 0.072, with 16 to 44 bytes of spills at two modes; two CTAs (48
//   to 60 registers, none spilled) take 0.512, 0.371, 0.350 and 0.087. CTAs of 1024 with the mode
//   count at run time took 0.538 (ML), 0.477 and 0.106 (blends);
// - two (up to 64) for rPIE's sums of two modes and more: 128² x 2 0.289, three CTAs 0.402 with 144
//   bytes of spills; at one mode three are ahead, 64² 0.127 to 0.138;
// - four (32) for one view of three or four modes: LSQML 128² x 3 0.218 with 24 bytes of spills,
//   three CTAs with two views 0.322 with 94.
template <int MODE, int K>
__host__ __device__ constexpr int tile_min_blocks() {
  return MODE == kGatherRpie ? (K == 1 ? 3 : 2) : K <= 2 || MODE == kGatherBlend ? 3 : 4;
}

template <int MODE, int K>
static __global__ void __launch_bounds__(kTileThreads, tile_min_blocks<MODE, K>())
    object_tile_kernel(GatherArgs a) {
  object_tile<MODE, K>(a);
}

// One launch of a.nprobe ≤ 4 modes over `tiles` object tiles.
template <int MODE>
static inline void launch_object_tiles(const GatherArgs& a, int tiles, cudaStream_t s) {
  switch (a.nprobe) {
    case 1: object_tile_kernel<MODE, 1><<<tiles, kTileThreads, 0, s>>>(a); break;
    case 2: object_tile_kernel<MODE, 2><<<tiles, kTileThreads, 0, s>>>(a); break;
    case 3: object_tile_kernel<MODE, 3><<<tiles, kTileThreads, 0, s>>>(a); break;
    default: object_tile_kernel<MODE, 4><<<tiles, kTileThreads, 0, s>>>(a);
  }
}

// Σ over `n` planes of `count` values at value i, in plane order, compensated; ten loads ahead of
// the additions (they alone took 7 of a 64² batch's 10.6 us with the loads one by one).
PTYB_D float2 plane_sum(const float2* planes, int n, int count, int i) {
  KahanC acc;
  acc.init();
  int ch = 0;
  for (; ch + 10 <= n; ch += 10) {
    float2 v[10];
#pragma unroll
    for (int k = 0; k < 10; ++k) v[k] = planes[(size_t)(ch + k) * count + i];
#pragma unroll
    for (int k = 0; k < 10; ++k) acc.add(v[k]);
  }
  for (; ch < n; ++ch) acc.add(planes[(size_t)ch * count + i]);
  return acc.value();
}

struct ProbeArgs {
  const float2* object;   // [nyo][nxo] object mode 0
  const float2* quad;     // [N][N]
  const float2* upd;      // [slot][K][N][N]
  const int* frames;
  const int2* corners;
  const float* omax;      // rPIE [slot]
  float2* partial;        // [nchunk][K][N][N]
  float* partial_den;     // modes 2 and 3: [nchunk][N][N] Σ_slots |O|² over the window
  float alpha;            // rPIE
  // probe_partial_kernel: 1 Σ conj(q·O)·upd, 2 also Σ|O|², 3 Σ|O|² alone
  int nslot, chunk, nxo, K, N, mode;
};

constexpr int kMaxProbeChunk = 256;
constexpr int kProbePixels = 512;  // probe pixels per CTA of the probe sums, rPIE's too
static_assert(kProbePixels == kTileThreads, "rpie_sums_kernel takes a probe pixel a thread");

// Chunk `blockIdx.y` of slots (at most kMaxProbeChunk), kProbePixels pixels per CTA of 256 threads:
// Σ_slots conj(q·O)·upd in slot order for a's K modes. Two neighbouring pixels a thread, the update
// planes and the phase read 16 bytes at a time: bound by the latency of those loads (84 % of the
// stalls with one pixel a thread).
template <int K>
static __global__ void __launch_bounds__(256) probe_partial_kernel(ProbeArgs a) {
  __shared__ int2 cs[kMaxProbeChunk];
  const int N = a.N;
  const size_t plane = (size_t)N * N;
  const int s0 = blockIdx.y * a.chunk, s1 = min(a.nslot, s0 + a.chunk);
  for (int i = threadIdx.x; i < s1 - s0; i += 256) cs[i] = a.corners[a.frames[s0 + i]];
  __syncthreads();
  const int pix = 2 * (blockIdx.x * 256 + threadIdx.x);
  if (pix >= N * N) return;
  const int yy = pix / N, xx = pix % N;
  const float4 qv = reinterpret_cast<const float4*>(a.quad)[pix / 2];
  const float2 q[2] = {make_float2(qv.x, qv.y), make_float2(qv.z, qv.w)};
  KahanC acc[2][K];
  Kahan den[2];
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    den[j].init();
#pragma unroll
    for (int m = 0; m < K; ++m) acc[j][m].init();
  }
  const float2* obj = a.object + (size_t)yy * a.nxo + xx;
#pragma unroll 4
  for (int s = s0; s < s1; ++s) {
    const int2 c = cs[s - s0];
    const float2* op = obj + (size_t)c.x * a.nxo + c.y;
    float2 o[2] = {op[0], op[1]};
    if (a.mode >= 2) {
      den[0].add(cnorm2(o[0]));
      den[1].add(cnorm2(o[1]));
    }
    if (a.mode == 3) continue;
    float2 w[2];  // conjugated in the products below
#pragma unroll
    for (int j = 0; j < 2; ++j) w[j] = cmul_rn(o[j], q[j]);
#pragma unroll
    for (int m = 0; m < K; ++m) {
      const float4 u =
          reinterpret_cast<const float4*>(a.upd + ((size_t)s * K + m) * plane)[pix / 2];
      acc[0][m].add(cmulc_rn2(w[0], make_float2(u.x, u.y)));
      acc[1][m].add(cmulc_rn2(w[1], make_float2(u.z, u.w)));
    }
  }
  if (a.mode != 3) {
#pragma unroll
    for (int m = 0; m < K; ++m) {
      const float2 v0 = acc[0][m].value(), v1 = acc[1][m].value();
      reinterpret_cast<float4*>(a.partial + ((size_t)blockIdx.y * K + m) * plane)[pix / 2] =
          make_float4(v0.x, v0.y, v1.x, v1.y);
    }
  }
  if (a.mode >= 2)
    reinterpret_cast<float2*>(a.partial_den + (size_t)blockIdx.y * plane)[pix / 2] =
        make_float2(den[0].s - den[0].c, den[1].s - den[1].c);
}

// rPIE's object sums (the first `ntiles` blocks, one object tile each) and probe sums (the rest:
// kProbePixels pixels of one chunk of slots, one a thread, Σ w·upd with the weight w =
// conj(q·O)/((1−α)|O|² + α·max|O|²)) of a batch in one launch. Both read the batch-start object and
// probe, and at 64² neither fills the GPU for more than the latency of a few views. With the
// maximum of the overlaps taken here and the updates in rpie_apply_kernel a batch is three launches
// instead of five: frame pass, sums, updates (46 -> 28 us for 100 frames of 64²).
template <int K>
static __global__ void __launch_bounds__(kTileThreads, tile_min_blocks<kGatherRpie, K>())
    rpie_sums_kernel(GatherArgs g, ProbeArgs a, int ntiles) {
  if (blockIdx.x < ntiles) {
    object_tile<kGatherRpie, K>(g);
    return;
  }
  __shared__ int2 cs[kMaxProbeChunk];
  __shared__ float om[kMaxProbeChunk];
  const int N = a.N, blocks = N * N / kProbePixels, block = blockIdx.x - ntiles;
  const int chunk = block / blocks;
  const size_t plane = (size_t)N * N;
  const int s0 = chunk * a.chunk, s1 = min(a.nslot, s0 + a.chunk);
  for (int i = threadIdx.x; i < s1 - s0; i += kTileThreads) {
    cs[i] = a.corners[a.frames[s0 + i]];
    om[i] = a.omax[s0 + i];
  }
  __syncthreads();
  const int pix = (block % blocks) * kProbePixels + threadIdx.x;
  const float2 q = a.quad[pix];
  const float2* obj = a.object + (size_t)(pix / N) * a.nxo + pix % N;
  KahanC acc[K];
#pragma unroll
  for (int m = 0; m < K; ++m) acc[m].init();
#pragma unroll 2
  for (int s = s0; s < s1; ++s) {
    const int2 c = cs[s - s0];
    const float2 o = obj[(size_t)c.x * a.nxo + c.y];
    float2 w = cconj(cmul(o, q));
    w = cscale(w, 1.f / ((1.f - a.alpha) * cnorm2(o) + a.alpha * om[s - s0]));
#pragma unroll
    for (int m = 0; m < K; ++m) acc[m].add(cmul(w, a.upd[((size_t)s * K + m) * plane + pix]));
  }
#pragma unroll
  for (int m = 0; m < K; ++m) a.partial[((size_t)chunk * K + m) * plane + pix] = acc[m].value();
}

static inline void launch_rpie_sums(const GatherArgs& g, const ProbeArgs& a, int ntiles,
                                    int blocks, cudaStream_t s) {
  switch (g.nprobe) {
    case 1: rpie_sums_kernel<1><<<blocks, kTileThreads, 0, s>>>(g, a, ntiles); break;
    case 2: rpie_sums_kernel<2><<<blocks, kTileThreads, 0, s>>>(g, a, ntiles); break;
    case 3: rpie_sums_kernel<3><<<blocks, kTileThreads, 0, s>>>(g, a, ntiles); break;
    default: rpie_sums_kernel<4><<<blocks, kTileThreads, 0, s>>>(g, a, ntiles);
  }
}

// rPIE's updates of a batch in one launch: the first `oblocks` blocks take the object,
// O += step·Σ_m num_m / ((1−α)·D_m + α·pmax) on covered pixels, the rest the probe,
// P += coef·Σ over the `nsum` planes in order. `pmax_next` is cleared for the batch that follows.
struct RpieApplyArgs {
  float2* object;
  const float2* num;  // [K][no]
  const float* den;   // [K][no], < 0 where no view covers the pixel
  const float* pmax;
  float* pmax_next;
  float2* probe;
  const float2* sums; // [nsum][count]
  size_t no;
  int K, nsum, count, oblocks;
  float alpha, step, coef;
};
static __global__ void __launch_bounds__(256) rpie_apply_kernel(RpieApplyArgs a) {
  if (blockIdx.x == 0 && threadIdx.x == 0) *a.pmax_next = 0.f;
  if (blockIdx.x < a.oblocks) {
    const size_t o = (size_t)blockIdx.x * 256 + threadIdx.x;
    if (o >= a.no || a.den[o] < 0.f) return;
    const float pmax = *a.pmax;
    float2 d = make_float2(0.f, 0.f);
#pragma unroll
    for (int m = 0; m < kMaxModes; ++m) {
      if (m >= a.K) break;
      const float w = (1.f - a.alpha) * a.den[m * a.no + o] + a.alpha * pmax;
      d = cadd(d, cscale(a.num[m * a.no + o], 1.f / w));
    }
    a.object[o] = cadd(a.object[o], cscale(d, a.step));
    return;
  }
  const int i = (blockIdx.x - a.oblocks) * 256 + threadIdx.x;
  if (i >= a.count) return;
  a.probe[i] = cadd(a.probe[i], cscale(plane_sum(a.sums, a.nsum, a.count, i), a.coef));
}

// One launch over `nchunk` chunks (K ≤ 4; N² is a multiple of 512 at every side).
static inline void launch_probe_partial(const ProbeArgs& a, int nchunk, cudaStream_t s) {
  const dim3 grid(a.N * a.N / kProbePixels, nchunk);
  switch (a.K) {
    case 1: probe_partial_kernel<1><<<grid, 256, 0, s>>>(a); break;
    case 2: probe_partial_kernel<2><<<grid, 256, 0, s>>>(a); break;
    case 3: probe_partial_kernel<3><<<grid, 256, 0, s>>>(a); break;
    default: probe_partial_kernel<4><<<grid, 256, 0, s>>>(a);
  }
}

// The object blend of AP / DM / RAAR (engine/ops.rs:371-381) from the sums kGatherBlend wrote:
// O = (num + reg·O) / max(norm + reg, 1e-12) with reg = inertia·max norm.
static __global__ void blend_apply_kernel(float2* object, const float2* num, const float* norm,
                                   const float* norm_max, float inertia, size_t n) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float reg = inertia * (*norm_max);
  object[i] = cscale(cadd(num[i], cscale(object[i], reg)), 1.f / fmaxf(norm[i] + reg, 1e-12f));
}

// The probe step of AP / DM / RAAR under the move (engine/features.rs:673-712), one block per
// probe mode m: with D = max(norm + reg, 1e-12) and reg = inertia·max norm, step = g / D,
// sums[m] = (Σ|g|²/D, reg·Σ|step|²) in double, added in a fixed order.
static __global__ void __launch_bounds__(1024) probe_pcg_step_kernel(const float2* g, const float* norm,
                                                              const float* norm_max,
                                                              float inertia, int plane,
                                                              float2* step, double* sums) {
  __shared__ double red[2][32];
  const int m = blockIdx.x;
  const float reg = inertia * (*norm_max);
  double slope = 0.0, curv = 0.0;
  for (int i = threadIdx.x; i < plane; i += 1024) {
    const float2 v = g[(size_t)m * plane + i];
    const float d = fmaxf(norm[i] + reg, 1e-12f);
    const float2 s = cscale(v, 1.f / d);
    step[(size_t)m * plane + i] = s;
    slope += ((double)v.x * v.x + (double)v.y * v.y) / d;
    curv += (double)reg * ((double)s.x * s.x + (double)s.y * s.y);
  }
  slope = warp_sum(slope);
  curv = warp_sum(curv);
  if (threadIdx.x % 32 == 0) {
    red[0][threadIdx.x / 32] = slope;
    red[1][threadIdx.x / 32] = curv;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0.0, b = 0.0;
    for (int w = 0; w < 32; ++w) {
      a += red[0][w];
      b += red[1][w];
    }
    sums[2 * m] = a;
    sums[2 * m + 1] = b;
  }
}

// Per slot and probe mode, Σ_pixels |O_window|²·|W|² in double (‖A·s‖² of one frame's view of
// the moved step W), added in a fixed order; grid (slots, K).
static __global__ void __launch_bounds__(256) weighted_norm_kernel(const float2* waves,
                                                            const float2* object,
                                                            const int* frames,
                                                            const int2* corners, int nxo, int N,
                                                            int K, double* out) {
  __shared__ double red[8];
  const int slot = blockIdx.x, m = blockIdx.y;
  const size_t plane = (size_t)N * N;
  const int2 c = corners[frames[slot]];
  const float2* w = waves + ((size_t)slot * K + m) * plane;
  double acc = 0.0;
  for (int pix = threadIdx.x; pix < N * N; pix += 256) {
    const int y = pix / N, x = pix % N;
    acc += (double)cnorm2(object[(size_t)(c.x + y) * nxo + c.y + x]) * cnorm2(w[pix]);
  }
  acc = warp_sum(acc);
  if (threadIdx.x % 32 == 0) red[threadIdx.x / 32] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int i = 0; i < 8; ++i) s += red[i];
    out[(size_t)slot * K + m] = s;
  }
}

// P_m += alpha_m·step_m over the K probe planes.
struct ModeCoefs {
  float c[kMaxModes];
};
static __global__ void probe_modes_axpy_kernel(float2* probe, const float2* step, ModeCoefs alpha,
                                        int plane, int count) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const float a = alpha.c[i / plane];
  if (a != 0.f) probe[i] = cadd(probe[i], cscale(step[i], a));
}

// The probe blend's norm Σ_frames |O|² per pixel: the chunks' sums in chunk order into `den`,
// and its maximum into *dmax (zeroed by the caller).
static __global__ void __launch_bounds__(256) probe_norm_kernel(const float* partial_den, int nchunk,
                                                         int plane, float* den, float* dmax) {
  __shared__ float red[8];
  const int i = blockIdx.x * 256 + threadIdx.x;
  float v = 0.f;
  if (i < plane) {
    Kahan acc;
    acc.init();
    for (int ch = 0; ch < nchunk; ++ch) acc.add(partial_den[(size_t)ch * plane + i]);
    v = acc.s - acc.c;
    den[i] = v;
  }
  v = warp_max(v);
  if (threadIdx.x % 32 == 0) red[threadIdx.x / 32] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    float mx = 0.f;
    for (int w = 0; w < 8; ++w) mx = fmaxf(mx, red[w]);
    atomic_max_nonneg(dmax, mx);
  }
}

// Σ over chunks in order; mode 1: out = coef·Σ; 2: out += Σ compensated; 3: the blend P = (Σ +
// reg·P) / max(norm + reg, 1e-12) with reg = coef·max norm (engine/ops.rs:371-381), `norm` one
// plane shared by the modes.
static __global__ void probe_finalize_kernel(const float2* partial, int nchunk, int count,
                                      float2* probe, float2* out, float2* comp, float coef,
                                      int mode, const float* norm = nullptr,
                                      const float* norm_max = nullptr, int plane = 1) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const float2 v = plane_sum(partial, nchunk, count, i);
  if (mode == 3) {
    const float reg = coef * (*norm_max);
    probe[i] = cscale(cadd(v, cscale(probe[i], reg)), 1.f / fmaxf(norm[i % plane] + reg, 1e-12f));
  } else if (mode == 1) {
    out[i] = cscale(v, coef);
  } else {
    float2 g = out[i], cc = comp[i];
    const float yr = v.x - cc.x, yi = v.y - cc.y;
    const float tr = g.x + yr, ti = g.y + yi;
    comp[i] = make_float2((tr - g.x) - yr, (ti - g.y) - yi);
    out[i] = make_float2(tr, ti);
  }
}

}  // namespace ptyb
