// rPIE on the GPU (reference engine/gpu/rpie.rs:31-63, 198-529; CPU twin
// engine/ptycho.rs:874-1085): per batch the frame pass, the overlap weights, the object and
// probe updates and, under the position model, pty-chi's position step.
#include "engine.cuh"

using namespace ptyb;

namespace ptyb::eng {
namespace {

// The arrays that take a batch's object sums and overlaps per mode, [K][nyo][nxo].
struct BatchSums {
  float2* num;
  float* den;
};

// For one mode they are LSQML's direction and preconditioner, which no call leaves a value in for
// another; for more, the part of the frames' planes (h->field) that batches of `batch` frames
// leave alone: all of it, or past the batch's own planes under the position model. Only where the
// object is larger than that (12·K bytes a pixel) do they get arrays of their own, made once.
BatchSums batch_sums(ptyb_handle* h, int batch) {
  if (h->K == 1) return {h->d_obj, h->pre};
  const size_t n = (size_t)h->K * h->nyo * h->nxo, planes = (size_t)h->K * h->N * h->N;
  const size_t used = h->have_offsets ? batch * planes : 0;
  if (8 * (h->slots * planes - used) >= 12 * n) {
    float2* num = h->field + used;
    return {num, reinterpret_cast<float*>(num + n)};
  }
  if (!h->rpie_num) {
    h->rpie_num = alloc<float2>(h, n);
    h->rpie_den = alloc<float>(h, n);
  }
  return {h->rpie_num, h->rpie_den};
}

// One rPIE batch (engine/ptycho.rs:904-1085; GPU launch sequence engine/gpu/rpie.rs:239-345):
// the frame pass, the object and probe sums from the batch-start arrays, the position model's
// passes, then both updates. `pmax` and `pmax_next` take the largest overlap of this batch and
// of the next in turn, each cleared by the updates of the batch before.
void rpie_batch(ptyb_handle* h, const ptyb_rpie_params& p, const int* frames, int nslot,
                const BatchSums& sums, float* pmax, float* pmax_next) {
  FrameArgs a = frame_args(h, frames);
  GatherArgs g = gather_args(h, frames, nslot);
  const int pstride = h->K * h->N * h->N;
  const bool moved = h->have_offsets, refine = h->have_offsets && h->refine_offsets;
  if (moved) {
    // every frame's probe moved by its offset from the batch-start probe (engine/ptycho.rs:
    // 920-935); the views' waves in the frame pass and the object gathers
    ensure_spec(h);
    spectrum_of(h, h->probe, h->spec);
    move_frames(h, frames, nslot, h->spec, h->wave);
    a.probe = h->wave;
    a.probe_stride = pstride;
    g.probe = h->wave;
    g.probe_stride = pstride;
  }
  check(h, launch_frame<kRpie>(h, a, nslot), "rpie frame pass");
  ++h->launches;
  const int count = h->K * h->N * h->N;
  // the probe's plain sums run beside the object's; under the move its directions go back first
  const bool sum_probe = p.update_probe && !moved;
  int nchunk = 0;
  const int chunk = sum_probe ? probe_chunk(h, nslot, &nchunk) : 0;
  const int tiles = p.update_object ? ntiles(h) : 0;
  const int pblocks = nchunk * (h->N * h->N / kProbePixels);
  if (tiles + pblocks > 0) {
    g.out = sums.num;
    g.pre = sums.den;
    g.pmax = pmax;
    ProbeArgs pa = {};
    pa.object = h->object;
    pa.quad = h->quad;
    pa.upd = h->upd;
    pa.frames = frames;
    pa.corners = h->corners;
    pa.omax = h->omax;
    pa.partial = h->partial;
    pa.alpha = (float)p.probe_alpha;
    pa.nslot = nslot;
    pa.chunk = chunk;
    pa.nxo = h->nxo;
    pa.K = h->K;
    pa.N = h->N;
    timed(h, kKRpieSums, [&] { launch_rpie_sums(g, pa, tiles, tiles + pblocks, h->stream); }, nslot);
    launched(h, "rpie sums");
  }
  if (refine) {
    // pty-chi's position sums from mode 0 of the batch-start state (engine/ptycho.rs:1037-1064)
    check(h, launch_move<kDerivWindow>(h, move_args(h, frames, h->field), nslot), "window derivative");
    ++h->launches;
    timed(h, kKPositionSums, [&] {
      position_sums_kernel<<<nslot, 256, 0, h->stream>>>(h->field, h->wave, pstride, h->quad,
                                                          h->upd, h->K, h->N, h->pos_sums);
    }, nslot);
    launched(h, "position sums");
  }
  if (p.update_probe && moved) {
    // each frame's rPIE probe direction moved back by −d (engine/ptycho.rs:1007-1035)
    timed(h, kKProbePartial, [&] {
      probe_terms_kernel<<<dim3((h->N * h->N + 255) / 256, nslot), 256, 0, h->stream>>>(
          h->object, h->quad, h->upd, frames, h->corners, h->nxo, h->K, h->N, h->field, h->omax,
          (float)p.probe_alpha);
    }, nslot);
    launched(h, "probe terms");
    check(h, launch_move<kMoveBack>(h, move_args(h, frames, h->field), nslot), "probe move back");
    ++h->launches;
  }
  // O and P += step/nbatch · Σ (frames in order)
  RpieApplyArgs u = {};
  u.object = h->object;
  u.num = sums.num;
  u.den = sums.den;
  u.pmax = pmax;
  u.pmax_next = pmax_next;
  u.probe = h->probe;
  u.sums = moved ? h->field : h->partial;
  u.no = (size_t)h->nyo * h->nxo;
  u.K = h->K;
  u.nsum = moved ? nslot : nchunk;
  u.count = p.update_probe ? count : 0;
  u.oblocks = p.update_object ? (int)blocks_for(u.no) : 0;
  u.alpha = (float)p.obj_alpha;
  u.step = (float)p.obj_step;
  u.coef = (float)(p.probe_step / nslot);
  if (u.oblocks + u.count > 0) {
    timed(h, kKRpieUpdates, [&] {
      rpie_apply_kernel<<<u.oblocks + blocks_for(u.count), 256, 0, h->stream>>>(u);
    });
    launched(h, "rpie updates");
  }
  if (refine) {
    const double eps = 1e-6 * ((double)h->N * h->N);
    timed(h, kKSolve, [&] {
      position_step_kernel<<<1, 1024, 0, h->stream>>>(h->pos_sums, nslot, h->P, eps, frames,
                                                    h->offsets);
    });
    launched(h, "position step");
  }
}

}  // namespace
}  // namespace ptyb::eng

using namespace ptyb::eng;

extern "C" {

int ptyb_rpie(ptyb_handle* h, const ptyb_rpie_params* p, int32_t nepoch) {
  if (!h || !p) return PTYB_INVALID;
  if (p->batch_size <= 0 || nepoch < 0) {
    h->err = "rPIE batch_size must be >= 1";
    return PTYB_INVALID;
  }
  if (h->nobj != 1) {
    h->err = "rPIE needs exactly one object mode";
    return PTYB_INVALID;
  }
  if (h->nslice > 1) {
    h->err = "rPIE runs on a single-slice object";
    return PTYB_INVALID;
  }
  return guarded(h, true, [&]() -> int {
    const int bs = std::min(p->batch_size, h->P);
    ensure_slots(h, std::max(bs, std::min(h->P, h->stack)));
    std::vector<std::vector<int32_t>> sizes;
    upload_orders(h, nepoch, p->batch_size, p->seed, h->cycle, &sizes, nullptr);
    const BatchSums sums = batch_sums(h, bs);
    float* overlap = h->scal + kScalOverlap;
    begin_call(h);
    check(h, cudaMemsetAsync(overlap, 0, 2 * sizeof(float), h->stream), "memset");
    int64_t batch = 0;
    for (int ic = 0; ic < nepoch; ++ic) {
      const int* order = h->order_all + (size_t)ic * h->P;
      int off = 0;
      for (int n : sizes[ic]) {
        rpie_batch(h, *p, order + off, n, sums, overlap + batch % 2, overlap + (batch + 1) % 2);
        off += n;
        ++batch;
      }
      if (llk_due(p->calc_llk, ic, nepoch)) record(h, kAlgRpie, llk_pass(h));
      ++h->cycle;
    }
    end_call(h, "rpie");
    return PTYB_OK;
  });
}

}  // extern "C"
