// dtb_kernels.cuh -- the GGDT tile visit (warp per 32x32 tile) and the kernels built from it.
//
// Kernels
//   ggdt_scan        seed-tile scan: reads every mask tile once, writes the tile states and queues the tiles
//                    that hold seeds (replaces initialize_generalised_distance_map + initialize_task_queue,
//                    reference dt/src/utils.cu:5-18, and the priority set-up of dt/src/block_priority.cu).
//   ggdt_persistent  cooperative persistent kernel: every warp pops tiles from the shared queue, visits them
//                    and re-activates neighbours whose halo it can still lower (replaces the task variant,
//                    reference dt/src/generalised_distance_transform_task.cu:129-150).  No grid barrier:
//                    termination is "queue empty and nothing in flight".
//   ggdt_round       one host-driven round over the active tiles (the plain per-image path; the round
//                    structure of reference dt/src/generalised_distance_transform_blocks.cu:156-163).
//   ggdt_finalize    writes v into tiles that were never reached (their memory was never initialised).
#pragma once

#include <type_traits>

#include "dtb_device.cuh"

namespace dtb {

constexpr int PHASE_LIMIT = 4096;
constexpr uint64_t TMA_TIMEOUT_NS = 2000000000ull;  // 2 s

// ------------------------------------------------------------------------------------------------------
// Schedulers: what "activate a neighbour" and "finish a visit" mean.
// ------------------------------------------------------------------------------------------------------
// Per-warp counters, flushed to the queue header in batches (the header lines are shared by all warps).
struct WarpStats {
  uint32_t visits = 0, phases = 0, activations = 0, unflushed = 0;
};

struct QueueSched {
  static constexpr bool any_change = false;  // ref-mode: activate the neighbours that the border can lower
  Queue q;
  uint32_t* states;
  // Optional: the warp's word for a tile it keeps.  Of the tiles a visit queues, one in the lowest bucket
  // (the one the workers take from: its activation value is among the smallest queued) is not pushed; the warp
  // visits it next, which saves the ring's push and pop (two to five L2 round trips) and reuses the halo just
  // written.  It stays counted in `pending` like a queued tile.  nullptr: every tile goes through the ring.
  uint32_t* keep_out = nullptr;
  // Start of a visit (whole warp): PENDING -> RUNNING; returns the state before.  Activations from here on belong to
  // the next queue entry.  `pending` takes as many tokens as the visit may activate neighbours, without waiting.
  static constexpr uint32_t TOKENS = 8;
  __device__ __forceinline__ uint32_t claim(uint32_t tile) const {
    uint32_t old = 0;
    if ((threadIdx.x & 31) == 0) {
      old = atomicXor(&states[tile], ST_PENDING | ST_RUNNING);
      if (q.keys) q.keys[tile] = KEY_NONE;
      atomicAdd(&q.hdr->pending.v, TOKENS);
    }
    return __shfl_sync(~0u, old, 0);
  }
  // Warp-level end of a visit.  Lanes with `want` ask for a re-run of neighbour `item`, bringing activation
  // value `key` (distance units; bucket width 1 / inv_width): idle -> queued; running -> running with a re-run
  // requested; queued -> unchanged.  Lane 31 clears RUNNING of the own tile (and sets / clears the xor_bits);
  // a re-run requested meanwhile re-queues it at the smallest value its activators left in keys[].
  // The tokens taken by claim() cover the pushes, so `pending` counts an item before it can be popped, and what is left
  // goes back without waiting; waiting workers look at `pending` themselves.  (A count before the pushes, its fence and
  // its result cost each visit three L2 round trips of 17.)
  // On a first visit the own-tile update is fenced before the activations: a woken neighbour takes this tile's
  // distances as halo only if it sees VISITED, and otherwise reads v in their place.  Seeing the activation without
  // the bit would consume the wake-up without the new distances.  Otherwise the two are in flight together.
  __device__ __forceinline__ void complete(uint32_t tile, uint32_t xor_bits, bool want, uint32_t want_item,
                                           float key = 0.0f, float inv_width = 0.0f) const {
    const int lane = threadIdx.x & 31;
    const uint32_t base = q.nb_mask ? ld_volatile(&q.hdr->base.v) : 0u;
    uint32_t own = 0, other = 0;
    if (lane == 31) own = atomicXor(&states[tile], xor_bits | ST_RUNNING);
    if (xor_bits & ST_VISITED) {
      fence_acq_rel();
      __syncwarp();
    }
    if (want && want_item >= q.total_tiles) {
      set_error(q, DERR_BAD_TILE, want_item);
      want = false;
    }
    if (want) {
      if (q.keys) atomicMin(&q.keys[want_item], __float_as_uint(key));
      other = atomicOr(&states[want_item], ST_PENDING);
    }
    const bool again = lane == 31 && (own & ST_PENDING) != 0u;
    const bool push = again || (want && !(other & (ST_PENDING | ST_RUNNING)));
    const uint32_t item = lane == 31 ? tile : want_item;
    float pkey = key;
    if (again && q.keys && !keep_out) {
      const uint32_t kb = ld_volatile(&q.keys[tile]);
      pkey = kb == KEY_NONE ? 0.0f : __uint_as_float(kb);
    }
    const uint32_t m = __ballot_sync(~0u, push);
    const uint32_t b = push ? bucket_at(q, pkey, inv_width, base) : 0u;
    int kept = -1;
    if (keep_out && m) {
      // The own tile first, whatever its bucket (lane 31 re-queues it when its halo dropped during the visit): its
      // re-run reuses the weights and distances in this warp's shared memory.  Else the smallest activation value
      // in the lowest bucket.
      if (m >> 31) {
        kept = 31;
      } else {
        const bool elig = push && b == (base & q.nb_mask);
        const uint32_t kmin = __reduce_min_sync(~0u, elig ? __float_as_uint(pkey) : 0xFFFFFFFFu);
        const uint32_t cand = __ballot_sync(~0u, elig && __float_as_uint(pkey) == kmin);
        if (cand) kept = __ffs(cand) - 1;
      }
      if (lane == kept) *keep_out = item;
    }
    if (push && lane != kept) slot_write(q, b, atomicAdd(&q.hdr->tails[b].v, 1u), item);
    __syncwarp();
    if (lane == 0) atomicSub(&q.hdr->pending.v, TOKENS + 1u - __popc(m));
  }
};

struct RoundSched {
  static constexpr bool any_change = true;  // ref-mode: activate the neighbours whose facing border changed
  Queue q;  // only the counters and error word are used
  uint32_t* states;
  uint8_t* next_active;
  uint32_t* changed;
  __device__ __forceinline__ void complete(uint32_t tile, uint32_t xor_bits, bool want, uint32_t want_item,
                                           float = 0.0f, float = 0.0f) const {
    if (want) {
      if (want_item >= q.total_tiles) {
        set_error(q, DERR_BAD_TILE, want_item);
      } else {
        next_active[want_item] = 1;
        *(volatile uint32_t*)changed = 1u;
      }
    }
    if ((threadIdx.x & 31) == 31 && xor_bits) atomicXor(&states[tile], xor_bits);
  }
};

// Adds a finished visit to the warp's counters; flushes `progress` every 16 visits (the watchdog and the
// visit cap only need it approximately).
__device__ __forceinline__ void count_visit(WarpStats& ws, const Queue& q, uint32_t nphase, uint32_t nact) {
  ws.visits += 1;
  ws.phases += nphase;
  ws.activations += nact;
  if (++ws.unflushed == 16) {
    if ((threadIdx.x & 31) == 0) atomicAdd(&q.hdr->progress.v, ws.unflushed);
    ws.unflushed = 0;
  }
}

__device__ __forceinline__ void flush_stats(WarpStats& ws, const Queue& q) {
  if ((threadIdx.x & 31) == 0) {
    if (ws.unflushed) atomicAdd(&q.hdr->progress.v, ws.unflushed);
    if (ws.phases) atomicAdd(&q.hdr->phases.v, ws.phases);
    if (ws.activations) atomicAdd(&q.hdr->activations.v, ws.activations);
  }
  ws = WarpStats{};
}

__device__ __forceinline__ float f_inf() { return __int_as_float(0x7f800000); }

__device__ __forceinline__ float* dist_row(const ImgDesc& dd, int y) {
  return reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(dd.dist) + (int64_t)y * dd.dist_pitch);
}

// Distance read of a pixel that another warp (on any SM) may have written during this launch: L2 only, so no
// line an SM cached earlier can be returned.
__device__ __forceinline__ float ld_dist(const ImgDesc& dd, int y, int x) { return __ldcg(dist_row(dd, y) + x); }

// Address of column x of row y0 of the distance map, passed through an empty asm that also takes `dep`.  A
// visit's tile loads and its write-back each take their row addresses from such a base, with different `dep`:
// the compiler then cannot keep the 32 row addresses of the loads live across the whole visit to reuse them in
// the write-back (64 registers).
__device__ __forceinline__ uint8_t* dist_base(const ImgDesc& dd, int y0, int x, uint32_t dep) {
  uint8_t* p = reinterpret_cast<uint8_t*>(dist_row(dd, y0) + x);
  asm("" : "+l"(p) : "r"(dep));
  return p;
}
__device__ __forceinline__ float ld_dist_at(const uint8_t* base, int64_t pitch, int y) {
  return __ldcg(reinterpret_cast<const float*>(base + (int64_t)y * pitch));
}

// Whether the seed mask holds a nonzero byte in columns x0 .. x0 + vw - 1 of row y (x0 a multiple of 32, vw <= 32).
__device__ __forceinline__ bool mask_row_any(const ImgDesc& dd, int x0, int y, int vw) {
  const uint8_t* row = dd.mask + (int64_t)y * dd.mask_pitch + x0;
  if (vw == TILE && (reinterpret_cast<uintptr_t>(row) & 15u) == 0) {
    const uint4 a = reinterpret_cast<const uint4*>(row)[0];
    const uint4 b = reinterpret_cast<const uint4*>(row)[1];
    return (a.x | a.y | a.z | a.w | b.x | b.y | b.z | b.w) != 0u;
  }
  bool nz = false;
  for (int c = 0; c < vw; ++c) nz |= row[c] != 0;
  return nz;
}

// 1 / bucket width of an image: one tile-width of path cost in bucket_tiles parts, 32 x the mean internal edge weight
// seen so far by first visits.
__device__ __forceinline__ float bucket_inv_width(const Queue& q, uint32_t img) {
  if (!q.wacc) return 0.0f;
  const volatile float* wa = q.wacc + 2 * img;
  const float s = wa[0], c = wa[1], w = q.bucket_tiles * (float)TILE;
  return (c > 0.0f && s > 0.0f) ? c / (w * s) : 1.0f / w;
}

// Waits for the TMA transactions on `bar`; its phase parity is bit `pmask` of `pbits`.  Bounded: after
// TMA_TIMEOUT_NS the error word is set and the wait goes on for as long again, to give a slow copy the chance
// to land before the warp leaves; after that the wait gives up, and a copy may then still be pending.  Either way
// STAGE_LOST is set in `pbits`: the warp visits nothing more and never arms its barriers again (one whose phase has
// not ended must not be armed twice).  The error word ends the launch for the warps that wait for work.
// `need`: false returns at once.  The wait is called outside of branches with that flag instead of inside of one: its
// loop has no exit that the compiler knows to be uniform, and a branch around it would make it guard every warp-wide
// operation that follows (see `uniform`).
// (Loops test it through `uniform`: a plain test of the bit, which the compiler takes for divergent, made the tile kernel
// 15 % slower.)
constexpr uint32_t STAGE_LOST = 0x80000000u;
__device__ __forceinline__ bool tma_wait(uint64_t* bar, uint32_t& pbits, uint32_t pmask, const Queue& q, uint32_t tile,
                                         bool need = true) {
  const uint32_t parity = (pbits & pmask) ? 1u : 0u;
  const uint64_t t0 = globaltimer();
  bool ok = true;
  while (need && !mbar_try_wait(bar, parity)) {
    const uint64_t dt = globaltimer() - t0;
    if (ok && dt > TMA_TIMEOUT_NS) { set_error(q, DERR_TMA_TIMEOUT, tile); ok = false; }
    if (dt > 2 * TMA_TIMEOUT_NS) break;
  }
  if (need) pbits ^= pmask;
  ok = __all_sync(~0u, ok);
  if (!ok) pbits |= STAGE_LOST;
  return ok;
}

// Shared memory of one visit.  A self-staging visit loads its image box and seed-mask box on `bar`; a visit
// staged ahead finds its image box issued on `bar` already and loads the mask box (seed visits only) on `mbar`.
struct VisitBufs {
  uint8_t* box;       // image box (TMA destination)
  void* mask;         // seed-mask box (TMA destination), used before the weights are computed
  TileBufs* t;
  uint64_t* bar;
  uint64_t* mbar;
  uint32_t pmask;     // bit of *pbits holding bar's phase parity
  uint32_t mmask;     // bit of *pbits holding mbar's phase parity
  uint32_t* pbits;
};

__device__ __forceinline__ VisitBufs visit_bufs(WarpSmem& sm, uint32_t& pbits) {
  return VisitBufs{sm.img, sm.t.Wv, &sm.t, &sm.bar, &sm.bar, 1u, 1u, &pbits};
}

// Issues one 2-D TMA box into this warp's shared memory on `bar` (whole warp; lane 0 issues).  Orders this
// warp's earlier generic accesses of the destination before the async-proxy writes.
__device__ __forceinline__ void stage_box(void* dst, uint64_t* bar, const CUtensorMap* tm, uint32_t bytes, int x, int y) {
  fence_proxy_async_smem();
  __syncwarp();
  if ((threadIdx.x & 31) == 0) {
    tmap_acquire(tm);
    mbar_arrive_expect_tx(bar, bytes);
    tma_load_2d(dst, tm, x, y, bar);
  }
}

// The image box of a tile (1-pixel halo; x starts 16 bytes left of the halo so that it stays 16-byte aligned).
__device__ __forceinline__ void stage_image_box(uint8_t* box, uint64_t* bar, const CUtensorMap* tm_img, bool rgb, int x0,
                                                int y0) {
  stage_box(box, bar, tm_img, (rgb ? IMG_BOX_RGB : IMG_BOX_GRAY) * IMG_BOX_ROWS, rgb ? 3 * x0 - 16 : x0 - 16, y0 - 1);
}

// Issues the image box of a warp's next tile ahead of its visit (the image index bits of a tile state never
// change, so reading them before the tile is claimed is safe).
__device__ __forceinline__ void stage_ahead(const ImgDesc* __restrict__ descs, const CUtensorMap* __restrict__ tmaps,
                                            const uint32_t* states, uint32_t tile, uint8_t* box, uint64_t* bar) {
  uint32_t st = 0;
  if ((threadIdx.x & 31) == 0) st = ld_volatile(&states[tile]);
  const uint32_t img = __shfl_sync(~0u, st, 0) >> ST_IMG_SHIFT;
  const ImgDesc& dd = descs[img];
  const uint32_t local = tile - dd.tile_base;
  const uint32_t tx = local % (uint32_t)dd.tiles_x, ty = local / (uint32_t)dd.tiles_x;
  stage_image_box(box, bar, tmaps + 2 * img, dd.channels == 3, (int)tx * TILE, (int)ty * TILE);
}

// Stages the image box (with 1-pixel halo) and, if needed, the seed-mask tile of a tile into shared memory,
// both on vb.bar.
__device__ __forceinline__ void stage_tile(const VisitBufs& vb, const CUtensorMap* tm_img, const CUtensorMap* tm_mask,
                                           bool rgb, bool with_mask, int x0, int y0) {
  // Order this warp's earlier generic reads of the slot before the async-proxy writes below.
  fence_proxy_async_smem();
  __syncwarp();
  if ((threadIdx.x & 31) == 0) {
    tmap_acquire(tm_img);
    if (with_mask) tmap_acquire(tm_mask);
    const uint32_t bytes = (rgb ? IMG_BOX_RGB : IMG_BOX_GRAY) * IMG_BOX_ROWS + (with_mask ? TILE * TILE : 0);
    mbar_arrive_expect_tx(vb.bar, bytes);
    tma_load_2d(vb.box, tm_img, rgb ? 3 * x0 - 16 : x0 - 16, y0 - 1, vb.bar);
    if (with_mask) tma_load_2d(vb.mask, tm_mask, x0, y0, vb.bar);
  }
}

// Packed pixel of the staged image box: box row r (tile row r - 1), tile column c in [-1, 32].
__device__ __forceinline__ uint32_t box_pix(const uint8_t* box, bool rgb, int r, int c) {
  if (!rgb) return box[r * IMG_BOX_GRAY + 16 + c];
  const int off = r * IMG_BOX_RGB + 16 + 3 * c;
  const uint32_t* wp = reinterpret_cast<const uint32_t*>(box + (off & ~3));
  return __funnelshift_r(wp[0], wp[1], (off & 3) * 8) & 0xFFFFFFu;
}

// Edge weights of a tile from its staged image box into Wh / Wv / E (lane = x; the left and right halo edges
// lane = y).  Returns this lane's sum of the tile's internal column edges (x < vw, 0 < y < vh).  UNROLL: rows in flight;
// the tile kernel, whose warps are all at different places of its code, runs faster with the smallest code (1 against 2:
// 512-image plan 4.41 against 4.70 ms), the block kernel, whose warps move together, with 2.
template <int UNROLL>
__device__ __forceinline__ float tile_weights(float g2, bool rgb, int vw, int vh, uint8_t* box, float* Wh, float* Wv, float* E) {
  const int lane = threadIdx.x & 31;
  const float INF = f_inf();
  float wsum = 0.0f;
  float et, eb, el, er;
  if (!rgb) {
    // Gray: the weight depends on |dI| in [0, 255] only.  A 256-entry table of the same expression (so the
    // same bits) costs 8 square roots per lane instead of 65; it sits in the part of the image box that the
    // 64-byte gray rows leave unused.
    float* lut = reinterpret_cast<float*>(box + GRAY_LUT_OFFSET);
#pragma unroll(UNROLL == 1 ? 2 : 8)
    for (int k = 0; k < 8; ++k) {
      const uint32_t a = (uint32_t)(lane + 32 * k);
      lut[a] = ns_weight_sq(a * a, g2);
    }
    __syncwarp();
    const uint8_t* col = box + 16 + lane;  // column `lane` of the box, row r at col[r * IMG_BOX_GRAY]
    int pprev = col[IMG_BOX_GRAY];
    et = lut[abs(pprev - (int)col[0])];
    Wv[lane] = INF;
    Wh[lane] = lane == 0 ? INF : lut[abs(pprev - (int)col[IMG_BOX_GRAY - 1])];
#pragma unroll UNROLL
    for (int y = 1; y < TILE; ++y) {
      const int pcur = col[(y + 1) * IMG_BOX_GRAY];
      const float w = lut[abs(pcur - pprev)];
      const float wx = lut[abs(pcur - (int)col[(y + 1) * IMG_BOX_GRAY - 1])];
      Wv[y * W_STRIDE + lane] = w;
      Wh[y * W_STRIDE + lane] = lane == 0 ? INF : wx;
      if (lane < vw && y < vh) wsum += w;
      pprev = pcur;
    }
    eb = lut[abs((int)col[(TILE + 1) * IMG_BOX_GRAY] - pprev)];
    const uint8_t* row = box + (lane + 1) * IMG_BOX_GRAY + 16;
    el = lut[abs((int)row[0] - (int)row[-1])];
    er = lut[abs((int)row[TILE] - (int)row[TILE - 1])];
  } else {
    uint32_t pprev = box_pix(box, true, 1, lane);
    et = ns_weight(box_pix(box, true, 0, lane), pprev, g2);
    Wv[lane] = INF;
    {
      const float wx = ns_weight(__shfl_up_sync(~0u, pprev, 1), pprev, g2);
      Wh[lane] = lane == 0 ? INF : wx;
    }
#pragma unroll UNROLL
    for (int y = 1; y < TILE; ++y) {
      const uint32_t pcur = box_pix(box, true, y + 1, lane);
      const float w = ns_weight(pprev, pcur, g2);
      const float wx = ns_weight(__shfl_up_sync(~0u, pcur, 1), pcur, g2);
      Wv[y * W_STRIDE + lane] = w;
      Wh[y * W_STRIDE + lane] = lane == 0 ? INF : wx;
      if (lane < vw && y < vh) wsum += w;
      pprev = pcur;
    }
    eb = ns_weight(pprev, box_pix(box, true, TILE + 1, lane), g2);
    el = ns_weight(box_pix(box, true, lane + 1, -1), box_pix(box, true, lane + 1, 0), g2);
    er = ns_weight(box_pix(box, true, lane + 1, TILE - 1), box_pix(box, true, lane + 1, TILE), g2);
  }
  if (vw < TILE || vh < TILE) {  // edges touching a pixel outside the image are INF
#pragma unroll 1
    for (int y = 0; y < TILE; ++y)
      if (lane >= vw || y >= vh) {
        Wh[y * W_STRIDE + lane] = INF;
        Wv[y * W_STRIDE + lane] = INF;
      }
    if (lane >= vw) et = INF;
    if (lane >= vw || vh < TILE) eb = INF;
    if (lane >= vh) el = INF;
    if (lane >= vh || vw < TILE) er = INF;
  }
  E[E_LEFT + lane] = el;
  E[E_RIGHT + lane] = er;
  E[E_TOP + lane] = et;
  E[E_BOTTOM + lane] = eb;
  return wsum;
}

// ------------------------------------------------------------------------------------------------------
// ns-mode visit (C4, w = sqrt(1 + g2 * dI2)), gray or rgb8.
//
// The tile's distances are relaxed from the halo once (values only decrease while the halo is fixed, so the halo
// edges stay satisfied), then by rounds of diagonal sweeps (skew_round) until a round changes nothing: every edge
// of the tile and its halo is then satisfied.  A visit whose halo lowers nothing runs no round unless it applies
// seeds.  The halo is an upper bound of the neighbours' values (values only decrease; never-visited neighbours read
// as v), so the visit never undershoots the fixpoint.  A neighbour is re-activated only if some border pixel plus
// its edge weight is below the halo value it was compared with.
//
// The rounds run in one of two skewed layouts (A: the down-right and up-left quadrants, B: the other two); the visit
// starts in the one whose corners hold the smallest border value, where the front comes in, and changes after
// LAYOUT_ROUNDS rounds without convergence (about one visit in five; changing after 2 rounds saved 5 % of the
// rounds and cost four times the reloads).
// Returns the number of rounds and activations through *nph / *nact.
//
// rerun: the warp visits again the tile it has just visited (its halo dropped while it ran, and the visit kept
// it).  The warp's shared memory still holds that tile's edge weights (Wh / Wv / E) and its final distances (B, equal
// to the tile in global memory: no other warp can have visited it in between), so the
// re-run reloads only the neighbour states and halos: no bulk copy, no weights, no tile loads.
// ------------------------------------------------------------------------------------------------------
constexpr int LAYOUT_ROUNDS = 3;

template <bool PRESTAGED, class Sched>
__device__ __forceinline__ void visit_ns(const ImgDesc& dd, const CUtensorMap* tm_img, const CUtensorMap* tm_mask,
                                         uint32_t tile, uint32_t old_state, const VisitBufs& vb, const Sched& sch,
                                         uint32_t* nph_out, uint32_t* nact_out, bool rerun = false) {
  const int lane = threadIdx.x & 31;
  const float INF = f_inf();
  const uint32_t local = tile - dd.tile_base;
  const int tx = (int)(local % (uint32_t)dd.tiles_x), ty = (int)(local / (uint32_t)dd.tiles_x);
  const int x0 = tx * TILE, y0 = ty * TILE;
  const int vw = min(TILE, dd.width - x0), vh = min(TILE, dd.height - y0);
  rerun = uniform(rerun);
  const bool first = !(old_state & ST_VISITED);
  const bool seed = (old_state & ST_SEED) != 0;
  const bool rgb = uniform(dd.channels == 3);
  const float v = dd.v;
  *nph_out = 0;
  *nact_out = 0;

  if (rerun) {
  } else if (!PRESTAGED) {
    stage_tile(vb, tm_img, tm_mask, rgb, seed, x0, y0);
  } else if (seed) {
    stage_box(vb.mask, vb.mbar, tm_mask, TILE * TILE, x0, y0);
  }

  // Neighbour states: lane 0 left, 1 right, 2 top, 3 bottom.
  const uint32_t nexist = (tx > 0 ? 1u : 0u) | (tx + 1 < dd.tiles_x ? 2u : 0u) | (ty > 0 ? 4u : 0u) |
                          (ty + 1 < dd.tiles_y ? 8u : 0u);
  const int nbx = tx + (lane == 0 ? -1 : lane == 1 ? 1 : 0);
  const int nby = ty + (lane == 2 ? -1 : lane == 3 ? 1 : 0);
  const uint32_t nb_tile = dd.tile_base + (uint32_t)(nby * dd.tiles_x + nbx);  // meaningful for lanes < 4
  uint32_t nvis;
  {
    bool vis = false;
    if (lane < 4 && ((nexist >> lane) & 1u)) vis = (ld_volatile(&sch.states[nb_tile]) & ST_VISITED) != 0;
    nvis = __ballot_sync(~0u, vis);
  }
  fence_acq_rel();  // acquire: distances were written before the VISITED bits / the activation we saw

  // Halo: column layout for top/bottom (lane = x), row layout for left/right (lane = y).
  float top = INF, bot = INF, lft = INF, rgt = INF;
  if (lane < vw) {
    if (nexist & 4u) top = (nvis & 4u) ? ld_dist(dd, y0 - 1, x0 + lane) : v;
    if (nexist & 8u) bot = (nvis & 8u) ? ld_dist(dd, y0 + TILE, x0 + lane) : v;
  }
  if (lane < vh) {
    if (nexist & 1u) lft = (nvis & 1u) ? ld_dist(dd, y0 + lane, x0 - 1) : v;
    if (nexist & 2u) rgt = (nvis & 2u) ? ld_dist(dd, y0 + lane, x0 + TILE) : v;
  }

  // Tile distances (lane = x): v on a first visit, else copied behind the weights' back.  The fence above orders the
  // copies after what the neighbours' states say, like the halo loads.
  float* B = vb.t->B;
  const int rows = lane < vw ? vh : 0;  // this lane's rows of the picture
  if (!rerun) {
    const uint8_t* src = dist_base(dd, y0, x0 + lane, 0u);
#pragma unroll 2
    for (int y = 0; y < TILE; ++y) {
      float* dst = B + y * W_STRIDE + lane;
      if (first || y >= rows) *dst = y < rows ? v : INF;
      else cp_async4(dst, src + (int64_t)y * dd.dist_pitch);
    }
  }

  if (!tma_wait(vb.bar, *vb.pbits, vb.pmask, sch.q, tile, !rerun)) {
    cp_async_wait();
    return;
  }
  if (PRESTAGED && !tma_wait(vb.mbar, *vb.pbits, vb.mmask, sch.q, tile, seed)) {
    cp_async_wait();
    return;
  }

  // Seeds first: the mask box shares memory with Wv.
  uint32_t seeds = 0;  // this lane's column of the mask tile
  if (seed) {
    const uint8_t* mbox = reinterpret_cast<const uint8_t*>(vb.mask);
#pragma unroll 2
    for (int y = 0; y < TILE; ++y) seeds |= (y < rows && mbox[y * TILE + lane] != 0 ? 1u : 0u) << y;
  }
  __syncwarp();

  // Edge weights into Wh / Wv / E (lane = x; the left and right halo edges lane = y).  A re-run has them.
  const uint32_t img_idx = old_state >> ST_IMG_SHIFT;
  const float* E = vb.t->E;
  float wsum = 0.0f;
  if (!rerun) {
    wsum = tile_weights<1>(dd.g2, rgb, vw, vh, vb.box, vb.t->Wh, vb.t->Wv, vb.t->E);
    vb.t->Wv[TILE * W_STRIDE + lane] = INF;
    cp_async_wait();
    if (seed) {
#pragma unroll 2
      for (int y = 0; y < TILE; ++y)
        if ((seeds >> y) & 1u) B[y * W_STRIDE + lane] = 0.0f;
    }
  }
  __syncwarp();

  // The image's mean edge weight, for its bucket width: each first visit adds its column edges.
  if (sch.q.wacc && first) {
    float* wa = sch.q.wacc + 2 * img_idx;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) wsum += __shfl_xor_sync(~0u, wsum, o);
    if (lane == 0 && vh > 1) {
      atomicAdd(&wa[0], wsum);
      atomicAdd(&wa[1], (float)(vw * (vh - 1)));
    }
  }

  // Relax the halo edges in B: top and bottom lane = x, then left and right lane = y.
  bool any, layout_a;
  {
    const float ct = __fadd_rn(top, E[E_TOP + lane]), cb = __fadd_rn(bot, E[E_BOTTOM + lane]);
    float dt = B[lane], db = B[(TILE - 1) * W_STRIDE + lane];
    bool low = ct < dt || cb < db;
    dt = fminf(dt, ct);
    db = fminf(db, cb);
    B[lane] = dt;
    B[(TILE - 1) * W_STRIDE + lane] = db;
    __syncwarp();
    const float cl = __fadd_rn(lft, E[E_LEFT + lane]), cr = __fadd_rn(rgt, E[E_RIGHT + lane]);
    float dl = B[lane * W_STRIDE], dr = B[lane * W_STRIDE + TILE - 1];
    low |= cl < dl || cr < dr;
    dl = fminf(dl, cl);
    dr = fminf(dr, cr);
    B[lane * W_STRIDE] = dl;
    B[lane * W_STRIDE + TILE - 1] = dr;
    any = __any_sync(~0u, low);
    // The smallest border value near the corners of either diagonal (float bits order like the values, all >= 0).
    const float tl = fminf(dt, dl), br = fminf(db, dr);
    const uint32_t ka = __reduce_min_sync(~0u, __float_as_uint(lane < TILE / 2 ? tl : br));
    const uint32_t kb = __reduce_min_sync(~0u, __float_as_uint(lane < TILE / 2 ? fminf(db, dr) : fminf(dt, dl)));
    layout_a = ka <= kb;
    __syncwarp();
  }
  uint32_t nph = 0;
  if (any || seed) {
    for (;;) {
      const int off = layout_a ? (TILE - lane) % TILE : lane;
      const int src_f = (layout_a ? lane + TILE - 1 : lane + 1) % TILE, src_r = (layout_a ? lane + 1 : lane + TILE - 1) % TILE;
      float d[TILE], wh[TILE], wv[TILE];
      load_skew_tile(d, wh, wv, *vb.t, lane, off, layout_a);
      bool ch;
      int r = 0;
#pragma unroll 1  // one copy of the round: the kernel's code is fetched through small instruction caches
      do {
        ch = __any_sync(~0u, skew_round(d, wh, wv, src_f, src_r));
        any |= ch;
        ++nph;
      } while (ch && ++r < LAYOUT_ROUNDS);
      store_skew(B + lane * W_STRIDE, off, d);
      __syncwarp();
      if (!ch || nph >= (uint32_t)PHASE_LIMIT) break;
      layout_a = !layout_a;
    }
    if (nph >= (uint32_t)PHASE_LIMIT && lane == 0) set_error(sch.q, DERR_PHASE_LIMIT, tile);
  }

  // Neighbours that can still decrease (bit 0 left, 1 right, 2 top, 3 bottom).
  uint32_t act = 0;
  float act_key = 0.0f;
  if (any || seed) {
    const float dt = B[lane], db = B[(TILE - 1) * W_STRIDE + lane];               // column layout
    const float dl = B[lane * W_STRIDE], dr = B[lane * W_STRIDE + TILE - 1];      // row layout
    const float wt = E[E_TOP + lane], wb = E[E_BOTTOM + lane], wl = E[E_LEFT + lane], wr = E[E_RIGHT + lane];
    // The activation value of a side: the smallest border value it can bring (its priority in the queue).
    const float vl = __fadd_rn(dl, wl), vr = __fadd_rn(dr, wr), vt = __fadd_rn(dt, wt), vb = __fadd_rn(db, wb);
    const uint32_t kl = __reduce_min_sync(~0u, vl < lft ? __float_as_uint(vl) : KEY_NONE);
    const uint32_t kr = __reduce_min_sync(~0u, vr < rgt ? __float_as_uint(vr) : KEY_NONE);
    const uint32_t kt = __reduce_min_sync(~0u, vt < top ? __float_as_uint(vt) : KEY_NONE);
    const uint32_t kbm = __reduce_min_sync(~0u, vb < bot ? __float_as_uint(vb) : KEY_NONE);
    act = (kl != KEY_NONE ? 1u : 0u) | (kr != KEY_NONE ? 2u : 0u) | (kt != KEY_NONE ? 4u : 0u) |
          (kbm != KEY_NONE ? 8u : 0u);
    // A missing neighbour has an INF halo, and fl(d + w) < INF holds for any finite d: mask by existence.
    act &= nexist;
    act_key = __uint_as_float(lane == 0 ? kl : lane == 1 ? kr : lane == 2 ? kt : kbm);
  }

  // The bucket width, read here so that the write-back covers the trip.
  const float inv_width = bucket_inv_width(sch.q, img_idx);

  // Write back (each row is one coalesced 128-byte store).  A seed visit always does: it may have lowered a pixel that
  // lowers nothing else.
  if (any || first || seed) {
    {
      uint8_t* wb = dist_base(dd, y0, x0 + lane, nph);
#pragma unroll 4
      for (int y = 0; y < TILE; ++y)
        if (y < rows) *reinterpret_cast<float*>(wb + (int64_t)y * dd.dist_pitch) = B[y * W_STRIDE + lane];
    }
  }
  fence_acq_rel();  // release: distances before activations and before the VISITED bit
  __syncwarp();
  sch.complete(tile, (first ? ST_VISITED : 0u) | (seed ? ST_SEED : 0u), lane < 4 && ((act >> lane) & 1u), nb_tile,
               act_key, inv_width);
  *nph_out = nph;
  *nact_out = (uint32_t)__popc(act);
}

// ------------------------------------------------------------------------------------------------------
// ref-mode visit (C8, reference weight), gray only.
//
// The edges' |dI| are computed once per visit into four shared arrays (RefTile); the tile's distances are relaxed from
// the halo once (values only decrease while the halo is fixed), then by phases that alternate between two layouts.
// Column phase: lane = x, position k = y; every pixel is relaxed from its three predecessors in the row above (forward
// chain) and below (backward chain).  Row phase: lane = y, position k = x, likewise from the columns beside it.  These are
// the passes of the reference (dt/src/dt_block_passes.cuh:12-127) with the reference's arithmetic per edge; all edges of
// a phase are in registers, so a step of a chain is two shuffles, five fused multiply-adds and three minima.
// The visit ends at a phase that changes nothing if the edges along the other layout's chains, which it does not see,
// hold too (the diagonal edges belong to both layouts).
// ------------------------------------------------------------------------------------------------------
constexpr float REF_SQ2 = 1.41421354f;  // sqrtf(2.f), reference generalised_distance_transform.cu:111

// D + l_eucl * {1, sqrt2} + l_grad * |dI| (ref_relax) with the parts that depend on the source alone taken out: `axial` /
// `diagonal` of the source's distance, then `grad` with the edge's word (|dI|, or l_grad * |dI| rounded by itself
// without FMA).  An edge that does not exist has an infinite word, so its candidate is infinite, or NaN when l_grad is
// 0, and fminf and < pass over both.
// (the host's pass over the constructor, whose arguments do not depend on the template, does not know __fmul_rn)
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
template <bool FMA>
struct RefEdge {
  float le, lg, le2;
  __device__ __forceinline__ RefEdge(float l_eucl, float l_grad) : le(l_eucl), lg(l_grad), le2(mul_rn(l_eucl, REF_SQ2)) {}
  __device__ __forceinline__ float axial(float q) const { return __fadd_rn(q, le); }  // l_eucl * 1 is exact
  __device__ __forceinline__ float diagonal(float q) const { return FMA ? __fmaf_rn(le, REF_SQ2, q) : __fadd_rn(q, le2); }
  __device__ __forceinline__ float grad(float e, float t) const { return FMA ? __fmaf_rn(lg, e, t) : __fadd_rn(t, e); }
  __device__ __forceinline__ float word(uint32_t absdi) const {
    const float f = __uint2float_rn(absdi);
    return FMA ? f : __fmul_rn(lg, f);
  }
};

// Edge words of a tile from its staged image box into t.V / Hh / DL / DR / E.  Returns this lane's sum of the axial
// costs of the tile's internal column edges.
template <bool FMA>
__device__ __forceinline__ float ref_tile_weights(const RefEdge<FMA>& re, int vw, int vh, RefTile& t) {
  const int lane = threadIdx.x & 31;
  const float INF = f_inf();
  const uint8_t* col = t.img + 16 + lane;  // column `lane` of the box, row r at col[r * IMG_BOX_GRAY]
  auto ad = [](int a, int b) { return (uint32_t)abs(a - b); };
  float wsum = 0.0f;
  int ul = col[-1], u = col[0], ur = col[1];
  {
    const int c = col[IMG_BOX_GRAY];
    t.E[E_TOP * 3 + lane] = re.word(ad(c, ul));
    t.E[E_TOP * 3 + TILE + lane] = re.word(ad(c, u));
    t.E[E_TOP * 3 + 2 * TILE + lane] = re.word(ad(c, ur));
  }
#pragma unroll 2
  for (int y = 0; y < TILE; ++y) {
    const uint8_t* pc = col + (y + 1) * IMG_BOX_GRAY;
    const int l = pc[-1], c = pc[0], r = pc[1];
    const bool in = lane < vw && y < vh;
    const float wv = re.word(ad(c, u));
    t.V[y * RS + lane] = in && y > 0 ? wv : INF;
    t.Hh[y * RS + lane] = in && lane > 0 ? re.word(ad(c, l)) : INF;
    t.DL[y * RS + lane] = in && y > 0 && lane > 0 ? re.word(ad(c, ul)) : INF;
    t.DR[y * RS + lane] = in && y > 0 && lane + 1 < vw ? re.word(ad(c, ur)) : INF;
    if (in && y > 0) wsum += re.grad(wv, re.le);
    ul = l;
    u = c;
    ur = r;
  }
  {
    const uint8_t* pb = col + (TILE + 1) * IMG_BOX_GRAY;
    t.E[E_BOTTOM * 3 + lane] = re.word(ad(u, pb[-1]));
    t.E[E_BOTTOM * 3 + TILE + lane] = re.word(ad(u, pb[0]));
    t.E[E_BOTTOM * 3 + 2 * TILE + lane] = re.word(ad(u, pb[1]));
  }
  const uint8_t* row = t.img + (lane + 1) * IMG_BOX_GRAY + 16;  // row `lane`
  const int cl = row[0], cr = row[TILE - 1];
#pragma unroll
  for (int o = 0; o < 3; ++o) {
    t.E[E_LEFT * 3 + o * TILE + lane] = re.word(ad(cl, row[(o - 1) * IMG_BOX_GRAY - 1]));
    t.E[E_RIGHT * 3 + o * TILE + lane] = re.word(ad(cr, row[(o - 1) * IMG_BOX_GRAY + TILE]));
  }
  t.DR[lane * RS + TILE] = INF;  // read as the word before the next row's first
  t.DR[TILE * RS + lane] = INF;
  return wsum;
}

// Halo of a tile in registers: the sides (lane = position along the side) and the corners (every lane).
struct RefHalo {
  float l, r, t, b, tl, tr, bl, br;
};

// The three halo pixels beside position `lane` of a side whose own pixel is h: before, at and after it.
__device__ __forceinline__ void halo3(float (&o)[3], float h, float before, float after) {
  const int lane = threadIdx.x & 31;
  const float up = __shfl_up_sync(~0u, h, 1), dn = __shfl_down_sync(~0u, h, 1);
  o[0] = lane == 0 ? before : up;
  o[1] = h;
  o[2] = lane == TILE - 1 ? after : dn;
}

// Relaxes the tile's border pixels in T from the halo; whether one of them fell.
template <bool FMA>
__device__ __forceinline__ bool ref_halo_relax(const RefEdge<FMA>& re, float* T, const float* E, const RefHalo& h, int vw, int vh) {
  const int lane = threadIdx.x & 31;
  bool low = false;
  auto side = [&](float hh, float before, float after, const float* e, float* px, bool in) {
    float o[3];
    halo3(o, hh, before, after);
    const float c = fminf(fminf(re.grad(e[lane], re.diagonal(o[0])), re.grad(e[TILE + lane], re.axial(o[1]))),
                          re.grad(e[2 * TILE + lane], re.diagonal(o[2])));
    if (in && c < *px) {
      *px = c;
      low = true;
    }
  };
  side(h.t, h.tl, h.tr, E + E_TOP * 3, T + lane, lane < vw);
  side(h.b, h.bl, h.br, E + E_BOTTOM * 3, T + (TILE - 1) * RS + lane, lane < vw && vh == TILE);
  __syncwarp();
  side(h.l, h.tl, h.bl, E + E_LEFT * 3, T + lane * RS, lane < vh);
  side(h.r, h.tr, h.br, E + E_RIGHT * 3, T + lane * RS + TILE - 1, lane < vh && vw == TILE);
  low = __any_sync(~0u, low);
  __syncwarp();
  return low;
}

// The smallest value the tile's border can bring to each neighbour below the halo it was compared with: lane k returns
// neighbour k's (left, right, top, bottom, then the corners tl, tr, bl, br) as float bits, KEY_NONE if nothing.  In a
// tile of vw x vh < 32 pixels the last pixel of a side has no diagonal neighbour after it: its halo is infinite there, and
// any value would be below it (lane 31's goes to a corner, which exists or not as a whole).
template <bool FMA>
__device__ __forceinline__ uint32_t ref_border_keys(const RefEdge<FMA>& re, const float* T, const float* E, const RefHalo& h, int vw,
                                                    int vh) {
  const int lane = threadIdx.x & 31;
  uint32_t kc[4] = {KEY_NONE, KEY_NONE, KEY_NONE, KEY_NONE};  // tl, tr, bl, br
  auto side = [&](float hh, float before, float after, const float* e, float px, int len, uint32_t& k0, uint32_t& k2) -> uint32_t {
    float o[3];
    halo3(o, hh, before, after);
    const float c0 = re.grad(e[lane], re.diagonal(px)), c1 = re.grad(e[TILE + lane], re.axial(px)),
                c2 = re.grad(e[2 * TILE + lane], re.diagonal(px));
    uint32_t k = c1 < o[1] ? __float_as_uint(c1) : KEY_NONE;
    const uint32_t u0 = c0 < o[0] ? __float_as_uint(c0) : KEY_NONE;
    const uint32_t u2 = c2 < o[2] && (lane + 1 < len || lane == TILE - 1) ? __float_as_uint(c2) : KEY_NONE;
    if (lane == 0) k0 = min(k0, u0); else k = min(k, u0);
    if (lane == TILE - 1) k2 = min(k2, u2); else k = min(k, u2);
    return __reduce_min_sync(~0u, k);
  };
  const uint32_t kt = side(h.t, h.tl, h.tr, E + E_TOP * 3, T[lane], vw, kc[0], kc[1]);
  const uint32_t kb = side(h.b, h.bl, h.br, E + E_BOTTOM * 3, T[(TILE - 1) * RS + lane], vw, kc[2], kc[3]);
  const uint32_t kl = side(h.l, h.tl, h.bl, E + E_LEFT * 3, T[lane * RS], vh, kc[0], kc[2]);
  const uint32_t kr = side(h.r, h.tr, h.br, E + E_RIGHT * 3, T[lane * RS + TILE - 1], vh, kc[1], kc[3]);
  const uint32_t ktl = __reduce_min_sync(~0u, kc[0]), ktr = __reduce_min_sync(~0u, kc[1]);
  const uint32_t kbl = __reduce_min_sync(~0u, kc[2]), kbr = __reduce_min_sync(~0u, kc[3]);
  return lane == 0 ? kl : lane == 1 ? kr : lane == 2 ? kt : lane == 3 ? kb : lane == 4 ? ktl : lane == 5 ? ktr
       : lane == 6 ? kbl : lane == 7 ? kbr : KEY_NONE;
}

// One phase.  c[k]: edge between positions k - 1 and k of the own line; p[k] / n[k]: between position k of the own line and
// position k - 1 of line l - 1 / l + 1.  The forward chain takes its diagonal predecessors from the neighbouring lanes;
// in the backward chain the neighbours send their candidates, whose edges they hold.
template <bool FMA>
__device__ __forceinline__ bool ref_phase(const RefEdge<FMA>& re, float (&d)[TILE], const float (&c)[TILE], const float (&p)[TILE],
                                          const float (&n)[TILE]) {
  const int lane = threadIdx.x & 31;
  const int lo = (lane + TILE - 1) % TILE, hi = (lane + 1) % TILE;  // edges across the warp's ends are infinite
  bool ch = false;
#pragma unroll
  for (int s = 1; s < TILE; ++s) {
    {
      const int k = s;
      const float q = d[k - 1], g = re.diagonal(q);
      const float gl = __shfl_sync(~0u, g, lo), gr = __shfl_sync(~0u, g, hi);
      const float a = fminf(d[k], re.grad(c[k], re.axial(q)));
      const float v = fminf(a, fminf(re.grad(p[k], gl), re.grad(n[k], gr)));
      ch |= v < d[k];
      d[k] = v;
    }
    {
      const int k = TILE - 1 - s;
      const float q = d[k + 1], g = re.diagonal(q);
      const float fl = __shfl_sync(~0u, re.grad(n[k + 1], g), lo), fr = __shfl_sync(~0u, re.grad(p[k + 1], g), hi);
      const float a = fminf(d[k], re.grad(c[k + 1], re.axial(q)));
      const float v = fminf(a, fminf(fl, fr));
      ch |= v < d[k];
      d[k] = v;
    }
  }
  return __any_sync(~0u, ch);
}

// Loads the tile in the column or row layout.
__device__ __forceinline__ void ref_load_tile(float (&d)[TILE], const float* T, bool col) {
  const int lane = threadIdx.x & 31;
  if (col) {
#pragma unroll
    for (int k = 0; k < TILE; ++k) d[k] = T[k * RS + lane];
  } else {
#pragma unroll
    for (int k = 0; k < TILE; ++k) d[k] = T[lane * RS + k];
  }
}
__device__ __forceinline__ void ref_store_tile(float* T, const float (&d)[TILE], bool col) {
  const int lane = threadIdx.x & 31;
  if (col) {
#pragma unroll
    for (int k = 0; k < TILE; ++k) T[k * RS + lane] = d[k];
  } else {
#pragma unroll
    for (int k = 0; k < TILE; ++k) T[lane * RS + k] = d[k];
  }
}
__device__ __forceinline__ void ref_load_edges(float (&c)[TILE], float (&p)[TILE], float (&n)[TILE], const RefTile& t, bool col) {
  const int lane = threadIdx.x & 31;
  if (col) {
#pragma unroll
    for (int k = 0; k < TILE; ++k) {
      c[k] = t.V[k * RS + lane];
      p[k] = t.DL[k * RS + lane];
      n[k] = t.DR[k * RS + lane];
    }
  } else {
#pragma unroll
    for (int k = 0; k < TILE; ++k) {
      c[k] = t.Hh[lane * RS + k];
      p[k] = t.DL[lane * RS + k];
      n[k] = t.DR[(lane + 1) * RS + k - 1];  // (x - 1, y + 1) - (x, y), kept with its lower pixel
    }
  }
}

// Whether an edge along the chains (c) of this layout can lower a pixel.
template <bool FMA>
__device__ __forceinline__ bool ref_chain_low(const RefEdge<FMA>& re, const float (&d)[TILE], const float* row, int stride) {
  bool low = false;
#pragma unroll
  for (int k = 1; k < TILE; ++k) {
    const float e = row[k * stride];
    low |= re.grad(e, re.axial(d[k - 1])) < d[k] || re.grad(e, re.axial(d[k])) < d[k - 1];
  }
  return __any_sync(~0u, low);
}

// Runs phases over the tile in t.img (T), a column phase first, until it is converged or PHASE_LIMIT phases have run; nph
// counts them.  Whether the tile is not converged; `changed` is set when a value fell.
template <bool FMA>
__device__ __forceinline__ bool ref_solve(const RefEdge<FMA>& re, RefTile& t, uint32_t& nph, bool& changed) {
  const int lane = threadIdx.x & 31;
  float* T = reinterpret_cast<float*>(t.img);
  float d[TILE], c[TILE], p[TILE], n[TILE];
  bool col = true;
  ref_load_tile(d, T, col);
  for (;;) {
    ref_load_edges(c, p, n, t, col);
    const bool ch = ref_phase<FMA>(re, d, c, p, n);
    changed |= ch;
    ++nph;
    if (ch) {
      ref_store_tile(T, d, col);
      __syncwarp();
    }
    col = !col;
    ref_load_tile(d, T, col);
    __syncwarp();
    // A phase without change: the other layout's chain edges decide.
    if (!ch && !ref_chain_low<FMA>(re, d, col ? t.V + lane : t.Hh + lane * RS, col ? RS : 1)) return false;
    if (nph >= (uint32_t)PHASE_LIMIT) return true;
  }
}

// Distances of a neighbour k (left, right, top, bottom, corners) at pixel (gx, gy): INF where there is no pixel, v where
// the neighbour has not been visited.
__device__ __forceinline__ float ref_halo_value(const ImgDesc& dd, uint32_t nexist, uint32_t nvis, int k, int gx, int gy, float v) {
  if (!((nexist >> k) & 1u) || gx >= dd.width || gy >= dd.height) return f_inf();
  return ((nvis >> k) & 1u) ? ld_dist(dd, gy, gx) : v;
}

template <bool FMA, class Sched>
__device__ __forceinline__ void visit_ref(const ImgDesc& dd, const CUtensorMap* tm_img, const CUtensorMap* tm_mask,
                                          uint32_t tile, uint32_t old_state, RefTile& sm, uint32_t& parity,
                                          const Sched& sch, uint32_t* nph_out, uint32_t* nact_out,
                                          bool rerun = false) {
  // rerun: as in visit_ns -- the edge words and the tile values (T) of this tile's previous visit are still in the warp's
  // shared memory; only the neighbour states and halos are read again.
  *nph_out = 0;
  *nact_out = 0;
  const int lane = threadIdx.x & 31;
  const float INF = f_inf();
  const uint32_t local = tile - dd.tile_base;
  const int tx = (int)(local % (uint32_t)dd.tiles_x), ty = (int)(local / (uint32_t)dd.tiles_x);
  const int x0 = tx * TILE, y0 = ty * TILE;
  const int vw = min(TILE, dd.width - x0), vh = min(TILE, dd.height - y0);
  rerun = uniform(rerun);
  const bool first = !(old_state & ST_VISITED);
  const bool seed = (old_state & ST_SEED) != 0;
  const float v = dd.v;
  const RefEdge<FMA> re(dd.l_eucl, dd.l_grad);

  const VisitBufs vb{sm.img, sm.V, nullptr, &sm.bar, &sm.bar, 1u, 1u, &parity};
  if (!rerun) stage_tile(vb, tm_img, tm_mask, false, seed, x0, y0);

  // Neighbour k = lane (0..7): (dx, dy) = L, R, T, B, TL, TR, BL, BR.
  // Offsets of neighbour k = lane, the tables {-1,1,0,0,-1,1,-1,1} and {0,0,-1,1,-1,-1,1,1} as bit masks (an
  // array indexed by the lane would live in local memory).
  const int ndx_l = (0xF3u >> lane) & 1u ? ((0xA2u >> lane) & 1u ? 1 : -1) : 0;
  const int ndy_l = (0xFCu >> lane) & 1u ? ((0xC8u >> lane) & 1u ? 1 : -1) : 0;
  uint32_t nvis, nexist;
  {
    bool vis = false, ex = false;
    if (lane < 8) {
      const int nx = tx + ndx_l, ny = ty + ndy_l;
      ex = nx >= 0 && ny >= 0 && nx < dd.tiles_x && ny < dd.tiles_y;
      if (ex) vis = (ld_volatile(&sch.states[dd.tile_base + (uint32_t)(ny * dd.tiles_x + nx)]) & ST_VISITED) != 0;
    }
    nvis = __ballot_sync(~0u, vis);
    nexist = __ballot_sync(~0u, ex);
  }
  fence_acq_rel();

  RefHalo h;
  h.t = lane < vw ? ref_halo_value(dd, nexist, nvis, 2, x0 + lane, y0 - 1, v) : INF;
  h.b = lane < vw ? ref_halo_value(dd, nexist, nvis, 3, x0 + lane, y0 + TILE, v) : INF;
  h.l = lane < vh ? ref_halo_value(dd, nexist, nvis, 0, x0 - 1, y0 + lane, v) : INF;
  h.r = lane < vh ? ref_halo_value(dd, nexist, nvis, 1, x0 + TILE, y0 + lane, v) : INF;
  h.tl = ref_halo_value(dd, nexist, nvis, 4, x0 - 1, y0 - 1, v);
  h.tr = ref_halo_value(dd, nexist, nvis, 5, x0 + TILE, y0 - 1, v);
  h.bl = ref_halo_value(dd, nexist, nvis, 6, x0 - 1, y0 + TILE, v);
  h.br = ref_halo_value(dd, nexist, nvis, 7, x0 + TILE, y0 + TILE, v);

  float* T = reinterpret_cast<float*>(sm.img);  // overlays the image box once the edge words are computed
  float wsum = 0.0f;
  float d[TILE];
  if (!rerun && !first) {
    const uint8_t* lb = dist_base(dd, y0, x0 + lane, 0u);
#pragma unroll
    for (int y = 0; y < TILE; ++y) d[y] = (lane < vw && y < vh) ? ld_dist_at(lb, dd.dist_pitch, y) : INF;
  }
  if (!tma_wait(&sm.bar, parity, 1u, sch.q, tile, !rerun)) return;
  if (!rerun) {
    uint32_t seeds = 0;  // this lane's column of the mask tile (its box shares memory with V)
    if (seed) {
      const uint8_t* mbox = reinterpret_cast<const uint8_t*>(sm.V);
#pragma unroll 4
      for (int y = 0; y < TILE; ++y) seeds |= (lane < vw && y < vh && mbox[y * TILE + lane] != 0 ? 1u : 0u) << y;
    }
    __syncwarp();
    wsum = ref_tile_weights<FMA>(re, vw, vh, sm);
    __syncwarp();
    if (first) {
#pragma unroll 4
      for (int y = 0; y < TILE; ++y) T[y * RS + lane] = (lane < vw && y < vh) ? (((seeds >> y) & 1u) ? 0.0f : v) : INF;
    } else {
#pragma unroll
      for (int y = 0; y < TILE; ++y) T[y * RS + lane] = ((seeds >> y) & 1u) ? 0.0f : d[y];
    }
    __syncwarp();
  }
  if constexpr (Sched::any_change) {  // the border as it was, lane = position along the side
    sm.B0[E_TOP + lane] = T[lane];
    sm.B0[E_BOTTOM + lane] = T[(TILE - 1) * RS + lane];
    sm.B0[E_LEFT + lane] = T[lane * RS];
    sm.B0[E_RIGHT + lane] = T[lane * RS + TILE - 1];
    __syncwarp();
  }

  // The image's mean axial edge cost, for its bucket width: each first visit adds its vertical edges.
  if (sch.q.wacc && first) {
    float* wa = sch.q.wacc + 2 * (old_state >> ST_IMG_SHIFT);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) wsum += __shfl_xor_sync(~0u, wsum, o);
    if (lane == 0 && vh > 1) {
      atomicAdd(&wa[0], wsum);
      atomicAdd(&wa[1], (float)(vw * (vh - 1)));
    }
  }

  bool any = ref_halo_relax<FMA>(re, T, sm.E, h, vw, vh);
  uint32_t nph = 0;
  if (any || seed) {
    if (ref_solve<FMA>(re, sm, nph, any) && lane == 0) set_error(sch.q, DERR_PHASE_LIMIT, tile);
  }

  // Neighbours to activate (bit k = neighbour k as in ndx_l / ndy_l) and the value each is activated at: the ones the
  // border can lower; in host-driven rounds the ones whose facing border changed (dt_block_passes.cuh:50-63), so that
  // the round counters count what the reference's do.
  uint32_t act = 0;
  float key = 0.0f;
  if (any || seed) {
    if constexpr (Sched::any_change) {
      const uint32_t ct = __ballot_sync(~0u, seed || T[lane] != sm.B0[E_TOP + lane]);
      const uint32_t cb = __ballot_sync(~0u, seed || T[(TILE - 1) * RS + lane] != sm.B0[E_BOTTOM + lane]);
      const uint32_t cl = __ballot_sync(~0u, seed || T[lane * RS] != sm.B0[E_LEFT + lane]);
      const uint32_t cr = __ballot_sync(~0u, seed || T[lane * RS + TILE - 1] != sm.B0[E_RIGHT + lane]);
      act = (cl ? 1u : 0u) | (cr ? 2u : 0u) | (ct ? 4u : 0u) | (cb ? 8u : 0u) | ((ct & 1u) ? 16u : 0u) |
            ((ct >> (TILE - 1)) & 1u ? 32u : 0u) | ((cb & 1u) ? 64u : 0u) | ((cb >> (TILE - 1)) & 1u ? 128u : 0u);
    } else {
      const uint32_t k = ref_border_keys<FMA>(re, T, sm.E, h, vw, vh);
      act = __ballot_sync(~0u, k != KEY_NONE);
      key = __uint_as_float(k);
    }
    act &= nexist;
  }

  const float inv_width = bucket_inv_width(sch.q, old_state >> ST_IMG_SHIFT);
  if (any || first || seed) {
    if (lane < vw) {
      uint8_t* wb = dist_base(dd, y0, x0 + lane, nph);
#pragma unroll 4
      for (int y = 0; y < TILE; ++y)
        if (y < vh) *reinterpret_cast<float*>(wb + (int64_t)y * dd.dist_pitch) = T[y * RS + lane];
    }
  }
  fence_acq_rel();
  __syncwarp();
  const bool want = lane < 8 && ((act >> lane) & 1u);
  const uint32_t item = want ? dd.tile_base + (uint32_t)((ty + ndy_l) * dd.tiles_x + tx + ndx_l) : 0u;
  sch.complete(tile, (first ? ST_VISITED : 0u) | (seed ? ST_SEED : 0u), want, item, key, inv_width);
  *nph_out = nph;
  *nact_out = (uint32_t)__popc(act);
}

// MODE is fixed per kernel instantiation: a launch covers images of one weight mode (and, in ref-mode, one
// rounding) only, so no kernel's register allocation is inflated by another mode's code.
template <int MODE>
using TileSmem = std::conditional_t<MODE == MODE_NS, WarpSmem, RefTile>;  // a warp's shared memory

template <int MODE, class Sched>
__device__ __forceinline__ void visit_tile(const ImgDesc& dd, const CUtensorMap* tmaps, uint32_t img, uint32_t tile,
                                           uint32_t old_state, TileSmem<MODE>& sm, uint32_t& parity, const Sched& sch,
                                           WarpStats& ws, bool rerun = false) {
  const CUtensorMap* tm_img = tmaps + 2 * img;
  const CUtensorMap* tm_mask = tmaps + 2 * img + 1;
  uint32_t nph, nact;
  if constexpr (MODE == MODE_NS)
    visit_ns<false>(dd, tm_img, tm_mask, tile, old_state, visit_bufs(sm, parity), sch, &nph, &nact, rerun);
  else if constexpr (MODE == MODE_REF)
    visit_ref<true>(dd, tm_img, tm_mask, tile, old_state, sm, parity, sch, &nph, &nact, rerun);
  else
    visit_ref<false>(dd, tm_img, tm_mask, tile, old_state, sm, parity, sch, &nph, &nact, rerun);
  count_visit(ws, sch.q, nph, nact);
}

template <class Smem = WarpSmem>
__device__ __forceinline__ Smem& warp_slot(uint8_t* smem_raw) {
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
  return reinterpret_cast<Smem*>(base)[threadIdx.x >> 5];
}

template <class Smem>
__device__ __forceinline__ void warp_slot_init(Smem& sm) {
  if ((threadIdx.x & 31) == 0) {
    mbar_init(&sm.bar, 1);
    fence_mbar_init();
  }
  __syncwarp();
}

__device__ __forceinline__ WarpSmemP& warp_slot_p(uint8_t* smem_raw) {
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
  return reinterpret_cast<WarpSmemP*>(base)[threadIdx.x >> 5];
}

__device__ __forceinline__ void warp_slot_init(WarpSmemP& sm) {
  if ((threadIdx.x & 31) == 0) {
    mbar_init(&sm.bar[0], 1);
    mbar_init(&sm.bar[1], 1);
    mbar_init(&sm.mbar, 1);
    fence_mbar_init();
  }
  __syncwarp();
}

// Image of a global tile id: binary search over the prefix array tile_base[0..n].
__device__ __forceinline__ uint32_t image_of_tile(const uint32_t* tile_base, int n, uint32_t t) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (tile_base[mid] <= t) lo = mid; else hi = mid - 1;
  }
  return (uint32_t)lo;
}

}  // namespace dtb
