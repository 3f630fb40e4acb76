// dtb_block.cuh -- the block kernel: a CTA per block of 2x2 tiles, for work that does not fill the GPU.
//
// With few tiles the time of a run is the length of its longest chain of dependent tile visits, and a visit through
// the tile queue (dtb_kernels.cuh) costs about 20,000 cycles of round trips around 4,000 cycles of sweeps: staging,
// weights, write-back, activation, queue.  Here the warps of a CTA hold the tiles of a block in shared memory, and a
// front crosses from tile to tile inside the block by shared memory alone; the round trips are paid once per block.
// Each block belongs to one CTA (block b to CTA b mod grid) and has one message word per side, written by the owner of
// the neighbouring block alone: a CTA polls the words of its own blocks, so there is no ring, no ticket and no atomic
// on the way from one block to the next, and a CTA whose last block is activated again finds the block's weights and
// distances still in shared memory.  A visit that finds them there takes about 16,000 cycles for 64 pixels of front,
// three quarters of it sweeps.  The seed scan and the fill of unreached blocks are part of the kernel.
#pragma once

#include "dtb_kernels.cuh"

namespace dtb {

constexpr int BLOCK_WARPS = BLOCK_TX * BLOCK_TY;
constexpr int BLOCK_OWNED_MAX = 32;                // blocks of one CTA at most
// Rounds a tile runs before its neighbours look at it: two complete a full sweep (1 and 3 were 25 % and 8 % slower on
// 2048^2 gray).
constexpr int BLOCK_ROUNDS = 2;
constexpr uint32_t BLOCK_CAP_CHECK = 16;           // visits of a CTA between its looks at the visit cap

struct alignas(128) BlockTile {
  uint8_t img[IMG_REGION];   // image box, then the tile buffer B[y * 34 + x]
  float Wh[TILE * W_STRIDE];
  float Wv[TILE * W_STRIDE];  // its first 1 KB receives the seed-mask box before the weights
  float E[4 * TILE];          // weights of the edges to the halo, per side
  float H[4 * TILE];          // halo of the sides that lie on the block's border (INF on the others), per side
  uint64_t bar;
};
constexpr int BLOCK_SIDES = 4;  // left, right, top, bottom
// Offset to the neighbour on side k (tables as bit masks: no array in local memory), and the side it sees us on.
__device__ __forceinline__ int side_dx(int k) { return (0x3 >> k) & 1 ? ((0x2 >> k) & 1 ? 1 : -1) : 0; }
__device__ __forceinline__ int side_dy(int k) { return (0xC >> k) & 1 ? ((0x8 >> k) & 1 ? 1 : -1) : 0; }
__device__ __forceinline__ int side_back(int k) { return k ^ 1; }

struct BlockCtl {
  uint32_t owned_img[BLOCK_OWNED_MAX];
  uint32_t sent[BLOCK_OWNED_MAX][BLOCK_SIDES];  // activations sent over each side of the owned blocks
  uint32_t seen[BLOCK_SIDES][BLOCK_OWNED_MAX];  // activations answered, per side
  uint32_t visited[BLOCK_OWNED_MAX / 32];  // bit i: owned block i has been visited
  uint32_t seeded[BLOCK_OWNED_MAX / 32];   // bit i: owned block i holds seeds not applied yet
  uint32_t next;       // index of the owned block to visit, or POP_NONE
  uint32_t first, seed, rerun;  // of this visit: no earlier visit; apply seeds; shared memory holds the block
  uint32_t nvis;       // bit k: the neighbouring block on side k holds valid distances
  uint32_t tokens;     // tokens the visit gives back at its end
  uint32_t side[BLOCK_SIDES];  // smallest value each side can bring to the neighbouring block (float bits), KEY_NONE if none
  uint32_t visits;     // tiles swept in this visit
  uint32_t done;       // visits of this CTA
  uint32_t phases, activations;  // counters of the run
  uint32_t img;        // the block's image
  ImgDesc desc;
};
struct BlockSmem {
  BlockTile tile[BLOCK_WARPS];
  BlockCtl ctl;
};
constexpr size_t BLOCK_SMEM = sizeof(BlockSmem) + 128;
static_assert(BLOCK_CTAS_MANY * (BLOCK_SMEM + 1024) <= 228 * 1024, "the blocks of an SM must fit its shared memory");

// Device words of a run.
struct BlockRun {
  QueueHdr* hdr;         // pending: tokens in use less `total`; the run has ended when all are back.  Every block starts
                         // out with one token, every activation under way carries one, and a visit holds four more
                         // from its start for those it may send: so the count never reaches zero early.
  uint2* msg;            // per block and side, from the neighbour there: x = 2 * activations sent + 1 (0: the neighbour
                         // has not been visited), y = the smallest value the last one brings (float bits)
  const uint32_t* base;  // block prefix of the images
  int n;                 // images
  uint32_t total;        // blocks
  uint32_t max_visits;
  uint64_t timeout_ns;
};

__device__ __forceinline__ uint4 ld_volatile4(const uint4* p) {
  uint4 v;
  asm volatile("ld.volatile.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

__device__ __forceinline__ void block_error(const BlockRun& a, uint32_t code, uint32_t info) {
  if (atomicCAS(&a.hdr->error.v, 0u, code) == 0u) atomicExch(&a.hdr->err_info.v, info);
}

// Waits until one of the CTA's blocks is to be visited and claims it (warp 0).  The block visited last comes first
// (its visit needs no staging), then the one with the smallest activation value.  Bounded: end of the run / error /
// watchdog.
__device__ __forceinline__ void block_next(const BlockRun& a, const ImgDesc* __restrict__ descs, BlockCtl& ctl, uint32_t first,
                                           uint32_t step, int count, uint32_t prev) {
  const int lane = threadIdx.x & 31;
  uint64_t t_check = globaltimer(), t_prog = t_check;
  uint32_t last = ld_volatile(&a.hdr->progress.v);
  for (;;) {
    // Each lane looks at every 32nd block: its best one, and the messages of that.
    uint32_t key = KEY_NONE, pick = POP_NONE, got[BLOCK_SIDES] = {};
    bool stop = ld_volatile(&a.hdr->pending.v) + a.total == 0u;
    // After an error no block is claimed any more, ready or not.  The word is on a line that nobody writes, so its load
    // comes back with the messages' (with the check of the copies in the visit, 512^2 gray takes 158.2 us instead of 157.9
    // and the 4096^2 maze 3.61 ms instead of 3.60).
    const uint32_t failed = ld_volatile(&a.hdr->error.v);
#pragma unroll 4
    for (int i = lane; i < count; i += 32) {
      const uint4* mine = reinterpret_cast<const uint4*>(a.msg + (uint64_t)BLOCK_SIDES * (first + (uint32_t)i * step));
      uint4 m[BLOCK_SIDES / 2];
#pragma unroll
      for (int s = 0; s < BLOCK_SIDES / 2; ++s) m[s] = ld_volatile4(mine + s);
      uint32_t k = KEY_NONE;
      bool ready = false;
      auto side = [&](uint32_t x, uint32_t y, int s) {
        if ((x >> 1) != ctl.seen[s][i]) {
          ready = true;
          k = min(k, y);
        }
      };
#pragma unroll
      for (int s = 0; s < BLOCK_SIDES / 2; ++s) {
        side(m[s].x, m[s].y, 2 * s);
        side(m[s].z, m[s].w, 2 * s + 1);
      }
      if ((ctl.seeded[i >> 5] >> lane) & 1u) {
        ready = true;
        k = 0u;
      }
      if (ready && ((uint32_t)i == prev || pick == POP_NONE || (pick != prev && k < key))) {
        key = k;
        pick = (uint32_t)i;
#pragma unroll
        for (int s = 0; s < BLOCK_SIDES / 2; ++s) {
          got[2 * s] = m[s].x;
          got[2 * s + 1] = m[s].z;
        }
      }
    }
    stop |= failed != 0u;
    if (__any_sync(~0u, pick != POP_NONE && !failed)) {
      // The block visited last, else the smallest value.
      if (pick == prev && pick != POP_NONE) key = 0u;
      const uint32_t best = __reduce_min_sync(~0u, pick == POP_NONE ? KEY_NONE : key);
      const uint32_t own = __ballot_sync(~0u, pick != POP_NONE && pick == prev);
      const int win = __ffs(own ? own : __ballot_sync(~0u, pick != POP_NONE && key == best)) - 1;
      if (!own) {
        // The visit's descriptor and tensor maps are read through this index: a map that is none would end in a device fault.
        const uint32_t img = ctl.owned_img[__shfl_sync(~0u, pick, win)];
        if (img >= (uint32_t)a.n) {
          if (lane == win) {
            block_error(a, DERR_BAD_TILE, pick);
            ctl.next = POP_NONE;
          }
          return;
        }
        if (lane == 0) ctl.img = img;
        const uint32_t* src = reinterpret_cast<const uint32_t*>(&descs[img]);
        uint32_t* dst = reinterpret_cast<uint32_t*>(&ctl.desc);
        for (int i = lane; i < (int)(sizeof(ImgDesc) / 4); i += 32) dst[i] = src[i];
        __syncwarp();
      }
      if (lane == win) {
        atomicAdd(&a.hdr->pending.v, (uint32_t)BLOCK_SIDES);
        uint32_t fresh = 0, nvis = 0;
#pragma unroll
        for (int s = 0; s < BLOCK_SIDES; ++s) {
          fresh += (got[s] >> 1) - ctl.seen[s][pick];
          nvis |= (got[s] ? 1u : 0u) << s;
          ctl.seen[s][pick] = got[s] >> 1;
        }
        const uint32_t bit = 1u << (pick & 31u), seed = ctl.seeded[pick >> 5] & bit;
        const bool warm = ctl.desc.warm != 0;
        ctl.nvis = warm ? ~0u : nvis;
        ctl.next = pick;
        ctl.tokens = (uint32_t)BLOCK_SIDES + fresh + (seed ? 1u : 0u);
        ctl.seed = seed ? 1u : 0u;
        ctl.first = warm || (ctl.visited[pick >> 5] & bit) ? 0u : 1u;
        ctl.rerun = pick == prev && !seed ? 1u : 0u;
        ctl.visited[pick >> 5] |= bit;
        ctl.seeded[pick >> 5] &= ~bit;
      }
      __syncwarp();
      fence_acq_rel();  // acquire, for the CTA: the messages before the neighbours' distances
      return;
    }
    const uint64_t now = globaltimer();
    if (now - t_check > POLL_CHECK_NS) {
      t_check = now;
      const uint32_t prog = ld_volatile(&a.hdr->progress.v);
      if (lane == 0 && !failed) {
        if (prog > a.max_visits) {
          block_error(a, DERR_VISIT_LIMIT, prog);
          stop = true;
        } else if (prog == last && now - t_prog > a.timeout_ns) {
          block_error(a, DERR_QUEUE_TIMEOUT, first);
          stop = true;
        }
      }
      if (prog != last) {
        last = prog;
        t_prog = now;
      }
    }
    if (__any_sync(~0u, stop)) {
      if (lane == 0) ctl.next = POP_NONE;
      return;
    }
  }
}

// End of a visit of block `blk` (warp 0, after the CTA's barrier): each side's lane tells the neighbouring block there, if
// there is one, that this block has been visited, and activates it if the visit found a value to bring (ctl.side).
__device__ __forceinline__ void block_complete(const BlockRun& a, BlockCtl& ctl, uint32_t blk) {
  const int lane = threadIdx.x & 31;
  const ImgDesc& dd = ctl.desc;
  const int bxn = dd.blocks_x, local = (int)(blk - dd.block_base), bx = local % bxn, by = local / bxn;
  const int nx = bx + side_dx(lane & 3), ny = by + side_dy(lane & 3);
  const bool exists = lane < BLOCK_SIDES && nx >= 0 && nx < bxn && ny >= 0 && ny < dd.blocks_y;
  const uint32_t key = lane < BLOCK_SIDES ? ctl.side[lane] : KEY_NONE;
  const bool want = exists && key != KEY_NONE;
  fence_acq_rel();  // release: the CTA's distances (and the visit's spare tokens) before the messages
  const uint32_t nsent = __popc(__ballot_sync(~0u, want));
  if (want || (exists && ctl.first)) {
    const uint32_t nb = dd.block_base + (uint32_t)(ny * bxn + nx);
    const uint32_t n = ctl.sent[ctl.next][lane] + (want ? 1u : 0u);
    ctl.sent[ctl.next][lane] = n;
    asm volatile("st.volatile.global.v2.u32 [%0], {%1, %2};" ::"l"(a.msg + (uint64_t)BLOCK_SIDES * nb + side_back(lane)), "r"(2u * n + 1u),
                 "r"(key)
                 : "memory");
  }
  if (lane < BLOCK_SIDES) ctl.side[lane] = KEY_NONE;
  if (lane == 0) {
    atomicSub(&a.hdr->pending.v, ctl.tokens - nsent);
    // The visit cap, also for a CTA that never waits: one look every BLOCK_CAP_CHECK visits (the add's way back costs a trip).
    if (++ctl.done % BLOCK_CAP_CHECK == 0u) {
      const uint32_t prog = atomicAdd(&a.hdr->progress.v, max(ctl.visits, 1u));
      if (prog > a.max_visits) block_error(a, DERR_VISIT_LIMIT, prog);
    } else {
      atomicAdd(&a.hdr->progress.v, max(ctl.visits, 1u));
    }
    ctl.visits = 0;
    ctl.activations += nsent;
  }
}

// Place of a warp's tile of block `blk`: origin, valid size, and its sides: bits 0..3 a neighbouring tile exists (left,
// right, top, bottom), bits 4..7 it lies in the same block, bits 8..11 in another one; bit 12 the tile itself exists.
struct BlockPlace {
  int x0, y0, vw, vh;
  uint32_t sides;
};
__device__ __forceinline__ BlockPlace block_place(const ImgDesc& dd, uint32_t blk) {
  const int warp = (int)uniform(threadIdx.x >> 5), wx = warp % BLOCK_TX, wy = warp / BLOCK_TX;
  const uint32_t local = blk - dd.block_base;
  BlockPlace p;
  p.x0 = (int)(local % (uint32_t)dd.blocks_x) * BLOCK_W + wx * TILE;
  p.y0 = (int)(local / (uint32_t)dd.blocks_x) * BLOCK_H + wy * TILE;
  p.vw = max(0, min(TILE, dd.width - p.x0));
  p.vh = max(0, min(TILE, dd.height - p.y0));
  p.sides = 0;
  if (p.vw > 0 && p.vh > 0) {
    const uint32_t ex = (p.x0 > 0 ? 1u : 0u) | (p.x0 + TILE < dd.width ? 2u : 0u) | (p.y0 > 0 ? 4u : 0u) |
                        (p.y0 + TILE < dd.height ? 8u : 0u);
    const uint32_t in = (wx > 0 ? 1u : 0u) | (wx + 1 < BLOCK_TX ? 2u : 0u) | (wy > 0 ? 4u : 0u) | (wy + 1 < BLOCK_TY ? 8u : 0u);
    p.sides = ex | (ex & in) << 4 | (ex & ~in) << 8 | 1u << 12;
  }
  return p;
}

// Writes the warp's tile to memory (row by row, coalesced).
__device__ __forceinline__ void block_store_tile(const ImgDesc& dd, const BlockPlace& p, const float* B) {
  const int lane = threadIdx.x & 31;
  if (lane < p.vw) {
    uint8_t* wb = dist_base(dd, p.y0, p.x0 + lane, 0u);
    const int64_t pitch = dd.dist_pitch;
#pragma unroll 4
    for (int y = 0; y < TILE; ++y)
      if (y < p.vh) *reinterpret_cast<float*>(wb + (int64_t)y * pitch) = B[y * W_STRIDE + lane];
  }
}

// Writes the lines of the warp's tile that lie on the block's border (`outer`: left, right, top, bottom) to memory.
__device__ __forceinline__ void block_store_border(const ImgDesc& dd, const BlockPlace& p, uint32_t outer, const float* B) {
  const int lane = threadIdx.x & 31;
  if (lane < p.vh) {
    float* row = dist_row(dd, p.y0 + lane) + p.x0;
    if (outer & 1u) row[0] = B[lane * W_STRIDE];
    if (outer & 2u) row[TILE - 1] = B[lane * W_STRIDE + TILE - 1];
  }
  if (lane < p.vw) {
    if (outer & 4u) dist_row(dd, p.y0)[p.x0 + lane] = B[lane];
    if (outer & 8u) dist_row(dd, p.y0 + TILE - 1)[p.x0 + lane] = B[(TILE - 1) * W_STRIDE + lane];
  }
}

// The warp's tile from memory (lane = x).
__device__ __forceinline__ void block_load_tile(const ImgDesc& dd, const BlockPlace& p, float (&d)[TILE]) {
  const int lane = threadIdx.x & 31;
  const uint8_t* lb = dist_base(dd, p.y0, p.x0 + lane, 0u);
  const int64_t pitch = dd.dist_pitch;
#pragma unroll
  for (int y = 0; y < TILE; ++y) d[y] = (lane < p.vw && y < p.vh) ? ld_dist_at(lb, pitch, y) : f_inf();
}

// Fills the warp's tile (distances, weights) from its staged boxes and, unless `first`, its distances d; whether a seed
// lowered a pixel.
__device__ __forceinline__ bool block_fill_ns(const ImgDesc& dd, const BlockPlace& p, BlockTile& t, bool first, bool seed,
                                              const float (&d)[TILE]) {
  const int lane = threadIdx.x & 31;
  const float INF = f_inf();
  uint32_t seeds = 0;  // this lane's column of the mask tile
  if (seed) {
    const uint8_t* mbox = reinterpret_cast<const uint8_t*>(t.Wv);
#pragma unroll 4
    for (int y = 0; y < TILE; ++y) seeds |= (lane < p.vw && y < p.vh && mbox[y * TILE + lane] != 0 ? 1u : 0u) << y;
  }
  __syncwarp();
  tile_weights<2>(dd.g2, uniform(dd.channels == 3), p.vw, p.vh, t.img, t.Wh, t.Wv, t.E);
  __syncwarp();
  float* pb = reinterpret_cast<float*>(t.img) + lane;
  if (first) {
    const float v = dd.v;
#pragma unroll 4
    for (int y = 0; y < TILE; ++y)
      pb[y * W_STRIDE] = (lane < p.vw && y < p.vh) ? (((seeds >> y) & 1u) ? 0.0f : v) : INF;
    return __any_sync(~0u, seeds != 0u);
  }
  bool low = false;  // a seed on a pixel that is 0 already asks for nothing
#pragma unroll
  for (int y = 0; y < TILE; ++y) {
    const bool s = ((seeds >> y) & 1u) != 0u;
    low |= s && d[y] > 0.0f;
    pb[y * W_STRIDE] = s ? 0.0f : d[y];
  }
  return __any_sync(~0u, low);
}

// A warp's flags: bit 0 the phase parity of its mbarrier; its tile of the block visited last differs from memory.
constexpr uint32_t BLOCK_UNSAVED = 2u;

// One visit of a block by its CTA (all warps; the barriers are CTA-wide); with `fill_only` it ends once the tiles are filled.  Tile (wx, wy) of the block is warp
// wy * BLOCK_TX + wx's.  The tiles relax their halo edges from their neighbours in the block (shared memory) and, on
// the block's border, from the halo read at the start; a tile whose border was lowered, or which had not converged,
// runs up to BLOCK_ROUNDS rounds (skew_round); this repeats until no tile has anything to do.  A tile may read a
// neighbour's border while the neighbour lowers it: values only decrease and each is one word, and the visit ends
// only after an iteration in which no tile changed.  Only the lines on the block's border are written to memory; the
// tiles stay in shared memory and are written when the CTA turns to another block (BLOCK_UNSAVED) or ends.
// Returns false when a copy into the block's tiles did not arrive: the CTA then visits nothing more (STAGE_LOST).
__device__ __forceinline__ bool block_visit_ns(const BlockRun& a, const CUtensorMap* __restrict__ tmaps, BlockSmem& sm,
                                               uint32_t blk, uint32_t& flags, const Queue& q, float (&wh)[TILE],
                                               float (&wv)[TILE], int& loaded, bool fill_only) {
  const int lane = threadIdx.x & 31, warp = (int)uniform(threadIdx.x >> 5);
  const float INF = f_inf();
  const ImgDesc& dd = sm.ctl.desc;
  BlockTile& t = sm.tile[warp];
  float* B = reinterpret_cast<float*>(t.img);
  uint32_t sides;
  bool todo = false;     // the tile has rounds to run whatever its halo
  bool changed = false;  // a value of the tile fell in this visit
  {
    const bool first = uniform(sm.ctl.first != 0u), seed = uniform(sm.ctl.seed != 0u), rerun = uniform(sm.ctl.rerun != 0u);
    const BlockPlace p = block_place(dd, blk);
    sides = uniform(p.sides);
    const bool exists = (sides & 0x1000u) != 0u;
    const VisitBufs vb{t.img, t.Wv, nullptr, &t.bar, &t.bar, 1u, 1u, &flags};
    if (exists && !rerun) stage_tile(vb, tmaps + 2 * sm.ctl.img, tmaps + 2 * sm.ctl.img + 1, dd.channels == 3, seed, p.x0, p.y0);
    {
      float top = INF, bot = INF, lft = INF, rgt = INF;
      const float v = dd.v;
      const uint32_t outer = sides >> 8, nvis = sm.ctl.nvis;
      if (lane < p.vw) {
        if (outer & 4u) top = (nvis & 4u) ? ld_dist(dd, p.y0 - 1, p.x0 + lane) : v;
        if (outer & 8u) bot = (nvis & 8u) ? ld_dist(dd, p.y0 + TILE, p.x0 + lane) : v;
      }
      if (lane < p.vh) {
        if (outer & 1u) lft = (nvis & 1u) ? ld_dist(dd, p.y0 + lane, p.x0 - 1) : v;
        if (outer & 2u) rgt = (nvis & 2u) ? ld_dist(dd, p.y0 + lane, p.x0 + TILE) : v;
      }
      t.H[E_LEFT + lane] = lft;
      t.H[E_RIGHT + lane] = rgt;
      t.H[E_TOP + lane] = top;
      t.H[E_BOTTOM + lane] = bot;
    }
    const bool fill = exists && !rerun;
    float td[TILE];
    if (fill && !first) block_load_tile(dd, p, td);
    const bool staged = tma_wait(&t.bar, flags, 1u, q, blk, fill);
    if (uniform(fill) && staged) todo = changed = block_fill_ns(dd, p, t, first, seed, td);
    if (!rerun) loaded = -1;
    // Every tile of the block is in place; with fill_only, ctl is block_next's from here on.
    if (__syncthreads_or(staged ? 0 : 1)) return false;
    if (fill_only) return true;
    if (first) flags |= BLOCK_UNSAVED;
  }
  uint32_t nph = 0;
  float d[TILE];
  for (uint32_t it = 0;; ++it) {
    bool layout_a = true;
    asm volatile("" : "+r"(sides));  // keeps the addresses below from being held in registers through the rounds
    if (sides & 0x1000u) {
      // The halo of each side, one word per lane: the neighbour's border in shared memory, or H.
      const BlockTile* pl = &t - 1;
      const BlockTile* pr = &t + 1;
      const BlockTile* pt = &t - BLOCK_TX;
      const BlockTile* pb = &t + BLOCK_TX;
      const volatile float* hl =
          (sides & 0x10u) ? reinterpret_cast<const float*>(pl->img) + lane * W_STRIDE + TILE - 1 : t.H + E_LEFT + lane;
      const volatile float* hr = (sides & 0x20u) ? reinterpret_cast<const float*>(pr->img) + lane * W_STRIDE : t.H + E_RIGHT + lane;
      const volatile float* ht =
          (sides & 0x40u) ? reinterpret_cast<const float*>(pt->img) + (TILE - 1) * W_STRIDE + lane : t.H + E_TOP + lane;
      const volatile float* hb = (sides & 0x80u) ? reinterpret_cast<const float*>(pb->img) + lane : t.H + E_BOTTOM + lane;
      const float ct = __fadd_rn(*ht, t.E[E_TOP + lane]), cb = __fadd_rn(*hb, t.E[E_BOTTOM + lane]);
      const float cl = __fadd_rn(*hl, t.E[E_LEFT + lane]), cr = __fadd_rn(*hr, t.E[E_RIGHT + lane]);
      float dt = B[lane], db = B[(TILE - 1) * W_STRIDE + lane];
      bool low = ct < dt || cb < db;
      dt = fminf(dt, ct);
      db = fminf(db, cb);
      B[lane] = dt;
      B[(TILE - 1) * W_STRIDE + lane] = db;
      __syncwarp();
      float dl = B[lane * W_STRIDE], dr = B[lane * W_STRIDE + TILE - 1];
      low |= cl < dl || cr < dr;
      dl = fminf(dl, cl);
      dr = fminf(dr, cr);
      B[lane * W_STRIDE] = dl;
      B[lane * W_STRIDE + TILE - 1] = dr;
      todo |= __any_sync(~0u, low);
      if (uniform(todo)) {
        const float tl = fminf(dt, dl), br = fminf(db, dr);
        const uint32_t ka = __reduce_min_sync(~0u, __float_as_uint(lane < TILE / 2 ? tl : br));
        const uint32_t kb = __reduce_min_sync(~0u, __float_as_uint(lane < TILE / 2 ? br : tl));
        layout_a = ka <= kb;
      }
      __syncwarp();
    }
    if (!__syncthreads_or(todo ? 1 : 0)) break;
    if (uniform(todo)) {
      const int off = layout_a ? (TILE - lane) % TILE : lane;
      const int src_f = (layout_a ? lane + TILE - 1 : lane + 1) % TILE, src_r = (layout_a ? lane + 1 : lane + TILE - 1) % TILE;
      if (loaded != (layout_a ? 1 : 0)) {
        loaded = layout_a ? 1 : 0;
        load_skew(wh, t.Wh + lane * W_STRIDE, off);
        load_skew(wv, t.Wv + (layout_a ? lane : src_f) * W_STRIDE, off);
      }
      load_skew(d, B + lane * W_STRIDE, off);
      int r = 0;
#pragma unroll 1
      do {
        todo = __any_sync(~0u, skew_round(d, wh, wv, src_f, src_r));
        ++nph;
      } while (todo && ++r < BLOCK_ROUNDS);
      changed = true;
      store_skew(B + lane * W_STRIDE, off, d);
      // The border lines go out at once: the checks that end the visit cover their way to L2.
      __syncwarp();
      block_store_border(dd, block_place(dd, blk), sides >> 8, B);
    }
    if (it >= (uint32_t)PHASE_LIMIT) {
      if (threadIdx.x == 0) set_error(q, DERR_PHASE_LIMIT, blk);
      break;
    }
    __syncthreads();
  }

  // What the block's border can bring to its neighbours, and the border lines that were never written.
  const uint32_t outer = (sides >> 8) & 15u;
  if (changed) flags |= BLOCK_UNSAVED;
  if (uniform(outer && (changed || sm.ctl.first))) {
    if (!nph) block_store_border(dd, block_place(dd, blk), outer, B);
    const float* E = t.E;
    const float bl = B[lane * W_STRIDE], br = B[lane * W_STRIDE + TILE - 1], bt = B[lane], bb = B[(TILE - 1) * W_STRIDE + lane];
    const float vl = __fadd_rn(bl, E[E_LEFT + lane]), vr = __fadd_rn(br, E[E_RIGHT + lane]);
    const float vt = __fadd_rn(bt, E[E_TOP + lane]), vbm = __fadd_rn(bb, E[E_BOTTOM + lane]);
    const uint32_t kl = __reduce_min_sync(~0u, vl < t.H[E_LEFT + lane] ? __float_as_uint(vl) : KEY_NONE);
    const uint32_t kr = __reduce_min_sync(~0u, vr < t.H[E_RIGHT + lane] ? __float_as_uint(vr) : KEY_NONE);
    const uint32_t kt = __reduce_min_sync(~0u, vt < t.H[E_TOP + lane] ? __float_as_uint(vt) : KEY_NONE);
    const uint32_t kb = __reduce_min_sync(~0u, vbm < t.H[E_BOTTOM + lane] ? __float_as_uint(vbm) : KEY_NONE);
    const uint32_t k = lane == 0 ? kl : lane == 1 ? kr : lane == 2 ? kt : kb;
    // Sides inside the block have an INF halo in H: mask them out.
    if (lane < 4 && ((outer >> lane) & 1u) && k != KEY_NONE) atomicMin(&sm.ctl.side[lane], k);
  }
  if (nph && lane == 0) {
    atomicAdd(&sm.ctl.visits, 1u);
    atomicAdd(&sm.ctl.phases, nph);
  }
  __syncthreads();
  if (warp == 0) block_complete(a, sm.ctl, blk);
  return true;
}

template <int CTAS>
__global__ void __launch_bounds__(BLOCK_WARPS * 32, CTAS)
    ggdt_block(const ImgDesc* __restrict__ descs, const CUtensorMap* __restrict__ tmaps, BlockRun a) {
  extern __shared__ uint8_t smem_raw[];
  BlockSmem& sm = *reinterpret_cast<BlockSmem*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
  const int lane = threadIdx.x & 31, warp = (int)uniform(threadIdx.x >> 5);
  const uint32_t first = blockIdx.x, step = gridDim.x;
  const int count = (int)((a.total - first + step - 1) / step);
  Queue q{};  // the header's error words only
  q.hdr = a.hdr;
  if (lane == 0) {
    mbar_init(&sm.tile[warp].bar, 1);
    fence_mbar_init();
  }
  for (int i = threadIdx.x; i < BLOCK_OWNED_MAX * BLOCK_SIDES; i += BLOCK_WARPS * 32) (&sm.ctl.sent[0][0])[i] = (&sm.ctl.seen[0][0])[i] = 0;
  for (int i = threadIdx.x; i < BLOCK_OWNED_MAX / 32; i += BLOCK_WARPS * 32) sm.ctl.seeded[i] = sm.ctl.visited[i] = 0;
  for (int i = threadIdx.x; i < count; i += BLOCK_WARPS * 32) sm.ctl.owned_img[i] = image_of_tile(a.base, a.n, first + (uint32_t)i * step);
  if (threadIdx.x < BLOCK_SIDES) sm.ctl.side[threadIdx.x] = KEY_NONE;
  if (threadIdx.x == 0) sm.ctl.visits = sm.ctl.done = sm.ctl.phases = sm.ctl.activations = 0;
  __syncthreads();
  // Seed scan of the owned blocks: one warp per tile, lane = row, the rows of several blocks in flight.
#pragma unroll 4
  for (int i = 0; i < count; ++i) {
    const uint32_t blk = first + (uint32_t)i * step;
    const ImgDesc& dd = descs[sm.ctl.owned_img[i]];
    const uint32_t local = blk - dd.block_base;
    const int x0 = (int)(local % (uint32_t)dd.blocks_x) * BLOCK_W + (warp % BLOCK_TX) * TILE;
    const int y0 = (int)(local / (uint32_t)dd.blocks_x) * BLOCK_H + (warp / BLOCK_TX) * TILE;
    const int vw = min(TILE, dd.width - x0);
    bool nz = false;
    if (vw > 0 && y0 + lane < dd.height) nz = mask_row_any(dd, x0, y0 + lane, vw);
    if (nz) atomicOr(&sm.ctl.seeded[i >> 5], 1u << (i & 31));
  }
  __syncthreads();
  // Blocks without seeds give their token back.
  if (warp == 0) {
    const uint32_t seeded = __reduce_add_sync(~0u, lane < BLOCK_OWNED_MAX / 32 ? (uint32_t)__popc(sm.ctl.seeded[lane]) : 0u);
    if (lane == 0) atomicSub(&a.hdr->pending.v, (uint32_t)count - seeded);
  }
  uint32_t flags = 0, prev = POP_NONE;
  float wh[TILE], wv[TILE];  // the tile's weights, in the layout `loaded`
  int loaded = -1;
  // The first block without seeds is filled before anything activates it, so that its first visit finds it in place: with
  // one block per CTA that takes 8,000 (gray) to 12,000 (rgb8) cycles off every step of the front into new blocks.
  int early = 0;
  while (early < count && ((sm.ctl.seeded[early >> 5] >> (early & 31)) & 1u)) ++early;
  if (uniform(early < count && descs[sm.ctl.owned_img[min(early, count - 1)]].warm == 0)) {
    if (warp == 0) {
      const uint32_t* src = reinterpret_cast<const uint32_t*>(&descs[sm.ctl.owned_img[early]]);
      for (int i = lane; i < (int)(sizeof(ImgDesc) / 4); i += 32) reinterpret_cast<uint32_t*>(&sm.ctl.desc)[i] = src[i];
      if (lane == 0) {
        sm.ctl.next = (uint32_t)early;
        sm.ctl.img = sm.ctl.owned_img[early];
        sm.ctl.first = 1u;
        sm.ctl.seed = sm.ctl.rerun = sm.ctl.nvis = 0u;
      }
    }
  } else {
    early = -1;
  }
  for (;;) {
    if (early < 0 && warp == 0) block_next(a, descs, sm.ctl, first, step, count, prev);
    __syncthreads();
    const uint32_t next = uniform(sm.ctl.next);
    if (next != prev && (flags & BLOCK_UNSAVED)) {
      const ImgDesc& dd = descs[sm.ctl.owned_img[prev]];
      block_store_tile(dd, block_place(dd, first + prev * step), reinterpret_cast<const float*>(sm.tile[warp].img));
      flags &= ~BLOCK_UNSAVED;
      __syncwarp();
    }
    if (next >= (uint32_t)count) {  // POP_NONE, or not an index at all
      if (next != POP_NONE && threadIdx.x == 0) block_error(a, DERR_BAD_TILE, next);
      break;
    }
    if (!block_visit_ns(a, tmaps, sm, first + next * step, flags, q, wh, wv, loaded, early >= 0)) break;
    prev = next;
    early = -1;
  }
  // Blocks never reached keep uninitialised memory: write v there.
  for (int i = 0; i < count; ++i) {
    const uint32_t blk = first + (uint32_t)i * step;
    if (((sm.ctl.visited[i >> 5] >> (i & 31)) & 1u) || sm.ctl.owned_img[i] >= (uint32_t)a.n) continue;
    const ImgDesc& dd = descs[sm.ctl.owned_img[i]];
    if (dd.warm) continue;
    const uint32_t local = blk - dd.block_base;
    const int x0 = (int)(local % (uint32_t)dd.blocks_x) * BLOCK_W + (warp % BLOCK_TX) * TILE;
    const int y0 = (int)(local / (uint32_t)dd.blocks_x) * BLOCK_H + (warp / BLOCK_TX) * TILE;
    if (x0 + lane < dd.width)
      for (int y = y0; y < min(y0 + TILE, dd.height); ++y) dist_row(dd, y)[x0 + lane] = dd.v;
  }
  if (threadIdx.x == 0) {
    atomicAdd(&a.hdr->phases.v, sm.ctl.phases);
    atomicAdd(&a.hdr->activations.v, sm.ctl.activations);
  }
}

}  // namespace dtb
