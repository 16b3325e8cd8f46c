// k_blend.cu — per-tile alpha blending (forward + adjoint), MSE, tonemap.
//
// Forward (rasterize.wgsl:48-118): one CTA per (view, tile), each warp on its
// own: a thread owns PPT vertically adjacent pixels (a warp an 8 x 4 PPT block
// of the tile), two of them in packed f32x2 arithmetic.  A warp walks the tile's
// depth-ordered list — its own pair list, or its super tile's item list filtered
// by the member masks — through a feed that stages 32 records (3 x 16 B each)
// ahead with cp.async, and leaves as soon as its pixels are saturated (T <
// 1e-4).  For an exact backward it writes down the entries that one of its pixels
// took.  The MSE of loss.rs:163-179 — dL/dC = scale * 2 (C - target) / (3 W H) per pixel, squared
// errors reduced per CTA in FP64 — runs in the forward's epilogue or in the
// backward's prologue.
//
// Backward (rasterize_backward.wgsl:73-210): same grid, each warp walking back
// over the entries that its pixels took (or, in the reference's mode and the
// stage calls, over the list from its last contributor or end).  Per (pixel,
// splat) a thread forms the opacity gradient h and T alpha; every 8 entries the
// warp turns its shared-memory rows round and sums h's moments (h, h dx, h dy,
// h dx^2, h dx dy, h dy^2) and the colour gradient over its 64 pixels, turns the
// sums into the splats' gradients (dmean.xy, dopacity, dconic.abc, dcolor.rgb)
// and sends them to global memory with one float4 vector atomic per lane, three
// per (warp, splat) — the reference issues nine CAS loops per (pixel, splat).
// The transmittance reconstruction T_i = T_{i+1} / (1 - alpha_i) uses one
// approximate reciprocal per (pixel, splat).
// Measured on the 1M-splat, 8-view 1080p step (BF16 storage): backward 2.86 -> 1.30 ms, and on
// one view of it 0.76 -> 0.20 ms, against a CTA walking the list together with a
// reduce-scatter over all lanes for every two entries and shared-memory sums.
#include "sc_internal.cuh"

#include <algorithm>
#include <type_traits>

namespace sck {

struct BlendArgs {
  uint32_t width, height, tw, th, tiles_x, tiles_y, num_tiles, stride;
  uint64_t pixels;  // per view
  uint32_t stage;   // entries the forward stages at a time, at most STAGE
  const SceneDev* scenes;  // per-view image sizes and MSE scales (many-scene steps), or null
  bool count_pairs;        // with work counters: also count contributing (pixel, entry) pairs
};

static BlendArgs blend_args(const sc_tiling* tl, uint32_t stride) {
  BlendArgs a;
  a.width = tl->width; a.height = tl->height; a.tw = tl->tile_w; a.th = tl->tile_h;
  a.tiles_x = (tl->width + tl->tile_w - 1) / tl->tile_w;
  a.tiles_y = (tl->height + tl->tile_h - 1) / tl->tile_h;
  a.num_tiles = a.tiles_x * a.tiles_y;
  a.stride = stride;
  a.pixels = (uint64_t)tl->width * tl->height;
  a.stage = 32;
  a.scenes = nullptr;
  a.count_pairs = false;
  return a;
}

// a view's image size and MSE scale: the scene's in a many-scene step
__device__ __forceinline__ void view_dims(const BlendArgs& a, uint32_t v, float gscale, uint32_t& W, uint32_t& H,
                                          float& gs) {
  W = a.width; H = a.height; gs = gscale;
  if (a.scenes) {
    const SceneDev& sd = a.scenes[v];
    W = sd.width; H = sd.height; gs = sd.gscale;
  }
}

// The pixels of thread threadIdx.x in tile (tx, ty): PPT vertically adjacent
// pixels from (px, py0).  Where the tile splits that way (tile_w a multiple of
// 8, tile_h / PPT of 4) a warp takes an 8 x 4 PPT block, else whole rows of the
// tile.  The compact block leaves more entries that no pixel of a warp takes
// (the backward skips their reduction) and lets a warp's pixels saturate
// together (1M splats, 8 views of 1920x1080, 16 x 16 tiles: forward 1.016 ->
// 0.985 ms, backward 2.563 -> 2.515 ms against warps of 16 x 4 pixels).
template <int PPT>
__device__ __forceinline__ void tile_pixel(const BlendArgs& a, uint32_t tx, uint32_t ty, uint32_t& px,
                                           uint32_t& py0) {
  const uint32_t wl = threadIdx.x >> 5, ln = threadIdx.x & 31;
  const bool blk = (a.tw & 7) == 0 && ((a.th / PPT) & 3) == 0;
  const uint32_t lx = blk ? (wl % (a.tw >> 3)) * 8 + (ln & 7) : threadIdx.x % a.tw;
  const uint32_t lr = blk ? (wl / (a.tw >> 3)) * 4 + (ln >> 3) : threadIdx.x / a.tw;
  px = tx * a.tw + lx;
  py0 = ty * a.th + PPT * lr;
}

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

#define ALPHA_MAX 0.99f
#define FULL_MASK 0xffffffffu

// e^(-q/2) = 2^(q * NEG_HALF_LOG2E), log2 e = 1 / ln 2
#define NEG_HALF_LOG2E (-0.72134752044448170368f)

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float2 f2(float x) { return make_float2(x, x); }

// The conic's quadratic form at (dx, dy) is A + B dy + c dy^2 with A = a dx^2
// and B = 2 b dx, shared by a thread's pixels in one column; per pixel it is
// evaluated as (c dy + B) dy + A.  Every rounding step is written out (no
// contraction left to the compiler), so the one-pixel path and the packed
// two-pixel path (sm_100 f32x2 instructions) produce the same bits.
struct EntryGeom {
  float dx, A, B;
};
__device__ __forceinline__ EntryGeom entry_geom(float fx, const float4 ra, const float4 rb) {
  EntryGeom e;
  e.dx = __fadd_rn(fx, -ra.x);
  e.A = __fmul_rn(__fmul_rn(rb.x, e.dx), e.dx);
  e.B = __fmul_rn(2.0f * rb.y, e.dx);
  return e;
}

// Gaussian weight and alpha of one (pixel, splat); false when the reference
// skips the pair (power = -quad/2 > 0, or alpha < 1/255).  Shared by forward
// and backward so both make identical skip decisions.
__device__ __forceinline__ bool eval_alpha(const EntryGeom& e, float c, float dy, float op, float& g,
                                           float& alpha_raw, float& alpha) {
  const float quad = __fmaf_rn(__fmaf_rn(c, dy, e.B), dy, e.A);
  g = ex2_approx(__fmul_rn(quad, NEG_HALF_LOG2E));
  alpha_raw = __fmul_rn(op, g);
  alpha = fminf(alpha_raw, ALPHA_MAX);
  return quad >= 0.0f && alpha >= ALPHA_MIN;
}

// The same for a thread's two pixels (rows fy.x, fy.y of one column) with
// packed arithmetic; v0, v1 are the per-pixel results of eval_alpha.  PLAIN:
// the record is plain_record, whose other two tests cannot fail.
template <bool PLAIN>
__device__ __forceinline__ void eval_alpha2(const EntryGeom& e, float c, float2 fy, float ry, float op, float2& dy,
                                            float2& g, float2& alpha_raw, float2& alpha, bool& v0, bool& v1) {
  dy = __fadd2_rn(fy, f2(-ry));
  const float2 quad = __ffma2_rn(__ffma2_rn(f2(c), dy, f2(e.B)), dy, f2(e.A));
  const float2 ex = __fmul2_rn(quad, f2(NEG_HALF_LOG2E));
  g = make_float2(ex2_approx(ex.x), ex2_approx(ex.y));
  alpha_raw = __fmul2_rn(f2(op), g);
  alpha = PLAIN ? alpha_raw : make_float2(fminf(alpha_raw.x, ALPHA_MAX), fminf(alpha_raw.y, ALPHA_MAX));
  v0 = (PLAIN || quad.x >= 0.0f) && alpha.x >= ALPHA_MIN;
  v1 = (PLAIN || quad.y >= 0.0f) && alpha.y >= ALPHA_MIN;
}

template <typename T>
__device__ __forceinline__ T block_sum(T x, T* sred) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(FULL_MASK, x, o);
  if (lane == 0) sred[warp] = x;
  __syncthreads();
  T r = 0;
  if (threadIdx.x == 0)
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) r += sred[w];
  return r;  // valid in thread 0
}

// MSE term of one pixel (loss.rs:163-179): returns dL/dC = gscale (C - target)
// and adds the squared error to sq.  The forward epilogue and the backward
// prologue both use it, so either pass can own the loss.
__device__ __forceinline__ float3 mse_pixel(float cr, float cg, float cb, const float* __restrict__ tgt, float gscale,
                                            double& sq) {
  const float dx = __fadd_rn(cr, -tgt[0]), dy = __fadd_rn(cg, -tgt[1]), dz = __fadd_rn(cb, -tgt[2]);
  sq += (double)__fmaf_rn(dx, dx, __fmaf_rn(dy, dy, __fmul_rn(dz, dz)));
  return make_float3(__fmul_rn(dx, gscale), __fmul_rn(dy, gscale), __fmul_rn(dz, gscale));
}

// Work counters of one blend launch (when given): per CTA, the list positions
// its furthest warp covered and the entries that one kept, added into one of
// BLEND_WORK_SLOTS (scanned, staged) pairs so that the atomics spread.
__device__ __forceinline__ void add_work(unsigned long long* work, uint32_t scanned, uint32_t staged) {
  if (work && threadIdx.x == 0 && scanned) {
    unsigned long long* w = work + 2 * (blockIdx.x % BLEND_WORK_SLOTS);
    atomicAdd(w, (unsigned long long)scanned);
    atomicAdd(w + 1, (unsigned long long)staged);
  }
}

// With COUNT, a blend launch also counts its contributing (pixel, entry)
// pairs (a pixel that takes an entry's alpha): the CTA's sum goes to the slot
// after the BLEND_WORK_SLOTS (scanned, staged) pairs.  Every thread of the CTA
// calls it; it ends with a barrier, so sred can be reused right after.
__device__ __forceinline__ void add_pixel_pairs(unsigned long long* work, uint32_t n, double* sred) {
  const double tot = block_sum((double)n, sred);
  if (threadIdx.x == 0 && tot > 0.0)
    atomicAdd(work + 2 * BLEND_WORK_SLOTS + blockIdx.x % BLEND_WORK_SLOTS, (unsigned long long)tot);
  __syncthreads();
}

// Where a CTA's depth-ordered splat list comes from.  LIST_PAIRS: the tile's
// pair list, ids[ranges[view * tiles + tile]].  LIST_ITEMS: its super tile's
// item list, ids[ranges[view * super tiles + super tile]], of which the CTA
// keeps the items whose member mask (bits 16..31 of keys; bit (ty % 4) * 4 +
// tx % 4 is tile (tx, ty)) holds its tile.  Both lists are in depth order, so
// a tile blends the same splats in the same order either way.
// LIST_TAKERS (backward): the entries that the forward wrote down per warp.
enum { LIST_PAIRS = 0, LIST_ITEMS = 1, LIST_TAKERS = 2 };
struct ListArgs {
  const uint32_t* ids;
  const uint2* ranges;
  const uint32_t* keys;  // LIST_ITEMS
  uint32_t super_x, super_per_view;
};

template <int LIST>
__device__ __forceinline__ uint2 list_range(const ListArgs& l, const BlendArgs& a, uint32_t v, uint32_t tx,
                                            uint32_t ty, uint32_t tile, uint32_t& bit) {
  if (LIST == LIST_PAIRS) {
    bit = 0;
    return l.ranges[(size_t)v * a.num_tiles + tile];
  }
  bit = (ty % SC_SUPER) * SC_SUPER + tx % SC_SUPER;
  return l.ranges[(size_t)v * l.super_per_view + (ty / SC_SUPER) * l.super_x + tx / SC_SUPER];
}

// A record whose pairs need only the alpha >= 1/255 test: finite and of ordinary
// size, its conic well away from singular (det > 2^-10 a c, so that the quadratic form,
// at least 2^-11 of its terms' magnitudes, cannot round below zero), and its
// opacity below 0.99, so that no alpha reaches the clamp.  The backward walks a
// stage of such entries without the other tests (1M splats, 8 views of 1080p: 1.405 -> 1.355
// ms with the 8 rows unrolled; the forward gained under 1 % and tests all).
__device__ __forceinline__ bool plain_record(const float4 ra, const float4 rb, float op) {
  const float det = rb.x * rb.z - rb.y * rb.y;
  return fabsf(ra.x) < 1e6f && fabsf(ra.y) < 1e6f && rb.x > 0.0f && rb.z > 0.0f && rb.x < 1e6f && rb.z < 1e6f &&
         det > 9.765625e-4f * (rb.x * rb.z) && op < ALPHA_MAX;
}

// Values whose products and sums over a list stay finite.
constexpr float ORDINARY = 1e15f;
__device__ __forceinline__ bool ordinary_record(const float4 ra, const float4 rb, const float4 rc) {
  return fabsf(ra.x) + fabsf(ra.y) + fabsf(rb.x) + fabsf(rb.y) + fabsf(rb.z) + fabsf(rc.x) + fabsf(rc.y) +
         fabsf(rc.z) + fabsf(rc.w) < ORDINARY;
}

// How a warp gets its entries, in stages of up to 32: gather() starts the copies
// of the next stage's records (3 float4 each, cp.async) and returns its size, 0
// at the end; ready() waits for them and returns how many of them are left to
// blend — the list feed drops those whose alpha stays below 1/255 over the
// warp's pixels.  The next gather() then runs beside the pixel loop.  Nothing is
// shared with another warp, so the warps of a CTA never wait for one another:
// with staging shared by the CTA and a barrier per batch, a tile's warps waited
// for the slowest of them, for the list words and for the gathers at every
// batch, about 500 cycles per kept entry in the backward and 200 in the forward (an
// item list keeps one position in about 5).
// (Records laid out anew with every operand of the packed arithmetic stored as a
// pair, 64 B an entry, were slower: backward 1.58 against 1.40 ms.)
constexpr uint32_t STAGE = 32;
struct StageSmem {
  float4 rec[2 * STAGE * 3];
  uint32_t id[2 * STAGE], pos[2 * STAGE];  // pos: the list feed's
};

// The pixel centres of a warp, as a rectangle.
struct WarpRect {
  float x0, x1, y0, y1;
};
__device__ __forceinline__ WarpRect warp_rect(uint32_t px, uint32_t py0, uint32_t rows) {
  WarpRect w;
  w.x0 = (float)__reduce_min_sync(FULL_MASK, px) + 0.5f;
  w.x1 = (float)__reduce_max_sync(FULL_MASK, px) + 0.5f;
  w.y0 = (float)__reduce_min_sync(FULL_MASK, py0) + 0.5f;
  w.y1 = (float)(__reduce_max_sync(FULL_MASK, py0) + rows) - 0.5f;
  return w;
}
// Whether the ellipse alpha >= 1/255 of a record may hold a pixel of the
// rectangle: its extent in x over the rectangle's band of rows (two square
// roots, as super_row_hull) against the rectangle's columns, with the binning
// test's margins, which cover the rounding here and in the blend.  A NaN
// anywhere keeps the entry.
__device__ __forceinline__ bool reaches(const float4 ra, const float4 rb, float op, const WarpRect& w) {
  const CullShape s = cull_shape(ra.x, ra.y, rb.x, rb.y, rb.z, op);
  const float w0 = w.y0 - s.my, w1 = w.y1 - s.my;
  const float a0 = fmaxf(w0, -s.yh), a1 = fminf(w1, s.yh);
  const float wr = fminf(fmaxf(-s.kx, a0), a1), wl = fminf(fmaxf(s.kx, a0), a1);
  const float ur = (-s.b * wr + cull_sqrt(fmaxf(s.L * s.a - wr * wr * s.det, 0.0f))) * s.inv_a;
  const float ul = (-s.b * wl - cull_sqrt(fmaxf(s.L * s.a - wl * wl * s.det, 0.0f))) * s.inv_a;
  const bool out = op < ALPHA_MIN ||
                   (!s.keep && op == op &&
                    (w1 < -s.yh || w0 > s.yh || s.mx + ur + 1e-2f < w.x0 || s.mx + ul - 1e-2f > w.x1));
  return !out;
}

__device__ __forceinline__ void copy_record(StageSmem& st, uint32_t slot, const float4* vrec, uint32_t id) {
  const float4* src = vrec + (size_t)3 * id;
  float4* dst = st.rec + 3 * slot;
  cp_async16(dst, src);
  cp_async16(dst + 1, src + 1);
  cp_async16(dst + 2, src + 2);
  st.id[slot] = id;
}

// List feed: the warp's list, front to back or (REV) back to front.  fill()
// takes 128 list positions (one 16-byte load of keys and of ids per lane,
// issued one chunk ahead) and appends the kept ones — the items of the warp's
// tile (LIST_ITEMS), or all of a pair list — to a queue that gather() takes
// the stages from.
constexpr uint32_t QCAP = 256;  // under one stage pending and a chunk, rounded up to a power of two
struct ListSmem {
  StageSmem st;
  uint2 q[QCAP];  // (id, list position)
};

template <int LIST, bool REV>
struct ListFeed {
  using Smem = ListSmem;
  ListSmem& sm;
  const uint32_t* ids;
  const uint32_t* keys;
  const float4* vrec;
  uint32_t mask;          // LIST_ITEMS: the tile's member bit
  uint32_t begin, end;    // the walked positions, as indices into ids
  uint32_t most;          // entries per stage
  uint32_t at;            // next chunk: [at, at + 128), REV: [at - 128, at); a multiple of 4
  uint32_t qtail, qhead;  // entries queued and gathered
  uint4 key, wid;         // this lane's four words of the next chunk
  bool odd;               // REV: the landed stage has a record that is not ordinary

  __device__ __forceinline__ ListFeed(ListSmem& smem, const ListArgs& l, const float4* rec, uint32_t b, uint32_t n,
                                      uint32_t bit, uint32_t stage)
      : sm(smem), ids(l.ids), keys(l.keys), vrec(rec), mask(0x10000u << bit), begin(b), end(b + n), most(stage),
        at(REV ? (b + n + 3u) & ~3u : b & ~3u), qtail(0), qhead(0), key(make_uint4(0, 0, 0, 0)), wid(key), odd(false) {
    load();
  }
  __device__ __forceinline__ bool more() const { return REV ? at > begin : at < end; }
  // first index of this lane's four, and whether they hold a walked position
  __device__ __forceinline__ uint32_t first() const {
    const uint32_t lane = threadIdx.x & 31;
    return REV ? at - 4 - 4 * lane : at + 4 * lane;
  }
  __device__ __forceinline__ bool mine() const {
    return REV ? at > begin + 4 * (threadIdx.x & 31) : first() < end;
  }
  // the lists' arrays are 16-byte aligned and hold whole groups of four words
  // (sc_list_bytes), so a group holding a walked position is readable whole
  __device__ __forceinline__ void load() {
    if (mine()) {
      if (LIST == LIST_ITEMS) key = __ldg(reinterpret_cast<const uint4*>(keys + first()));
      wid = __ldg(reinterpret_cast<const uint4*>(ids + first()));
    }
  }
  __device__ __forceinline__ void fill() {
    const uint32_t lt = (1u << (threadIdx.x & 31)) - 1u, i = first();
    const bool any = mine();
    const uint32_t k4[4] = {key.x, key.y, key.z, key.w}, w4[4] = {wid.x, wid.y, wid.z, wid.w};
    bool keep[4];
    uint32_t slot = qtail;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      keep[e] = any && i + e >= begin && i + e < end && (LIST == LIST_PAIRS || (k4[e] & mask));
      const uint32_t bal = __ballot_sync(FULL_MASK, keep[e]);
      slot += __popc(bal & lt);
      qtail += __popc(bal);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {  // in walking order
      const int c = REV ? 3 - e : e;
      if (keep[c]) sm.q[slot++ % QCAP] = make_uint2(w4[c], i + c - begin);
    }
    at = REV ? at - min(at, 128u) : at + 128;
    if (more()) load();
    __syncwarp();
  }
  __device__ __forceinline__ uint32_t gather() {
    while (qtail - qhead < most && more()) fill();
    const uint32_t n = min(most, qtail - qhead), lane = threadIdx.x & 31;
    if (lane < n) {
      const uint2 w = sm.q[(qhead + lane) % QCAP];
      copy_record(sm.st, lane, vrec, w.x);
      sm.st.pos[lane] = w.y;
    }
    qhead += n;
    return n;
  }
  // the landed stage, culled, moves from the buffer's first half to its second
  __device__ __forceinline__ uint32_t ready(uint32_t n, const WarpRect& w) {
    cp_async_wait_all();
    __syncwarp();
    const uint32_t lane = threadIdx.x & 31;
    const float4* r = sm.st.rec + 3 * lane;
    const float4 ra = r[0], rb = r[1], rc = r[2];
    const uint32_t id = sm.st.id[lane], pos = sm.st.pos[lane];
    const bool keep = lane < n && reaches(ra, rb, rc.w, w);
    const uint32_t bal = __ballot_sync(FULL_MASK, keep);
    if constexpr (REV) odd = __any_sync(FULL_MASK, keep && !ordinary_record(ra, rb, rc));
    if (keep) {
      const uint32_t slot = STAGE + __popc(bal & ((1u << lane) - 1u));
      float4* d = sm.st.rec + 3 * slot;
      d[0] = ra; d[1] = rb; d[2] = rc;
      sm.st.id[slot] = id;
      sm.st.pos[slot] = pos;
    }
    __syncwarp();
    return __popc(bal);
  }
  // records, ids and list positions of the entries to blend
  __device__ __forceinline__ const float4* rec() const { return sm.st.rec + 3 * STAGE; }
  __device__ __forceinline__ const uint32_t* id() const { return sm.st.id + STAGE; }
  __device__ __forceinline__ uint32_t pos(uint32_t i) const { return sm.st.pos[STAGE + i]; }
};

// Taker feed: the entries that some pixel of the warp took in the forward, which
// wrote them down (TakerOut) in chunks of 32 ids, each chunk naming the one
// before it; walked back to front.  pos is the entry's index among them.  An
// exact backward fed so evaluates no entry in vain (30 % of the kept entries of the
// 1M-splat, 8-view workload have no taker in a warp of 8 x 8 pixels) and scans no list.
struct TakerFeed {
  using Smem = StageSmem;
  StageSmem& sm;
  const TakerChunks& ch;
  const float4* vrec;
  uint32_t left;    // entries not gathered
  uint32_t n_next;  // size of the next stage (its ids are in wid), and the chunk before it
  uint32_t wid, prev;
  uint32_t base, base_next;  // pos of the first entry of the landed stage, and of the one gathered
  uint32_t par;              // buffer half the next gather fills: 0 or STAGE

  __device__ __forceinline__ TakerFeed(StageSmem& smem, const TakerChunks& c, const float4* rec, uint2 head)
      : sm(smem), ch(c), vrec(rec), left(head.y), n_next(0), wid(0), prev(head.x), base(0), base_next(0), par(0) {
    load();
  }
  __device__ __forceinline__ void load() {
    n_next = left ? ((left - 1) & (STAGE - 1)) + 1 : 0;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t c = prev;
    if (lane < n_next) wid = __ldg(ch.ids + (size_t)c * STAGE + (n_next - 1 - lane));
    if (left > STAGE) prev = __ldg(ch.prev + c);
  }
  __device__ __forceinline__ uint32_t gather() {
    const uint32_t n = n_next, lane = threadIdx.x & 31;
    if (lane < n) copy_record(sm, par + lane, vrec, wid);
    base_next = left - 1;
    left -= n;
    if (n) load();
    return n;
  }
  __device__ __forceinline__ uint32_t ready(uint32_t n, const WarpRect&) {
    base = base_next;
    par ^= STAGE;
    cp_async_wait_all();
    __syncwarp();
    return n;
  }
  __device__ __forceinline__ const float4* rec() const { return sm.rec + 3 * (par ^ STAGE); }
  __device__ __forceinline__ const uint32_t* id() const { return sm.id + (par ^ STAGE); }
  __device__ __forceinline__ uint32_t pos(uint32_t i) const { return base - i; }
};

// The forward's side: a warp appends its takers' ids to a small ring and writes
// every 32 of them to a chunk of its own.  A chunk number is drawn when the one
// before it is written, so that its latency is hidden; the draws go to
// TAKER_POOLS counters, each with its share of the chunks.  A pool that runs out
// raises an error: the step's later kernels then do nothing, and the caller runs
// it again with the chunks it needs.
struct TakerOut {
  const TakerChunks& ch;
  uint32_t* ring;        // 64 ids
  uint32_t count;        // takers so far
  uint32_t chunk, last;  // chunk being filled, and the one before it
  bool ok;

  // neighbouring tiles and the tiles of a column go to different pools
  static __device__ __forceinline__ uint32_t pool() {
    return (blockIdx.x * 2654435761u) >> 16 & (TAKER_POOLS - 1);
  }
  __device__ __forceinline__ uint32_t draw() {
    uint32_t c = 0;
    if ((threadIdx.x & 31) == 0) c = atomicAdd(ch.drawn + pool(), 1u);
    return c;
  }
  __device__ __forceinline__ TakerOut(const TakerChunks& c, uint32_t* r)
      : ch(c), ring(r), count(0), chunk(0), last(0), ok(true) {
    chunk = draw();
  }
  // the chunk drawn, as every lane's number
  __device__ __forceinline__ uint32_t number() {
    const uint32_t c = __shfl_sync(FULL_MASK, chunk, 0);
    ok = ok && c < ch.pool_cap;
    return pool() * ch.pool_cap + min(c, ch.pool_cap - 1);
  }
  // append the entries of a stage whose bit in m is set (this lane's entry has id)
  __device__ __forceinline__ void append(uint32_t m, uint32_t id) {
    const uint32_t lane = threadIdx.x & 31, n = __popc(m), at = count % STAGE;
    if (m >> lane & 1u) ring[(count + __popc(m & ((1u << lane) - 1u))) % (2 * STAGE)] = id;
    __syncwarp();
    if (at + n >= STAGE) {
      const uint32_t c = number();
      ch.ids[(size_t)c * STAGE + lane] = ring[(count - at + lane) % (2 * STAGE)];
      if (lane == 0) ch.prev[c] = last;
      last = c;
      chunk = draw();
      __syncwarp();
    }
    count += n;
  }
  // the last chunk, and where the walk back starts: (chunk, takers)
  __device__ __forceinline__ uint2 finish(uint32_t* err) {
    const uint32_t lane = threadIdx.x & 31, at = count % STAGE;
    uint32_t head = last;
    if (at) {
      const uint32_t c = number();
      if (lane < at) ch.ids[(size_t)c * STAGE + lane] = ring[(count - at + lane) % (2 * STAGE)];
      if (lane == 0) ch.prev[c] = last;
      head = c;
    }
    if (!ok && lane == 0) atomicOr(err, SC_DEVERR_TAKERS);
    return make_uint2(head, ok ? count : 0u);
  }
};

struct NoTakers {
  __device__ __forceinline__ NoTakers(const TakerChunks&, uint32_t*) {}
};

// The CTA's warps meet only for the work counters: the list positions the
// furthest warp covered and the entries it kept.
__device__ __forceinline__ void add_tile_work(unsigned long long* work, uint32_t scanned, uint32_t staged,
                                              uint32_t* s_work) {
  if (!work) return;
  if (threadIdx.x < 2) s_work[threadIdx.x] = 0;
  __syncthreads();
  if ((threadIdx.x & 31) == 0) {
    atomicMax(&s_work[0], scanned);
    atomicMax(&s_work[1], staged);
  }
  __syncthreads();
  add_work(work, s_work[0], s_work[1]);
}

// ---------------------------------------------------------------- forward
// TAKERS: write down each warp's takers (TakerOut); aux then holds a pixel's last
// contributor as its index among them plus one, else as its list position plus one.
struct TakerRing { uint32_t id[2 * STAGE]; };
template <int PPT, int LIST, bool COUNT, bool TAKERS>
__global__ void __launch_bounds__(256) k_composite(const float4* __restrict__ rec, ListArgs l, BlendArgs a,
                                                   float4* __restrict__ image, uint2* __restrict__ aux,
                                                   const float* __restrict__ target, float gscale,
                                                   float4* __restrict__ dl_dc, double* __restrict__ loss,
                                                   uint32_t* __restrict__ skip, unsigned long long* __restrict__ work,
                                                   TakerChunks takers) {
  sc_after_previous();
  extern __shared__ float4 sbuf[];  // one ListSmem per warp, then one TakerRing per warp
  __shared__ double sred[8];
  __shared__ uint32_t s_work[2];
  if (skip && (*skip & SC_DEVERR_CAPACITY)) return;  // the lists of this step are incomplete
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n_warps = blockDim.x >> 5;
  ListSmem& sm = reinterpret_cast<ListSmem*>(sbuf)[warp];
  const uint32_t vt = blockIdx.x;
  const uint32_t v = vt / a.num_tiles, tile = vt - v * a.num_tiles;
  const uint32_t ty = tile / a.tiles_x, tx = tile - ty * a.tiles_x;
  uint32_t px, py0;
  tile_pixel<PPT>(a, tx, ty, px, py0);
  const float fx = (float)px + 0.5f;
  uint32_t W, H;
  float gs;
  view_dims(a, v, gscale, W, H, gs);
  uint32_t bit;
  const uint2 r = list_range<LIST>(l, a, v, tx, ty, tile, bit);
  const uint32_t begin = r.x, len = r.y > r.x ? r.y - r.x : 0u;
  const float4* vrec = rec + (size_t)3 * v * a.stride;

  float T[PPT], cr[PPT], cg[PPT], cb[PPT], fy[PPT];
  uint32_t last[PPT];
  bool in[PPT];
  bool all_done = true;
#pragma unroll
  for (int k = 0; k < PPT; ++k) {
    cr[k] = cg[k] = cb[k] = 0.f; last[k] = 0;
    fy[k] = (float)(py0 + k) + 0.5f;
    in[k] = px < W && py0 + k < H;
    // a pixel is done exactly when its T < 1e-4: one outside the image, never
    // written, runs with T = 0
    T[k] = in[k] ? 1.0f : 0.0f;
    all_done &= !in[k];
  }
  uint32_t w_pix = 0, scanned = 0, staged = 0;
  uint2 taken = make_uint2(0u, 0u);
  if (len > 0 && !__all_sync(FULL_MASK, all_done)) {
    ListFeed<LIST, false> feed(sm, l, vrec, begin, len, bit, a.stage);
    TakerRing* rings = reinterpret_cast<TakerRing*>(reinterpret_cast<ListSmem*>(sbuf) + n_warps);
    typename std::conditional<TAKERS, TakerOut, NoTakers>::type out(takers, rings[warp].id);
    float2 T2 = make_float2(T[0], T[PPT - 1]);
    float2 R2 = f2(0.f), G2 = R2, B2 = R2;
    const float2 fy2 = make_float2(fy[0], fy[PPT - 1]);
    bool sat = false;
    const WarpRect rect = warp_rect(px, py0, PPT);
    for (uint32_t n_raw = feed.gather(); n_raw > 0 && !sat;) {
      const uint32_t n = feed.ready(n_raw, rect);
      n_raw = feed.gather();
      const float4* sr = feed.rec();
      uint32_t took[PPT];  // this stage's entries that the pixels took
#pragma unroll
      for (int q = 0; q < PPT; ++q) took[q] = 0;
      auto blend = [&](const float4* r, uint32_t b) {
        const float4 ra = r[0], rb = r[1], rc = r[2];
        const EntryGeom e = entry_geom(fx, ra, rb);
        if constexpr (PPT == 2) {
          // both pixels, without a branch: a pixel that skips the splat gets
          // alpha 0, which leaves its colour and T bit for bit unchanged
          float2 dy, g, araw, al;
          bool v0, v1;
          eval_alpha2<false>(e, rb.z, fy2, ra.y, rc.w, dy, g, araw, al, v0, v1);
          v0 &= T2.x >= 1e-4f;
          v1 &= T2.y >= 1e-4f;
          const float2 am = make_float2(v0 ? al.x : 0.0f, v1 ? al.y : 0.0f);
          const float2 ta = __fmul2_rn(T2, am);
          R2 = __ffma2_rn(ta, f2(rc.x), R2);
          G2 = __ffma2_rn(ta, f2(rc.y), G2);
          B2 = __ffma2_rn(ta, f2(rc.z), B2);
          T2 = __fmul2_rn(T2, __ffma2_rn(am, f2(-1.0f), f2(1.0f)));
          if constexpr (COUNT) w_pix += (uint32_t)v0 + (uint32_t)v1;
          if (v0) took[0] |= b;
          if (v1) took[PPT - 1] |= b;
        } else {
          float g, araw, alpha;
          if (eval_alpha(e, rb.z, __fadd_rn(fy2.x, -ra.y), rc.w, g, araw, alpha) && T2.x >= 1e-4f) {
            const float ta = __fmul_rn(T2.x, alpha);
            R2.x = __fmaf_rn(ta, rc.x, R2.x);
            G2.x = __fmaf_rn(ta, rc.y, G2.x);
            B2.x = __fmaf_rn(ta, rc.z, B2.x);
            T2.x = __fmul_rn(T2.x, __fadd_rn(1.0f, -alpha));
            if constexpr (COUNT) ++w_pix;
            took[0] |= b;
          }
        }
      };
      // one saturation test per four entries: an entry past a pixel's
      // saturation gives it alpha 0 and changes nothing
      auto saturated = [&]() {
        return __all_sync(FULL_MASK, T2.x < 1e-4f && (PPT == 1 || T2.y < 1e-4f));
      };
      uint32_t i = 0;
      for (; i + 3 < n; i += 4, sr += 12) {
        blend(sr, 1u << i);
        blend(sr + 3, 2u << i);
        blend(sr + 6, 4u << i);
        blend(sr + 9, 8u << i);
        if ((sat = saturated())) break;
      }
      if (!sat && i < n) {
        for (; i < n; ++i, sr += 3) blend(sr, 1u << i);
        sat = saturated();
      }
      if constexpr (TAKERS) {
        uint32_t mine = took[0];
        if constexpr (PPT == 2) mine |= took[1];
        const uint32_t m = __reduce_or_sync(FULL_MASK, mine);
#pragma unroll
        for (int q = 0; q < PPT; ++q)
          if (took[q]) last[q] = out.count + __popc(m & (0xFFFFFFFFu >> __clz(took[q])));
        out.append(m, feed.id()[lane]);
      } else {
#pragma unroll
        for (int q = 0; q < PPT; ++q)
          if (took[q]) last[q] = feed.pos(31 - __clz(took[q])) + 1;
      }
      __syncwarp();  // the stage may be written again
    }
    cp_async_wait_all();
    if constexpr (TAKERS) taken = out.finish(skip);
    scanned = min(feed.at, begin + len) - begin;
    staged = feed.qtail;
    T[0] = T2.x; cr[0] = R2.x; cg[0] = G2.x; cb[0] = B2.x;
    if constexpr (PPT == 2) { T[1] = T2.y; cr[1] = R2.y; cg[1] = G2.y; cb[1] = B2.y; }
  }
  if constexpr (TAKERS) {
    if (lane == 0) takers.head[(size_t)vt * n_warps + warp] = taken;
  }
  add_tile_work(work, scanned, staged, s_work);
  if constexpr (COUNT) add_pixel_pairs(work, w_pix, sred);
  double sq = 0.0;
#pragma unroll
  for (int q = 0; q < PPT; ++q) {
    const uint32_t py = py0 + q;
    if (in[q]) {
      const size_t pix = (size_t)v * a.pixels + (size_t)py * a.width + px;
      image[pix] = make_float4(cr[q], cg[q], cb[q], 1.0f - T[q]);
      if (aux) aux[pix] = make_uint2(__float_as_uint(T[q]), last[q]);
      if (target) {
        const float3 d = mse_pixel(cr[q], cg[q], cb[q], target + 3 * pix, gs, sq);
        dl_dc[pix] = make_float4(d.x, d.y, d.z, 0.0f);
      }
    }
  }
  if (target && loss) {
    const double s = block_sum(sq, sred);
    if (threadIdx.x == 0 && s != 0.0) atomicAdd(&loss[v], s);
  }
}

template <int PPT, int LIST>
static sc_status composite_ppt(sc_ctx* ctx, const BlendArgs& a, uint32_t grid, uint32_t threads, const float4* rec,
                               const ListArgs& l, float4* image, uint2* aux, const float* target, float gscale,
                               float4* dl_dc, double* loss, uint32_t* d_skip, uint64_t* work,
                               const TakerChunks& takers) {
  const bool count = work && a.count_pairs;
  auto kern = takers.head ? (count ? k_composite<PPT, LIST, true, true> : k_composite<PPT, LIST, false, true>)
                          : (count ? k_composite<PPT, LIST, true, false> : k_composite<PPT, LIST, false, false>);
  const size_t smem = threads / 32 * (sizeof(ListSmem) + (takers.head ? sizeof(TakerRing) : 0));
  if (smem > 48 * 1024)
    SC_CUDA_TRY(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), "smem attr");
  sc_launch(ctx, kern, grid, threads, smem, rec, l, a, image, aux, target, gscale, dl_dc, loss, d_skip,
            reinterpret_cast<unsigned long long*>(work), takers);
  return sc_check_launch(ctx, "k_composite");
}

// pixels per thread: 2 when the tile splits into whole warps that way (4 per
// thread measured slower in both kernels at 16x16 tiles: fewer warps per tile
// to hide the entry loop's latency, more registers)
static int pick_ppt(const sc_tiling* tl) {
  const uint32_t px = tl->tile_w * tl->tile_h;
  return (tl->tile_h % 2 == 0 && (px / 2) % 32 == 0) ? 2 : 1;
}

template <int LIST>
static sc_status composite_list(sc_ctx* ctx, const float4* rec, uint32_t stride, uint32_t n_views, const ListArgs& l,
                                const sc_tiling* tl, float4* image, uint2* aux, const float* target, float mse_scale,
                                float4* dl_dc, double* loss, uint32_t* d_skip, uint64_t* work,
                                uint32_t batch, const SceneDev* scenes, bool count_pairs,
                                const TakerChunks* takers) {
  BlendArgs a = blend_args(tl, stride);
  // an item list keeps about a quarter of its positions
  if (batch) a.stage = std::min(std::max(batch / 4, 8u), STAGE) & ~3u;
  a.scenes = scenes;
  a.count_pairs = count_pairs;
  const uint32_t pixels = tl->tile_w * tl->tile_h;
  if (pixels > 512 || pixels % 32 != 0) return sc_fail(ctx, SC_ERR_INVALID_ARG, "tile must hold 32..512 pixels, multiple of 32");
  const uint64_t grid = (uint64_t)n_views * a.num_tiles;
  if (grid == 0) return SC_OK;
  const float n_scalars = (float)tl->width * (float)tl->height * 3.0f;
  const float gscale = (2.0f / n_scalars) * mse_scale;
  const int ppt = pick_ppt(tl);
  if (ppt == 1 && pixels > 256) return sc_fail(ctx, SC_ERR_INVALID_ARG, "tile too large for one pixel per thread");
  const TakerChunks tk = takers ? *takers : TakerChunks{};
  return (ppt == 2 ? composite_ppt<2, LIST> : composite_ppt<1, LIST>)(
      ctx, a, (uint32_t)grid, pixels / ppt, rec, l, image, aux, target, gscale, dl_dc, loss, d_skip, work, tk);
}

sc_status launch_composite(sc_ctx* ctx, const float4* rec, uint32_t stride, uint32_t n_views, const uint32_t* payloads,
                           const uint32_t* ranges, const sc_tiling* tl, float4* image, uint2* aux, const float* target,
                           float mse_scale, float4* dl_dc, double* loss, uint32_t* d_skip,
                           const TakerChunks* takers) {
  ListArgs l{payloads, reinterpret_cast<const uint2*>(ranges), nullptr, 0, 0};
  return composite_list<LIST_PAIRS>(ctx, rec, stride, n_views, l, tl, image, aux, target, mse_scale, dl_dc, loss,
                                    d_skip, nullptr, 0, nullptr, false, takers);
}

sc_status launch_composite_items(sc_ctx* ctx, const float4* rec, uint32_t stride, uint32_t n_views,
                                 const uint32_t* item_keys, const uint32_t* item_ids, const uint32_t* item_ranges,
                                 const sc_tiling* tl, float4* image, uint2* aux, const float* target, float mse_scale,
                                 float4* dl_dc, double* loss, uint32_t* d_skip, uint64_t* work,
                                 uint32_t batch, const SceneDev* scenes, bool count_pairs,
                                 const TakerChunks* takers) {
  const BlendArgs a = blend_args(tl, stride);
  ListArgs l{item_ids, reinterpret_cast<const uint2*>(item_ranges), item_keys, (a.tiles_x + SC_SUPER - 1) / SC_SUPER,
             super_tiles_per_view(tl)};
  return composite_list<LIST_ITEMS>(ctx, rec, stride, n_views, l, tl, image, aux, target, mse_scale, dl_dc, loss,
                                    d_skip, work, batch, scenes, count_pairs, takers);
}

// warps per (view, tile) of a blend launch: one takers' head each
uint32_t blend_warps_per_tile(const sc_tiling* tl) { return tl->tile_w * tl->tile_h / pick_ppt(tl) / 32; }

// Classes from 1024, 512 and 192 takers up, 256 tiles each: four classes of 128
// from 2048, 1024, 512 and 256 left the 3M-splat step at 1.67 ms, a last class from
// 256 the 200k-splat one at 134 us.
__global__ void __launch_bounds__(256) k_heavy_tiles(TakerChunks t, uint32_t tiles, uint32_t warps,
                                                     const uint32_t* __restrict__ skip) {
  sc_after_previous();
  const uint32_t vt = blockIdx.x * 256 + threadIdx.x;
  if (vt >= tiles || (skip && (*skip & SC_DEVERR_SKIP))) return;
  uint32_t most = 0;
  for (uint32_t w = 0; w < warps; ++w) most = max(most, t.head[(size_t)vt * warps + w].y);
  const uint32_t c = most >= 1024 ? 0 : most >= 512 ? 1 : 2;
  uint32_t at = HEAVY_CAP;
  if (most >= 192) at = atomicAdd(t.n_heavy + c, 1u);
  if (at < HEAVY_CAP) t.heavy[c * HEAVY_CAP + at] = vt;
  t.is_heavy[vt] = at < HEAVY_CAP;
}

sc_status launch_heavy_tiles(sc_ctx* ctx, const TakerChunks& takers, uint32_t tiles, uint32_t warps_per_tile,
                             const uint32_t* d_skip) {
  if (tiles == 0) return SC_OK;
  sc_launch(ctx, k_heavy_tiles, (tiles + 255) / 256, 256, 0, takers, tiles, warps_per_tile, d_skip);
  return sc_check_launch(ctx, "k_heavy_tiles");
}

// ---------------------------------------------------------------- MSE (standalone)
__global__ void k_mse_views(const float4* __restrict__ pred, const float* __restrict__ target, uint64_t P,
                            float gscale, float4* __restrict__ dl_dc, double* __restrict__ loss) {
  __shared__ double sred[8];
  const uint32_t v = blockIdx.y;
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  double sq = 0.0;
  if (i < P) {
    const uint64_t q = (uint64_t)v * P + i;
    const float4 p = pred[q];
    const float dx = p.x - target[3 * q], dy = p.y - target[3 * q + 1], dz = p.z - target[3 * q + 2];
    dl_dc[q] = make_float4(dx * gscale, dy * gscale, dz * gscale, 0.0f);
    sq = (double)(dx * dx + dy * dy + dz * dz);
  }
  if (loss) {
    const double s = block_sum(sq, sred);
    if (threadIdx.x == 0 && s != 0.0) atomicAdd(&loss[v], s);
  }
}

sc_status launch_mse(sc_ctx* ctx, const float4* pred, const float* target, uint64_t P, uint32_t n_views, float scale,
                     float4* dl_dc, double* loss) {
  if (P == 0 || n_views == 0) return SC_OK;
  const float n_scalars = (float)P * 3.0f;
  const float gscale = (2.0f / n_scalars) * scale;
  dim3 grid((unsigned)sc_div_up(P, 256), n_views);
  k_mse_views<<<grid, 256, 0, ctx->stream>>>(pred, target, P, gscale, dl_dc, loss);
  return sc_check_launch(ctx, "k_mse_views");
}

// ---------------------------------------------------------------- backward
// Reduce-scatter of N values over the warp by recursive halving: at the level
// of lane bit O a lane keeps one half of its slots and sends the other half to
// lane ^ O, which keeps the opposite half (2 selects and 1 shuffle per slot
// pair, ceil(n / 2) slots left; the adds go two at a time as packed f32x2
// adds, the same roundings); after the 5 levels every lane holds one slot.
// rs_owner<N>(lane) is the value index that slot totals (-1: a padding
// slot).  N = 9: 12 shuffles; N = 18: 20.
template <int N, int O>
__device__ __forceinline__ void rs_half(const float* x, float* y, int lane) {
  constexpr int M = (N + 1) / 2;
  float kp[M], rv[M];
  const bool bit = lane & O;
#pragma unroll
  for (int i = 0; i < M; ++i) {
    const float lo = x[i];
    const float hi = i + M < N ? x[i + M] : 0.0f;
    const float send = bit ? lo : hi;
    kp[i] = bit ? hi : lo;
    rv[i] = __shfl_xor_sync(FULL_MASK, send, O);
  }
#pragma unroll
  for (int i = 0; i + 1 < M; i += 2) {
    const float2 t = __fadd2_rn(make_float2(kp[i], kp[i + 1]), make_float2(rv[i], rv[i + 1]));
    y[i] = t.x; y[i + 1] = t.y;
  }
  if constexpr (M & 1) y[M - 1] = kp[M - 1] + rv[M - 1];
}
template <int N, int O>
__device__ __forceinline__ float rs_level(const float* x, int lane) {
  constexpr int M = (N + 1) / 2;
  float y[M];
  rs_half<N, O>(x, y, lane);
  if constexpr (O == 1) {
    static_assert(M == 1, "at most 32 values");
    return y[0];
  } else {
    return rs_level<M, O / 2>(y, lane);
  }
}
template <int N>
__device__ __forceinline__ float warp_reduce_scatter(const float (&x)[N], int lane) {
  return rs_level<N, 16>(x, lane);
}
template <int N>
__device__ __forceinline__ int rs_owner(int lane) {
  int lo = 0, len = N, n = N;
  for (int o = 16; o >= 1; o >>= 1) {
    const int m = (n + 1) / 2;
    if (lane & o) { lo += m; len = max(len - m, 0); } else { len = min(len, m); }
    n = m;
  }
  return len >= 1 ? lo : -1;
}

// Entries per warp reduction of the general path: 2 (an 18-value
// reduce-scatter, 20 shuffles for two entries).  3 entries (27 values, 28
// shuffles) measured slower at 80 registers; more than 3 do not fit the 32
// lanes.
constexpr int RS_E = 2;

// Octet reduction (two pixels per thread, tile width a multiple of 8: the 8
// lanes of an octet own 8 consecutive columns of one row pair).  While a warp
// walks its entries, each lane writes its two pixels' h and T alpha of an entry
// that some pixel of the warp takes into one row of a warp-private shared
// buffer; every OCT_E rows the warp turns round: lane (q, e) sums entry e over
// the 8 columns and 2 rows of octet q, in packed f32x2 over the two rows, so
// the 64-pixel sums of 9 quantities cost 8 row loads and 7 packed operations a
// column for 8 entries at once, and the four octets' partial sums meet in a
// two-level reduce-scatter (8 shuffles for 8 entries).  Per entry and warp that
// is about 17 instructions instead of the about 50 of the reduce-scatter over
// all 32 lanes.  A row is padded by one float4, so both the rows' stores and
// the turned loads (8 lanes, 8 rows, one column) touch all banks once.
constexpr int OCT_E = 8;
constexpr int OCT_ROW = 33;  // float4 per row: 32 lanes and the pad

// shared memory of one backward warp
struct OctSmem {
  float4 row[OCT_E * OCT_ROW];
  float4 rg[36];  // dL/dC red and green of a lane's two pixels; octet q at 9 q
  float2 b[36];   // blue
};
struct SumSmem {
  float sum[20];  // a reduce-scatter's 18 totals
};
template <typename FEED, bool OCT>
struct BwdSmem {
  typename FEED::Smem feed;
  typename std::conditional<OCT, OctSmem, SumSmem>::type red;
};

// Compensated accumulation of x into the sum *s, the rounding error of the
// addition going to *c: the atomic returns the old sum, the device forms the
// same rounded sum again (an atomic float add rounds to nearest) and Knuth's
// TwoSum gives the exact error of that addition.  *s + *c then carries the
// total to within about one rounding of the final value, whatever the number
// and the order of the tiles that add to it (plain float atomics: an error
// growing with the number of additions and their magnitudes).
__device__ __forceinline__ void twosum_atomic_add(float* s, float* c, float x) {
  if (x == 0.0f) return;
  const float old = atomicAdd(s, x);
  const float sum = __fadd_rn(old, x);
  const float bp = __fsub_rn(sum, old);
  const float err = __fadd_rn(__fsub_rn(old, __fsub_rn(sum, bp)), __fsub_rn(x, bp));
  if (err != 0.0f) atomicAdd(c, err);
}
__device__ __forceinline__ void twosum_atomic_add4(float4* s, float4* c, float4 x) {
  float* sp = reinterpret_cast<float*>(s);
  float* cp = reinterpret_cast<float*>(c);
  twosum_atomic_add(sp, cp, x.x);
  twosum_atomic_add(sp + 1, cp + 1, x.y);
  twosum_atomic_add(sp + 2, cp + 2, x.z);
}

// MODE is the sc_bwd_mode.  In exact mode a pixel takes part from its last
// contributor down to the start of the tile's list and never stops early, so
// the early-exit bookkeeping exists only in reference mode.
// With a target, the MSE's dL/dC (and the loss, added to loss[view]) is formed
// here from the forward image instead of being read from dl_dc.
// COMP: the per-(view, splat) totals across tiles are accumulated with
// twosum_atomic_add into proj_grad and the compensation records proj_comp.
// OCT: the octet reduction (PPT 2 and a tile width that is a multiple of 8).
// LIST_TAKERS: exact mode over the entries that the forward wrote down per warp.
// A warp sends its sums of an entry to global memory itself, one float4 atomic
// per part of the entry's record.
// The tiles with the longest walks (at silhouettes, where pixels never saturate:
// thousands of takers against some 60 on average) start first: in tile order the
// last of them began half-way, and a one-view step waited for it alone (1M
// splats, one 1080p view: 272 -> 208 us; 200k splats at 1024x1024: 142 -> 127 us;
// 3M splats, 4 views: 1.62 -> 1.50 ms; 8 views of 1M 1.372 -> 1.369 ms).
template <int PPT, int MODE, int LIST, bool COMP, bool COUNT, bool OCT>
__global__ void __launch_bounds__(256) k_composite_backward(const float4* __restrict__ rec, ListArgs l, BlendArgs a,
                                                            const float4* __restrict__ fwd,
                                                            const float4* __restrict__ dl_dc,
                                                            const float* __restrict__ target, float gscale,
                                                            double* __restrict__ loss,
                                                            const uint2* __restrict__ aux,
                                                            float4* __restrict__ proj_grad,
                                                            const uint32_t* __restrict__ skip,
                                                            unsigned long long* __restrict__ work,
                                                            float4* __restrict__ proj_comp, TakerChunks takers) {
  sc_after_previous();
  static_assert(!OCT || PPT == 2, "the octet reduction takes two pixels per thread");
  static_assert(LIST != LIST_TAKERS || MODE == SC_BWD_EXACT, "the takers are the exact mode's entries");
  using FEED = typename std::conditional<LIST == LIST_TAKERS, TakerFeed, ListFeed<LIST, true>>::type;
  extern __shared__ float4 sbuf[];  // one BwdSmem per warp
  __shared__ double s_red[8];
  __shared__ uint32_t s_work[2];
  if (skip && (*skip & SC_DEVERR_SKIP)) return;
  const uint32_t warp = threadIdx.x >> 5;
  BwdSmem<FEED, OCT>& sm = reinterpret_cast<BwdSmem<FEED, OCT>*>(sbuf)[warp];
  uint32_t vt = blockIdx.x;
  if (LIST == LIST_TAKERS && takers.heavy) {  // the heavy tiles' blocks come first
    constexpr uint32_t H = HEAVY_CLASSES * HEAVY_CAP;
    if (vt < H) {
      if (vt % HEAVY_CAP >= takers.n_heavy[vt / HEAVY_CAP]) return;
      vt = takers.heavy[vt];
    } else {
      vt -= H;
      if (takers.is_heavy[vt]) return;
    }
  }
  const uint32_t v = vt / a.num_tiles, tile = vt - v * a.num_tiles;
  const uint32_t ty = tile / a.tiles_x, tx = tile - ty * a.tiles_x;
  uint32_t px, py0;
  tile_pixel<PPT>(a, tx, ty, px, py0);
  const float fx = (float)px + 0.5f;
  uint32_t W, H;
  float gs;
  view_dims(a, v, gscale, W, H, gs);
  uint32_t begin = 0, len = 0, bit = 0;
  uint2 head = make_uint2(0u, 0u);
  if constexpr (LIST == LIST_TAKERS) {
    head = takers.head[(size_t)vt * (blockDim.x >> 5) + warp];
    len = head.y;
  } else {
    const uint2 r = list_range<LIST>(l, a, v, tx, ty, tile, bit);
    begin = r.x;
    len = r.y > r.x ? r.y - r.x : 0u;
  }
  const float4* vrec = rec + (size_t)3 * v * a.stride;
  float4* vgrad = proj_grad + (size_t)3 * v * a.stride;

  // GS = dL/dC . S, the accumulated colour behind the pixel dotted with its
  // colour gradient: dL/dalpha_i = (T_{i+1} (dL/dC . c_i) - GS) / (1 - alpha_i)
  float T[PPT], gr[PPT], gg[PPT], gb[PPT], GS[PPT], fy[PPT];
  uint32_t stop[PPT];
  bool done[PPT];
  uint32_t tstop = 0;
  bool all_done = true;
  double sq = 0.0;
#pragma unroll
  for (int q = 0; q < PPT; ++q) {
    const uint32_t py = py0 + q;
    fy[q] = (float)py + 0.5f;
    T[q] = 1.0f; gr[q] = gg[q] = gb[q] = 0.f; GS[q] = 0.f;
    stop[q] = 0;
    done[q] = !(px < W && py < H);
    if (!done[q]) {
      const size_t pix = (size_t)v * a.pixels + (size_t)py * a.width + px;
      float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
      if (target || MODE == SC_BWD_REF) c = fwd[pix];
      if (target) {
        const float3 d = mse_pixel(c.x, c.y, c.z, target + 3 * pix, gs, sq);
        gr[q] = d.x; gg[q] = d.y; gb[q] = d.z;
      } else {
        const float4 d = dl_dc[pix];
        gr[q] = d.x; gg[q] = d.y; gb[q] = d.z;
      }
      if (MODE == SC_BWD_REF) {
        T[q] = 1.0f - c.w;
        stop[q] = len;
      } else {
        const uint2 x = aux[pix];
        T[q] = __uint_as_float(x.x);
        stop[q] = min(x.y, len);
      }
      tstop = max(tstop, stop[q]);
    }
    all_done &= done[q];
  }
  if (target && loss) {  // every CTA, the ones with an empty list too
    const double sum = block_sum(sq, s_red);
    if (threadIdx.x == 0 && sum != 0.0) atomicAdd(&loss[v], sum);
  }
  // the walk starts at the warp's last contributor
  const uint32_t hi0 = __reduce_max_sync(FULL_MASK, tstop);
  uint32_t staged = 0, w_pix = 0;
  if (hi0 > 0) {
    const int lane = threadIdx.x & 31;
    // general path: after the 18-value reduce-scatter of two entries this lane
    // holds one value: value rs_idx % 9 of entry rs_idx / 9
    const int rs_idx = rs_owner<9 * RS_E>(lane);
    // octet reduction: this lane turns to entry row oe of octet oq, and holds
    // after the two levels the three sums of part oq of that entry's gradient
    const int oe = lane & 7, oq = lane >> 3;
    const float fx_oct = fx - (float)oe;  // the octet's first column (the lane's own octet is oq)
    if constexpr (OCT) {  // warp-private: read after the __syncwarp of the first turn
      sm.red.rg[oq * 9 + oe] = make_float4(gr[0], gr[PPT - 1], gg[0], gg[PPT - 1]);
      sm.red.b[oq * 9 + oe] = make_float2(gb[0], gb[PPT - 1]);
    }
    // the positions below lo0 are behind no pixel's last contributor; none with a
    // pixel outside the image, whose walk must stay empty
    uint32_t low = stop[0];
#pragma unroll
    for (int q = 1; q < PPT; ++q) low = min(low, stop[q]);
    const uint32_t lo0 = MODE == SC_BWD_EXACT ? __reduce_min_sync(FULL_MASK, low) : 0u;
    FEED feed = [&]() {
      if constexpr (LIST == LIST_TAKERS) return TakerFeed(sm.feed, takers, vrec, head);
      else return ListFeed<LIST, true>(sm.feed, l, vrec, begin, hi0, bit, STAGE);
    }();
    // part `part` of the gradient record of the stage's entry i, from its sums m
    // over the warp's pixels of h = dL/dalpha * gauss and its moments in (dx,
    // dy): with the splat's opacity and conic (a, b, c)
    // (rasterize_backward.wgsl:174-185) dpower = op h, dmean = dpower (a dx +
    // b dy, b dx + c dy), dconic = dpower (-1/2)(dx^2, 2 dx dy, dy^2); the
    // opacity and colour gradients are the sums themselves
    auto send = [&](uint32_t i, int part, float3 m) {
      float4 g = make_float4(m.x, m.y, m.z, 0.0f);
      if (part < 2) {
        const float4 cb = feed.rec()[3 * i + 1];
        const float op = feed.rec()[3 * i + 2].w;
        if (part == 0) {
          g.x = op * (cb.x * m.x + cb.y * m.y);
          g.y = op * (cb.y * m.x + cb.z * m.y);
        } else {
          g.x = -0.5f * op * m.x; g.y = -op * m.y; g.z = -0.5f * op * m.z;
        }
      }
      const size_t o = (size_t)3 * feed.id()[i] + part;
      if constexpr (COMP)
        twosum_atomic_add4(vgrad + o, proj_comp + (size_t)3 * v * a.stride + o, g);
      else if (g.x != 0.f || g.y != 0.f || g.z != 0.f)
        atomicAdd(vgrad + o, g);
    };
    float2 T2 = make_float2(T[0], T[PPT - 1]), NG2 = f2(0.f);  // NG = -GS
    const float2 gr2 = make_float2(gr[0], gr[PPT - 1]), gg2 = make_float2(gg[0], gg[PPT - 1]);
    const float2 gb2 = make_float2(gb[0], gb[PPT - 1]), fy2 = make_float2(fy[0], fy[PPT - 1]);
    bool stopped = false;
    // A pixel that skips an entry carries zeros for it, which add nothing unless
    // they meet a value that is not finite: a pixel's dL/dC or T, or the entry's
    // record.  The entries of a list that some pixel need not have taken are then
    // walked with `gate`: a skipping pixel leaves its state alone and adds an
    // exact zero, and an entry that no pixel of the warp takes sends nothing.
    // (On every entry the gate cost a stage-by-stage step of 100k splats at 800x600
    // 12 us of 508, apart 1; one of 61k at 1013x571, 3 views, in the reference's
    // mode 6 of 798 either way.)
    uint32_t took = 0;  // with gate: the rows that this thread's pixels took
    bool odd = false;   // the warp has such a pixel
    if constexpr (PPT == 2 && (LIST != LIST_TAKERS || !OCT)) {
      float s = 0.0f;
#pragma unroll
      for (int q = 0; q < PPT; ++q) s += fabsf(gr[q]) + fabsf(gg[q]) + fabsf(gb[q]) + fabsf(T[q]);
      odd = __any_sync(FULL_MASK, !(s < ORDINARY));
    }
    // octet path: a thread's two pixels' (h, -T alpha) of entry i (zeros where a
    // pixel skips it).  Alpha is carried negated, which needs no negations in
    // the packed operations; a skipping pixel gets alpha 0, so it keeps its T
    // (1 / 1 is exact) and its sums.
    // `plain`: the stage's records are plain and no pixel of the warp stops
    // behind its entries, which leaves the alpha >= 1/255 test alone.
    auto entry2 = [&](auto plain, auto gate, uint32_t i, uint32_t row, const float4* r) -> float4 {
      constexpr bool PLAIN = decltype(plain)::value;
      const float4 ra = r[0], rb = r[1], rc = r[2];
      const EntryGeom e = entry_geom(fx, ra, rb);
      float2 dy, g, araw, al;
      bool v0, v1;
      eval_alpha2<PLAIN>(e, rb.z, fy2, ra.y, rc.w, dy, g, araw, al, v0, v1);
      const uint32_t j = PLAIN ? 0u : feed.pos(i);
      if (!PLAIN) {
        v0 &= (MODE == SC_BWD_EXACT || !done[0]) && j < stop[0];
        v1 &= (MODE == SC_BWD_EXACT || !done[PPT - 1]) && j < stop[PPT - 1];
      }
      float2 am = make_float2(v0 ? -al.x : 0.0f, v1 ? -al.y : 0.0f);
      const float2 oma = __fadd2_rn(f2(1.0f), am);
      const float2 inv = make_float2(rcp_approx(oma.x), rcp_approx(oma.y));
      float2 Tn = __fmul2_rn(T2, inv);  // T_i = T_{i+1} / (1 - alpha_i)
      if (MODE == SC_BWD_REF) {
        if (v0 && Tn.x > 1.0001f) { done[0] = true; v0 = false; am.x = 0.0f; Tn.x = T2.x; }
        if (v1 && Tn.y > 1.0001f) { done[PPT - 1] = true; v1 = false; am.y = 0.0f; Tn.y = T2.y; }
      }
      const float2 gm = make_float2(v0 && (PLAIN || araw.x < ALPHA_MAX) ? g.x : 0.0f,
                                    v1 && (PLAIN || araw.y < ALPHA_MAX) ? g.y : 0.0f);
      float2 ta = __fmul2_rn(Tn, am);
      // dC/dalpha = T_i c - S / (1 - alpha) = (T_{i+1} c - S) / (1 - alpha)
      const float2 dc = make_float2(fmaf(gb2.x, rc.z, fmaf(gg2.x, rc.y, gr2.x * rc.x)),
                                    fmaf(gb2.y, rc.z, fmaf(gg2.y, rc.y, gr2.y * rc.x)));
      float2 h = __fmul2_rn(__fmul2_rn(inv, __ffma2_rn(T2, dc, NG2)), gm);
      float2 ng = __ffma2_rn(ta, dc, NG2);
      if constexpr (decltype(gate)::value) {
        if (!v0) { h.x = ta.x = 0.0f; ng.x = NG2.x; Tn.x = T2.x; }
        if (!v1) { h.y = ta.y = 0.0f; ng.y = NG2.y; Tn.y = T2.y; }
        if (v0 || v1) took |= 1u << row;
      }
      NG2 = ng;
      T2 = Tn;
      if constexpr (COUNT) w_pix += (uint32_t)v0 + (uint32_t)v1;
      if (MODE == SC_BWD_REF) all_done = (done[0] || j == 0) && (done[PPT - 1] || j == 0);
      return make_float4(h.x, h.y, ta.x, ta.y);
    };
    // turn round: the sums of entries i0 .. i0 + rows - 1 over the warp's pixels, and out
    auto turn = [&](auto gate, uint32_t i0, uint32_t rows) {
      if constexpr (OCT) {
        constexpr bool GATE = decltype(gate)::value;
        uint32_t taken = 0xFFFFFFFFu;
        if constexpr (GATE) {
          taken = __reduce_or_sync(FULL_MASK, took);
          took = 0;
        }
        __syncwarp();
        const float4* w = sm.red.row + oe * OCT_ROW + oq * 8;
        const float4 m = feed.rec()[3 * (i0 + oe)];
        float2 sh = f2(0.f), shx = sh, shxx = sh, cr = sh, cg = sh, cb = sh;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float4 x = w[j];
          const float2 h = make_float2(x.x, x.y), ta = make_float2(x.z, x.w);
          float4 rg = sm.red.rg[oq * 9 + j];
          float2 b = sm.red.b[oq * 9 + j];
          if constexpr (GATE) {  // T alpha of a pixel that skips the entry is 0
            if (ta.x == 0.0f) rg.x = rg.z = b.x = 0.0f;
            if (ta.y == 0.0f) rg.y = rg.w = b.y = 0.0f;
          }
          const float2 dx = f2(__fadd_rn(fx_oct + (float)j, -m.x));
          const float2 hx = __fmul2_rn(h, dx);
          sh = __fadd2_rn(sh, h);
          shx = __fadd2_rn(shx, hx);
          shxx = __ffma2_rn(hx, dx, shxx);
          cr = __ffma2_rn(ta, make_float2(rg.x, rg.y), cr);
          cg = __ffma2_rn(ta, make_float2(rg.z, rg.w), cg);
          cb = __ffma2_rn(ta, b, cb);
        }
        const float2 dy = __fadd2_rn(fy2, f2(-m.y));
        const float2 hy = __fmul2_rn(sh, dy), hxy = __fmul2_rn(shx, dy);
        const float c[12] = {shx.x + shx.y,   hy.x + hy.y,   sh.x + sh.y,
                             shxx.x + shxx.y, hxy.x + hxy.y, fmaf(hy.x, dy.x, hy.y * dy.y),
                             -(cr.x + cr.y),  -(cg.x + cg.y), -(cb.x + cb.y), 0.f, 0.f, 0.f};
        float c6[6], c3[3];
        rs_half<12, 16>(c, c6, lane);
        rs_half<6, 8>(c6, c3, lane);
        if (oe < rows && oq < 3 && (!GATE || (taken >> oe & 1u))) send(i0 + oe, oq, make_float3(c3[0], c3[1], c3[2]));
        __syncwarp();  // the rows may be written again
      }
    };
    // general path: this thread's raw sums of entry i over its pixels into
    // c[0..8]: h = dL/dalpha * gauss (the opacity gradient), its first and second
    // moments in (dx, dy), and the colour gradient; whether one of them took it.
    // Two pixels go through entry2's packed arithmetic (tiles of 4x16, 50k splats at
    // 640x480, backward over lists: 141 us pixel by pixel, 124 so; with the
    // reference's mode 203 and 167)
    auto entry = [&](auto gate, uint32_t i, const float4* r, float* c) -> bool {
      const float4 ra = r[0], rb = r[1];
      const EntryGeom e = entry_geom(fx, ra, rb);
      if constexpr (PPT == 2) {
        const float4 x = entry2(std::false_type{}, gate, i, 0, r);
        const float2 h = make_float2(x.x, x.y), ta = make_float2(-x.z, -x.w);
        const float2 dy = __fadd2_rn(fy2, f2(-ra.y)), hy = __fmul2_rn(h, dy);
        c[2] = h.x + h.y;
        c[1] = hy.x + hy.y;
        c[5] = fmaf(hy.x, dy.x, hy.y * dy.y);
        c[0] = c[2] * e.dx;  // both pixels share dx
        c[3] = c[0] * e.dx;
        c[4] = c[1] * e.dx;
        // T alpha of a skipping pixel is a zero without a sign here, of a taking one never
        const bool t0 = __float_as_uint(x.z) != 0u, t1 = __float_as_uint(x.w) != 0u;
        const bool m0 = !decltype(gate)::value || t0, m1 = !decltype(gate)::value || t1;
        c[6] = fmaf(ta.x, m0 ? gr2.x : 0.0f, ta.y * (m1 ? gr2.y : 0.0f));
        c[7] = fmaf(ta.x, m0 ? gg2.x : 0.0f, ta.y * (m1 ? gg2.y : 0.0f));
        c[8] = fmaf(ta.x, m0 ? gb2.x : 0.0f, ta.y * (m1 ? gb2.y : 0.0f));
        return t0 || t1;
      } else {
        const float4 rc = r[2];
        const uint32_t j = feed.pos(i);
        bool contrib = false;
#pragma unroll
        for (int q = 0; q < 9; ++q) c[q] = 0.0f;
        if ((MODE == SC_BWD_EXACT || !done[0]) && j < stop[0]) {
          const float dy = __fadd_rn(fy[0], -ra.y);
          float g, araw, alpha;
          if (eval_alpha(e, rb.z, dy, rc.w, g, araw, alpha)) {
            const float inv = rcp_approx(__fadd_rn(1.0f, -alpha));
            const float Tn = __fmul_rn(T2.x, inv);  // T_i = T_{i+1} / (1 - alpha_i)
            if (MODE == SC_BWD_REF && Tn > 1.0001f) {
              done[0] = true;
            } else {
              const float ta = __fmul_rn(Tn, alpha);
              c[6] = gr[0] * ta; c[7] = gg[0] * ta; c[8] = gb[0] * ta;
              const float dc = gr[0] * rc.x + gg[0] * rc.y + gb[0] * rc.z;
              const float galpha = inv * (T2.x * dc + NG2.x);
              const float h = araw < ALPHA_MAX ? galpha * g : 0.0f;
              const float hx = h * e.dx, hy = h * dy;
              c[0] = hx; c[1] = hy; c[2] = h;
              c[3] = hx * e.dx; c[4] = hx * dy; c[5] = hy * dy;
              NG2.x -= ta * dc;
              T2.x = Tn;
              contrib = true;
              if constexpr (COUNT) ++w_pix;
            }
          }
        }
        if (MODE == SC_BWD_REF) all_done = done[0] || j == 0;
        return contrib;
      }
    };
    const WarpRect rect = LIST == LIST_TAKERS ? WarpRect{} : warp_rect(px, py0, PPT);
    for (uint32_t n_raw = feed.gather(); n_raw > 0 && !stopped;) {
      const uint32_t n = feed.ready(n_raw, rect);
      n_raw = feed.gather();
      const float4* sr = feed.rec();
      staged += n;
      uint32_t i = 0;
      if constexpr (OCT) {
        float4* row = sm.red.row + lane;
        auto walk = [&](auto plain, auto gate) {
          constexpr int U = decltype(gate)::value ? 1 : OCT_E;  // the rare walk stays small
          for (; i + OCT_E <= n && !stopped; i += OCT_E) {
#pragma unroll U
            for (int e = 0; e < OCT_E; ++e) row[e * OCT_ROW] = entry2(plain, gate, i + e, e, sr + 3 * (i + e));
            turn(gate, i, OCT_E);
            if (MODE == SC_BWD_REF) stopped = __all_sync(FULL_MASK, all_done);
          }
          if (i < n && !stopped) {
            for (uint32_t e = 0; i + e < n; ++e) row[e * OCT_ROW] = entry2(plain, gate, i + e, e, sr + 3 * (i + e));
            turn(gate, i, n - i);
            if (MODE == SC_BWD_REF) stopped = __all_sync(FULL_MASK, all_done);
          }
        };
        bool plain = MODE == SC_BWD_EXACT && n > 0 && feed.pos(0) < lo0;
        if (plain) {
          const float4* r = sr + 3 * lane;
          plain = __all_sync(FULL_MASK, lane >= (int)n || plain_record(r[0], r[1], r[2].w));
        }
        bool gate = false;
        if constexpr (LIST != LIST_TAKERS) gate = odd || feed.odd;
        if (LIST != LIST_TAKERS && gate) walk(std::false_type{}, std::true_type{});
        else if (plain) walk(std::true_type{}, std::false_type{});
        else walk(std::false_type{}, std::false_type{});
      } else {
        // two entries together: one 18-value reduce-scatter, unless no pixel took them
        auto walk = [&](auto gate) {
          for (; i < n && !stopped; i += 2) {
            const bool two = i + 1 < n;
            float c[9 * RS_E];
#pragma unroll
            for (int q = 9; q < 9 * RS_E; ++q) c[q] = 0.0f;
            const bool any0 = __any_sync(FULL_MASK, entry(gate, i, sr + 3 * i, c));
            const bool any1 = two && __any_sync(FULL_MASK, entry(gate, i + 1, sr + 3 * i + 3, c + 9));
            if (any0 || any1) {
              const float w = warp_reduce_scatter<9 * RS_E>(c, lane);
              if (rs_idx >= 0) sm.red.sum[rs_idx] = w;
              __syncwarp();
              if (lane < 3 ? any0 : lane < 6 && any1) {
                const float* m = sm.red.sum + 3 * lane;
                send(i + lane / 3, lane % 3, make_float3(m[0], m[1], m[2]));
              }
              __syncwarp();
            }
            if (MODE == SC_BWD_REF) stopped = __all_sync(FULL_MASK, all_done);
          }
        };
        bool gate = odd;
        if constexpr (LIST != LIST_TAKERS) gate = gate || feed.odd;
        if (PPT == 2 && gate) walk(std::true_type{});
        else walk(std::false_type{});
      }
      __syncwarp();  // the stage may be written again
    }
    cp_async_wait_all();
  }
  add_tile_work(work, hi0, staged, s_work);
  if constexpr (COUNT) add_pixel_pairs(work, w_pix, s_red);
}

template <int PPT, int LIST, int MODE, bool OCT>
static sc_status backward_ppt(sc_ctx* ctx, const BlendArgs& a, uint32_t grid, uint32_t threads, const float4* rec,
                              const ListArgs& l, const float4* fwd, const float4* dl_dc, const float* target,
                              float gscale, double* loss, const uint2* aux, float4* proj_grad,
                              const uint32_t* d_skip, uint64_t* work, float4* proj_comp, const TakerChunks& takers) {
  using FEED = typename std::conditional<LIST == LIST_TAKERS, TakerFeed, ListFeed<LIST, true>>::type;
  const bool count = work && a.count_pairs;
  auto kern = proj_comp ? (count ? k_composite_backward<PPT, MODE, LIST, true, true, OCT>
                                 : k_composite_backward<PPT, MODE, LIST, true, false, OCT>)
                        : (count ? k_composite_backward<PPT, MODE, LIST, false, true, OCT>
                                 : k_composite_backward<PPT, MODE, LIST, false, false, OCT>);
  const size_t smem = threads / 32 * sizeof(BwdSmem<FEED, OCT>);
  if (smem > 48 * 1024)
    SC_CUDA_TRY(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), "smem attr");
  if (LIST == LIST_TAKERS && takers.heavy) grid += HEAVY_CLASSES * HEAVY_CAP;
  sc_launch(ctx, kern, grid, threads, smem, rec, l, a, fwd, dl_dc, target, gscale, loss, aux, proj_grad, d_skip,
            reinterpret_cast<unsigned long long*>(work), proj_comp, takers);
  return sc_check_launch(ctx, "k_composite_backward");
}

static sc_status backward_list(sc_ctx* ctx, const float4* rec, uint32_t stride, uint32_t n_views, int list,
                               const ListArgs& l, const sc_tiling* tl, const float4* fwd, const float4* dl_dc,
                               const float* target, float mse_scale, double* loss, int mode, const uint2* aux,
                               float4* proj_grad, const uint32_t* d_skip, uint64_t* work, float4* proj_comp,
                               const SceneDev* scenes, bool count_pairs, const TakerChunks* takers) {
  BlendArgs a = blend_args(tl, stride);
  a.scenes = scenes;
  a.count_pairs = count_pairs;
  const float gscale = (2.0f / ((float)tl->width * (float)tl->height * 3.0f)) * mse_scale;
  const uint32_t pixels = tl->tile_w * tl->tile_h;
  if (pixels > 512 || pixels % 32 != 0) return sc_fail(ctx, SC_ERR_INVALID_ARG, "tile must hold 32..512 pixels, multiple of 32");
  if (mode == SC_BWD_EXACT && !aux) return sc_fail(ctx, SC_ERR_INVALID_ARG, "exact backward needs the forward aux buffer");
  const uint64_t grid = (uint64_t)n_views * a.num_tiles;
  if (grid == 0) return SC_OK;
  const int ppt = pick_ppt(tl);
  if (ppt == 1 && pixels > 256) return sc_fail(ctx, SC_ERR_INVALID_ARG, "tile too large for one pixel per thread");
  // the octet reduction needs an octet's lanes in one row pair of the tile
  const bool oct = ppt == 2 && tl->tile_w % 8 == 0;
  const TakerChunks tk = takers ? *takers : TakerChunks{};
#define SC_BWD_SHAPES(LIST, MODE) \
  (oct ? backward_ppt<2, LIST, MODE, true> : ppt == 2 ? backward_ppt<2, LIST, MODE, false> \
                                                      : backward_ppt<1, LIST, MODE, false>)
  auto launch = takers && mode == SC_BWD_EXACT ? SC_BWD_SHAPES(LIST_TAKERS, SC_BWD_EXACT)
                : list == LIST_ITEMS ? (mode == SC_BWD_EXACT ? SC_BWD_SHAPES(LIST_ITEMS, SC_BWD_EXACT)
                                                             : SC_BWD_SHAPES(LIST_ITEMS, SC_BWD_REF))
                                     : (mode == SC_BWD_EXACT ? SC_BWD_SHAPES(LIST_PAIRS, SC_BWD_EXACT)
                                                             : SC_BWD_SHAPES(LIST_PAIRS, SC_BWD_REF));
#undef SC_BWD_SHAPES
  return launch(ctx, a, (uint32_t)grid, pixels / ppt, rec, l, fwd, dl_dc, target, gscale, loss, aux, proj_grad, d_skip,
                work, proj_comp, tk);
}

sc_status launch_composite_backward(sc_ctx* ctx, const float4* rec, uint32_t stride, uint32_t n_views,
                                    const uint32_t* payloads, const uint32_t* ranges, const sc_tiling* tl,
                                    const float4* fwd, const float4* dl_dc, int mode, const uint2* aux,
                                    float4* proj_grad, const uint32_t* d_skip, const float* target,
                                    float mse_scale, double* loss, float4* proj_comp, const TakerChunks* takers) {
  ListArgs l{payloads, reinterpret_cast<const uint2*>(ranges), nullptr, 0, 0};
  return backward_list(ctx, rec, stride, n_views, LIST_PAIRS, l, tl, fwd, dl_dc, target, mse_scale, loss, mode, aux,
                       proj_grad, d_skip, nullptr, proj_comp, nullptr, false, takers);
}

sc_status launch_composite_backward_items(sc_ctx* ctx, const float4* rec, uint32_t stride, uint32_t n_views,
                                          const uint32_t* item_keys, const uint32_t* item_ids,
                                          const uint32_t* item_ranges, const sc_tiling* tl, const float4* fwd,
                                          const float4* dl_dc, int mode, const uint2* aux, float4* proj_grad,
                                          const uint32_t* d_skip, const float* target, float mse_scale,
                                          double* loss, uint64_t* work, float4* proj_comp, const SceneDev* scenes,
                                          bool count_pairs, const TakerChunks* takers) {
  const BlendArgs a = blend_args(tl, stride);
  ListArgs l{item_ids, reinterpret_cast<const uint2*>(item_ranges), item_keys, (a.tiles_x + SC_SUPER - 1) / SC_SUPER,
             super_tiles_per_view(tl)};
  return backward_list(ctx, rec, stride, n_views, LIST_ITEMS, l, tl, fwd, dl_dc, target, mse_scale, loss, mode, aux,
                       proj_grad, d_skip, work, proj_comp, scenes, count_pairs, takers);
}

// proj_grad += proj_comp over n float4 (the compensated totals rounded once)
__global__ void k_fold_comp(float4* __restrict__ g, const float4* __restrict__ c, uint64_t n) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 x = g[i], y = c[i];
  g[i] = make_float4(x.x + y.x, x.y + y.y, x.z + y.z, x.w + y.w);
}

sc_status launch_fold_comp(sc_ctx* ctx, float4* proj_grad, const float4* proj_comp, uint64_t n_float4) {
  if (n_float4 == 0) return SC_OK;
  k_fold_comp<<<(unsigned)sc_div_up(n_float4, 256), 256, 0, ctx->stream>>>(proj_grad, proj_comp, n_float4);
  return sc_check_launch(ctx, "k_fold_comp");
}

// ---------------------------------------------------------------- tonemap (tonemap.wgsl:27-41)
__device__ __forceinline__ float srgb(float c) {
  c = fminf(fmaxf(c, 0.0f), 1.0f);
  return c > 0.0031308f ? 1.055f * powf(c, 1.0f / 2.4f) - 0.055f : c * 12.92f;
}
__device__ __forceinline__ uint8_t unorm8(float x) {
  x = fminf(fmaxf(x, 0.0f), 1.0f);
  return (uint8_t)__float2int_rn(x * 255.0f);
}
__global__ void k_tonemap(const float4* __restrict__ img, uint32_t w, uint32_t h, uchar4* __restrict__ out) {
  const uint32_t x = blockIdx.x * 16 + threadIdx.x, y = blockIdx.y * 16 + threadIdx.y;
  if (x >= w || y >= h) return;
  const size_t i = (size_t)y * w + x;
  const float4 p = img[i];
  const float r = p.x / (1.0f + fmaxf(p.x, 0.0f)), g = p.y / (1.0f + fmaxf(p.y, 0.0f)), b = p.z / (1.0f + fmaxf(p.z, 0.0f));
  out[i] = make_uchar4(unorm8(srgb(r)), unorm8(srgb(g)), unorm8(srgb(b)), unorm8(p.w));
}

sc_status launch_tonemap(sc_ctx* ctx, const float4* img, uint32_t w, uint32_t h, uint8_t* out) {
  if (w == 0 || h == 0) return SC_OK;
  dim3 grid((w + 15) / 16, (h + 15) / 16), block(16, 16);
  k_tonemap<<<grid, block, 0, ctx->stream>>>(img, w, h, reinterpret_cast<uchar4*>(out));
  return sc_check_launch(ctx, "k_tonemap");
}

}  // namespace sck
