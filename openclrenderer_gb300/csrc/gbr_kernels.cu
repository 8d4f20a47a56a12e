// gbr_kernels.cu — sm_103a kernels of the triangle pipeline.
//
// Compiled with --fmad=false: every fused multiply-add below is an explicit
// fmaf() standing for a `mad` of cl2.cl; all other float expressions round
// after each operation, as the determinism contract in gbr_math.h requires.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "gbr_internal.h"
#include "gbr_shade_math.h"

namespace gbr {
namespace {

__device__ __forceinline__ f3 ld3(const float* p) { return mk3(__ldg(p), __ldg(p + 1), __ldg(p + 2)); }
__device__ __forceinline__ f4 ld4(const float* p) {
  float4 v = __ldg(reinterpret_cast<const float4*>(p));
  f4 r; r.x = v.x; r.y = v.y; r.z = v.z; r.w = v.w;
  return r;
}

// Warp-aggregated "atomicAdd(&counter[key], 1)": lanes with the same key
// share one atomic.  Every lane of the warp must call it; inactive lanes pass
// active = false.  Returns this lane's old value + its rank within its key.
__device__ __forceinline__ uint32_t agg_inc(uint32_t* counter, uint32_t key, bool active) {
  const unsigned act = __ballot_sync(0xFFFFFFFFu, active);
  uint32_t res = 0;
  if (active) {
    const int lane = threadIdx.x & 31;
    const unsigned grp = __match_any_sync(act, key);
    const int leader = __ffs(grp) - 1;
    uint32_t old = 0;
    if (lane == leader) old = atomicAdd(&counter[key], (uint32_t)__popc(grp));
    old = __shfl_sync(grp, old, leader);
    res = old + (uint32_t)__popc(grp & ((1u << lane) - 1u));
  }
  return res;
}

// Colour-only arithmetic of the light loop: every use below feeds the colour
// continuously (no comparison, rounding or index depends on it), so the
// approximate division is covered by the 1/255 colour tolerance.  The
// hardware's approximations, taken as single instructions that flush subnormal
// operands and results to 0: a flushed result is far below a colour level, and
// where an operand can be subnormal (csqrt) it is dealt with.  (1080p kernel3
// 3,350 -> 3,060 instructions per pixel, 223 -> 210 us, against __fdividef,
// rsqrtf and __expf.)
__device__ __forceinline__ float ex2_ftz(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float rsqrt_ftz(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float crcp(float b) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(b));
  return r;
}

// A visible clipped triangle before it becomes a record.  (The second
// triangle of a split at the near clip, which is rare, is made after the first
// one is done with, so that only one is held at a time.)
struct Cand {
  f3 p[3];
  float mm[4];  // bbox4, or the smaller box of tight_box
  float area;   // of bbox4
  int box;      // tight_box
  bool inside;  // on_surface
  uint32_t key;
};

// prearrange's per-output culls (cl2.cl:4352-4377): returns false when the
// output is culled or its bbox is empty (ceil(area/op_size) == 0).
__device__ __forceinline__ bool cull_candidate(Cand& c, bool two_sided, float w, float h) {
  const f3* p = c.p;
  int valid = two_sided || backface_front(p[0], p[1], p[2]);
  int cond = (p[0].x < 0 && p[1].x < 0 && p[2].x < 0) ||
             (p[0].x >= w && p[1].x >= w && p[2].x >= w) ||
             (p[0].y < 0 && p[1].y < 0 && p[2].y < 0) ||
             (p[0].y >= h && p[1].y >= h && p[2].y >= h);
  if (!valid || cond) return false;
  f3 xpv = mk3(roundf(p[0].x), roundf(p[1].x), roundf(p[2].x));
  f3 ypv = mk3(roundf(p[0].y), roundf(p[1].y), roundf(p[2].y));
  bbox4(p[0], p[1], p[2], w, h, c.mm);
  c.area = (c.mm[1] - c.mm[0]) * (c.mm[3] - c.mm[2]);
  c.box = tight_box(xpv, ypv, w, h, c.mm);
  c.inside = on_surface(xpv, ypv, w, h);
  return c.area > 0.0f;
}

// rc: rconstant of the rounded vertices, which kernel3's plane reads too
__device__ __forceinline__ void make_rec(const Cand& c, uint32_t surface, RasterRec& R, float* rc) {
  const f3* p = c.p;
  f3 xpv = mk3(roundf(p[0].x), roundf(p[1].x), roundf(p[2].x));
  f3 ypv = mk3(roundf(p[0].y), roundf(p[1].y), roundf(p[2].y));
  f3 depths = mk3(rcp(over_far(p[0].z)), rcp(over_far(p[1].z)), rcp(over_far(p[2].z)));
  *rc = rconstant(xpv, ypv);
  plane_const(depths, xpv, ypv, *rc, &R.A, &R.B, &R.C);
  EdgeTest e = make_edge(xpv.x, ypv.x, xpv.y, ypv.y, xpv.z, ypv.z);
  // (a sign change commutes with rounding: the sign is folded in)
  R.s0 = e.s0 * e.sign; R.sa = e.sa * e.sign; R.sb = e.sb * e.sign;
  R.t0 = e.t0 * e.sign; R.ta = e.ta * e.sign; R.tb = e.tb * e.sign;
  R.bound = e.bound;
  R.key = c.key;
  R.xr = (uint32_t)c.mm[0] | ((uint32_t)c.mm[1] << 16);
  R.yr = (uint32_t)c.mm[2] | ((uint32_t)c.mm[3] << 16);
  R.surface = surface;
  R.kind = (c.box == kBoxTight ? kRecTight : 0u) | (c.inside ? kRecInside : near_surface(xpv, ypv) ? kRecNear : 0u);
}

__device__ __forceinline__ void store_rec(RasterRec* dst, const RasterRec& R) {
  float4* d = reinterpret_cast<float4*>(dst);
  d[0] = make_float4(R.A, R.B, R.C, R.bound);
  d[1] = make_float4(R.s0, R.sa, R.sb, 0.0f);
  d[2] = make_float4(R.t0, R.ta, R.tb, __uint_as_float(R.key));
  d[3] = make_float4(__uint_as_float(R.xr), __uint_as_float(R.yr), __uint_as_float(R.surface),
                     __uint_as_float(R.kind));
}

// Tile footprint of a record: inclusive fine tiles, or coarse tiles when its
// bbox4 touches more than ws.fine_max fine tiles (tiles of kTile <<
// ws.coarse_shift pixels).  A tight box counts and places only the tiles it
// touches itself; *ref is the number of tiles of the bbox4, what a scratch
// limit is measured against.
struct Foot {
  int tx0, tx1, ty0, ty1;
  bool coarse;
};
__device__ __forceinline__ int foot_count(const Foot& f) { return (f.tx1 - f.tx0 + 1) * (f.ty1 - f.ty0 + 1); }
__device__ __forceinline__ Foot footprint(uint32_t xr, uint32_t yr, uint32_t kind, const Workspace& ws, int* ref) {
  const uint32_t tight = kind & kRecTight;
  const int minx = xr & 0xFFFF, maxx = xr >> 16, miny = yr & 0xFFFF, maxy = yr >> 16;
  int bx0 = (minx - (int)tight) >> 4, by0 = max(miny - (int)tight, 0) >> 4;  // tight: minx >= 1
  Foot f;
  f.tx0 = minx >> 4; f.tx1 = (maxx - 1) >> 4;
  f.ty0 = miny >> 4; f.ty1 = (maxy - 1) >> 4;
  f.coarse = (f.tx1 - bx0 + 1) * (f.ty1 - by0 + 1) > ws.fine_max;
  const int sh = f.coarse ? ws.coarse_shift : 0;
  f.tx0 >>= sh; f.tx1 >>= sh; bx0 >>= sh;
  f.ty0 >>= sh; f.ty1 >>= sh; by0 >>= sh;
  *ref = (f.tx1 - bx0 + 1) * (f.ty1 - by0 + 1);
  return f;
}
static_assert(kTile == 16, "footprint shifts by 4");
// The tiles of a footprint one after another, as indices into the fine or
// coarse counters.
struct FootWalk {
  int tx, ty;
  __device__ __forceinline__ FootWalk(const Foot& f) : tx(f.tx0), ty(f.ty0) {}
  __device__ __forceinline__ uint32_t fine(const Surface& S) const { return S.tile_base + ty * S.tiles_x + tx; }
  __device__ __forceinline__ void next(const Foot& f) {
    if (++tx > f.tx1) {
      tx = f.tx0;
      ty++;
    }
  }
};
// Calls go(record, fine tile) for every (record, fine tile) pair of a warp's
// lanes, each with a record r and `mine' tiles (0: none).  Footprints of up to
// kLockstep tiles go lane by lane in lockstep, so that neighbouring triangles,
// which usually share tiles, can share an atomic (agg: go_agg(tile, on) for all
// lanes); larger ones are laid end to end and dealt out to the lanes, 32 pairs
// at a time (a lane walking its own 16 tiles is a chain of 16 atomics).
constexpr int kLockstep = 4;
template <class GoAgg, class Go>
__device__ __forceinline__ void each_fine_tile(const Foot& f, int mine, const Surface* S, uint32_t r, GoAgg go_agg,
                                               Go go) {
  constexpr unsigned full = 0xFFFFFFFFu;
  const bool big = mine > kLockstep;
  const int most = (int)__reduce_max_sync(full, big ? 0u : (uint32_t)mine);
  FootWalk walk(f);
  for (int it = 0; it < most; it++) {
    const bool on = !big && it < mine;
    go_agg(on ? walk.fine(*S) : 0u, on);
    walk.next(f);
  }
  if (!__any_sync(full, big)) return;
  const int lane = threadIdx.x & 31;
  int start = big ? mine : 0;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(full, start, o);
    if (lane >= o) start += v;
  }
  const int total = __shfl_sync(full, start, 31);
  start -= big ? mine : 0;  // exclusive
  const int w = f.tx1 - f.tx0 + 1, row = big ? S->tiles_x : 0;
  const uint32_t base = big ? S->tile_base + f.ty0 * row + f.tx0 : 0u;
#pragma unroll 2
  for (int t0 = 0; t0 < total; t0 += 32) {
    const int t = t0 + lane;
    int src = 0;  // the last lane whose pairs start at or before t
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      if (__shfl_sync(full, start, src + o) <= t) src += o;
    const int k = t - __shfl_sync(full, start, src), sw = __shfl_sync(full, w, src), srow = __shfl_sync(full, row, src);
    const uint32_t sbase = __shfl_sync(full, base, src), sr = __shfl_sync(full, r, src);
    if (t < total) {
      const int ky = k / sw;
      go(sr, sbase + (uint32_t)(ky * srow + (k - ky * sw)));
    }
  }
}
// Calls go(lane's record index, coarse tile) for every (record, coarse tile)
// pair of the lanes that have a coarse footprint: the warp takes one record
// after another, its lanes the tiles.  (A lane looping over its own record's
// tiles, 240 at 2560x1440, made the setup and the fill wait for the few warps
// of large records.)  Every lane of the warp calls it.
template <class Go>
__device__ __forceinline__ void each_coarse_tile(const Foot& f, bool coarse, const Surface* S, uint32_t r, Go go) {
  for (unsigned todo = __ballot_sync(0xFFFFFFFFu, coarse); todo; todo &= todo - 1) {
    const int src = __ffs(todo) - 1;
    const int tx0 = __shfl_sync(0xFFFFFFFFu, f.tx0, src), w = __shfl_sync(0xFFFFFFFFu, f.tx1, src) - tx0 + 1;
    const int ty0 = __shfl_sync(0xFFFFFFFFu, f.ty0, src), h = __shfl_sync(0xFFFFFFFFu, f.ty1, src) - ty0 + 1;
    const uint32_t row = (uint32_t)__shfl_sync(0xFFFFFFFFu, coarse ? S->ctiles_x : 0, src);
    const uint32_t base = __shfl_sync(0xFFFFFFFFu, coarse ? S->ctile_base : 0u, src) + ty0 * row + tx0;
    const uint32_t rr = __shfl_sync(0xFFFFFFFFu, r, src);
    // k / w as a product: exact while k * w < 2^20 (w <= 60, h <= 34: 64-pixel tiles of 3840x2160)
    const uint32_t inv = ((1u << 20) + (uint32_t)w - 1u) / (uint32_t)w;
#pragma unroll 1
    for (int k = threadIdx.x & 31; k < w * h; k += 32) {
      const uint32_t ky = ((uint32_t)k * inv) >> 20;
      go(rr, base + ky * row + ((uint32_t)k - ky * (uint32_t)w));
    }
  }
}

// point_in_tri of a record at pixel (fx, fy).
__device__ __forceinline__ bool rec_in_tri(const float4 q[3], float fx, float fy) {
  const float s = (q[1].x + q[1].y * fx) + q[1].z * fy;
  const float t = (q[2].x + q[2].y * fx) + q[2].z * fy;
  return s > -0.0001f && t > -0.0001f && (s + t) < q[0].w;
}

// One candidate as a record (and shade record for views).
__device__ __forceinline__ void write_rec(const Cand& c, uint32_t r, uint32_t surface, const Workspace& ws,
                                          bool view) {
  RasterRec R;
  float rc;
  make_rec(c, surface, R, &rc);
  store_rec(ws.rec + r, R);
  if (view) {  // what prep_shade needs, in the record's first 48 bytes
    uint32_t tri = c.key >> 1;
    float4* q = reinterpret_cast<float4*>(ws.srec + r);
    q[0] = make_float4(c.p[0].x, c.p[0].y, c.p[0].z, rc);
    q[1] = make_float4(c.p[1].x, c.p[1].y, c.p[1].z, __uint_as_float(tri));
    q[2] = make_float4(c.p[2].x, c.p[2].y, c.p[2].z, 0.0f);
  }
}

// Depth-only passes (cube faces): a candidate whose bbox has at most this
// many pixels is rasterised by its setup thread straight into the face with
// global atomicMin -- the same coverage tests and depths as the tile raster,
// and a minimum does not depend on order -- instead of becoming a record.
constexpr float kDirectArea = 64.0f;

// kernel1 of one small candidate into its cube face; returns the covered
// pixel count.  (Rows narrowed to their exact spans, with no test per pixel,
// were 5 % fewer instructions and 8 us slower on a 1M-triangle terrain: the
// lanes' spans differ more than their rows.)
__device__ __forceinline__ uint32_t direct_raster(const Cand& c, uint32_t* __restrict__ face) {
  RasterRec R;
  float rc;
  make_rec(c, 0u, R, &rc);
  const float4 q[3] = {make_float4(R.A, R.B, R.C, R.bound), make_float4(R.s0, R.sa, R.sb, 0.0f),
                       make_float4(R.t0, R.ta, R.tb, 0.0f)};
  const int x0 = (int)(R.xr & 0xFFFF), x1 = (int)(R.xr >> 16), y0 = (int)(R.yr & 0xFFFF), y1 = (int)(R.yr >> 16);
  uint32_t hits = 0;
  // row by row: the walk rule of the row's left-column pixel, then point_in_tri
  // (walk_skip_rows: 0 at once unless the bbox touches the top of the face;
  // a bbox of at most 64 pixels has at most 64 rows)
  uint64_t skip = 0;
  if (!(R.kind & kRecTight))
    skip = (uint64_t)walk_skip_rows(R.xr, R.yr, y0, min(y1, y0 + 32), y0, kOpSizeLight) |
           ((uint64_t)walk_skip_rows(R.xr, R.yr, y0 + 32, y1, y0 + 32, kOpSizeLight) << 32);
  for (int y = y0; y < y1; y++) {
    for (int x = x0 + (int)((skip >> (y - y0)) & 1u); x < x1; x++)
      if (rec_in_tri(q, (float)x, (float)y)) {
        atomicMin(face + (y * kLightBufferDim + x), depth_at(R.A, R.B, R.C, (float)x, (float)y));
        hits++;
      }
  }
  return hits;
}

// What the setup threads of a block add up before it reaches the pass's
// counters: one global atomic per counter and block instead of one per warp.
struct SetupSums {
  unsigned long long frags;
  uint32_t bins, vis, samples, warps;
  __device__ __forceinline__ void clear() {
    frags = 0;
    bins = vis = samples = warps = 0;
  }
};
struct SetupCounts {
  uint32_t frags = 0, bins = 0, vis = 0, samples = 0;  // of this lane
};
// Adds the lanes' counts to the block's.  (A lane's fragments of up to 12
// triangles: below 2^18.)
__device__ __forceinline__ void setup_add(SetupSums* b, const SetupCounts& c) {
  const uint32_t frags = __reduce_add_sync(0xFFFFFFFFu, c.frags), bins = __reduce_add_sync(0xFFFFFFFFu, c.bins);
  const uint32_t vis = __reduce_add_sync(0xFFFFFFFFu, c.vis), samples = __reduce_add_sync(0xFFFFFFFFu, c.samples);
  if ((threadIdx.x & 31) != 0) return;
  if (frags) atomicAdd(&b->frags, (unsigned long long)frags);
  if (bins) atomicAdd(&b->bins, bins);
  if (vis) atomicAdd(&b->vis, vis);
  if (samples) atomicAdd(&b->samples, samples);
}
// Every warp of the block calls it once, when it is done; the last one writes
// the block's sums.
__device__ __forceinline__ void setup_done(SetupSums* b, const Workspace& ws) {
  if ((threadIdx.x & 31) != 0) return;
  __threadfence_block();
  if (atomicAdd(&b->warps, 1u) + 1u != blockDim.x / 32) return;
  __threadfence_block();
  volatile SetupSums* v = b;
  if (v->frags) atomicAdd(&ws.ctr->frag_ref, (unsigned long long)v->frags);
  if (v->bins) atomicAdd(&ws.ctr->bins, (unsigned long long)v->bins);
  if (v->vis) atomicAdd(&ws.ctr->vis, (uint32_t)v->vis);
  if (v->samples) atomicAdd(&ws.ctr->samples, (unsigned long long)v->samples);
}

// Append this lane's candidate (act: it has one) as a record and count its
// bins (depth-only passes rasterise small ones directly).  A candidate without
// a pixel (kBoxEmpty) is counted as visible, but not stored.  Every lane of
// the warp must call it.
template <bool VIEW>
__device__ __forceinline__ void emit(const Cand& c, bool act, uint32_t surface, const Surface& S, const Workspace& ws,
                                     SetupCounts& cnt) {
  constexpr unsigned full = 0xFFFFFFFFu;
  const bool direct = !VIEW && act && c.area <= kDirectArea, rec = act && !direct;
  if (act) {  // ceil(area / chunk)
    const float chunk = (float)S.chunk;
    cnt.frags += c.area <= chunk ? 1u : (uint32_t)ceilf(fdiv(c.area, chunk));
  }
  if (direct && c.box != kBoxEmpty) cnt.samples += direct_raster(c, S.depth);
  if (!__any_sync(full, rec)) return;
  const bool store = rec && c.box != kBoxEmpty;
  Foot f{0, -1, 0, -1, false};
  if (rec) {
    int ref;
    f = footprint((uint32_t)c.mm[0] | ((uint32_t)c.mm[1] << 16), (uint32_t)c.mm[2] | ((uint32_t)c.mm[3] << 16),
                  c.box != kBoxAny ? kRecTight : 0u, ws, &ref);
    cnt.vis++;
    cnt.bins += (uint32_t)ref;
  }
  const unsigned who = __ballot_sync(full, store);
  const int lane = threadIdx.x & 31;
  uint32_t slot = 0;
  if (lane == 0 && who) slot = atomicAdd(&ws.ctr->nrec, (uint32_t)__popc(who));
  slot = __shfl_sync(full, slot, 0) + (uint32_t)__popc(who & ((1u << lane) - 1u));
  const bool stored = store && slot < ws.rec_cap;
  if (stored)
    write_rec(c, slot, surface, ws, VIEW);
  else if (store)
    atomicOr(&ws.ctr->overflow, 1u);
  // tile counts
  each_fine_tile(f, stored && !f.coarse ? foot_count(f) : 0, &S, slot,
                 [&](uint32_t tile, bool on) { agg_inc(ws.fine_count, tile, on); },
                 [&](uint32_t, uint32_t tile) { atomicAdd(&ws.fine_count[tile], 1u); });
  const bool coarse = stored && f.coarse;
  each_coarse_tile(f, coarse, &S, slot, [&](uint32_t, uint32_t tile) { atomicAdd(&ws.coarse_count[tile], 1u); });
  // the list of coarse records, from the end of the bins down (k_fill)
  const unsigned listed = __ballot_sync(full, coarse);
  if (listed) {
    uint32_t at = 0;
    if (lane == 0) at = atomicAdd(&ws.ctr->ncoarse, (uint32_t)__popc(listed));
    at = __shfl_sync(full, at, 0) + (uint32_t)__popc(listed & ((1u << lane) - 1u));
    if (coarse && at < ws.bin_cap) ws.bins[ws.bin_cap - 1 - at] = slot;
  }
}

__device__ __forceinline__ void load_tri_pos(const gbr_triangle* T, f3 v[3], uint32_t* o_id) {
  const float* base = reinterpret_cast<const float*>(T);
  float4 a = __ldg(reinterpret_cast<const float4*>(base));       // v0.pos
  float4 b = __ldg(reinterpret_cast<const float4*>(base + 8));   // v0.vt, object_id, col
  float4 c = __ldg(reinterpret_cast<const float4*>(base + 12));  // v1.pos
  float4 d = __ldg(reinterpret_cast<const float4*>(base + 24));  // v2.pos
  v[0] = mk3(a.x, a.y, a.z);
  v[1] = mk3(c.x, c.y, c.z);
  v[2] = mk3(d.x, d.y, d.z);
  *o_id = __float_as_uint(b.z);
}


// World-space vertices of every triangle: rot_quat(v * scale, q) + world_pos,
// the object half of full_rotate_quat (cl2.cl:700-710).  It does not depend on
// the camera, so one pass serves the view and all cube faces until the
// triangles or descriptors change.
// Also the radius of each object's world-space vertices around its
// world_pos (objr, float bits, zeroed before): the bounding sphere of the
// object cull.
__global__ void __launch_bounds__(256) k_world(SceneDev sc, float4* __restrict__ world, uint32_t* __restrict__ objr) {
  const uint32_t tri = blockIdx.x * blockDim.x + threadIdx.x;
  const bool valid = tri < sc.ntris;
  uint32_t o_id = 0;
  float rmax = 0.0f;
  if (valid) {
    f3 v[3];
    load_tri_pos(sc.tris + tri, v, &o_id);
    const gbr_obj_g_descriptor* G = sc.descs + o_id;
    const f4 qn = fast_normalize4(ld4(G->world_rot_quat));
    const f3 wp = ld3(G->world_pos);
    const float scale = __ldg(&G->scale);
    const int flags = __ldg(&G->feature_flag);
    float4* out = world + (size_t)tri * 3;
#pragma unroll
    for (int k = 0; k < 3; k++) {
      f3 r = add3(rot_quat_n(mul3s(v[k], scale), qn), wp);
      out[k] = make_float4(r.x, r.y, r.z, k == 0 ? __uint_as_float(o_id) : k == 1 ? __int_as_float(flags) : 0.0f);
      const float d = fast_length3(sub3(r, wp));
      rmax = d == d ? fmax_(rmax, d) : __int_as_float(0x7F800000);  // a NaN vertex disables the cull
    }
  }
  // the largest radius per object, aggregated over the warp's lanes of that object
  const unsigned act = __ballot_sync(0xFFFFFFFFu, valid);
  if (valid) {
    const unsigned grp = __match_any_sync(act, o_id);
    const uint32_t m = __reduce_max_sync(grp, __float_as_uint(rmax));  // non-negative floats order as integers
    if ((threadIdx.x & 31) == (uint32_t)(__ffs(grp) - 1)) atomicMax(objr + o_id, m);
  }
}

// Object cull of a view pass: bit o of row v is 0 when every triangle of
// object o is culled by prearrange's own tests in view v, so its setup
// threads stop after reading the object id.  Object o lies within radius
// objr[o] of its world_pos.  It is culled when it is farther than depth_far
// (the reference's object test, exactly), or when its bounding sphere lies
// entirely behind the near clip (z <= 20) or beyond the far clip (z >
// 350000) -- every vertex is then clipped away -- or, lying entirely nearer
// than the far clip, beyond one side plane of the view.  In that last case a
// clipped vertex lies on an edge between a vertex behind the near clip and
// one in front of it, inside the same half-space, so every projected vertex
// is off-screen on that side and the off-screen cull removes the triangle
// (cl2.cl:4352-4377).  (A vertex beyond the far clip is also clipped against
// z = 20, by extrapolation along its edge, which can leave the half-space:
// hence the far-clip condition.)  The margins (a relative 1e-3 of the radius
// and of the distance, plus one unit) are orders of magnitude above the
// float rounding of the per-triangle transform.
//
// The first kernel of a view pass: cull_blocks blocks do that (0: no object
// cull), the others clear the pass's counters (ncounts words) and, for a pass
// of one view given with the launch (one), write its parameters where the
// other kernels read them.  One launch instead of three clears, two copies and
// the cull.
__global__ void __launch_bounds__(256) k_begin_views(SceneDev sc, const __grid_constant__ ViewParams one_view,
                                                     const __grid_constant__ Surface one_surf, bool one,
                                                     ViewParams* __restrict__ views, Surface* __restrict__ surfs,
                                                     uint32_t nviews, const uint32_t* __restrict__ objr,
                                                     uint32_t words, uint32_t* __restrict__ vis,
                                                     uint32_t cull_blocks, uint32_t* __restrict__ counts,
                                                     uint32_t ncounts) {
  if (blockIdx.x >= cull_blocks) {
    const uint32_t b = blockIdx.x - cull_blocks;
    for (uint32_t i = b * blockDim.x + threadIdx.x; i < ncounts; i += (gridDim.x - cull_blocks) * blockDim.x)
      counts[i] = 0;
    if (one && b == 0) {
      static_assert(sizeof(ViewParams) % 4 == 0 && sizeof(ViewParams) / 4 <= 256 && sizeof(Surface) / 4 <= 256, "");
      if (threadIdx.x < sizeof(ViewParams) / 4)
        reinterpret_cast<uint32_t*>(views)[threadIdx.x] = reinterpret_cast<const uint32_t*>(&one_view)[threadIdx.x];
      if (threadIdx.x < sizeof(Surface) / 4)
        reinterpret_cast<uint32_t*>(surfs)[threadIdx.x] = reinterpret_cast<const uint32_t*>(&one_surf)[threadIdx.x];
    }
    return;
  }
  const uint32_t per_view = cull_blocks / nviews, v = blockIdx.x / per_view;
  const uint32_t o = (blockIdx.x % per_view) * blockDim.x + threadIdx.x;
  bool keep = false;
  if (o < sc.ndescs) {
    const ViewParams& V = one ? one_view : views[v];
    const Surface& S = one ? one_surf : surfs[V.surface];
    const f3 cpos = mk3(V.cpos[0], V.cpos[1], V.cpos[2]);
    const float4 q2 = __ldg(sc.objq + (size_t)o * kObjQuads + 2);
    const f3 wp = mk3(q2.x, q2.y, q2.z);
    const float dist = fast_length3(sub3(wp, cpos));
    if (!(dist > kDepthFar)) {
      const float r = __uint_as_float(__ldg(objr + o));
      const float m = r * 1.001f + dist * 1e-3f + 1.0f;
      const f3 q = rot_cs(wp, cpos, mk3(V.ccos[0], V.ccos[1], V.ccos[2]), mk3(V.csin[0], V.csin[1], V.csin[2]));
      // side planes through the camera: x * fov = -+ z * W/2, y * fov = -+ z * H/2
      const float hw = (float)S.width * 0.5f, hh = (float)S.height * 0.5f;
      const float nx = rsqrtf(V.fov * V.fov + hw * hw), ny = rsqrtf(V.fov * V.fov + hh * hh);
      const bool side = (q.x * V.fov + q.z * hw) * nx < -m || (q.x * V.fov - q.z * hw) * nx > m ||
                        (q.y * V.fov + q.z * hh) * ny < -m || (q.y * V.fov - q.z * hh) * ny > m;
      const bool out = q.z + m < kDepthCutoff || q.z - m > kDepthFar || (q.z + m < kDepthFar && side);
      keep = !out || !(m < 1e30f);  // an infinite or NaN radius culls nothing
    }
  }
  const unsigned bits = __ballot_sync(0xFFFFFFFFu, keep);
  if ((threadIdx.x & 31) == 0 && (o >> 5) < words) vis[(size_t)v * words + (o >> 5)] = bits;
}

// Per object: the normalised rotation quaternion rot_quat applies, and the
// normalised inverse back_rot_quat applies (conjugate / |q|^2, normalised by
// rot_quat) -- the same arithmetic every pixel of kernel3 would repeat.
__device__ __forceinline__ f4 quat_inverse_n(f4 q) {
  f4 conj; conj.x = -q.x; conj.y = -q.y; conj.z = -q.z; conj.w = q.w;
  float len_sq = dot4(conj, conj);
  f4 n; n.x = fdiv(conj.x, len_sq); n.y = fdiv(conj.y, len_sq);
  n.z = fdiv(conj.z, len_sq); n.w = fdiv(conj.w, len_sq);
  return fast_normalize4(n);
}

// and the material terms kernel3 reads (kObjQuads float4 per object).
__global__ void __launch_bounds__(256) k_objects(SceneDev sc, float4* __restrict__ objq) {
  const uint32_t o = blockIdx.x * blockDim.x + threadIdx.x;
  if (o >= sc.ndescs) return;
  const gbr_obj_g_descriptor* G = sc.descs + o;
  const f4 q = ld4(G->world_rot_quat);
  const f4 qn = fast_normalize4(q), qi = quat_inverse_n(q);
  float4* d = objq + (size_t)kObjQuads * o;
  d[0] = make_float4(qn.x, qn.y, qn.z, qn.w);
  d[1] = make_float4(qi.x, qi.y, qi.z, qi.w);
  d[2] = make_float4(__ldg(&G->world_pos[0]), __ldg(&G->world_pos[1]), __ldg(&G->world_pos[2]), __ldg(&G->diffuse));
  d[3] = make_float4(__ldg(&G->spec_mult), clampf_(1.0f - __ldg(&G->specular), 0.001f, 10.0f),
                     __int_as_float(__ldg(&G->feature_flag)), __uint_as_float(__ldg(&G->tid)));
}

// The atlas slot of level L of texture t (slot descriptor nums[...] = page <<
// 16 | slot; pages are powers of two, 16..2048, so the slot's row and column
// within its page are exact in integers): the texture level table entry.
__global__ void __launch_bounds__(256) k_texture_levels(const uint32_t* __restrict__ nums,
                                                        const uint32_t* __restrict__ sizes, uint32_t mipmap_start,
                                                        float4* __restrict__ texlv) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= mipmap_start * kTexLevels) return;
  const uint32_t t = i / kTexLevels, L = i % kTexLevels;
  const uint32_t nv = nums[L == 0 ? t : mipmap_start + t * kMipLevels + (L - 1)];
  const uint32_t page = nv >> 16, which = nv & 0xFFFFu;
  const uint32_t w = sizes[page];
  const uint32_t hnum = (uint32_t)kTexPage / w;
  const uint32_t row = which / hnum, col = which - row * hnum;
  texlv[i] = make_float4(__uint_as_float(col * w), __uint_as_float(row * w), (float)w, __uint_as_float(page));
}

// World-space vertices of a triangle, its object and the object's feature
// flags: from the scene's cache when there is one, else computed here with the
// same arithmetic as k_world.
__device__ __forceinline__ void load_world(const SceneDev& sc, uint32_t tri, f3 w[3], uint32_t* o_id, int* flags) {
  if (!sc.world) {
    f3 v[3];
    load_tri_pos(sc.tris + tri, v, o_id);
    const gbr_obj_g_descriptor* G = sc.descs + *o_id;
    const f4 qn = fast_normalize4(ld4(G->world_rot_quat));
    const f3 wp = ld3(G->world_pos);
    const float scale = __ldg(&G->scale);
    *flags = __ldg(&G->feature_flag);
#pragma unroll
    for (int k = 0; k < 3; k++) w[k] = add3(rot_quat_n(mul3s(v[k], scale), qn), wp);
    return;
  }
  const float4* p = sc.world + (size_t)tri * 3;
  float4 a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2);
  w[0] = mk3(a.x, a.y, a.z);
  w[1] = mk3(b.x, b.y, b.z);
  w[2] = mk3(c.x, c.y, c.z);
  *o_id = __float_as_uint(a.w);
  *flags = __float_as_int(b.w);
}

// The camera half of full_rotate_quat (cl2.cl:700-729): world -> camera
// space, near/far clip, projection of clip output k (0 or 1).  Returns the
// number of clip outputs; o is only written for k below it.
__device__ __forceinline__ int transform_clip(const f3 w[3], f3 cpos, f3 c, f3 s, float fov, float width,
                                              float height, int k, f3 o[3]) {
  f3 t0[3], t1[3];
  const int n = clip_tri_reg(rot_cs(w[0], cpos, c, s), rot_cs(w[1], cpos, c, s), rot_cs(w[2], cpos, c, s), t0, t1);
  if (k < n) {
#pragma unroll
    for (int j = 0; j < 3; j++) o[j] = depth_project1(k ? t1[j] : t0[j], width, height, fov);
  }
  return n;
}

// prearrange's handling of clip output k of one (triangle, surface): *num is
// the number of clip outputs; returns whether output k survives the culls.
__device__ __forceinline__ bool make_cand(const f3 w[3], f3 cpos, f3 c, f3 s, float fov, float width, float height,
                                          bool two, uint32_t tri, int k, Cand& out, int* num) {
  *num = transform_clip(w, cpos, c, s, fov, width, height, k, out.p);
  out.key = tri * 2u + (uint32_t)k;
  return k < *num && cull_candidate(out, two, width, height);
}

// The second clip outputs of a warp's triangles (has: the lane has one), from
// their vertices again: a near-clip split is rare, and the common path keeps
// no registers for it.  Every lane of the warp must call it.
template <bool VIEW>
__device__ __noinline__ void emit_second(const SceneDev& sc, const Workspace& ws, uint32_t tri, bool has, f3 pos, f3 c,
                                         f3 s, float fov, uint32_t surface, const Surface* surfs, SetupSums* sums) {
  const Surface& S = surfs[surface];
  Cand cand;
  bool act = false;
  if (has) {
    f3 wv[3];
    uint32_t o_id;
    int num, flags;
    load_world(sc, tri, wv, &o_id, &flags);
    act = make_cand(wv, pos, c, s, fov, (float)S.width, (float)S.height, (flags & kFlagTwoSided) > 0, tri, 1, cand,
                    &num);
  }
  SetupCounts cnt;
  emit<VIEW>(cand, act, surface, S, ws, cnt);
  setup_add(sums, cnt);
}

// prearrange (cl2.cl:4271-4409), one thread per (triangle, view).  Bound by
// latency and issue together (51 % active, 45 % of the warps; more CTAs per SM
// spill): 1M-triangle terrain 36 us, 64 views of 500k triangles 280 us.
__global__ void __launch_bounds__(256, 5) k_setup_views(const __grid_constant__ SceneDev sc,
                                                     const ViewParams* __restrict__ views,
                                                     const Surface* __restrict__ surfs,
                                                     const __grid_constant__ Workspace ws) {
  __shared__ SetupSums sums;
  if (threadIdx.x == 0) sums.clear();
  __syncthreads();
  uint32_t tri = blockIdx.x * blockDim.x + threadIdx.x;
  const ViewParams& V = views[blockIdx.y];
  const Surface& S = surfs[V.surface];
  SetupCounts cnt;
  // the object cull (k_begin_views), when the pass has one, includes the
  // reference's own object test.  A pass of one view reads the whole triangle
  // at once (two rounds of loads); a pass of many views, which skips most
  // objects in each, reads the object id alone first.
  bool live = tri < sc.ntris;
  f3 wv[3];
  uint32_t o_id = 0;
  int flags = 0;
  const f3 cpos = mk3(V.cpos[0], V.cpos[1], V.cpos[2]);
  const bool whole = gridDim.y == 1;
  if (live && (whole || !ws.vis)) load_world(sc, tri, wv, &o_id, &flags);
  if (live && ws.vis) {
    if (!whole) o_id = __float_as_uint(__ldg(&sc.world[(size_t)tri * 3].w));
    live = (__ldg(ws.vis + (size_t)blockIdx.y * ws.vis_words + (o_id >> 5)) >> (o_id & 31)) & 1u;
  } else if (live) {
    live = !(fast_length3(sub3(ld3(sc.descs[o_id].world_pos), cpos)) > kDepthFar);
  }
  // a warp with nothing to set up (objects are mostly contiguous runs of
  // triangles) leaves before emit's warp-wide work
  if (!__any_sync(0xFFFFFFFFu, live)) {
    setup_done(&sums, ws);
    return;
  }
  Cand cand;
  int num = 0;
  bool act = false;
  const f3 c = mk3(V.ccos[0], V.ccos[1], V.ccos[2]), s = mk3(V.csin[0], V.csin[1], V.csin[2]);
  if (live) {
    if (!whole && ws.vis) load_world(sc, tri, wv, &o_id, &flags);
    act = make_cand(wv, cpos, c, s, V.fov, (float)S.width, (float)S.height, (flags & kFlagTwoSided) > 0, tri, 0, cand,
                    &num);
  }
  emit<true>(cand, act, V.surface, S, ws, cnt);
  if (__any_sync(0xFFFFFFFFu, num > 1))
    emit_second<true>(sc, ws, tri, num > 1, cpos, c, s, V.fov, V.surface, surfs, &sums);
  setup_add(&sums, cnt);
  setup_done(&sums, ws);
}

// prearrange_realtime_shadowing (cl2.cl:4419-4636), one thread per (triangle, light job).
// Bound by the direct rasters: lanes' boxes differ (20 of 32 active) and their
// atomics wait; 52 % issue active.  1M-triangle terrain 136 -> 76 us;
// 128 x 7 measured best of blocks of 32 to 256 threads.
__global__ void __launch_bounds__(128, 7) k_setup_shadow(const __grid_constant__ SceneDev sc,
                                                      const ShadowJob* __restrict__ jobs,
                                                      const Surface* __restrict__ surfs,
                                                      const __grid_constant__ Workspace ws) {
  __shared__ SetupSums sums;
  if (threadIdx.x == 0) sums.clear();
  __syncthreads();
  uint32_t tri = blockIdx.x * blockDim.x + threadIdx.x;
  const ShadowJob& J = jobs[blockIdx.y];
  SetupCounts cnt;
  const float L = (float)kLightBufferDim;
  int mask = 0;
  f3 wv[3];
  f3 lpos = mk3(J.lpos[0], J.lpos[1], J.lpos[2]);
  bool two = false;
  if (tri < sc.ntris) {
    uint32_t o_id;
    int ff;
    load_world(sc, tri, wv, &o_id, &ff);
    bool is_static = (ff & kFlagIsStatic) > 0;
    two = (ff & kFlagTwoSided) > 0;
    f3 wp = ld3(sc.descs[o_id].world_pos);
    if (is_static == (J.only_static != 0) && !(fast_length3(sub3(wp, lpos)) > kDepthFar)) {
      for (int k = 0; k < 3; k++) mask |= 1 << ret_cubeface(wv[k], lpos);
    }
  }
  for (int face = 0; face < 6; face++) {
    if (!__any_sync(0xFFFFFFFFu, mask & (1 << face))) continue;  // warp-uniform
    const f3 c = mk3(sc.face_cos[face][0], sc.face_cos[face][1], sc.face_cos[face][2]);
    const f3 s = mk3(sc.face_sin[face][0], sc.face_sin[face][1], sc.face_sin[face][2]);
    const uint32_t surface = J.surface_base + face;
    Cand cand;
    int num = 0;
    bool act = false;
    if (mask & (1 << face)) act = make_cand(wv, lpos, c, s, kLFov, L, L, two, tri, 0, cand, &num);
    emit<false>(cand, act, surface, surfs[surface], ws, cnt);
    if (__any_sync(0xFFFFFFFFu, num > 1))
      emit_second<false>(sc, ws, tri, num > 1, lpos, c, s, kLFov, surface, surfs, &sums);
  }
  setup_add(&sums, cnt);
  setup_done(&sums, ws);
}

// Warp-aggregated allocation of n slots from *counter; every lane of the
// warp must call it (n may be 0).  Returns this lane's first slot.
__device__ __forceinline__ uint32_t warp_alloc(uint32_t* counter, uint32_t n) {
  const unsigned full = 0xFFFFFFFFu;
  const int lane = threadIdx.x & 31;
  uint32_t incl = n;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(full, incl, o);
    if (lane >= o) incl += v;
  }
  const uint32_t total = __shfl_sync(full, incl, 31);
  uint32_t base = 0;
  if (lane == 31 && total) base = atomicAdd(counter, total);
  return __shfl_sync(full, base, 31) + incl - n;
}

// Bin offsets: every fine tile's bin, and every coarse tile's, gets its place
// from a counter, a warp's tiles at a time (the order of the bins is free:
// what a tile resolves does not depend on it, so no scan is needed).  fine_off
// and coarse_off then serve as the fill's cursors: after it they are the
// bins' ends.  Also, where asked for,
//   ws.tiles  each fine tile's surface (binary search over tile_base) and
//             global coarse tile: the first loads of the raster and kernel3;
//   ws.list   depth-only passes with per_surface tiles on every surface: the
//             tiles that have records (a cube face's are mostly empty).
// One launch for the scan's one or two and the tile table's: 3 us where the
// one-block scan of a 1080p view took 8 and the chunked one 15.
__global__ void __launch_bounds__(256) k_offsets(Workspace ws, const Surface* __restrict__ surfs, uint32_t nsurf,
                                                 uint32_t per_surface) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t c = t < ws.nfine ? ws.fine_count[t] : 0u;
  const uint32_t off = warp_alloc(&ws.ctr->fine_total, c);
  if (t < ws.nfine) ws.fine_off[t] = off;
  const uint32_t cc = t < ws.ncoarse ? ws.coarse_count[t] : 0u;
  if ((t & ~31u) < ws.ncoarse) {  // warp-uniform
    const uint32_t coff = warp_alloc(&ws.ctr->coarse_total, cc);
    if (t < ws.ncoarse) ws.coarse_off[t] = coff;
  }
  if (t == 0) {
    // the scratch must hold every visible triangle and every tile of its
    // bbox4 (the limits callers know), although fewer are stored
    if (ws.ctr->vis > ws.rec_cap) ws.ctr->overflow |= 1u;
    if (ws.ctr->bins > ws.bin_cap) ws.ctr->overflow |= 2u;
  }
  if (!ws.tiles && !ws.list) return;
  bool busy = false;
  if (t < ws.nfine) {
    uint32_t s = 0;
    if (per_surface) {
      s = t / per_surface;
    } else {
      uint32_t hi = nsurf - 1;
      while (s < hi) {
        const uint32_t mid = (s + hi + 1) >> 1;
        if (surfs[mid].tile_base <= t) s = mid; else hi = mid - 1;
      }
    }
    const Surface& S = surfs[s];
    const uint32_t lt = t - S.tile_base;
    const int tx = lt % S.tiles_x, ty = lt / S.tiles_x;
    const uint32_t ct = S.ctile_base + (ty >> ws.coarse_shift) * S.ctiles_x + (tx >> ws.coarse_shift);
    if (ws.tiles) ws.tiles[t] = make_uint2(s, ct);
    busy = c > 0 || ws.coarse_count[ct] > 0;
  }
  if (!ws.list) return;
  const unsigned who = __ballot_sync(0xFFFFFFFFu, busy);
  const uint32_t at = warp_alloc(&ws.ctr->nlist, (threadIdx.x & 31) == 0 ? (uint32_t)__popc(who) : 0u);
  const uint32_t first = __shfl_sync(0xFFFFFFFFu, at, 0);
  if (busy) ws.list[first + (uint32_t)__popc(who & ((1u << (threadIdx.x & 31)) - 1u))] = t;
}

// Barycentrics (cl2.cl:5372-5384) split into the per-triangle part and the
// per-point part; bary_exact is barycentric() bit for bit.
struct BaryFrame {
  f3 a, v0, v1;
  float d00, d01, d11, denom;
};
__device__ __forceinline__ BaryFrame bary_frame(f3 a, f3 b, f3 c) {
  BaryFrame f;
  f.a = a;
  f.v0 = sub3(b, a);
  f.v1 = sub3(c, a);
  f.d00 = dot3(f.v0, f.v0);
  f.d01 = dot3(f.v0, f.v1);
  f.d11 = dot3(f.v1, f.v1);
  f.denom = f.d00 * f.d11 - f.d01 * f.d01;
  return f;
}
__device__ __forceinline__ void bary_exact(const BaryFrame& f, f3 p, float* u, float* v, float* w) {
  f3 v2 = sub3(p, f.a);
  float d20 = dot3(v2, f.v0), d21 = dot3(v2, f.v1);
  *v = fdiv(f.d11 * d20 - f.d01 * d21, f.denom);
  *w = fdiv(f.d00 * d21 - f.d01 * d20, f.denom);
  *u = (1.0f - *v) - *w;
}
// kernel3's per-triangle arithmetic for one view record, in place: the
// setup's projected vertices, rconst and triangle index become the
// barycentric frame (cl2.cl:5372-5384) of the scaled object-space vertices,
// get_vtdiff's 1/z plane through the rounded vertices (cl2.cl:5691-5760), the
// vertex normals, UVs and colours, and the facing (cl2.cl:491-494).  Every
// value is computed with the arithmetic kernel3 applies per pixel in the
// reference, so the pixels read exactly what they would compute.
// q0, q1, q2: the setup's output; R: the triangle (per vertex pos, normal,
// (vt, object_id, vertex_col)), made the record in place: the normals stay
// where they are.
__device__ __forceinline__ void prep_shade(const SceneDev& sc, float4 q0, float4 q1, float4 q2, ShadeRec* R) {
  const f3 tp0 = mk3(q0.x, q0.y, q0.z), tp1 = mk3(q1.x, q1.y, q1.z), tp2 = mk3(q2.x, q2.y, q2.z);
  const uint32_t tri = __float_as_uint(q1.w);
  const float4 vc0 = R->plane, vc1 = R->t, vc2 = R->col;
  const uint32_t o_id = __float_as_uint(vc0.z);
  const float scale = __ldg(&sc.descs[o_id].scale);
  const uint32_t back = backface_front(tp0, tp1, tp2) ? 0u : 0x80000000u;
  R->n1.w = vc0.x;
  R->n2.w = vc0.y;
  R->n3.w = vc1.x;
  R->t = make_float4(vc1.y, vc2.x, vc2.y, __uint_as_float(o_id | back));
  R->col = make_float4(vc0.w, vc1.w, vc2.w, __uint_as_float(tri));
  const f3 xpv = mk3(roundf(tp0.x), roundf(tp1.x), roundf(tp2.x));
  const f3 ypv = mk3(roundf(tp0.y), roundf(tp1.y), roundf(tp2.y));
  const f3 depths = mk3(rcp(tp0.z), rcp(tp1.z), rcp(tp2.z));
  float DA, DB, DC;
  plane_const(depths, xpv, ypv, q0.w, &DA, &DB, &DC);
  const float4 va0 = R->a, va1 = R->e0, va2 = R->e1;
  const BaryFrame bf = bary_frame(mul3s(mk3(va0.x, va0.y, va0.z), scale), mul3s(mk3(va1.x, va1.y, va1.z), scale),
                                  mul3s(mk3(va2.x, va2.y, va2.z), scale));
  R->a = make_float4(bf.a.x, bf.a.y, bf.a.z, bf.d00);
  R->e0 = make_float4(bf.v0.x, bf.v0.y, bf.v0.z, bf.d01);
  R->e1 = make_float4(bf.v1.x, bf.v1.y, bf.v1.z, bf.d11);
  R->plane = make_float4(DA, DB, DC, bf.denom);
}

// The shade constants of 32 records, R[0 .. n), by a warp.  A record and a
// triangle are 144 bytes: a lane that loads and stores its own touches 32
// sectors an instruction, half of each unused, and the load and store units
// were the bound.  Here the warp moves the runs together, by way of shared
// memory (buf: kPrepQuads; a stride of 9 float4 has no bank conflicts).  A pass
// of 64 views: 117 -> 90 us (5.5 of the 6.8 TB/s a copy reaches); 9 views: 67
// -> 49 us; the raster with these blocks in front: 4K 241 -> 228 us.
constexpr int kShadeQuads = sizeof(ShadeRec) / 16, kPrepQuads = 32 * kShadeQuads;
static_assert(sizeof(gbr_triangle) == sizeof(ShadeRec) && kShadeQuads == 9, "one buffer for both");
__device__ __forceinline__ void copy16_async(float4* shared, const float4* global) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(shared)), "l"(global)
               : "memory");
}
// The warp's copies by copy16_async are done and visible to all of its lanes.
__device__ __forceinline__ void copies_done() {
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncwarp();
}
__device__ __forceinline__ void prep_records(const SceneDev& sc, ShadeRec* R, uint32_t n, float4* buf) {
  const uint32_t lane = threadIdx.x & 31;
  float4* rec = reinterpret_cast<float4*>(R);
  const float4* tris = reinterpret_cast<const float4*>(sc.tris);
#pragma unroll
  for (uint32_t i = lane; i < 96; i += 32)  // the setup's output: 3 float4 of each record
    if (i < 3 * n) copy16_async(buf + i, rec + i / 3 * kShadeQuads + i % 3);
  copies_done();
  const float4 q0 = buf[3 * lane], q1 = buf[3 * lane + 1], q2 = buf[3 * lane + 2];
  __syncwarp();
  const uint32_t tri = __float_as_uint(q1.w);
  // (quotient and remainder by steps: 9 of each, kept over the records, spill)
  uint32_t of = lane / kShadeQuads, at = lane % kShadeQuads;
#pragma unroll 3
  for (uint32_t i = lane; i < kPrepQuads; i += 32) {
    const uint32_t t = __shfl_sync(0xFFFFFFFFu, tri, of);
    if (of < n) copy16_async(buf + i, tris + (size_t)t * kShadeQuads + at);
    of += 32 / kShadeQuads, at += 32 % kShadeQuads;
    if (at >= kShadeQuads) at -= kShadeQuads, of++;
  }
  copies_done();
  if (lane < n) prep_shade(sc, q0, q1, q2, reinterpret_cast<ShadeRec*>(buf) + lane);
  __syncwarp();
#pragma unroll
  for (uint32_t i = lane; i < kPrepQuads; i += 32)
    if (i < kShadeQuads * n) rec[i] = buf[i];
  __syncwarp();
}

// The shade constants of every record of a pass of several views (after the
// setup; the raster does not read them).
__global__ void __launch_bounds__(256, 4) k_prep(SceneDev sc, Workspace ws) {
  __shared__ float4 buf[8][kPrepQuads];
  if (ws.ctr->overflow) return;
  const uint32_t nrec = min(ws.ctr->nrec, ws.rec_cap), warp = threadIdx.x / 32;
  for (uint32_t r = (blockIdx.x * 8 + warp) * 32; r < nrec; r += gridDim.x * 256)
    prep_records(sc, ws.srec + r, min(32u, nrec - r), buf[warp]);
}

// Scatter record indices into their tile bins (cursor atomics aggregated
// across the warp).  Records in coarse bins are taken one per warp from the
// setup's list at the end of the bins, as long as the list and the bins do not
// meet: large triangles often follow one another, and 32 of them in one warp
// are a chain of hundreds of atomics (1,000 screen-covering triangles at
// 2560x1440: fill 220 -> 15 us).
__global__ void __launch_bounds__(256) k_fill(Workspace ws, const Surface* __restrict__ surfs) {
  const uint32_t nrec = min(ws.ctr->nrec, ws.rec_cap);
  if (ws.ctr->overflow) return;
  const uint32_t coarse_base = ws.ctr->fine_total;
  const uint32_t stride = gridDim.x * blockDim.x, ncoarse = ws.ctr->ncoarse;
  const bool list = (uint64_t)coarse_base + ws.ctr->coarse_total + ncoarse <= ws.bin_cap;
  for (uint32_t r0 = blockIdx.x * blockDim.x; r0 < nrec; r0 += stride) {
    const uint32_t r = r0 + threadIdx.x;
    const bool valid = r < nrec;
    Foot f{0, -1, 0, -1, false};
    const Surface* S = surfs;
    if (valid) {
      const float4 q = __ldg(reinterpret_cast<const float4*>(ws.rec + r) + 3);
      S = surfs + __float_as_uint(q.z);
      int ref;
      f = footprint(__float_as_uint(q.x), __float_as_uint(q.y), __float_as_uint(q.w), ws, &ref);
    }
    each_fine_tile(
        f, valid && !f.coarse ? foot_count(f) : 0, S, r,
        [&](uint32_t tile, bool on) {
          const uint32_t pos = agg_inc(ws.fine_off, tile, on);
          if (on) ws.bins[pos] = r;
        },
        [&](uint32_t rr, uint32_t tile) { ws.bins[atomicAdd(&ws.fine_off[tile], 1u)] = rr; });
    each_coarse_tile(f, valid && f.coarse && !list, S, r, [&](uint32_t rr, uint32_t tile) {
      ws.bins[coarse_base + atomicAdd(&ws.coarse_off[tile], 1u)] = rr;
    });
  }
  if (!list) return;
  const uint32_t warps = stride / 32, lane = threadIdx.x & 31;
  for (uint32_t i = blockIdx.x + gridDim.x * (threadIdx.x / 32); i < ncoarse; i += warps) {
    const uint32_t r = ws.bins[ws.bin_cap - 1 - i];
    const float4 q = __ldg(reinterpret_cast<const float4*>(ws.rec + r) + 3);
    const Surface& S = surfs[__float_as_uint(q.z)];
    int ref;
    const Foot f = footprint(__float_as_uint(q.x), __float_as_uint(q.y), __float_as_uint(q.w), ws, &ref);
    const uint32_t w = (uint32_t)(f.tx1 - f.tx0 + 1), n = (uint32_t)foot_count(f);
    for (uint32_t k = lane; k < n; k += 32) {
      const uint32_t tile = S.ctile_base + (f.ty0 + k / w) * S.ctiles_x + f.tx0 + k % w;
      ws.bins[coarse_base + atomicAdd(&ws.coarse_off[tile], 1u)] = r;
    }
  }
}

// kernel1 + kernel2 for one 16x16 tile: depth min, then the canonical id.
//
// The tile's records (its fine bin, then its coarse tile's bin) are staged NT
// at a time in shared memory, keeping those whose bbox meets the tile.  Each
// contributes the rows of its bbox in the tile; one block scan (packing the
// record count and the row count) compacts the records and lays all rows of
// the chunk end to end.  Each warp takes one contiguous share of that list, 32
// rows at a time: it maps rows to records with one ballot of the record starts
// inside the window (every staged record has a row, so at most 32 start
// there), narrows each lane's row to the span that the three edges leave
// (row_span, with more slack for records with vertices off the surface),
// and lays the spans' horizontal pixel pairs end to end in turn.  Those are
// tested 32 at a time, mapped to spans as rows are to records: a pair costs
// one decode and record load for two exact tests, and small, large and thin
// triangles are load-balanced alike.  Pass 0 resolves the minimum depth with
// shared-memory atomicMin; pass 1 the minimum packed (key << 32 | record)
// among tests within +-20 of the final depth.  Both are minima, so neither bin
// order nor thread order changes the result.  Pass 0 keeps its covered pixels
// in a list per warp (hit_cap, compacted in place when it fills: an entry 20
// or more behind the pixel's depth so far never passes), and pass 1 runs over
// those lists; only a tile whose lists overflow all the same tests its records
// again.
//
// Measured (launch alone, before -> now; bound by instruction issue, 72 %
// active, and by the barriers between chunks): 1080p terrain 114 -> 81 us, 9
// ragged views of a 500k-triangle scene 689 -> 431 us (tiles of several chunks
// no longer stage and test everything twice; the walk rule costs a comparison
// per record), 2560x1440 under 1,000 screen-covering triangles 22.4 -> 0.43 ms
// (the depth cull at staging).  Then tight boxes and fewer records: 69 us
// (terrain).  Rows narrowed to spans instead of all pairs of the bbox: 64
// sphere views 1.01 -> 0.97 ms, 4K 210 -> 191 us, cube faces with large walls
// 141 -> 121 us, 1080p terrain 68 -> 67 us.  Records with vertices off the surface
// as well (whole rows, on top of the pairs, were slower than the pairs alone):
// cube faces of 3,762, 2,750 and 2,471 large triangles at one depth 1,468 ->
// 450, 1,349 -> 734 and 1,037 -> 434 us (1,031, 1,123 and 892 by pairs).
//
// A view pass of many tiles (kManyWaves of them) takes CTAs of 64 threads for
// the default 128: a warp's fixed work per tile is paid half as often, two
// warps wait less for one another than four, and more tiles are in flight
// behind the first loads of each.  At 128 and at 64 threads: 64 sphere views
// (253k tiles) 981 and 763 us (instructions 784M and 591M), 4K (32k) 228 and
// 185, nine ragged views (25k) 200 and 195, 1,000 screen-covering triangles at
// 1440p (14k) 360 to 460 and 305, 1080p (8k) 80 and 84, 1279x721 (3.7k) 30.5
// and 33.4: the last wave counts there.
constexpr uint32_t kManyWaves = 4;
// Entries of a warp's list: about 100 are used in a tile of 1.2 layers by each
// of four warps, and twice that by each of two.  At least what compaction can
// leave and one window of tests can add: one entry for each of the tile's
// pixels (more only where layers lie within kernel2's window of one another)
// and 64.  With room for 256 alone, tiles of dozens of layers over all their
// pixels gave their lists up and tested everything again: 4,000 overlapping
// triangles of 30 pixels along a row of tiles at 720p, raster 196 us, 128 with
// 320 entries, 161 without lists; 1,000 of them 59, 42 and 54.  512-thread CTAs
// keep no lists (their static shared memory stays under 48 KB) and re-test in
// the id pass.
template <int NT>
__host__ __device__ constexpr int hit_cap() { return NT == 64 ? 352 : 320; }
static_assert(hit_cap<64>() >= kTilePixels + 64 && hit_cap<128>() >= kTilePixels + 64, "");
// The fused pass keeps 256: with 320 its blocks leave kernel3 less of the L1 (16
// sphere views 948 -> 1,000 us).
constexpr int kFusedHits = 256;
// View CTAs per SM, by registers and (64 threads) shared memory.
template <int NT>
__host__ __device__ constexpr int raster_ctas() { return NT == 64 ? 15 : 1024 / NT; }
// A list entry's second word: pixel | record << 8, so records below 2^24
// (passes with room for more re-test tiles of several chunks).
constexpr uint32_t kHitRecords = 1u << 24;
constexpr uint32_t kSlotBits = 9;  // staged slots of a one-chunk tile: below 512

// Barrier of a tile's NT threads: the block, or (PART) one of its groups.
template <int NT, bool PART>
__device__ __forceinline__ void tile_barrier() {
  if (!PART)
    __syncthreads();
  else if (threadIdx.x < NT)  // (constant numbers: with one in a register a block holds all 16 barriers)
    asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory");
  else
    asm volatile("bar.sync 2, %0;" ::"n"(NT) : "memory");
}

// Exclusive block scan with a single barrier: each warp scans its lanes,
// publishes its total, and after the barrier every thread adds up the totals
// of the warps before its own (and of all warps, the block total).
// The NT threads are a block, or (PART) one of the block's groups of NT.
template <int NT, bool PART>
__device__ __forceinline__ uint32_t block_excl_scan1(uint32_t v, uint32_t* swarp, uint32_t* total) {
  const int lane = threadIdx.x & 31, warp = (threadIdx.x & (NT - 1)) >> 5;
  uint32_t incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) swarp[warp] = incl;
  tile_barrier<NT, PART>();
  uint32_t before = 0, all = 0;
#pragma unroll
  for (int w = 0; w < NT / 32; w++) {
    const uint32_t t = swarp[w];
    all += t;
    if (w < warp) before += t;
  }
  *total = all;
  return before + incl - v;
}


// Shared-memory slot of tile pixel p = ly * 16 + lx in the per-pixel depth
// (32-bit words) and id (64-bit words) arrays: a row of 16 pixels fills 16
// of the 32 banks, so rows y and y + 2 (64-bit: y and y + 1) would share
// banks and a narrow triangle's tests collide.  32-bit: each 32-word line
// (a row pair) is rotated by 4 banks per line, so that a footprint up to 4
// pixels wide and 8 rows tall falls on distinct banks; 64-bit: the column is
// XOR-ed with the row.  Permutations within each line (row).
__device__ __forceinline__ int swz32(int p) {
  const int line = p >> 5;
  return (line << 5) | ((p + 4 * line) & 31);
}
__device__ __forceinline__ int swz64(int p) { return p ^ ((p >> 4) & 15); }

// kernel3's RGBA8 output word
// (quant8 of each channel: saturation is the clamp, NaN included, and the
// truncation to a byte is the low byte of an addition of 2^23 rounded toward zero)
__device__ __forceinline__ uint32_t pack_rgba(float r, float g, float b, float a) {
  auto q = [](float v) { return __float_as_uint(__fadd_rz(__saturatef(v) * 255.0f + 0.5f, 8388608.0f)); };
  return __byte_perm(__byte_perm(q(r), q(g), 0x0040), __byte_perm(q(b), q(a), 0x0040), 0x5410);
}

// Drops the entries of a warp's list that are 20 or more behind their pixel's
// depth so far (the final depth is at most that, and kernel2's window ends 20
// behind it).  Every lane of the warp calls it; returns the new length.
__device__ __noinline__ uint32_t compact_hits(uint2* hits, uint32_t n, const uint32_t* sdepth) {
  const int lane = threadIdx.x & 31;
  uint32_t kept = 0;
  __syncwarp();  // the entries are other lanes' stores, and a vote orders no memory
  for (uint32_t g0 = 0; g0 < n; g0 += 32) {
    const uint32_t g = g0 + lane;
    uint2 e = make_uint2(0, 0);
    bool keep = false;
    if (g < n) {
      e = hits[g];
      const uint32_t fd = sdepth[swz32((int)(e.y & 0xFF))];
      keep = fd > kDepthClear - kBufError || e.x < fd + kBufError;
    }
    const unsigned b = __ballot_sync(0xFFFFFFFFu, keep);  // (every lane has read its entry)
    if (keep) hits[kept + (uint32_t)__popc(b & ((1u << lane) - 1u))] = e;
    kept += (uint32_t)__popc(b);
    __syncwarp();
  }
  return kept;
}

// Spans a warp holds at once: fewer than 32 that wait, and those of 32 rows.
constexpr uint32_t kSpanRing = 64;

// Shared memory of one tile's raster (NT threads; ID: views; lists of CAP).
template <int NT, bool ID, int CAP = hit_cap<NT>()>
struct RasterSmem {
  static constexpr int kHits = ID && NT <= 256 ? CAP : 0;  // entries of a warp's list, 0: none
  float4 srec[3][NT];  // the staged records' first three float4, one array each (conflict-free stores)
  uint32_t sidx[NT];
  uint32_t soff[NT + 1];
  uint32_t sgeo[NT];   // lx0 | ly0 << 4 | bw << 8 | kind << 13
  float2 sinv[NT];     // reciprocal x slopes of t and of bound - s - t (that of s: srec[1].w)
  uint2 spans[NT / 32][kSpanRing];  // per warp: spans of rows that can be covered
  // bit ly: the walk skips the record's left-column pixel in tile row ly (0
  // when that column lies left of the tile)
  uint16_t sskip[NT];
  // the covered pixels of pass 0 kept for the id pass: depth, and pixel |
  // record << 8 (the staged slot in one-chunk tiles, else the pass's record);
  // warp w's list at w * kHits
  uint2 hits[kHits ? kHits * (NT / 32) : 1];
  uint32_t sdepth[kTilePixels];
  unsigned long long sid[kTilePixels];
  uint32_t swarp[NT / 32];
  uint32_t sscan;
  uint32_t ssamples;
  uint32_t szcap;  // every coverable pixel of the tile ends at this depth or nearer
  Surface S;
  uint32_t s;  // the tile's surface
  uint32_t lists[4];
};

// NT threads per tile: a CTA of 64, 128, 256 or 512, or (PART) one of a CTA's
// two halves of 64; ID: resolve the canonical id too (views) or only the depth
// (cube faces, tiles with records); CC: see chunk below.  surface: the tile's
// surface when the caller knows it, else -1 (ws.tiles, or the pass's only
// surface).  Every thread of the block calls it; the caller synchronises before
// reusing the shared memory.
template <int NT, bool ID, bool CC = false, bool PART = false, int CAP = hit_cap<NT>()>
__device__ __forceinline__ void raster_tile(const Workspace& ws, const Surface* __restrict__ surfs, uint32_t tile,
                                            int surface, RasterSmem<NT, ID, CAP>& sm) {
  constexpr uint32_t kHits = RasterSmem<NT, ID, CAP>::kHits;
  static_assert(!(ID && PART), "the id pass votes across the block");
  constexpr bool with_id = ID;
  constexpr int NW = NT / 32;
  constexpr uint32_t kCountShift = 18;  // scan word: pixels (< 2^18) | records << 18
  float4 (&srec)[3][NT] = sm.srec;
  uint32_t* sidx = sm.sidx;
  uint32_t* soff = sm.soff;
  uint32_t* sgeo = sm.sgeo;
  uint16_t* sskip = sm.sskip;
  uint32_t* sdepth = sm.sdepth;
  unsigned long long* sid = sm.sid;
  uint32_t* swarp = sm.swarp;
  uint32_t& sscan = sm.sscan;
  uint32_t& ssamples = sm.ssamples;
  Surface& S = sm.S;
  uint32_t* lists = sm.lists;
  const int tid = threadIdx.x & (NT - 1), lane = tid & 31, warp = tid >> 5;
  if (tid == 0) {  // the tile's surface and bins
    const uint32_t fcnt = ws.fine_count[tile], foff = ws.fine_off[tile] - fcnt, ftot = ws.ctr->fine_total;
    uint32_t s, ct;
    if (ws.tiles) {  // two rounds of loads
      const uint2 tt = ws.tiles[tile];
      s = surface >= 0 ? (uint32_t)surface : tt.x;
      ct = tt.y;
      S = surfs[s];
    } else {  // the surface is known (a cube face, or the pass's only one)
      s = surface >= 0 ? (uint32_t)surface : 0u;
      S = surfs[s];
      const uint32_t lt = tile - S.tile_base;
      const int tx = lt % S.tiles_x, ty = lt / S.tiles_x;
      ct = S.ctile_base + (ty >> ws.coarse_shift) * S.ctiles_x + (tx >> ws.coarse_shift);
    }
    sm.s = s;
    lists[0] = foff;
    lists[1] = fcnt;
    lists[3] = ws.coarse_count[ct];
    lists[2] = ftot + ws.coarse_off[ct] - lists[3];
    ssamples = 0;
    sm.szcap = kDepthClear;
  }
  if (with_id) {
    for (int p = tid; p < kTilePixels; p += NT) {
      sdepth[p] = kDepthClear;
      sid[p] = ~0ull;
    }
  }
  tile_barrier<NT, PART>();
  const uint32_t lt = tile - S.tile_base;
  const int tx0 = (lt % S.tiles_x) * kTile, ty0 = (lt / S.tiles_x) * kTile;
  if (with_id && lists[1] + lists[3] == 0) {  // no records: an empty tile
    // kernel3's output here is the clear colour and zero normals, unless the
    // view blends in another context's colour: write it, and mark the tile
    // (kernel3 then reads nothing of it, the record map included)
    uint32_t* rgba = nullptr;
    uint32_t* nrm = nullptr;
    uint32_t* rmap = S.rec;
    uint32_t clear = 0;
    if (ws.tile_empty) {
      const ViewParams& V = ws.views[sm.s];
      const bool direct = V.blend_depth == nullptr;
      if (direct) {
        rgba = reinterpret_cast<uint32_t*>(V.rgba);
        nrm = reinterpret_cast<uint32_t*>(V.normals);
        rmap = nullptr;
        clear = pack_rgba(V.clear[0], V.clear[1], V.clear[2], V.clear[3]);
      }
      if (tid == 0) ws.tile_empty[tile] = direct ? 1 : 0;
    }
    for (int lp = tid; lp < kTilePixels; lp += NT) {
      const int px = tx0 + (lp & (kTile - 1)), py = ty0 + (lp / kTile);
      if (px < S.width && py < S.height) {
        const size_t p = (size_t)py * S.width + px;
        S.depth[p] = kDepthClear;
        if (S.id) S.id[p] = kNoId;
        if (rmap) rmap[p] = kNoId;
        if (rgba) rgba[p] = clear;
        if (nrm) nrm[p] = 0;
      }
    }
    return;
  }
  if (with_id && ws.tile_empty && tid == 0) ws.tile_empty[tile] = 0;
  if (!with_id) {
    // depth-only passes: the surface was cleared and holds the small
    // triangles the setup rasterised (a tile without records is not listed)
    for (int p = tid; p < kTilePixels; p += NT) {
      const int px = tx0 + (p & (kTile - 1)), py = ty0 + p / kTile;
      sdepth[swz32(p)] = (px < S.width && py < S.height) ? S.depth[(size_t)py * S.width + px] : kDepthClear;
    }
  }
  // the walk's fragment size (Surface.chunk: op_size for views, op_size_light
  // for cube faces).  CC (passes of several view surfaces) takes it as the
  // constant op_size, so that the walk rule's modulos are multiplications:
  // 1.8 % faster batches; the one-view raster measured faster with the
  // runtime value
  const int chunk = CC ? kOpSize : S.chunk;
  const uint32_t nfine = lists[1], ntotal = lists[1] + lists[3];
  const int passes = ntotal == 0 ? 0 : (with_id ? 2 : 1);
  const bool resident = ntotal <= (uint32_t)NT;
  // A tile resolved in one chunk keeps the canonical id as 32 bits, key <<
  // kSlotBits | staged slot (keys of the scene below ws.pack_keys): a record
  // has one key, so the minimum of these picks the same record as the
  // minimum of (key << 32 | record), with half the shared-memory traffic.
  const bool packed = with_id && resident && ws.pack_keys;
  uint32_t* sid32 = reinterpret_cast<uint32_t*>(sid);
  // the warp's list of covered pixels and its length
  uint2* hits = sm.hits + warp * kHits;
  uint32_t nh = 0;
  bool listing = kHits > 0 && (resident || ws.rec_cap <= kHitRecords);
  uint32_t wsamples = 0;  // covered tests of pass 0 seen by this warp
  bool cached = false;
  for (int pass = 0; pass < passes; pass++) {
    for (uint32_t c0 = 0; c0 < ntotal; c0 += NT) {
      const uint32_t m = min((uint32_t)NT, ntotal - c0);
      if (cached) {
        // pass 1 from the lists of pass 0
        if (c0 == 0) {
          for (uint32_t g = lane; g < nh; g += 32) {
            const uint2 e = hits[g];
            const int p = (int)(e.y & 0xFF);
            const uint32_t lo = e.y >> 8;
            const uint32_t d = e.x, fd = sdepth[swz32(p)];
            if (d > fd - kBufError && d < fd + kBufError) {
              if (!resident)
                atomicMin(&sid[swz64(p)], ((unsigned long long)__ldg(&ws.rec[lo].key) << 32) | lo);
              else if (packed)
                atomicMin(sid32 + swz32(p), (__float_as_uint(srec[2][lo].w) << kSlotBits) | lo);
              else
                atomicMin(&sid[swz64(p)], ((unsigned long long)__float_as_uint(srec[2][lo].w) << 32) | sidx[lo]);
            }
          }
        }
        break;
      }
      if (!(resident && pass == 1)) {
        if (pass != 0 || c0 != 0) tile_barrier<NT, PART>();  // the previous chunk's readers are done
        uint32_t rows = 0, r = 0, geo = 0, skip = 0;
        int bx0 = 0, bx1 = 0, by0 = 0, by1 = 0;
        float4 q0, q1, q2, q3;
        if ((uint32_t)tid < m) {
          const uint32_t e = c0 + tid;
          r = e < nfine ? ws.bins[lists[0] + e] : ws.bins[lists[2] + (e - nfine)];
          const float4* src = reinterpret_cast<const float4*>(ws.rec + r);
          q0 = __ldg(src);
          q1 = __ldg(src + 1);
          q2 = __ldg(src + 2);
          q3 = __ldg(src + 3);
          const uint32_t xr = __float_as_uint(q3.x), yr = __float_as_uint(q3.y);
          bx0 = max((int)(xr & 0xFFFF), tx0), bx1 = min((int)(xr >> 16), tx0 + kTile);
          by0 = max((int)(yr & 0xFFFF), ty0), by1 = min((int)(yr >> 16), ty0 + kTile);
          if (bx1 > bx0 && by1 > by0) {
            const uint32_t kind = __float_as_uint(q3.w);
            rows = (uint32_t)(by1 - by0);
            geo = (uint32_t)(bx0 - tx0) | ((uint32_t)(by0 - ty0) << 4) | ((uint32_t)(bx1 - bx0) << 8) | (kind << 13);
            // the walk rule of the bbox's left column, once per row of this
            // tile (a tight box has left that column out)
            if ((int)(xr & 0xFFFF) >= tx0 && !(kind & kRecTight)) skip = walk_skip_rows(xr, yr, by0, by1, ty0, chunk);
          }
        }
        // Depth cull.  A record that covers every coverable pixel of the tile
        // bounds their final depths by its own farthest depth here; a record
        // whose nearest depth lies 20 or more behind such a bound changes
        // neither the depths nor (outside kernel2's window) the ids, so when
        // it covers its whole box its pixels are only counted.  The bound
        // comes from the chunks before this one and the warp's own records.
        // (Coverable: a bbox ends at the surface's last column and row, which
        // stay clear.)
        const bool whole = rows && bx0 == tx0 && by0 == ty0 && bx1 == min(tx0 + kTile, S.width - 1) &&
                           by1 == min(ty0 + kTile, S.height - 1) && !skip;
        uint32_t zcap = __shfl_sync(0xFFFFFFFFu, sm.szcap, 0);
        if (__any_sync(0xFFFFFFFFu, whole) || zcap != kDepthClear) {
          bool full = false;
          uint32_t dlo = 0, dhi = kDepthClear;
          if (rows)
            full = box_bounds(q0.x, q0.y, q0.z, EdgeTest{q1.x, q1.y, q1.z, q2.x, q2.y, q2.z, 1.0f, q0.w}, bx0, by0,
                              bx1 - 1, by1 - 1, &dlo, &dhi);
          const uint32_t bound = __reduce_min_sync(0xFFFFFFFFu, full && whole ? dhi : kDepthClear);
          if (bound < zcap) {
            zcap = bound;
            if (lane == 0) atomicMin(&sm.szcap, bound);
          }
          uint32_t hidden = 0;
          if (full && zcap < kDepthClear - kBufError && dlo >= zcap + kBufError) {
            hidden = (uint32_t)((bx1 - bx0) * (by1 - by0)) - (uint32_t)__popc(skip);
            rows = 0;
          }
          if (pass == 0) wsamples += __reduce_add_sync(0xFFFFFFFFu, hidden);
        }
        const uint32_t word = rows ? (rows | (1u << kCountShift)) : 0u;
        uint32_t tot = 0;
        const uint32_t off = block_excl_scan1<NT, PART>(word, swarp, &tot);
        if (rows) {
          const uint32_t slot = off >> kCountShift;
          srec[0][slot] = q0;
          srec[1][slot] = make_float4(q1.x, q1.y, q1.z, span_slope(q1.y));
          srec[2][slot] = q2;
          sm.sinv[slot] = make_float2(span_slope(q2.y), span_slope(-(q1.y + q2.y)));
          sidx[slot] = r;
          sgeo[slot] = geo;
          sskip[slot] = (uint16_t)skip;
          soff[slot] = off & ((1u << kCountShift) - 1);
        }
        if (tid == 0) {
          soff[tot >> kCountShift] = tot & ((1u << kCountShift) - 1);
          sscan = tot;
        }
        tile_barrier<NT, PART>();
      }
      const uint32_t nstaged = sscan >> kCountShift;
      const uint32_t total = soff[nstaged];
      // this warp's contiguous share of the row list, in windows of 32 (a
      // few rows may hold many pixels: shares are equal, not whole windows)
      const uint32_t per = (total + NW - 1) / NW;
      const uint32_t start = min(total, (uint32_t)warp * per), end = min(total, start + per);
      if (start < end) {
        // first record: the last staged record with soff <= start (warp-uniform;
        // soff increases, so that is their number)
        int rec = -1;
        for (uint32_t k = lane; k < nstaged + lane; k += 32)
          rec += __popc(__ballot_sync(0xFFFFFFFFu, k < nstaged && soff[k] <= start));
        uint2* spans = sm.spans[warp];
        // spans appended and the pixel pairs in them; pairs done, and the span
        // the next one lies in
        uint32_t nspans = 0, npairs = 0, done = 0, cur = 0;
        const unsigned below = (1u << lane) - 1u, upto_lane = (2u << lane) - 1u;
#pragma unroll 1
        for (uint32_t base = start; base < end; base += 32) {
          // record starts inside (base, base + 32): at most 32 records
          const uint32_t nxt = (uint32_t)rec + 1 + lane;
          const uint32_t pos = nxt < nstaged ? soff[nxt] - base : 32u;
          const uint32_t starts = __reduce_or_sync(0xFFFFFFFFu, pos < 32u ? (1u << pos) : 0u);
          uint32_t pairs = 0, span = 0;
          if (base + lane < end) {
            // the lane's row of a record, and the span of it that can be covered
            const uint32_t row_rec = (uint32_t)rec + __popc(starts & upto_lane), geo = sgeo[row_rec];
            const int ly = (int)((geo >> 4) & 0xF) + (int)(base + lane - soff[row_rec]);
            int xa = (int)(geo & 0xF), xb = xa + (int)((geo >> 8) & 0x1F) - 1;
            // the walk rule: only a row's first pixel can be the bbox's left column
            xa += (int)((sskip[row_rec] >> ly) & 1u);
            if (geo & ((kRecInside | kRecNear) << 13)) {
              const float4 q1 = srec[1][row_rec], q2 = srec[2][row_rec];
              const float2 inv = sm.sinv[row_rec];
              const float ftx = (float)tx0, fy = (float)(ty0 + ly);
              const float bound = srec[0][row_rec].w;
              float slack = 0.5f, slack_u = (geo & (kRecTight << 13)) ? 0.5f : 4.0f;  // row_span's
              if (geo & (kRecNear << 13))
                slack = slack_u = span_slack(q1.x, q1.y, q1.z, q2.x, q2.y, q2.z, bound, ftx + (float)kTile, fy);
              row_span_slack((q1.x + q1.z * fy) + q1.y * ftx, (q2.x + q2.z * fy) + q2.y * ftx, bound, q1.w, inv.x,
                             inv.y, slack, slack_u, &xa, &xb);
            }
            if (xb >= xa) {
              pairs = (uint32_t)(xb - xa + 2) >> 1;
              span = row_rec | ((uint32_t)ly << 10) | ((uint32_t)xa << 14) | ((uint32_t)xb << 18);
            }
          }
          // the record of row base + 32: lane 31's, or the next one if it starts there
          rec += __popc(starts);
          if ((uint32_t)rec + 1 < nstaged && soff[rec + 1] == base + 32) rec++;
          // append the spans, their pixel pairs laid end to end
          uint32_t first = pairs;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, first, o);
            if (lane >= o) first += v;
          }
          const unsigned who = __ballot_sync(0xFFFFFFFFu, pairs != 0);
          __syncwarp();  // (readers of the spans overwritten here are done)
          if (pairs)
            spans[(nspans + __popc(who & below)) % kSpanRing] = make_uint2(npairs + first - pairs, span);
          npairs += __shfl_sync(0xFFFFFFFFu, first, 31);
          nspans += (uint32_t)__popc(who);
          __syncwarp();
          // test them 32 at a time; fewer wait for the next rows
          const uint32_t least = base + 32 < end ? 32u : 1u;
#pragma unroll 1
          for (; npairs - done >= least; done += min(32u, npairs - done)) {
            if (cur + 1 < nspans && spans[(cur + 1) % kSpanRing].x <= done) cur++;
            const uint32_t sn = cur + 1 + lane;
            const uint32_t sp = sn < nspans ? spans[sn % kSpanRing].x - done : 32u;
            const uint32_t sstarts = __reduce_or_sync(0xFFFFFFFFu, sp < 32u ? (1u << sp) : 0u);
            const uint2 e = spans[(cur + (uint32_t)__popc(sstarts & upto_lane)) % kSpanRing];
            cur += (uint32_t)__popc(sstarts);
            const uint32_t lo = e.y & 0x3FF;
            const int ly = (int)((e.y >> 10) & 0xF), lx = (int)((e.y >> 14) & 0xF) + 2 * (int)(done + lane - e.x);
            const int p = ly * kTile + lx;
            const float4 q[3] = {srec[0][lo], srec[1][lo], srec[2][lo]};
            const float fx = (float)(tx0 + lx), fy = (float)(ty0 + ly);
            const bool on = done + lane < npairs;
            const bool h0 = on && rec_in_tri(q, fx, fy);
            const bool h1 = on && lx < (int)(e.y >> 18) && rec_in_tri(q, fx + 1.0f, fy);
            const unsigned b0 = __ballot_sync(0xFFFFFFFFu, h0), b1 = __ballot_sync(0xFFFFFFFFu, h1);
            const uint32_t n0 = (uint32_t)__popc(b0), n1 = (uint32_t)__popc(b1);
            if (pass == 0) {
              wsamples += n0 + n1;
              if (listing && nh + n0 + n1 > kHits) {  // warp-uniform
                nh = compact_hits(hits, nh, sdepth);
                listing = nh + n0 + n1 <= kHits;
              }
            }
            auto resolve = [&](float px, int pp, uint32_t slot) {
              const uint32_t d = depth_at(q[0].x, q[0].y, q[0].z, px, fy);
              if (pass == 0) {
                atomicMin(&sdepth[swz32(pp)], d);
                if (listing) hits[slot] = make_uint2(d, (uint32_t)pp | ((resident ? lo : sidx[lo]) << 8));
              } else {
                const uint32_t fd = sdepth[swz32(pp)];
                if (d > fd - kBufError && d < fd + kBufError) {
                  if (packed)
                    atomicMin(sid32 + swz32(pp), (__float_as_uint(q[2].w) << kSlotBits) | lo);
                  else
                    atomicMin(&sid[swz64(pp)], ((unsigned long long)__float_as_uint(q[2].w) << 32) | sidx[lo]);
                }
              }
            };
            if (h0) resolve(fx, p, nh + (uint32_t)__popc(b0 & below));
            if (h1) resolve(fx + 1.0f, p + 1, nh + n0 + (uint32_t)__popc(b1 & below));
            if (pass == 0 && listing) nh += n0 + n1;
          }
        }
      }
    }
    if (pass == 0 && lane == 0 && wsamples) atomicAdd(&ssamples, wsamples);
    // the id pass reads pass 0's lists when every warp's held (block-uniform)
    if (with_id && pass == 0)
      cached = __syncthreads_and(listing) != 0;
    else
      tile_barrier<NT, PART>();
  }
  if (tid == 0 && ssamples) atomicAdd(&ws.ctr->samples, (unsigned long long)ssamples);
  for (int lp = tid; lp < kTilePixels; lp += NT) {
    const int px = tx0 + (lp & (kTile - 1)), py = ty0 + (lp / kTile);
    if (px < S.width && py < S.height) {
      const size_t p = (size_t)py * S.width + px;
      S.depth[p] = sdepth[swz32(lp)];
      if (with_id && packed) {
        const uint32_t v = sid32[swz32(lp)];
        if (S.id) S.id[p] = v == ~0u ? kNoId : v >> kSlotBits;
        S.rec[p] = v == ~0u ? kNoId : sidx[v & ((1u << kSlotBits) - 1)];
      } else if (with_id) {
        const unsigned long long v = sid[swz64(lp)];
        if (S.id) S.id[p] = v == ~0ull ? kNoId : (uint32_t)(v >> 32);
        S.rec[p] = v == ~0ull ? kNoId : (uint32_t)v;
      }
    }
  }
}

// prep_blocks (one view that shades): the first blocks of the grid compute the
// shade constants instead, beside the tiles, which do not read them.
template <int NT, bool CC>
__global__ void __launch_bounds__(NT, raster_ctas<NT>())
    k_raster(Workspace ws, const Surface* __restrict__ surfs, uint32_t tile0, uint32_t prep_blocks,
             const __grid_constant__ SceneDev sc) {
  __shared__ RasterSmem<NT, true> sm;
  if (ws.ctr->overflow) return;
  if (!CC && blockIdx.x < prep_blocks) {
    // (as many warps as the tile's shared memory has buffers for)
    constexpr uint32_t kWarps = NT / 32 < sizeof(sm) / (16 * kPrepQuads) ? NT / 32 : sizeof(sm) / (16 * kPrepQuads);
    const uint32_t nrec = min(ws.ctr->nrec, ws.rec_cap), warp = threadIdx.x / 32;
    if (warp < kWarps)
      for (uint32_t r = (blockIdx.x * kWarps + warp) * 32; r < nrec; r += prep_blocks * kWarps * 32)
        prep_records(sc, ws.srec + r, min(32u, nrec - r), reinterpret_cast<float4*>(&sm) + warp * kPrepQuads);
    return;
  }
  raster_tile<NT, true, CC>(ws, surfs, tile0 + blockIdx.x - prep_blocks, -1, sm);
}

// The tiles of ws.list (surfaces of per_surface tiles each) of a depth-only
// pass, by as many blocks as fit at once: 24,576 tiles of a cubemap of which
// some 4,000 have records took 30 us as a block each, mostly to start them.
// A long list (kPartWaves tiles a block of 128) goes to the blocks' halves, a
// tile each, as in view passes of many tiles: three lights among large walls
// 123 -> 98 us.  A list of some 6,000 tiles took 32.5 us by blocks and 34.8 by
// halves, one that the blocks take at once (4K) 13.5 and 17.
constexpr uint32_t kPartWaves = 6;
constexpr int kPart = 64;
template <int NT>
__global__ void __launch_bounds__(NT, 1280 / NT) k_raster_list(Workspace ws, const Surface* __restrict__ surfs,
                                                               uint32_t per_surface) {
  constexpr uint32_t kParts = NT == 128 ? NT / kPart : 1;
  __shared__ union {
    RasterSmem<NT, false> one;
    RasterSmem<kPart, false> part[kParts];
  } sm;
  if (ws.ctr->overflow) return;
  const uint32_t n = ws.ctr->nlist;
  if (kParts > 1 && n >= kPartWaves * gridDim.x) {
    const uint32_t part = threadIdx.x / kPart % kParts;
    for (uint32_t i = kParts * blockIdx.x + part; i < n; i += kParts * gridDim.x) {
      const uint32_t tile = ws.list[i];
      raster_tile<kPart, false, false, true>(ws, surfs, tile, (int)(tile / per_surface), sm.part[part]);
      tile_barrier<kPart, true>();
    }
    return;
  }
  for (uint32_t i = blockIdx.x; i < n; i += gridDim.x) {
    const uint32_t tile = ws.list[i];
    raster_tile<NT, false>(ws, surfs, tile, (int)(tile / per_surface), sm.one);
    __syncthreads();  // the next tile reuses the shared memory
  }
}

// ---- kernel3 ------------------------------------------------------------------
// Byte -> float: one conversion that selects its byte (kernel3 0.6 % fewer
// instructions than 2^23 + b, minus 2^23; the conversion pipe is a third busy).
__device__ __forceinline__ float u8f(uint32_t b) { return (float)(uint8_t)b; }

// read_tex_array_all_precalculated (cl2.cl:823-851) in one atlas slot of the
// texture level table: (ox, oy) is the slot origin in its page, tnum * width
// in the reference, an integer below 2048 and so exact in float, which makes
// its fma(tnum, width, c) = ox + c.
struct TexSlot {
  int ox, oy;
  float width;
  const uchar4* page;
};
__device__ __forceinline__ TexSlot level_slot(const SceneDev& sc, float4 lv) {
  TexSlot t;
  t.ox = __float_as_int(lv.x);
  t.oy = __float_as_int(lv.y);
  t.width = lv.z;
  t.page = sc.atlas + (size_t)__float_as_uint(lv.w) * kTexPage * kTexPage;
  return t;
}
__device__ __forceinline__ f4 texel(const TexSlot& ts, int ix, int iy) {
  const uint32_t t = __ldg(reinterpret_cast<const uint32_t*>(ts.page) + ((size_t)iy * kTexPage + ix));
  f4 r; r.x = u8f(t & 0xFF); r.y = u8f((t >> 8) & 0xFF); r.z = u8f((t >> 16) & 0xFF); r.w = u8f(t >> 24);
  return r;
}

// The four texels of a bilinear footprint at (mx, my) of a slot, and its
// weights.  The reference clamps the float coordinates floor(m) and floor(m) +
// 1 to [0.001, w - 0.001] and truncates o + c, o the slot origin: in integers
// that is o + clamp(floor(m), 0, w - 1) (0.001 truncates to 0, w - 0.001 to w
// - 1; o + w <= 2048 keeps o + w - 0.001 below o + w in float).  Coordinates
// come from texture_mod, so floor(m) is not negative; the conversion and the
// clamps keep any other in the slot all the same, and a NaN, whose weights
// make the result NaN whatever the texels are.
struct Footprint {
  int x0, x1, y0, y1;
  float ux, uy;
};
__device__ __forceinline__ Footprint footprint_at(const TexSlot& ts, float mx, float my) {
  Footprint f;
  const float posx = floorf(mx), posy = floorf(my);
  const int w = (int)ts.width;
  const int px = __vimin_s32_relu((int)posx, w), py = __vimin_s32_relu((int)posy, w);
  f.x0 = ts.ox + min(px, w - 1), f.x1 = ts.ox + __viaddmin_s32(px, 1, w - 1);
  f.y0 = ts.oy + min(py, w - 1), f.y1 = ts.oy + __viaddmin_s32(py, 1, w - 1);
  f.ux = mx - posx, f.uy = my - posy;
  return f;
}

// The bilinear fetch of the normal map and the reflection map, which feed
// decisions: plain products.
__device__ f4 bilinear_exact(const TexSlot& ts, float mx, float my) {
  const Footprint f = footprint_at(ts, mx, my);
  const f4 c0 = texel(ts, f.x0, f.y0), c1 = texel(ts, f.x1, f.y0), c2 = texel(ts, f.x0, f.y1),
           c3 = texel(ts, f.x1, f.y1);
  const float ux = f.ux, uy = f.uy, bx = 1.0f - ux, by = 1.0f - uy;
  f4 r;
  r.x = fma_(c0.x, bx, c1.x * ux) * by + fma_(c2.x, bx, c3.x * ux) * uy;
  r.y = fma_(c0.y, bx, c1.y * ux) * by + fma_(c2.y, bx, c3.y * ux) * uy;
  r.z = fma_(c0.z, bx, c1.z * ux) * by + fma_(c2.z, bx, c3.z * ux) * uy;
  r.w = fma_(c0.w, bx, c1.w * ux) * by + fma_(c2.w, bx, c3.w * ux) * uy;
  return r;
}

// The bilinear fetch of a texel colour, which only scales the colour: the
// blend is contracted, and two channels go through one packed instruction.
__device__ __forceinline__ float2 dup2(float v) { return make_float2(v, v); }
struct Texel2 {
  float2 rg, ba;
};
__device__ __forceinline__ Texel2 texel2(const TexSlot& ts, int ix, int iy) {
  const uint32_t t = __ldg(reinterpret_cast<const uint32_t*>(ts.page) + ((size_t)iy * kTexPage + ix));
  Texel2 r;
  r.rg = make_float2(u8f(t & 0xFF), u8f((t >> 8) & 0xFF));
  r.ba = make_float2(u8f((t >> 16) & 0xFF), u8f(t >> 24));
  return r;
}
__device__ __forceinline__ Texel2 bilinear_colour(const TexSlot& ts, float mx, float my) {
  const Footprint f = footprint_at(ts, mx, my);
  const Texel2 c0 = texel2(ts, f.x0, f.y0), c1 = texel2(ts, f.x1, f.y0), c2 = texel2(ts, f.x0, f.y1),
               c3 = texel2(ts, f.x1, f.y1);
  const float2 u = dup2(f.ux), v = dup2(f.uy), bx = dup2(1.0f - f.ux), by = dup2(1.0f - f.uy);
  auto blend = [&](float2 a0, float2 a1, float2 a2, float2 a3) {
    return __ffma2_rn(__ffma2_rn(a2, bx, __fmul2_rn(a3, u)), v, __fmul2_rn(__ffma2_rn(a0, bx, __fmul2_rn(a1, u)), by));
  };
  Texel2 r;
  r.rg = blend(c0.rg, c1.rg, c2.rg, c3.rg);
  r.ba = blend(c0.ba, c1.ba, c2.ba, c3.ba);
  return r;
}

// texture_filter_diff (cl2.cl:1511-1573); COLOUR: bilinear_colour's blend, in
// packed channels (1080p kernel3 1 % fewer instructions).  The
// two mip levels come from the texture level table: level mip_lower (the
// texture itself at 0) and level min(mip_lower, 3) + 1, the slots the
// reference's tid_lower / tid_higher name.
template <bool COLOUR>
__device__ f4 texture_filter_diff(const SceneDev& sc, f2 vt, f2 vtdiff, int tid2) {
  const float4* lv = sc.texlv + (size_t)tid2 * kTexLevels;
  const float tsize = __ldg(&lv[0].z);
  f2 vtm = texture_mod(vt);
  float wx = vtdiff.x * tsize, wy = vtdiff.y * tsize;
  float worst = fsqrt(wx * wx + wy * wy);
  float wif = fmax_(log2_approx(worst), 0.0f);  // finite for every input
  float mip_lower = clampf_(floorf(wif), 0.0f, (float)kMipLevels);
  float fmd = wif - mip_lower;
  const int lo = (int)mip_lower, hi = min(lo, kMipLevels - 1) + 1;
  const TexSlot sl = level_slot(sc, __ldg(lv + lo)), sh = level_slot(sc, __ldg(lv + hi));
  const float i255 = 1.0f / 255.0f;
  f4 r;
  if (COLOUR) {
    const Texel2 c1 = bilinear_colour(sl, vtm.x * sl.width, vtm.y * sl.width);
    const Texel2 c2 = bilinear_colour(sh, vtm.x * sh.width, vtm.y * sh.width);
    const float2 f = dup2(fmd), k = dup2(i255), neg = dup2(-1.0f);  // fma(c1, -1, c2) = c2 - c1
    const float2 rg = __fmul2_rn(__ffma2_rn(__ffma2_rn(c1.rg, neg, c2.rg), f, c1.rg), k);
    const float2 ba = __fmul2_rn(__ffma2_rn(__ffma2_rn(c1.ba, neg, c2.ba), f, c1.ba), k);
    r.x = rg.x; r.y = rg.y; r.z = ba.x; r.w = ba.y;
  } else {
    const f4 c1 = bilinear_exact(sl, vtm.x * sl.width, vtm.y * sl.width);
    const f4 c2 = bilinear_exact(sh, vtm.x * sh.width, vtm.y * sh.width);
    r.x = (c1.x + (c2.x - c1.x) * fmd) * i255;
    r.y = (c1.y + (c2.y - c1.y) * fmd) * i255;
    r.z = (c1.z + (c2.z - c1.z) * fmd) * i255;
    r.w = (c1.w + (c2.w - c1.w) * fmd) * i255;
  }
  return r;
}

// A tap coordinate of generate_ssao: clamped to [1, n - 2] as the reference
// does; for views 1 or 2 pixels wide (high), where that range is empty and the
// reference reads outside its buffer, clamped into the view (0).
__device__ __forceinline__ int ssao_coord(float v, int n) {
  return max((int)clampf_(v, 1.0f, (float)n - 2.0f), 0);
}

// The 25 taps' counts with the thresholds as the reference adds them up: the
// few pixels for which ssao_tap is not exact (within 2 units below a power of
// two, or nearer than 8).
__device__ __noinline__ int ssao_taps_any(int x, int y, float dep, float world_rad, const uint32_t* depth, int W,
                                          int H) {
  // the thresholds dep + z, z = -2..2, scaled by 2^32 (depth_scaled)
  const float t0 = (dep + -2.0f) * kTwo32, t1 = (dep + -1.0f) * kTwo32, t2 = dep * kTwo32,
              t3 = (dep + 1.0f) * kTwo32, t4 = (dep + 2.0f) * kTwo32;
  int acc = 0;
  const float r1 = roundf(world_rad), r2 = roundf(2.0f * world_rad), r0 = roundf(0.0f * world_rad);
  for (int yy = -2; yy <= 2; yy++) {
    const float oy = yy == 0 ? r0 : copysignf(yy == 2 || yy == -2 ? r2 : r1, (float)yy);
    const uint32_t* row = depth + (size_t)ssao_coord((float)y + oy, H) * W;
    for (int xx = -2; xx <= 2; xx++) {
      const float ox = xx == 0 ? r0 : copysignf(xx == 2 || xx == -2 ? r2 : r1, (float)xx);
      acc += ssao_count(depth_scaled(__ldca(row + ssao_coord((float)x + ox, W))), t0, t1, t2, t3, t4);
    }
  }
  return acc;
}

// ssao_coord(v + off) for an integer offset: max(v + off, 1), then min with
// n - 2 and max with 0, an instruction each.
__device__ __forceinline__ int ssao_coord_int(int v, int off, int n) {
  return __vimin_s32_relu(__viaddmax_s32(v, off, 1), n - 2);
}

// generate_ssao (cl2.cl:2194-2260) for a pixel of depth d.  The 25 taps share
// 5 rows and 5 columns, whose offsets round(k * world_rad), k = -2..2, are the
// same five values: round is odd-symmetric (half away from zero) and 1 * r,
// 2 * r and -r, -2 * r are exact, so two roundings give all of them; they and
// the coordinates are small integers.  The count (at most 125, exact in float)
// is kept in an integer.  Far from the camera (world_rad < 0.25) every offset
// rounds to 0 and all 25 taps read the same pixel; when that holds for the
// whole warp, the pixel is read once and its count taken 25 times.
// seed2 = rand_xorshift(wang_hash(x + W*H*y)), the pixel's first random
// number, which kernel3's normal jitter also draws.
// depth is read with plain (coherent) loads: in the fused pass other blocks
// wrote it during the same launch.
__device__ float generate_ssao(int x, int y, uint32_t seed2, uint32_t d, const uint32_t* depth, int W, int H,
                               float fov) {
  float foffset = (float)seed2 * kInvMulInt;
  const float dep = depth_to_dist(d);
  float rad = kSsaoRad + foffset * 0.5f;  // foffset / 2, exact
  float world_rad = fdiv(rad * fov, dep);
  int acc = 0;
  const float c8 = (2.0f - dep) * 0.125f;
  if (!ssao_exact(dep)) {
    acc = ssao_taps_any(x, y, dep, world_rad, depth, W, H);
  } else if (__all_sync(__activemask(), world_rad < 0.25f)) {
    acc = 25 * (int)(ssao_tap(__ldca(depth + (size_t)ssao_coord_int(y, 0, H) * W + ssao_coord_int(x, 0, W)), c8) -
                     kSsaoTapZero);
  } else {
    // roundf of a value >= 0: the truncation of v + 0.5, that sum rounded toward
    // zero (it never passes an integer).  Views are below 4096.
    const int i1 = min(__float2int_rz(__fadd_rz(world_rad, 0.5f)), 8192);
    const int i2 = min(__float2int_rz(__fadd_rz(2.0f * world_rad, 0.5f)), 8192);
    const int off[5] = {-i2, -i1, 0, i1, i2};
    int wx[5];
#pragma unroll
    for (int k = 0; k < 5; k++) wx[k] = ssao_coord_int(x, off[k], W);
    uint32_t sum = 0;
#pragma unroll
    for (int k = 0; k < 5; k++) {
      const uint32_t* row = depth + (size_t)ssao_coord_int(y, off[k], H) * W;
#pragma unroll
      for (int xx = 0; xx < 5; xx++) sum += ssao_tap(__ldca(row + wx[xx]), c8);
    }
    acc = (int)(sum - 25u * kSsaoTapZero);
  }
  // the occlusion scales the colour only: approximate divisions
  const float facc = (float)acc * (1.0f / 125.0f);
  return 1.0f - (1.0f - facc) * (1.0f / kSsaoDiv);
}


// generate_hard_occlusion (cl2.cl:2536-2701), SMOOTH_SHADOWS.  Inlined: as
// a call it cost kernel3 spills around it (1080p kernel3 0.236 -> 0.233 ms
// inlined).  ptl: pixel to light, rinv: its approximate reciprocal length.
__device__ __forceinline__ float hard_occlusion(const SceneDev& sc, f3 lpos, f3 normal, f3 ptl, float rinv,
                                                const uint32_t* buf, int face, f3 gpos, int shnum) {
  f3 c = mk3(sc.face_cos[face][0], sc.face_cos[face][1], sc.face_cos[face][2]);
  f3 s = mk3(sc.face_sin[face][0], sc.face_sin[face][1], sc.face_sin[face][2]);
  f3 local = rot_cs(gpos, lpos, c, s);
  f3 post = depth_project1(local, (float)kLightBufferDim, (float)kLightBufferDim, kLFov);
  float dpth = post.z;
  const uint32_t* map = buf + (size_t)(face + shnum * 6) * kLightBufferDim * kLightBufferDim;
  float px = clampf_(post.x, 3.0f, kLightBufferDim - 4.0f);
  float py = clampf_(post.y, 3.0f, kLightBufferDim - 4.0f);
  int ix = f2i_sat(px), iy = f2i_sat(py);
  // The bias is 50 tan(angle of incidence), at most 50: with the cosine below
  // kBiasFullCos it is 50 whatever the cosine is, so neither the exact unit
  // vector nor its arc cosine and tangent are needed.
  float bias = kShadowBias;
  if (!(dot3(normal, ptl) * rinv <= kBiasFullCos - 0.01f)) bias = shadow_bias(dot3(normal, fast_normalize3(ptl)));
  // The taps' test dpth > depth_to_dist(d) + bias in depth units: it holds
  // below lo and fails above hi; a tap between them (next to none) has all of
  // them tested as they stand.
  uint32_t lo, hi;
  const bool limits = shadow_limits(dpth, bias, &lo, &hi);
  const uint32_t* row = map + (iy - 1) * kLightBufferDim + ix - 1;
  uint32_t cond = 0, near = 0xFFFFFFFFu;  // bit (yy+1)*4 + (xx+1)
#pragma unroll
  for (int k = 0; k < 16; k++) {
    const uint32_t d = __ldg(row + (k >> 2) * kLightBufferDim + (k & 3));
    if (d < lo) cond |= 1u << k;
    near = min(near, d - lo);
  }
  if (near <= hi - lo || !limits) {
    cond = 0;
#pragma unroll 1
    for (int k = 0; k < 16; k++) {
      const float ldp = depth_to_dist(__ldg(row + (k >> 2) * kLightBufferDim + (k & 3)));
      if (dpth > ldp + bias) cond |= 1u << k;
    }
  }
  // The 3x3 bilinear blend of the 4x4 tests: every tap has the same
  // fractional offsets (ux, uy), so the sum of the nine bilinear_interpolate
  // calls is separable, with column weights (1 - ux, 1, 1, ux) and row
  // weights (1 - uy, 1, 1, uy).  The occlusion scales the colour only.
  const float mx = (px + 0.5f) - 0.5f, my = (py + 0.5f) - 0.5f;
  const float ux = mx - floorf(mx), uy = my - floorf(my);
  const float by = 1.0f - uy;
  // per column group (left, middle two, right): tests of the top row, the
  // middle two rows and the bottom row
  auto rows = [&](uint32_t top, uint32_t mid, uint32_t bot) {
    return fma_(uy, (float)__popc(cond & bot), fma_(by, (float)__popc(cond & top), (float)__popc(cond & mid)));
  };
  const float sl = rows(0x0001u, 0x0110u, 0x1000u);
  const float sm = rows(0x0006u, 0x0660u, 0x6000u);
  const float sr = rows(0x0008u, 0x0880u, 0x8000u);
  const float shadow = fma_(ux, sr, fma_(1.0f - ux, sl, sm));
  return shadow * (1.0f / 9.0f);
}

// Vertex colour channels (colour path: multiplication by 1/255).
__device__ __forceinline__ f4 vertex_col(uint32_t c) {
  const float k = 1.0f / 255.0f;
  f4 r;
  r.x = u8f(c >> 24) * k;
  r.y = u8f((c >> 16) & 0xFF) * k;
  r.z = u8f((c >> 8) & 0xFF) * k;
  r.w = u8f(c & 0xFF) * k;
  return r;
}


__device__ __forceinline__ f3 cnormalize(f3 a) {
  float r = rsqrt_ftz(dot3(a, a));
  return mk3(a.x * r, a.y * r, a.z * r);
}
// Colour-path dot product with contraction.
__device__ __forceinline__ float cdot3(f3 a, f3 b) { return fma_(a.z, b.z, fma_(a.y, b.y, a.x * b.x)); }
// rational_acos (cl2.cl:1919-1936) in Horner form: x (a + b x^2) / (1 + c x^2 + d x^4) + pi/2.
__device__ __forceinline__ float c_rational_acos(float x) {
  const float a = -0.939115566365855f, b = 0.9217841528914573f, c = -1.2845906244690837f,
              d = 0.295624144969963174f;
  const float x2 = x * x;
  return fma_(x * fma_(b, x2, a), crcp(fma_(x2, fma_(d, x2, c), 1.0f)), kPi / 2.0f);
}


// Colour-only square root: 0 for 0 and for subnormals (whose root is below
// 1.1e-19; rsqrt_ftz takes them for 0, and x * inf is infinite), NaN for a
// negative normal input.  (An infinite input gives NaN as well; gamma_inv's sum
// of infinities of both signs is NaN either way.)
__device__ __forceinline__ float csqrt(float x) {
  const float s = x * rsqrt_ftz(x);
  return fabsf(x) < 1.17549435e-38f ? 0.0f : s;
}
// gamma_inv (cl2.cl:5778-5782) on the colour path.
__device__ __forceinline__ float c_gamma_inv(float c) {
  float s1 = csqrt(c);
  float s2 = csqrt(s1);
  float s3 = csqrt(s2);
  return fma_(-0.368262736f, s3, fma_(0.783140355f, s2, 0.585122381f * s1));
}
// gamma_fwd (cl2.cl:5763-5770) in Horner form, for colours
__device__ __forceinline__ float c_gamma_fwd(float c) {
  return c * fma_(fma_(0.305306011f, c, 0.682171111f), c, 0.012522878f);
}

// kernel3's attenuation cutoff: a light adds (illum - 0.1) / 0.9 where that is positive
constexpr float kLightCutoff = 0.1f;

// A light as the shade loop reads it, staged once per CTA in shared memory
// as three float4: (pos, cut2), (colour, brightness, divided by 1 - cutoff
// for lights without shadows), (radius, 1 / radius approximated, diffuse,
// shadow | is_static << 1).  The colour is already in
// linear space when the view renders linearly (the same gamma_fwd every pixel
// would apply).  cut2 is a conservative squared distance beyond which a light
// without shadows stays under kernel3's attenuation cutoff, so the pixel
// skips it without computing the attenuation: brightness / (d / radius + 1)^2
// <= 0.1 holds beyond d = radius * (sqrt(10 * brightness) - 1), and the
// margins below cover the approximate colour-path arithmetic of that test
// (relative errors of a few 1e-7).  -1: always under the cutoff; +inf: no
// early test (shadow lights, whose cutoff decides the cubemap later shadow
// lights read, and lights whose radius or brightness is not finite); at most
// the largest float for all others: a squared distance that overflows is past
// any finite radius.
constexpr int kLightQuads = 3;
__device__ __forceinline__ void stage_light(const gbr_light* L, bool linear, float4* dst) {
  f3 c = mk3(L->col[0], L->col[1], L->col[2]);
  if (linear) c = mk3(gamma_fwd(c.x), gamma_fwd(c.y), gamma_fwd(c.z));
  const float radius = L->radius, brightness = L->brightness;
  const float b10 = 10.0f * brightness;
  const float largest = 3.4028235e38f;
  float cut2 = __int_as_float(0x7F800000);
  if (!L->shadow && radius > 0.0f && b10 == b10) {
    if (b10 <= 1.0f) {
      cut2 = -1.0f;
    } else {
      const float rs = radius * ((sqrtf(b10) * 1.00001f - 1.0f) * 1.00001f);
      cut2 = (rs * rs) * 1.00001f;
    }
  }
  if (!L->shadow && fabsf(radius) <= largest && fabsf(b10) <= largest) cut2 = fmin_(cut2, largest);
  // lights without shadows fold kernel3's cutoff into the brightness:
  // (b / tt^2 - 0.1) / 0.9 = (b / 0.9) / tt^2 - 0.1 / 0.9 (colour only)
  const float bw = L->shadow ? brightness : brightness * (1.0f / (1.0f - kLightCutoff));
  dst[0] = make_float4(L->pos[0], L->pos[1], L->pos[2], cut2);
  dst[1] = make_float4(c.x, c.y, c.z, bw);
  dst[2] = make_float4(radius, __fdividef(1.0f, radius), L->diffuse,
                       __uint_as_float((L->shadow ? 1u : 0u) | (L->is_static ? 2u : 0u)));
}

// kernel3 (cl2.cl:5792-6408) for one pixel of a view.
// ENABLE_NORMAL_MAPPING (cl2.cl:5987-6027): the tangent-space normal from the
// object's normal map, in object space through the triangle's tangent frame,
// then rotated into world space.  It feeds the shadow bias, so it keeps the
// IEEE contract (normalize as fast_normalize).
// dp1 = p2 - p1 and dp2 = p3 - p1 are the barycentric frame's edges.
__device__ __forceinline__ f3 normal_map(const SceneDev& sc, f2 vt, f2 vtdiff, uint32_t rid, f3 dp1, f3 dp2,
                                      f2 vt1, f2 vt2, f2 vt3, f3 model_normal, f4 qn) {
  const f4 t4 = texture_filter_diff<false>(sc, vt, vtdiff, (int)rid);
  f3 tn = mk3(2.0f * t4.x - 1.0f, 2.0f * t4.y - 1.0f, 2.0f * t4.z - 1.0f);
  tn = fast_normalize3(tn);
  const f2 duv1 = mk2(vt2.x - vt1.x, vt2.y - vt1.y), duv2 = mk2(vt3.x - vt1.x, vt3.y - vt1.y);
  const float r = fdiv(1.0f, duv1.x * duv2.y - duv1.y * duv2.x);
  f3 tangent = mk3((dp1.x * duv2.y - dp2.x * duv1.y) * r, (dp1.y * duv2.y - dp2.y * duv1.y) * r,
                   (dp1.z * duv2.y - dp2.z * duv1.y) * r);
  f3 bitangent = mk3((dp2.x * duv1.x - dp1.x * duv2.x) * r, (dp2.y * duv1.x - dp1.y * duv2.x) * r,
                     (dp2.z * duv1.x - dp1.z * duv2.x) * r);
  tangent = fast_normalize3(tangent);
  bitangent = fast_normalize3(bitangent);
  tangent = fast_normalize3(sub3(tangent, mul3s(model_normal, dot3(model_normal, tangent))));
  if (dot3(cross3(model_normal, tangent), bitangent) < 0.0f) tangent = mul3s(tangent, -1.0f);
  const f3 ms = mk3((tangent.x * tn.x + bitangent.x * tn.y) + model_normal.x * tn.z,
                    (tangent.y * tn.x + bitangent.y * tn.y) + model_normal.y * tn.z,
                    (tangent.z * tn.x + bitangent.z * tn.y) + model_normal.z * tn.z);
  return rot_quat_n(ms, qn);
}

// generate_outline (cl2.cl:2315-2362): the largest depth step to the four
// neighbours, over 100, at most 1.
__device__ __forceinline__ float generate_outline(int x, int y, const uint32_t* depth, int W, int H) {
  const float d0 = depth_to_dist(__ldca(depth + (size_t)y * W + x));
  float furthest = d0;
  for (int xx = -1; xx <= 1; xx++) {
    const int px = x + xx;
    if (px < 0 || px >= W) continue;
    const float nd = depth_to_dist(__ldca(depth + (size_t)y * W + px));
    if (nd > furthest) furthest = nd;
  }
  for (int yy = -1; yy <= 1; yy++) {
    const int py = y + yy;
    if (py < 0 || py >= H) continue;
    const uint32_t d = __ldca(depth + (size_t)py * W + x);
    const float nd = depth_to_dist(d);
    if (fabsf(nd - d0) > fabsf(furthest - d0) && nd > kDepthCutoff && d != 0) furthest = nd;
  }
  return fmin_(fdiv(fabsf(furthest - d0), 100.0f), 1.0f);
}

// One RGBA8 texel of the blend source as read_imagef returns it (c / 255).
__device__ __forceinline__ f4 blend_texel(const uint8_t* __restrict__ rgba, size_t p) {
  const uchar4 t = reinterpret_cast<const uchar4*>(rgba)[p];
  f4 o;
  o.x = u8_over_255(t.x); o.y = u8_over_255(t.y);  // fdiv(t, 255.0f)
  o.z = u8_over_255(t.z); o.w = u8_over_255(t.w);
  return o;
}

// kernel3's output for a pixel with nothing to shade (depth d): the clear
// colour and zero normals.  FEAT: kernel3's optional switches (view flags)
// compiled in.
template <bool FEAT>
__device__ __forceinline__ void shade_clear(const ViewParams& V, size_t p, uint32_t d) {
  uint32_t* out = reinterpret_cast<uint32_t*>(V.rgba);
  if (out) {
    f4 c;
    c.x = V.clear[0]; c.y = V.clear[1]; c.z = V.clear[2]; c.w = V.clear[3];
    // CAN_INTEGRATED_BLEND (cl2.cl:5839-5851): the other context's colour
    // over the clear colour where it has depth; its .xyzz swizzle gives
    // alpha = blue
    if (FEAT && V.blend_depth && V.blend_depth[p] < d) {
      const f4 o = blend_texel(V.blend_rgba, p);
      c.x = fma_(o.x, o.w, c.x * (1.0f - o.w));
      c.y = fma_(o.y, o.w, c.y * (1.0f - o.w));
      c.z = fma_(o.z, o.w, c.z * (1.0f - o.w));
      c.w = c.z;
    }
    out[p] = pack_rgba(c.x, c.y, c.z, c.w);
  }
  if (V.normals) reinterpret_cast<uint32_t*>(V.normals)[p] = 0;
}

// kernel3 for a covered pixel: depth d, record r (< the pass's record count).
// colx[i] = ((float)(x0 + i) - W/2) / fov and rowy[j] likewise for the tile's
// 17 columns and rows: the per-column / per-row divisions of get_vtdiff.
template <bool FEAT>
__device__ void shade_covered(const SceneDev& sc, const ViewParams& V, const Surface& S,
                              const ShadeRec* __restrict__ srec, const float4* __restrict__ lights, int x, int y,
                              uint32_t d, uint32_t r, const float* __restrict__ colx,
                              const float* __restrict__ rowy) {
  const int W = S.width, H = S.height;
  const size_t p = (size_t)y * W + x;
  uint32_t* out = reinterpret_cast<uint32_t*>(V.rgba);
  const float fov = V.fov;
  const f3 cpos = mk3(V.cpos[0], V.cpos[1], V.cpos[2]);
  const f3 cc = mk3(V.ccos[0], V.ccos[1], V.ccos[2]);
  const f3 cs = mk3(V.csin[0], V.csin[1], V.csin[2]);
  // the triangle's shade constants (prep_shade) and its object's terms
  const ShadeRec* R = srec + r;
  BaryFrame bf;
  {
    const float4 fa = __ldg(&R->a), f0 = __ldg(&R->e0), f1 = __ldg(&R->e1), fp = __ldg(&R->plane);
    bf.a = mk3(fa.x, fa.y, fa.z);
    bf.v0 = mk3(f0.x, f0.y, f0.z);
    bf.v1 = mk3(f1.x, f1.y, f1.z);
    bf.d00 = fa.w; bf.d01 = f0.w; bf.d11 = f1.w; bf.denom = fp.w;
  }
  const float4 fn1 = __ldg(&R->n1), fn2 = __ldg(&R->n2), fn3 = __ldg(&R->n3), ft = __ldg(&R->t);
  const f2 vt1 = mk2(fn1.w, fn2.w), vt2 = mk2(fn3.w, ft.x), vt3 = mk2(ft.y, ft.z);
  const uint32_t obits = __float_as_uint(ft.w);
  const uint32_t o_id = obits & 0x7FFFFFFFu;
  const float4* OQ = sc.objq + (size_t)o_id * kObjQuads;
  const float4 oq0 = __ldg(OQ), oq1 = __ldg(OQ + 1), oq2 = __ldg(OQ + 2), oq3 = __ldg(OQ + 3);
  f4 qn, qi;  // rot_quat's and back_rot_quat's normalised quaternions
  qn.x = oq0.x; qn.y = oq0.y; qn.z = oq0.z; qn.w = oq0.w;
  qi.x = oq1.x; qi.y = oq1.y; qi.z = oq1.z; qi.w = oq1.w;
  const f3 wpos = mk3(oq2.x, oq2.y, oq2.z);

  const float ldepth = depth_to_dist(d);
  const float fx = (float)x, fy = (float)y;
  f3 local = mk3(fdiv((fx - (float)W / 2.0f) * ldepth, fov), fdiv((fy - (float)H / 2.0f) * ldepth, fov),
                 ldepth);
  const f3 zero = mk3(0, 0, 0);
  const f3 gpos = add3(back_rot_cs(local, zero, cc, cs), cpos);
  f3 olocal = rot_quat_n(sub3(gpos, wpos), qi);
  float l1, l2, l3;
  bary_exact(bf, olocal, &l1, &l2, &l3);
  f2 vt = mk2(fma_(vt1.x, l1, fma_(vt2.x, l2, vt3.x * l3)), fma_(vt1.y, l1, fma_(vt2.y, l2, vt3.y * l3)));
  f3 normal = mk3(fma_(fn1.x, l1, fma_(fn2.x, l2, fn3.x * l3)), fma_(fn1.y, l1, fma_(fn2.y, l2, fn3.y * l3)),
                  fma_(fn1.z, l1, fma_(fn2.z, l2, fn3.z * l3)));
  const f3 model_normal = normal;
  normal = rot_quat_n(normal, qn);

  f4 col;
  const float4 fcol = __ldg(&R->col);
  const uint32_t vc0 = __float_as_uint(fcol.x);
  // normal map of the object (ENABLE_NORMAL_MAPPING), 0xFFFFFFFF if none
  const uint32_t rid = (FEAT && (V.flags & GBR_VIEW_NORMAL_MAPPING)) ? __ldg(&sc.descs[o_id].rid) : 0xFFFFFFFFu;
  f2 vtdiff = mk2(0.0f, 0.0f);
  if (vc0 == 0 || rid != 0xFFFFFFFFu) {
    // get_vtdiff (cl2.cl:5691-5760), its 1/z plane from the shade constants.
    // The plane extrapolated to the neighbouring pixels is ill-conditioned
    // for triangles seen edge-on (it can cross zero), so this stays in IEEE
    // arithmetic: rounding differences there would pick other mip levels.
    const float4 fp = __ldg(&R->plane);
    float dmx = fma_(fp.x, fx + 1.0f, fma_(fp.y, fy, fp.z));
    float dmy = fma_(fp.x, fx, fma_(fp.y, fy + 1.0f, fp.z));
    const int lx = x & (kTile - 1), ly = y & (kTile - 1);
    f3 lmx = mk3(colx[lx + 1], rowy[ly], 1.0f);  // fdiv((fx + 1) - hw, fov), fdiv(fy - hh, fov)
    f3 lmy = mk3(colx[lx], rowy[ly + 1], 1.0f);  // fdiv(fx - hw, fov), fdiv((fy + 1) - hh, fov)
    lmx = mk3(fdiv(lmx.x, dmx), fdiv(lmx.y, dmx), fdiv(lmx.z, dmx));
    lmy = mk3(fdiv(lmy.x, dmy), fdiv(lmy.y, dmy), fdiv(lmy.z, dmy));
    f3 gmx = rot_quat_n(sub3(add3(back_rot_cs(lmx, zero, cc, cs), cpos), wpos), qi);
    f3 gmy = rot_quat_n(sub3(add3(back_rot_cs(lmy, zero, cc, cs), cpos), wpos), qi);
    float lx1, lx2, lx3, ly1, ly2, ly3;
    bary_exact(bf, gmx, &lx1, &lx2, &lx3);
    bary_exact(bf, gmy, &ly1, &ly2, &ly3);
    f2 vtx = mk2(fma_(vt1.x, lx1, fma_(vt2.x, lx2, vt3.x * lx3)), fma_(vt1.y, lx1, fma_(vt2.y, lx2, vt3.y * lx3)));
    f2 vty = mk2(fma_(vt1.x, ly1, fma_(vt2.x, ly2, vt3.x * ly3)), fma_(vt1.y, ly1, fma_(vt2.y, ly2, vt3.y * ly3)));
    const float mip_bias = 1.0f / kMipBias;
    vtdiff = mk2((fabsf(vtx.x - vt.x) + fabsf(vty.x - vt.x)) * mip_bias,
                 (fabsf(vtx.y - vt.y) + fabsf(vty.y - vt.y)) * mip_bias);
  }
  // (the reference replaces the normal after its colour and jitter seeds,
  // neither of which reads it)
  if (FEAT && rid != 0xFFFFFFFFu)
    normal = normal_map(sc, vt, vtdiff, rid, bf.v0, bf.v1, vt1, vt2, vt3, model_normal, qn);
  if (vc0 != 0) {
    f4 c0 = vertex_col(vc0), c1 = vertex_col(__float_as_uint(fcol.y)), c2 = vertex_col(__float_as_uint(fcol.z));
    col.x = fma_(c0.x, l1, fma_(c1.x, l2, c2.x * l3));
    col.y = fma_(c0.y, l1, fma_(c1.y, l2, c2.y * l3));
    col.z = fma_(c0.z, l1, fma_(c1.z, l2, c2.z * l3));
    col.w = fma_(c0.w, l1, fma_(c1.w, l2, c2.w * l3));
  } else {
    col = texture_filter_diff<true>(sc, vt, vtdiff, (int)__float_as_uint(oq3.w));
  }
  if (V.use_linear) {
    col.x = c_gamma_fwd(col.x);
    col.y = c_gamma_fwd(col.y);
    col.z = c_gamma_fwd(col.z);
  }
  uint32_t seed2 = rand_xorshift(wang_hash((uint32_t)x + (uint32_t)y * (uint32_t)W * (uint32_t)H));
  uint32_t seed3 = rand_xorshift(seed2);
  uint32_t seed4 = rand_xorshift(seed3);
  f3 rseed = mk3(((float)seed2 * kInvMulInt - 0.5f) * 2.0f, ((float)seed3 * kInvMulInt - 0.5f) * 2.0f,
                 ((float)seed4 * kInvMulInt - 0.5f) * 2.0f);
  const f3 l2p = cnormalize(sub3(cpos, gpos));
  const int ff = (int)__float_as_uint(oq3.z);
  const bool two = (ff & kFlagTwoSided) > 0;
  const bool recv_dyn = !((ff & kFlagNoDynShadows) > 0);
  if ((obits >> 31) && two) normal = neg3(normal);  // back-facing (cl2.cl:491-494)
  const float ssao = generate_ssao(x, y, seed2, d, S.depth, W, H, fov);
  normal = fast_normalize3(normal);
  const f3 lnormal = cnormalize(add3(normal, mk3(rseed.x * 0.01f, rseed.y * 0.01f, rseed.z * 0.01f)));
  const float ambient = V.use_linear ? gamma_fwd(kAmbient) : kAmbient;
  const float g_diffuse = oq2.w, g_spec_mult = oq3.x;
  const float rough = oq3.y;  // clamp(1 - specular, 0.001, 10)
  // per-pixel factors of the light loop (colour only)
  const float ndv_raw = cdot3(normal, l2p);
  const float ndv = fmax_(0.0f, ndv_raw);
  const float r_pndv = crcp(kPi * ndv);  // spec / (pi ndv)
  const float nr2 = -crcp(rough * rough);  // Gaussian exponent -alpha^2 / rough^2
  const float spec_k = 0.4f * g_spec_mult;
  const float amb1 = 1.0f - ambient;
  f3 dsum = mk3(0, 0, 0), ssum = mk3(0, 0, 0);
  int shnum = 0, static_num = 0;
  for (uint32_t i = 0; i < sc.nlights; i++) {
    const float4 LA = lights[kLightQuads * i];
    const f3 lpos = mk3(LA.x, LA.y, LA.z);
    f3 ptl = sub3(lpos, gpos);
    // The distance only feeds the colour, except through the cutoff below,
    // which for a shadow light also decides which cubemap later shadow lights
    // read (shnum): IEEE arithmetic for shadow lights (a warp-uniform branch),
    // approximate otherwise, after the conservative early test (whose margins
    // cover the contracted dot product).
    const float d2 = cdot3(ptl, ptl);
    if (d2 > LA.w) continue;
    const float4 LB = lights[kLightQuads * i + 1], LC = lights[kLightQuads * i + 2];
    const uint32_t lflags = __float_as_uint(LC.w);
    const f3 lcol = mk3(LB.x, LB.y, LB.z);
    const float rinv = rsqrt_ftz(d2);
    if (lflags & 1u) {  // a shadow light: its distance in IEEE arithmetic
      const float d2s = dot3(ptl, ptl);
      float occlusion = 1.0f;
      if (lflags & 2u) {  // is_static
        int face = ret_cubeface(gpos, lpos);
        occlusion = 1.0f - hard_occlusion(sc, lpos, normal, ptl, rinv, sc.shadow_static, face, gpos, static_num);
        static_num++;
      }
      const float tt = fdiv(fsqrt(d2s), LC.x) + 1.0f;
      float illum = fdiv(LB.w, tt * tt);
      illum -= kLightCutoff;
      illum *= 1.0f / (1.0f - kLightCutoff);
      if (illum <= 0) continue;
      if (recv_dyn) {
        int face = ret_cubeface(gpos, lpos);
        float dyn = 1.0f - hard_occlusion(sc, lpos, normal, ptl, rinv, sc.shadow_dyn, face, gpos, shnum);
        occlusion = fmin_(occlusion, dyn);
        shnum++;
      }
      ptl = mul3s(ptl, rinv);  // cnormalize(ptl), the dot contracted (colour only)
      // Lambert + ambient
      const float light = fmax_(cdot3(ptl, lnormal) * occlusion, 0.0f);
      const float dscale = fma_(amb1, light, ambient) * ((LC.z * g_diffuse) * illum);
      dsum = mk3(fma_(lcol.x, dscale, dsum.x), fma_(lcol.y, dscale, dsum.y), fma_(lcol.z, dscale, dsum.z));
      // Cook-Torrance: F0 0.4, Gaussian microfacet 0.8346, geometric term
      const f3 Hv = cnormalize(add3(l2p, ptl));
      const float ndh = fmax_(0.0f, cdot3(normal, Hv));
      const float vdh = fmax_(0.0f, cdot3(l2p, Hv));
      const float ndl = fmax_(0.0f, cdot3(normal, ptl));
      const float omv = 1.0f - vdh, omv2 = omv * omv;
      const float fresnel = fma_(0.6f, (omv2 * omv2) * omv, 0.4f);
      const float alpha = c_rational_acos(ndh);
      const float microfacet = 0.8346f * ex2_ftz(((alpha * alpha) * nr2) * 1.4426950408889634f);
      const float sv = (2.0f * ndh) * crcp(vdh);
      const float geometric = min3f(1.0f, sv * ndv, sv * ndl);
      const float spec = ((fresnel * microfacet) * geometric) * r_pndv;
      const float sscale = spec * (spec_k * illum);
      ssum = mk3(fmax_(fma_(lcol.x, sscale, ssum.x), 0.0f) * occlusion,
                 fmax_(fma_(lcol.y, sscale, ssum.y), 0.0f) * occlusion,
                 fmax_(fma_(lcol.z, sscale, ssum.z), 0.0f) * occlusion);
      continue;
    }
    // a light without shadows: its occlusion is 1
    // the approximate square root: 2^63 is the reciprocal root of the smallest
    // normal float, so the minimum only matters at 0 (and at subnormals), where
    // rinv is infinite; infinite and NaN squares give NaN
    const float distance = d2 * fmin_(rinv, 0x1p63f);
    const float tt = fma_(distance, LC.y, 1.0f);
    const float illum = fma_(LB.w, crcp(tt * tt), -kLightCutoff / (1.0f - kLightCutoff));
    // (turned into 0 by a select instead: 1080p frame 395 us against 391, and a
    // NaN specular term of a dark light cleared the sum of the others)
    if (illum <= 0.0f) continue;
    ptl = mul3s(ptl, rinv);
    const float light = fmax_(cdot3(ptl, lnormal), 0.0f);
    const float dscale = fma_(amb1, light, ambient) * ((LC.z * g_diffuse) * illum);
    dsum = mk3(fma_(lcol.x, dscale, dsum.x), fma_(lcol.y, dscale, dsum.y), fma_(lcol.z, dscale, dsum.z));
    // the half vector H = (v + l) / |v + l| of the unit vectors v (l2p) and l
    // (ptl) through dot products: |v + l|^2 = 2 + 2 v.l, n.H = (n.v + n.l) /
    // |v + l|, v.H = (1 + v.l) / |v + l|
    const float nl = cdot3(normal, ptl), vl = cdot3(l2p, ptl);
    const float rh = rsqrt_ftz(fma_(2.0f, vl, 2.0f));
    const float vdh = fmax_(0.0f, (1.0f + vl) * rh);
    const float ndh = fmax_(0.0f, (ndv_raw + nl) * rh);
    const float ndl = fmax_(0.0f, nl);
    const float alpha = c_rational_acos(ndh);
    const float ex = ((alpha * alpha) * nr2) * 1.4426950408889634f;
    const float microfacet = 0.8346f * ex2_ftz(ex);
    const float omv = 1.0f - vdh, omv2 = omv * omv;
    const float fresnel = fma_(0.6f, (omv2 * omv2) * omv, 0.4f);
    const float sv = (2.0f * ndh) * crcp(vdh);
    const float geometric = min3f(1.0f, sv * ndv, sv * ndl);
    const float spec = ((fresnel * microfacet) * geometric) * r_pndv;
    const float sscale = spec * (spec_k * illum);
    ssum = mk3(fmax_(fma_(lcol.x, sscale, ssum.x), 0.0f), fmax_(fma_(lcol.y, sscale, ssum.y), 0.0f),
               fmax_(fma_(lcol.z, sscale, ssum.z), 0.0f));
  }
  ssum = mul3s(ssum, ssao);
  dsum = mul3s(dsum, ssao);
  const float rsc = 0.7f;
  f3 colclamp = add3(add3(mk3(col.x, col.y, col.z), zero), mul3s(ssum, rsc));
  f3 sp2 = mul3s(ssum, 1.0f - rsc);
  f3 fin = mk3(fma_(colclamp.x, dsum.x, sp2.x), fma_(colclamp.y, dsum.y, sp2.y), fma_(colclamp.z, dsum.z, sp2.z));
  // CAN_INTEGRATED_BLEND (cl2.cl:6339-6351): alpha_blend of the other
  // context's colour where it is nearer, before the output gamma
  if (FEAT && V.blend_depth && V.blend_depth[p] < d) {
    const f4 o = blend_texel(V.blend_rgba, p);
    fin = mk3(fma_(o.x, o.w, fin.x * (1.0f - o.w)), fma_(o.y, o.w, fin.y * (1.0f - o.w)),
              fma_(o.z, o.w, fin.z * (1.0f - o.w)));
  }
  if (V.use_linear) fin = mk3(c_gamma_inv(fin.x), c_gamma_inv(fin.y), c_gamma_inv(fin.z));
  if (FEAT && (V.flags & GBR_VIEW_OUTLINE) && (ff & kFlagOutline) > 0) {
    const float o = generate_outline(x, y, S.depth, W, H);
    fin = mk3(fin.x + o, fin.y + o, fin.z + o);
  }
  if (out) out[p] = pack_rgba(fin.x, fin.y, fin.z, col.w);
  if (V.normals) {
    // encode_normal (cl2.cl:5618-5628)
    float nx = normal.x, ny = normal.y, nz = normal.z;
    if (nx * nx + ny * ny < 0.0001f) nx = 0.01f;
    float l = fsqrt(nx * nx + ny * ny);
    float sq = fsqrt(fmax_(nz * 0.5f + 0.5f, 0.0f));
    // (v / 2 = v * 0.5 exactly: both are the correctly rounded v / 2)
    float ex = ((fdiv(nx, l) * sq + 1.0f) * 0.5f) * 65536.0f - 1.0f;
    float ey = ((fdiv(ny, l) * sq + 1.0f) * 0.5f) * 65536.0f - 1.0f;
    uint32_t ux = min(f2u_sat(ex), 65535u), uy = min(f2u_sat(ey), 65535u);
    reinterpret_cast<uint32_t*>(V.normals)[p] = ux | (uy << 16);
  }
}

// kernel3 for one pixel.  nrec: the records this pass wrote; the raster
// stores only indices below it in the record map, and any other value is
// treated as an empty pixel, so no index read from the map can leave the
// record arrays.
template <bool FEAT>
__device__ __forceinline__ void shade_pixel(const SceneDev& sc, const ViewParams& V, const Surface& S,
                                            const ShadeRec* __restrict__ srec, uint32_t nrec,
                                            const float4* __restrict__ lights, int x, int y,
                                            const float* __restrict__ colx, const float* __restrict__ rowy) {
  const size_t p = (size_t)y * S.width + x;
  const uint32_t d = S.depth[p];
  const uint32_t r = S.rec[p];
  if (d == kDepthClear || r >= nrec)
    shade_clear<FEAT>(V, p, d);
  else
    shade_covered<FEAT>(sc, V, S, srec, lights, x, y, d, r, colx, rowy);
}

// Shared memory of one tile's shading.
struct ShadeSmem {
  float4 lights[kMaxLights * kLightQuads];
  float colx[kTile + 1], rowy[kTile + 1];
};

// kernel3 over one 16x16 tile of view surface `sid` (NT threads, 256 / NT
// pixels each).  Every thread of the block calls it; the caller synchronises
// before reusing the shared memory.
template <bool FEAT, int NT>
__device__ __forceinline__ void shade_tile(const SceneDev& sc, const ViewParams* __restrict__ views,
                                           const Surface* __restrict__ surfs, const ShadeRec* __restrict__ srec,
                                           uint32_t nrec, uint32_t tile, uint32_t sid, ShadeSmem& sm) {
  const Surface& S = surfs[sid];
  const ViewParams& V = views[sid];
  const uint32_t lt = tile - S.tile_base;
  const int x0 = (lt % S.tiles_x) * kTile, y0 = (lt / S.tiles_x) * kTile;
  const bool linear = V.use_linear != 0;
  for (uint32_t i = threadIdx.x; i < sc.nlights; i += NT) stage_light(sc.lights + i, linear, sm.lights + kLightQuads * i);
  if (threadIdx.x < 2 * (kTile + 1)) {
    const int i = threadIdx.x % (kTile + 1);
    if (threadIdx.x <= kTile)
      sm.colx[i] = fdiv((float)(x0 + i) - (float)S.width / 2.0f, V.fov);
    else
      sm.rowy[i] = fdiv((float)(y0 + i) - (float)S.height / 2.0f, V.fov);
  }
  __syncthreads();
  if (NT == kTilePixels) {  // one pixel per thread
    const int x = x0 + (threadIdx.x & (kTile - 1)), y = y0 + threadIdx.x / kTile;
    if (x < S.width && y < S.height) shade_pixel<FEAT>(sc, V, S, srec, nrec, sm.lights, x, y, sm.colx, sm.rowy);
    return;
  }
#pragma unroll 1
  for (int lp = threadIdx.x; lp < kTilePixels; lp += NT) {
    const int x = x0 + (lp & (kTile - 1)), y = y0 + lp / kTile;
    if (x < S.width && y < S.height) shade_pixel<FEAT>(sc, V, S, srec, nrec, sm.lights, x, y, sm.colx, sm.rowy);
  }
}

// kernel3 over the tiles of a pass, one 256-thread CTA per 16x16 tile.
// tile_empty (or null): tiles whose output the raster wrote, which return at
// once; tiles (null for one view): each tile's surface (Workspace).  Each
// thread reads its pixel; empty pixels get the clear colour, covered ones are
// compacted in pixel order into the first threads, which shade them.
// ONE: a pass of one view whose parameters come with the launch (one_view,
// one_surf: constant-bank operands instead of loads that hold registers);
// otherwise they are read from views / surfs.
//
// A pass whose setup or binning overflowed its scratch leaves the depth and
// record map unwritten (the raster returns at once); shading returns too, and
// the host re-runs the pass with grown scratch.
//
// Bound by instruction issue (79 % active; 73 % in batches).  1080p terrain:
// 2,690 instructions per pixel (3,350 before the approximations as single
// instructions, the SSAO counts without compares, packed texel blends, integer
// texel coordinates and the view in the constant bank), 182 us (223); 64 sphere
// views 1.79 ms (2.24).  The lights' shared memory is sized by the scene: with
// room for kMaxLights the L1 lost 3 points of its hit rate (1.4 % of the batch's
// time).  Tiles of 128 or 64 pixels per block were slower (203 / 212 us): their
// blocks share less in the L1 and start more often.
template <bool FEAT, bool ONE>
__global__ void __launch_bounds__(kTilePixels, 4) k_shade(SceneDev sc,
                                               const __grid_constant__ ViewParams one_view,
                                               const __grid_constant__ Surface one_surf,
                                               const ViewParams* __restrict__ views,
                                               const Surface* __restrict__ surfs, const ShadeRec* __restrict__ srec,
                                               const Counters* __restrict__ ctr,
                                               uint32_t rec_cap, uint32_t tile0,
                                               const uint8_t* __restrict__ tile_empty,
                                               const uint2* __restrict__ tiles, Counters* __restrict__ host_ctr) {
  constexpr int NW = kTilePixels / 32;
  extern __shared__ float4 s_lights[];  // kLightQuads per light of the scene
  __shared__ float s_colx[kTile + 1], s_rowy[kTile + 1];
  __shared__ uint32_t s_warp[NW];
  __shared__ uint32_t s_px[kTilePixels], s_d[kTilePixels], s_r[kTilePixels];
  // (the counters are final: a copy in mapped host memory saves the pass a
  // transfer at its end)
  if (ONE && host_ctr && blockIdx.x == 0 && threadIdx.x < sizeof(Counters) / 4)
    reinterpret_cast<uint32_t*>(host_ctr)[threadIdx.x] = reinterpret_cast<const uint32_t*>(ctr)[threadIdx.x];
  if (ctr->overflow) return;
  const uint32_t nrec = min(ctr->nrec, rec_cap);
  const uint32_t tile = tile0 + blockIdx.x;
  // every thread reads the tile's flag and surface (the same words): the
  // return is block-uniform and needs no barrier
  if (tile_empty && tile_empty[tile]) return;
  const uint32_t sid = !ONE && tiles ? tiles[tile].x : 0u;  // null: one view
  const Surface& S = ONE ? one_surf : surfs[sid];
  const ViewParams& V = ONE ? one_view : views[sid];
  const uint32_t lt = tile - S.tile_base;
  const int x0 = (lt % S.tiles_x) * kTile, y0 = (lt / S.tiles_x) * kTile;
  // the thread's own pixel: empty pixels are written at once; covered ones
  // are compacted (in pixel order) so that whole warps shade them
  const int lp = threadIdx.x, lane = lp & 31, warp = lp >> 5;
  const int x = x0 + (lp & (kTile - 1)), y = y0 + lp / kTile;
  const bool inside = x < S.width && y < S.height;
  const size_t p = (size_t)y * S.width + x;
  uint32_t d = kDepthClear, r = kNoId;
  if (inside) {
    d = S.depth[p];
    r = S.rec[p];
  }
  const bool cov = inside && d != kDepthClear && r < nrec;
  const unsigned m = __ballot_sync(0xFFFFFFFFu, cov);
  if (lane == 0) s_warp[warp] = __popc(m);
  if (inside && !cov) shade_clear<FEAT>(V, p, d);
  const bool linear = V.use_linear != 0;
  for (uint32_t i = threadIdx.x; i < sc.nlights; i += kTilePixels)
    stage_light(sc.lights + i, linear, s_lights + kLightQuads * i);
  if (threadIdx.x < 2 * (kTile + 1)) {
    const int i = threadIdx.x % (kTile + 1);
    if (threadIdx.x <= kTile)
      s_colx[i] = fdiv((float)(x0 + i) - (float)S.width / 2.0f, V.fov);
    else
      s_rowy[i] = fdiv((float)(y0 + i) - (float)S.height / 2.0f, V.fov);
  }
  __syncthreads();
  const uint32_t wc = lane < NW ? s_warp[lane] : 0u;
  const uint32_t base = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? wc : 0u);
  const uint32_t total = __reduce_add_sync(0xFFFFFFFFu, wc);
  if (cov) {
    const uint32_t k = base + __popc(m & ((1u << lane) - 1u));
    s_px[k] = (uint32_t)lp;
    s_d[k] = d;
    s_r[k] = r;
  }
  __syncthreads();
  if (threadIdx.x < total) {
    const uint32_t q = s_px[threadIdx.x];
    shade_covered<FEAT>(sc, V, S, srec, s_lights, x0 + (int)(q & (kTile - 1)), y0 + (int)(q / kTile),
                        s_d[threadIdx.x], s_r[threadIdx.x], s_colx, s_rowy);
  }
}

// ---- the fused raster -> shade pass of many views ------------------------------
// One persistent, cooperative launch (every block resident) takes the pass's
// tiles from a work queue: each view's raster tiles (kernel1 + kernel2), and
// each view's shade tiles (kernel3), which the host orders after at least a
// grid's worth of later views' raster tiles.  kernel3's SSAO reads depth
// anywhere in its view (its tap offsets grow as the depth shrinks), so a
// shade tile waits until every raster tile of its view is done: a per-view
// counter, polled with a bounded wait.  Every item depends only on items
// taken before it, so the waits always end; a wait that reaches its limit
// anyway sets bit 2 of the pass's overflow word and leaves that tile
// unshaded (the host reports GBR_DEVICE_TIMEOUT).  One view's shading thus
// overlaps later views' rasters: the raster waits on block barriers, the
// shading is bound by instruction issue.
//
// queue: [0] next item, [1] unused, [2 + v] raster tiles done of view v
// (zeroed by the host before the launch).  sched: seg_start[nseg + 1] (first
// item of each segment; seg_start[nseg] = item count), then seg_view[nseg]
// (view | 1 << 31 for shade segments).
constexpr uint32_t kWaitPolls = 1u << 22;  // with ~0.25 us sleeps: about a second

__device__ __forceinline__ uint32_t ld_acquire_gpu(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

template <int NT, bool FEAT>
__global__ void __launch_bounds__(NT, 1024 / NT) k_raster_shade(Workspace ws, const Surface* __restrict__ surfs,
                                                                uint32_t nsurf, SceneDev sc,
                                                                const ViewParams* __restrict__ views,
                                                                const uint32_t* __restrict__ sched, uint32_t nseg,
                                                                uint32_t* __restrict__ queue) {
  union Smem {
    RasterSmem<NT, true, kFusedHits> r;
    ShadeSmem s;
  };
  __shared__ Smem sm;
  __shared__ uint32_t s_item[2];
  __shared__ int s_ok;
  if (ws.ctr->overflow) return;
  const uint32_t nrec = min(ws.ctr->nrec, ws.rec_cap);
  const uint32_t total = __ldg(sched + nseg);
  if (threadIdx.x == 0) s_item[0] = atomicAdd(&queue[0], 1u);
  __syncthreads();
#pragma unroll 1
  for (int cur = 0;; cur ^= 1) {
    const uint32_t item = s_item[cur];
    if (item >= total) break;
    if (threadIdx.x == 0) s_item[cur ^ 1] = atomicAdd(&queue[0], 1u);  // the next item, taken early
    int seg = 0, hi = (int)nseg - 1;
    while (seg < hi) {
      const int mid = (seg + hi + 1) >> 1;
      if (__ldg(sched + mid) <= item) seg = mid; else hi = mid - 1;
    }
    const uint32_t info = __ldg(sched + nseg + 1 + seg);
    const uint32_t v = info & 0x7FFFFFFFu;
    const uint32_t tile = surfs[v].tile_base + (item - __ldg(sched + seg));
    if (!(info >> 31)) {
      raster_tile<NT, true, false, false, kFusedHits>(ws, surfs, tile, (int)v, sm.r);
      __threadfence();  // this thread's depth / id / record-map writes, before the count
      __syncthreads();
      if (threadIdx.x == 0) atomicAdd(&queue[2 + v], 1u);
    } else {
      if (threadIdx.x == 0) {
        const uint32_t need = (uint32_t)(surfs[v].tiles_x * surfs[v].tiles_y);
        int ok = 1;
        for (uint32_t polls = 0; ld_acquire_gpu(&queue[2 + v]) < need; polls++) {
          if (polls >= kWaitPolls) {
            ok = 0;
            atomicOr(&ws.ctr->overflow, 4u);
            break;
          }
          __nanosleep(256);
        }
        s_ok = ok;
      }
      __syncthreads();
      if (s_ok) shade_tile<FEAT, NT>(sc, views, surfs, ws.srec, nrec, tile, v, sm.s);
    }
    __syncthreads();
  }
}

// ---- texture atlas ----------------------------------------------------------------
// Slot origin of texture descriptor tid as write_tex_array computes it
// (cl2.cl:856-889).
__device__ __forceinline__ void tex_slot(const uint32_t* nums, const uint32_t* sizes, uint32_t tid,
                                         float* tnx, float* tny, int* slice, float* width) {
  uint32_t nv = nums[tid];
  *slice = (int)(nv >> 16);
  int which = (int)(nv & 0xFFFF);
  *width = (float)sizes[*slice];
  float hnum = floorf(fdiv(2048.0f, *width));
  float tnumy = floorf(fdiv((float)which, hnum));
  *tny = tnumy;
  *tnx = fma_(-tnumy, hnum, (float)which);
}

__device__ __forceinline__ void write_tex(uchar4* atlas, const uint32_t* nums, const uint32_t* sizes,
                                          uint32_t tid, float cx, float cy, uchar4 c) {
  float tnx, tny, w;
  int slice;
  tex_slot(nums, sizes, tid, &tnx, &tny, &slice, &w);
  float tx = tnx * w, ty = tny * w;
  cx = clampf_(fmodf(cx, w), 0.001f, w - 0.001f);
  cy = clampf_(fmodf(cy, w), 0.001f, w - 0.001f);
  int ix = (int)(tx + cx), iy = (int)(ty + cy);
  atlas[(size_t)slice * kTexPage * kTexPage + (size_t)iy * kTexPage + ix] = c;
}

__device__ __forceinline__ float4 read_tex(const uchar4* atlas, const uint32_t* nums, const uint32_t* sizes,
                                           uint32_t tid, float cx, float cy) {
  float tnx, tny, w;
  int slice;
  tex_slot(nums, sizes, tid, &tnx, &tny, &slice, &w);
  cx = clampf_(cx, 0.001f, w - 0.001f);
  cy = clampf_(cy, 0.001f, w - 0.001f);
  int ix = f2i_sat(fma_(tnx, w, cx)), iy = f2i_sat(fma_(tny, w, cy));
  uchar4 t = atlas[(size_t)slice * kTexPage * kTexPage + (size_t)iy * kTexPage + ix];
  return make_float4(t.x, t.y, t.z, t.w);
}

// update_gpu_tex with flip (cl2.cl:923-953); blockIdx.z = texture.
__global__ void k_tex_upload(uchar4* atlas, const uint32_t* nums, const uint32_t* sizes, const uint8_t* pixels,
                             const uint64_t* offsets, const int32_t* tsizes) {
  const uint32_t t = blockIdx.z;
  const int s = tsizes[t];
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= s || y >= s) return;
  uchar4 c = reinterpret_cast<const uchar4*>(pixels + offsets[t])[(size_t)y * s + x];
  float w = (float)sizes[nums[t] >> 16];
  write_tex(atlas, nums, sizes, t, (float)x, w - (float)y, c);
}

// generate_mips / generate_mip_mips (cl2.cl:1070-1189): level src -> src+1
// for every texture (blockIdx.z), grid over the base texture size.
__global__ void k_mip(uchar4* atlas, const uint32_t* nums, const uint32_t* sizes, uint32_t mipmap_start,
                      const int32_t* tsizes, int level) {
  const uint32_t t = blockIdx.z;
  const int s = tsizes[t];
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= s || y >= s) return;
  uint32_t src = level == 0 ? t : t * kMipLevels + mipmap_start + (uint32_t)(level - 1);
  uint32_t dst = t * kMipLevels + mipmap_start + (uint32_t)level;
  float w = (float)sizes[nums[src] >> 16];
  if ((float)x >= w || (float)y >= w) return;
  const float g[3] = {1.f, 2.f, 1.f};
  float a0 = 0, a1 = 0, a2 = 0, a3 = 0, div = 0;
  for (int j = -1; j <= 1; j++)
    for (int i = -1; i <= 1; i++) {
      float4 c = read_tex(atlas, nums, sizes, src, (float)(x * 2 + i), (float)(y * 2 + j));
      c.w = fdiv(c.w, 255.f);
      c.x *= c.w; c.y *= c.w; c.z *= c.w;
      float gw = g[j + 1] * g[i + 1];
      a0 += c.x * gw; a1 += c.y * gw; a2 += c.z * gw; a3 += c.w * gw;
      div += gw;
    }
  a0 = fdiv(a0, div); a1 = fdiv(a1, div); a2 = fdiv(a2, div); a3 = fdiv(a3, div);
  if (a3 > 0.00000001f) { a0 = fdiv(a0, a3); a1 = fdiv(a1, a3); a2 = fdiv(a2, a3); }
  a3 *= 255.f;
  float nw = (float)sizes[nums[dst] >> 16];
  float yx0 = fdiv((float)(x * 2), w) * nw, yx1 = fdiv((float)(y * 2), w) * nw;
  if (yx0 >= nw || yx1 >= nw) return;
  uchar4 c = make_uchar4((unsigned char)f2u_sat(a0), (unsigned char)f2u_sat(a1), (unsigned char)f2u_sat(a2),
                         (unsigned char)f2u_sat(a3));
  write_tex(atlas, nums, sizes, dst, yx0, yx1, c);
}

// object::g_flush's writes (object.cpp:652-860): pose, scale, texture id and
// feature flags of the listed descriptors.
__global__ void k_flush_objects(gbr_obj_g_descriptor* descs, const gbr_object_flush* objs, uint32_t n) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const gbr_object_flush f = objs[i];
  gbr_obj_g_descriptor* G = descs + f.index;
  for (int k = 0; k < 4; k++) {
    G->world_pos[k] = f.world_pos[k];
    G->world_rot_quat[k] = f.world_rot_quat[k];
  }
  G->scale = f.scale;
  G->tid = f.tid;
  G->feature_flag = f.feature_flag;
}

// The first kernel of a depth-only pass: every surface to UINT_MAX before the
// setup rasterises small candidates into it (blockIdx.y = surface), and the
// pass's counters to 0 (the last grid row).
__global__ void __launch_bounds__(256) k_begin_faces(const Surface* __restrict__ surfs, uint32_t nsurf,
                                                     uint32_t* __restrict__ counts, uint32_t ncounts) {
  const size_t first = (size_t)blockIdx.x * blockDim.x + threadIdx.x, step = (size_t)gridDim.x * blockDim.x;
  if (blockIdx.y == nsurf) {
    for (size_t i = first; i < ncounts; i += step) counts[i] = 0;
    return;
  }
  const Surface& S = surfs[blockIdx.y];
  const size_t n = (size_t)S.width * S.height;
  uint4* d4 = reinterpret_cast<uint4*>(S.depth);
  const uint4 v = make_uint4(kDepthClear, kDepthClear, kDepthClear, kDepthClear);
  for (size_t i = first; i < n / 4; i += step) d4[i] = v;
  if (blockIdx.x == 0 && threadIdx.x < (n & 3)) S.depth[(n & ~(size_t)3) + threadIdx.x] = kDepthClear;
}

// Atomic-rate probe (diagnostics): every thread issues `iters` 32-bit
// atomicMin.  Shared mode: each lane its own word of the block's 256 (a lane
// XOR keeps a warp's 32 words distinct, in 32 banks).  Global mode: words
// spread over an L2-resident array of nwords.
__global__ void __launch_bounds__(256) k_atomic_rate(uint32_t* g, uint32_t nwords, int iters, int shared_mode) {
  __shared__ uint32_t s[256];
  s[threadIdx.x] = 0xFFFFFFFFu;
  __syncthreads();
  const uint32_t v = blockIdx.x * 256u + threadIdx.x;
  if (shared_mode) {
    for (int i = 0; i < iters; i++) atomicMin(&s[threadIdx.x ^ (uint32_t)(i & 31)], v - (uint32_t)i);
    __syncthreads();
    if (s[threadIdx.x] == 0x12345u) g[0] = 0;  // keeps the shared result live
  } else {
    const uint32_t base = v % nwords;
    for (int i = 0; i < iters; i++) atomicMin(g + (base + (uint32_t)i * 4099u) % nwords, v - (uint32_t)i);
  }
}

__global__ void k_fill_u32(uint32_t* p, uint32_t v, size_t n) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    p[i] = v;
}

int g_num_sms = 0;
int num_sms() {
  if (!g_num_sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
    if (g_num_sms <= 0) g_num_sms = 152;
  }
  return g_num_sms;
}

}  // namespace

cudaError_t launch_world(const SceneDev& sc, float4* world, float4* objq, uint32_t* objr, cudaStream_t st) {
  if (sc.ndescs) k_objects<<<(sc.ndescs + 255) / 256, 256, 0, st>>>(sc, objq);
  if (sc.ntris && world) {
    if (!objr) return cudaErrorInvalidValue;
    cudaError_t e = cudaMemsetAsync(objr, 0, sizeof(uint32_t) * sc.ndescs, st);
    if (e != cudaSuccess) return e;
    k_world<<<(sc.ntris + 255) / 256, 256, 0, st>>>(sc, world, objr);
  }
  return cudaGetLastError();
}

cudaError_t launch_begin_views(const SceneDev& sc, const ViewParams* one_view, const Surface* one_surf,
                               ViewParams* d_views, Surface* d_surf, uint32_t nviews, const uint32_t* objr,
                               const Workspace& ws, cudaStream_t st) {
  if (!nviews) return cudaErrorInvalidValue;
  const bool one = nviews == 1 && one_view && one_surf;
  uint32_t cull_blocks = 0;
  if (ws.vis && ws.vis_words) {
    if (!sc.objq || !objr) return cudaErrorInvalidValue;
    cull_blocks = (ws.vis_words * 32 + 255) / 256 * nviews;
  }
  const uint32_t clear_blocks = std::min<uint32_t>((ws.ncounts + 1023) / 1024, (uint32_t)num_sms() * 2);
  k_begin_views<<<cull_blocks + std::max<uint32_t>(clear_blocks, 1), 256, 0, st>>>(
      sc, one ? *one_view : ViewParams{}, one ? *one_surf : Surface{}, one, d_views, d_surf, nviews, objr,
      ws.vis_words, const_cast<uint32_t*>(ws.vis), cull_blocks, reinterpret_cast<uint32_t*>(ws.ctr), ws.ncounts);
  return cudaGetLastError();
}

cudaError_t launch_texture_levels(const uint32_t* nums, const uint32_t* sizes, uint32_t mipmap_start, float4* texlv,
                                  cudaStream_t st) {
  const uint32_t n = mipmap_start * kTexLevels;
  if (n) k_texture_levels<<<(n + 255) / 256, 256, 0, st>>>(nums, sizes, mipmap_start, texlv);
  return cudaGetLastError();
}

cudaError_t launch_setup_views(const SceneDev& sc, const ViewParams* d_views, uint32_t nviews,
                               const Surface* d_surf, const Workspace& ws, cudaStream_t st) {
  if (!sc.ntris || !nviews) return cudaSuccess;
  dim3 grid((sc.ntris + 255) / 256, nviews);
  k_setup_views<<<grid, 256, 0, st>>>(sc, d_views, d_surf, ws);
  return cudaGetLastError();
}

cudaError_t launch_setup_shadow(const SceneDev& sc, const ShadowJob* d_jobs, uint32_t njobs,
                                const Surface* d_surf, const Workspace& ws, cudaStream_t st) {
  if (!sc.ntris || !njobs) return cudaSuccess;
  dim3 grid((sc.ntris + 127) / 128, njobs);  // small blocks: lanes' direct rasters differ in length
  k_setup_shadow<<<grid, 128, 0, st>>>(sc, d_jobs, d_surf, ws);
  return cudaGetLastError();
}

cudaError_t launch_offsets(const Workspace& ws, const Surface* d_surf, uint32_t nsurf, uint32_t per_surface,
                           cudaStream_t st) {
  if ((ws.tiles || ws.list) && !nsurf) return cudaErrorInvalidValue;
  const uint32_t n = std::max(std::max(ws.nfine, ws.ncoarse), 1u);
  k_offsets<<<(n + 255) / 256, 256, 0, st>>>(ws, d_surf, nsurf, per_surface);
  return cudaGetLastError();
}

cudaError_t launch_prep(const SceneDev& sc, const Workspace& ws, cudaStream_t st) {
  if (!ws.srec) return cudaErrorInvalidValue;
  k_prep<<<num_sms() * 4, 256, 0, st>>>(sc, ws);
  return cudaGetLastError();
}

cudaError_t launch_fill(const Workspace& ws, const Surface* d_surf, cudaStream_t st) {
  k_fill<<<num_sms() * 8, 256, 0, st>>>(ws, d_surf);
  return cudaGetLastError();
}

cudaError_t launch_raster_faces(const Workspace& ws, const Surface* d_surf, uint32_t ntiles, int threads,
                                cudaStream_t st, uint32_t tiles_per_surface) {
  if (!ntiles) return cudaSuccess;
  if (!ws.list || !tiles_per_surface) return cudaErrorInvalidValue;
  const uint32_t blocks = std::min<uint32_t>(ntiles, (uint32_t)num_sms() * (1280 / threads));
  switch (threads) {
    case 128: k_raster_list<128><<<blocks, 128, 0, st>>>(ws, d_surf, tiles_per_surface); break;
    case 512: k_raster_list<512><<<blocks, 512, 0, st>>>(ws, d_surf, tiles_per_surface); break;
    default: k_raster_list<256><<<blocks, 256, 0, st>>>(ws, d_surf, tiles_per_surface); break;
  }
  return cudaGetLastError();
}

cudaError_t launch_raster(const Workspace& ws, const Surface* d_surf, uint32_t ntiles, int threads, cudaStream_t st,
                          uint32_t tile0, const SceneDev* prep) {
  if (!ntiles) return cudaSuccess;
  if (prep && (!ws.srec || ws.tiles)) return cudaErrorInvalidValue;
  if (threads == 128 && ntiles >= kManyWaves * num_sms() * raster_ctas<64>()) threads = 64;
  const uint32_t pb = prep ? std::min<uint32_t>((prep->ntris + threads - 1) / threads, (uint32_t)num_sms() * 4) : 0;
  const SceneDev sc = prep ? *prep : SceneDev{};
#define GBR_RASTER(NT, CC) k_raster<NT, CC><<<ntiles + pb, NT, 0, st>>>(ws, d_surf, tile0, pb, sc)
  if (ws.tiles) {
    switch (threads) {
      case 64: GBR_RASTER(64, true); break;
      case 128: GBR_RASTER(128, true); break;
      case 512: GBR_RASTER(512, true); break;
      default: GBR_RASTER(256, true); break;
    }
  } else {
    switch (threads) {
      case 64: GBR_RASTER(64, false); break;
      case 128: GBR_RASTER(128, false); break;
      case 512: GBR_RASTER(512, false); break;
      default: GBR_RASTER(256, false); break;
    }
  }
#undef GBR_RASTER
  return cudaGetLastError();
}

cudaError_t launch_shade(const SceneDev& sc, const ViewParams* d_views, uint32_t nviews, const Surface* d_surf,
                         uint32_t ntiles, const Workspace& ws, cudaStream_t st, bool features, uint32_t tile0,
                         const ViewParams* one_view, const Surface* one_surf, Counters* host_ctr) {
  if (!ntiles) return cudaSuccess;
  if (!sc.objq || !sc.texlv || !ws.srec || (nviews > 1 && !ws.tiles)) return cudaErrorInvalidValue;
  const bool one = nviews == 1 && one_view && one_surf;
  auto go = [&](auto kernel) {
    kernel<<<ntiles, kTilePixels, sizeof(float4) * kLightQuads * sc.nlights, st>>>(
        sc, one ? *one_view : ViewParams{}, one ? *one_surf : Surface{}, d_views, d_surf, ws.srec, ws.ctr, ws.rec_cap,
        tile0, ws.tile_empty, ws.tiles, host_ctr);
  };
  if (features)
    one ? go(k_shade<true, true>) : go(k_shade<true, false>);
  else
    one ? go(k_shade<false, true>) : go(k_shade<false, false>);
  return cudaGetLastError();
}

// Blocks of the fused pass that fit on the device at once (cooperative grid).
template <int NT, bool FEAT>
uint32_t fused_grid() {
  static uint32_t cached[2] = {0, 0};
  int dev = 0;
  cudaGetDevice(&dev);
  uint32_t& g = cached[dev > 0 ? 1 : 0];
  if (!g || dev > 1) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_raster_shade<NT, FEAT>, NT, 0) != cudaSuccess)
      per_sm = 0;
    g = (uint32_t)std::max(per_sm, 0) * (uint32_t)num_sms();
  }
  return g;
}

template <int NT, bool FEAT>
cudaError_t launch_fused_t(const SceneDev& sc, const ViewParams* d_views, const Surface* d_surf, uint32_t nsurf,
                           const Workspace& ws, const uint32_t* sched, uint32_t nseg, uint32_t* queue,
                           cudaStream_t st) {
  const uint32_t grid = fused_grid<NT, FEAT>();
  if (!grid) return cudaErrorInvalidConfiguration;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(NT);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_raster_shade<NT, FEAT>, ws, d_surf, nsurf, sc, d_views, sched, nseg, queue);
}

cudaError_t launch_raster_shade(const SceneDev& sc, const ViewParams* d_views, const Surface* d_surf, uint32_t nsurf,
                                const Workspace& ws, const uint32_t* sched, uint32_t nseg, uint32_t* queue,
                                int threads, cudaStream_t st, bool features) {
  if (!sc.objq || !sc.texlv || !ws.srec || !sched || !queue || !nseg) return cudaErrorInvalidValue;
  if (threads == 128)
    return features ? launch_fused_t<128, true>(sc, d_views, d_surf, nsurf, ws, sched, nseg, queue, st)
                    : launch_fused_t<128, false>(sc, d_views, d_surf, nsurf, ws, sched, nseg, queue, st);
  return features ? launch_fused_t<256, true>(sc, d_views, d_surf, nsurf, ws, sched, nseg, queue, st)
                  : launch_fused_t<256, false>(sc, d_views, d_surf, nsurf, ws, sched, nseg, queue, st);
}

uint32_t fused_blocks(int threads, bool features) {
  if (threads == 128) return features ? fused_grid<128, true>() : fused_grid<128, false>();
  return features ? fused_grid<256, true>() : fused_grid<256, false>();
}

cudaError_t launch_texture_upload(uchar4* atlas, const uint32_t* nums, const uint32_t* sizes,
                                  const uint8_t* pixels, const uint64_t* offsets, const int32_t* tsizes,
                                  uint32_t ntex, int32_t max_size, cudaStream_t st) {
  if (!ntex) return cudaSuccess;
  dim3 block(16, 16), grid((max_size + 15) / 16, (max_size + 15) / 16, ntex);
  k_tex_upload<<<grid, block, 0, st>>>(atlas, nums, sizes, pixels, offsets, tsizes);
  return cudaGetLastError();
}

cudaError_t launch_mips(uchar4* atlas, const uint32_t* nums, const uint32_t* sizes, uint32_t mipmap_start,
                        const int32_t* tsizes, uint32_t ntex, int32_t max_size, cudaStream_t st) {
  if (!ntex) return cudaSuccess;
  dim3 block(16, 16), grid((max_size + 15) / 16, (max_size + 15) / 16, ntex);
  for (int level = 0; level < kMipLevels; level++) {
    k_mip<<<grid, block, 0, st>>>(atlas, nums, sizes, mipmap_start, tsizes, level);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t launch_flush_objects(gbr_obj_g_descriptor* descs, const gbr_object_flush* objs, uint32_t n,
                                 cudaStream_t st) {
  if (!n) return cudaSuccess;
  k_flush_objects<<<(n + 255) / 256, 256, 0, st>>>(descs, objs, n);
  return cudaGetLastError();
}

cudaError_t launch_begin_faces(const Surface* d_surf, uint32_t nsurf, const Workspace& ws, cudaStream_t st) {
  if (!nsurf) return cudaErrorInvalidValue;
  k_begin_faces<<<dim3(64, nsurf + 1), 256, 0, st>>>(d_surf, nsurf, reinterpret_cast<uint32_t*>(ws.ctr), ws.ncounts);
  return cudaGetLastError();
}

cudaError_t launch_atomic_rate(uint32_t* g, uint32_t nwords, int iters, int shared_mode, uint32_t blocks,
                               cudaStream_t st) {
  k_atomic_rate<<<blocks, 256, 0, st>>>(g, nwords, iters, shared_mode);
  return cudaGetLastError();
}

cudaError_t launch_fill_u32(uint32_t* p, uint32_t v, size_t n, cudaStream_t st) {
  if (!n) return cudaSuccess;
  k_fill_u32<<<num_sms() * 4, 256, 0, st>>>(p, v, n);
  return cudaGetLastError();
}

}  // namespace gbr

// Post passes over a rendered view (godrays, pseudo-AA, motion blur,
// reflections): they share the device helpers above.
#include "gbr_post.cuh"
