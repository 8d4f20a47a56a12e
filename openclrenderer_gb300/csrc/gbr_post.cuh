// gbr_post.cuh -- post passes over a rendered view: the reference's
// screenspace_godrays, do_pseudo_aa, do_motion_blur and
// screenspace_reflections (cl2.cl:1792-1917, 6437-7356), behind
// engine::draw_godrays / do_pseudo_aa / do_motion_blur /
// draw_screenspace_reflections (engine.cpp:1463-1536).  Included at the end
// of gbr_kernels.cu, whose device helpers they use.  Every pass reads one
// RGBA8 image and writes another; a pixel the reference leaves unwritten keeps
// its input colour.
#pragma once

namespace gbr {

// A light with shafts as the marches read it: its projection (screen x, y and
// camera z) and its colour times its intensity.
struct ShaftLight {
  f3 spos, col;
};

// screenspace_godrays (cl2.cl:1792-1917) for pixel (x, y) of a view: light
// shafts of every light with godray_intensity > 0 (nshafts of them), marched
// from the pixel towards the light's screen position over the depth buffer.
// my_depth, my_col: the pixel's own.  Returns the RGBA colour before
// quantisation.
__device__ f4 godrays_pixel(int x, int y, uint32_t my_depth, f4 my_col, const uint32_t* __restrict__ depth, int W, int H,
                            const ShaftLight* shafts, uint32_t nshafts) {
  const float samples = 80.f;
  const float decay_factor = 0.97f, weight = 0.01f;
  const float step = 400.f / samples;  // max_length / samples
  const f3 original = mk3((float)x, (float)y, depth_to_dist(my_depth));
  // a step is occluded where its distance is below the pixel's own - 5: in
  // depth units, one integer comparison.  (The reference also requires cdepth
  // != UINT_MAX; an empty pixel is at 350000, never below 349995.)
  const uint32_t occluded_below = nshafts ? depth_below(original.z - 5.0f) : 0u;
  const float xmax = (float)W - 1.0f, ymax = (float)H - 1.0f;
  for (uint32_t i = 0; i < nshafts; i++) {
    float idecay = 1.f;
    f3 iter_col = mk3(0, 0, 0);
    f3 dest = shafts[i].spos;
    const f3 cval = shafts[i].col;
    if (dest.z < 0) dest = add3(sub3(original, dest), original);
    const float vx = fabsf(original.x - dest.x), vy = fabsf(original.y - dest.y);
    const float mnum = vx > vy ? vx : vy;
    f3 dir = sub3(dest, original);
    const float dx = fdiv(dir.x, mnum) * step, dy = fdiv(dir.y, mnum) * step;
    // steps j with (float)j < mnum and j < samples
    const int n = mnum > 0.0f ? (int)fminf(ceilf(mnum), samples) : 0;
    float cx = original.x, cy = original.y;
    // A march whose whole segment, one step past its end, keeps 0.05 px inside
    // the screen needs no bounds tests: the positions move monotonically along
    // dir, and 80 float additions below 4096 stray from the exact line by less
    // than 0.01 px.  (Every comparison fails on NaN.)
    const float ex = cx + (float)n * dx, ey = cy + (float)n * dy;
    const bool inside = cx >= 0.05f && ex >= 0.05f && cx <= xmax - 0.05f && ex <= xmax - 0.05f &&
                        cy >= 0.05f && ey >= 0.05f && cy <= ymax - 0.05f && ey <= ymax - 0.05f;
    // Eight steps at a time: their positions (the same running sums as the
    // reference's current += dir), then their depth loads in flight together,
    // then the decay chain in order.  The reference skips the rest of the
    // march once it leaves the screen; an unoccluded step adds exactly 0.
    auto resolve = [&](const uint32_t (&dv)[8], int m) {
#pragma unroll
      for (int k = 0; k < 8; k++) {
        if (k < m) {
          if (dv[k] < occluded_below) {
            idecay *= 0.9f;
            iter_col = add3(iter_col, mul3s(mul3s(cval, idecay), weight));
          }
          idecay *= decay_factor;
        }
      }
    };
    int j0 = 0;
    if (__all_sync(__activemask(), inside)) {  // (else the warp would march twice, once each way)
      // positions in [0, 4096): truncated by adding 2^23 rounded toward zero
      // (the low bits are the integer), off the conversion pipe, which three
      // conversions a step kept as busy as the issue slots
      const uint32_t magic = 0x4B000000u * (uint32_t)W + 0x4B000000u;
      for (; j0 + 8 <= n; j0 += 8) {
        uint32_t dv[8];
#pragma unroll
        for (int k = 0; k < 8; k++) {
          const uint32_t ix = __float_as_uint(__fadd_rz(cx, 8388608.0f)), iy = __float_as_uint(__fadd_rz(cy, 8388608.0f));
          dv[k] = __ldg(depth + (iy * (uint32_t)W + ix - magic));
          cx += dx;
          cy += dy;
        }
        uint32_t nearest = dv[0];
#pragma unroll
        for (int k = 1; k < 8; k++) nearest = min(nearest, dv[k]);
        if (nearest < occluded_below) {
          resolve(dv, 8);
        } else {  // nothing in the way: the decay alone
#pragma unroll
          for (int k = 0; k < 8; k++) idecay *= decay_factor;
        }
      }
    }
    for (; j0 < n; j0 += 8) {
      int m = min(8, n - j0);
      uint32_t dv[8];
      {
        float px[8], py[8];
#pragma unroll
        for (int k = 0; k < 8; k++) {
          px[k] = cx;
          py[k] = cy;
          cx += dx;
          cy += dy;
        }
        if (!inside) {
#pragma unroll
          for (int k = 7; k >= 0; k--)
            if (px[k] < 0 || py[k] < 0 || px[k] >= xmax || py[k] >= ymax) m = min(m, k);
        }
#pragma unroll
        // (cvt.rzi: truncation, NaN -> 0, so a NaN march stays in bounds as in the oracle)
        for (int k = 0; k < 8; k++)
          dv[k] = k < m ? __ldg(depth + (size_t)__float2int_rz(py[k]) * W + __float2int_rz(px[k])) : 0u;
      }
      resolve(dv, m);
      if (m < 8) break;
    }
    my_col.x += iter_col.x;
    my_col.y += iter_col.y;
    my_col.z += iter_col.z;
  }
  my_col.w = 1.0f;
  const float exposure = 0.99f;
  f4 r;
  r.x = my_col.x * exposure; r.y = my_col.y * exposure; r.z = my_col.z * exposure; r.w = my_col.w * exposure;
  return r;
}

// engine::draw_godrays (engine.cpp:1463-1482): one thread per pixel.  The
// lights with shafts, in order, are projected once per block, while the
// pixels' own loads are in flight (569x406, one light: 22 us, 26 with the loads
// after the barrier and 23 with a projection per pixel).  Bound by instruction
// issue (the decay chain of a march is sequential).
__global__ void __launch_bounds__(256) k_godrays(const uint32_t* __restrict__ depth, const uint8_t* __restrict__ in,
                                                 uint8_t* __restrict__ out, int W, int H, float fov,
                                                 const gbr_light* __restrict__ lights, uint32_t nlights, f3 cpos,
                                                 f3 cc, f3 cs) {
  __shared__ ShaftLight shafts[kMaxLights];
  __shared__ uint32_t nshafts;
  const int x = blockIdx.x * 16 + (threadIdx.x & 15), y = blockIdx.y * 16 + (threadIdx.x >> 4);
  const bool inside = x < W && y < H;
  uint32_t my_depth = 0;
  f4 my_col{0.0f, 0.0f, 0.0f, 0.0f};
  if (inside) {  // (in flight while the first warp projects the lights)
    my_depth = depth[(size_t)y * W + x];
    my_col = read_linear_rgba8(in, W, H, (float)x - 0.25f, (float)y - 0.25f);
  }
  if (threadIdx.x < 32) {
    uint32_t n = 0;
    for (uint32_t i0 = 0; i0 < nlights; i0 += 32) {
      const uint32_t i = i0 + threadIdx.x;
      const bool on = i < nlights && !(lights[i].godray_intensity <= 0);
      const unsigned who = __ballot_sync(0xFFFFFFFFu, on);
      if (on) {
        const gbr_light& L = lights[i];
        ShaftLight& s = shafts[n + __popc(who & ((1u << threadIdx.x) - 1u))];
        s.spos = depth_project1(rot_cs(mk3(L.pos[0], L.pos[1], L.pos[2]), cpos, cc, cs), (float)W, (float)H, fov);
        s.col = mul3s(mk3(L.col[0], L.col[1], L.col[2]), L.godray_intensity);
      }
      n += (uint32_t)__popc(who);
    }
    if (threadIdx.x == 0) nshafts = n;
  }
  __syncthreads();
  if (!inside) return;
  const f4 c = godrays_pixel(x, y, my_depth, my_col, depth, W, H, shafts, nshafts);
  reinterpret_cast<uint32_t*>(out)[(size_t)y * W + x] = pack_rgba(c.x, c.y, c.z, c.w);
}

cudaError_t launch_godrays(const uint32_t* depth, const uint8_t* in, uint8_t* out, int W, int H, float fov,
                           const gbr_light* lights, uint32_t nlights, const float cpos[3], const float cc[3],
                           const float cs[3], cudaStream_t st) {
  dim3 grid((W + 15) / 16, (H + 15) / 16);
  k_godrays<<<grid, 256, 0, st>>>(depth, in, out, W, H, fov, lights, nlights, mk3(cpos[0], cpos[1], cpos[2]),
                                  mk3(cc[0], cc[1], cc[2]), mk3(cs[0], cs[1], cs[2]));
  return cudaGetLastError();
}

// ---- do_pseudo_aa (cl2.cl:6437-6657) ---------------------------------------
// Pixel (x, y) is an edge when exactly one horizontal and one vertical
// neighbour, and at least one diagonal, differ from it: by more than 100 depth
// units (test 0), or by more than 20 degrees of normal (test 1).  The first
// test that finds an edge replaces the colour with 0.65 x the mean of the
// similar neighbours + 0.35 x the mean of the differing ones.
// The 8 neighbours in the reference's order (dy = -1..1, then dx = -1..1),
// bit j of an edge mask: diagonals j = 0, 2, 5, 7; horizontal 3, 4; vertical
// 1, 6.
constexpr uint32_t kAADiag = 0xA5u, kAAHoriz = 0x18u, kAAVert = 0x42u;
// A block covers 32x8 pixels, one row per warp (so that a warp's halo reads
// are 32 consecutive words, free of bank conflicts); with their neighbours,
// a 34x10 halo.
constexpr int kAABlockW = 32, kAABlockH = 8;
constexpr int kAAHalo = kAABlockW + 2, kAAHaloH = kAABlockH + 2;

// The pixel at halo index h (distances and decoded normals staged in shared
// memory): the edge masks of both tests, then, for the first test that
// finds an edge, the colour means in the reference's accumulation order.
// The colours are read only for edge pixels: the other test's sums never
// reach the output.
__device__ __forceinline__ bool pseudo_aa_pixel(int x, int y, int W, int h, const float* sd, const float* snx,
                                                const float* sny, const float* snz,
                                                const uchar4* __restrict__ in, f3* out) {
  const float here = sd[h];
  const f3 n0 = fast_normalize3(mk3(snx[h], sny[h], snz[h]));
  uint32_t e0 = 0, e1 = 0;
  int j = 0;
#pragma unroll
  for (int dy = -1; dy <= 1; dy++) {
#pragma unroll
    for (int dx = -1; dx <= 1; dx++) {
      if (dx == 0 && dy == 0) continue;
      const int hq = h + dy * kAAHalo + dx;
      if (fabsf(sd[hq] - here) > 100.0f) e0 |= 1u << j;
      if (dot3(n0, mk3(snx[hq], sny[hq], snz[hq])) < kAACos) e1 |= 1u << j;
      j++;
    }
  }
  auto is_edge = [](uint32_t e) {
    return __popc(e & kAAHoriz) == 1 && __popc(e & kAAVert) == 1 && (e & kAADiag) != 0;
  };
  uint32_t e;
  if (is_edge(e0)) e = e0;
  else if (is_edge(e1)) e = e1;
  else return false;
  f3 same = mk3(0, 0, 0), other = mk3(0, 0, 0);
  float nsame = 0, nother = 0;
  j = 0;
#pragma unroll
  for (int dy = -1; dy <= 1; dy++) {
#pragma unroll
    for (int dx = -1; dx <= 1; dx++) {
      if (dx == 0 && dy == 0) continue;
      const uchar4 t = in[(size_t)(y + dy) * W + (x + dx)];
      const f3 c = mk3(u8_over_255(t.x), u8_over_255(t.y), u8_over_255(t.z));  // fdiv(t, 255.0f)
      if ((e >> j) & 1u) {
        other = add3(other, c);
        nother += 1.0f;
      } else {
        same = add3(same, c);
        nsame += 1.0f;
      }
      j++;
    }
  }
  const f3 m = mk3(fdiv(same.x, nsame), fdiv(same.y, nsame), fdiv(same.z, nsame));
  const f3 o = mk3(fdiv(other.x, nother), fdiv(other.y, nother), fdiv(other.z, nother));
  *out = add3(mul3s(m, 0.65f), mul3s(o, 0.35f));
  return true;
}

// engine::do_pseudo_aa (engine.cpp:1513-1516): one thread per pixel, 32x8
// pixels per block.  The block's 34x10 neighbourhood of distances and
// decoded normals is staged in shared memory first: each is decoded once
// instead of by each of its nine readers.
__global__ void __launch_bounds__(256) k_pseudo_aa(const uint32_t* __restrict__ depth, const uint32_t* __restrict__ ids,
                                                   const ushort2* __restrict__ nrm, const uchar4* __restrict__ in,
                                                   uchar4* __restrict__ out, int W, int H) {
  constexpr int E = kAAHalo, N = kAAHalo * kAAHaloH;
  __shared__ float sd[N], snx[N], sny[N], snz[N];
  const int bx = blockIdx.x * kAABlockW, by = blockIdx.y * kAABlockH;
  for (int i = threadIdx.x; i < N; i += blockDim.x) {
    const int hx = bx - 1 + i % E, hy = by - 1 + i / E;
    float d = 0.0f;
    f3 n = mk3(0, 0, 0);
    if (hx >= 0 && hy >= 0 && hx < W && hy < H) {
      const size_t q = (size_t)hy * W + hx;
      d = depth_to_dist(depth[q]);
      const ushort2 nq = nrm[q];
      n = decode_normal(nq.x, nq.y);
    }
    sd[i] = d;
    snx[i] = n.x;
    sny[i] = n.y;
    snz[i] = n.z;
  }
  __syncthreads();
  const int lx = threadIdx.x % kAABlockW, ly = threadIdx.x / kAABlockW;
  const int x = bx + lx, y = by + ly;
  if (x >= W || y >= H) return;
  const size_t p = (size_t)y * W + x;
  f3 c;
  const bool inner = x >= 1 && y >= 1 && x < W - 1 && y < H - 1;
  if (inner && depth[p] != kDepthClear && ids[p] != kNoId &&
      pseudo_aa_pixel(x, y, W, (ly + 1) * E + lx + 1, sd, snx, sny, snz, in, &c)) {
    reinterpret_cast<uint32_t*>(out)[p] = pack_rgba(c.x, c.y, c.z, 1.0f);
  } else {
    out[p] = in[p];
  }
}

cudaError_t launch_pseudo_aa(const uint32_t* depth, const uint32_t* ids, const uint16_t* normals, const uint8_t* in,
                             uint8_t* out, int W, int H, cudaStream_t st) {
  dim3 grid((W + kAABlockW - 1) / kAABlockW, (H + kAABlockH - 1) / kAABlockH);
  k_pseudo_aa<<<grid, kAABlockW * kAABlockH, 0, st>>>(depth, ids, reinterpret_cast<const ushort2*>(normals),
                                    reinterpret_cast<const uchar4*>(in), reinterpret_cast<uchar4*>(out), W, H);
  return cudaGetLastError();
}

// ---- do_motion_blur (cl2.cl:6714-6860) ---------------------------------------
// Bytes LO and HI of t over 255, as RN(x * hi + RN(x * lo)) with 1 / 255 = hi +
// lo: equal to u8_over_255 for every byte (two packed operations, not three).
template <int LO, int HI>
__device__ __forceinline__ float2 over_255(uint32_t t) {
  const float2 m = make_float2(__uint_as_float(__byte_perm(t, 0x4B000000u, 0x7440 | LO)),
                               __uint_as_float(__byte_perm(t, 0x4B000000u, 0x7440 | HI)));
  const float2 x = __fadd2_rn(m, dup2(-8388608.0f));
  return __ffma2_rn(x, dup2(kInv255Hi), __fmul2_rn(x, dup2(kInv255Lo)));
}
// o (+)= w * texel t
__device__ __forceinline__ void add_texel(uint32_t t, float w, bool first, f4& o) {
  const float2 w2 = dup2(w), rg = __fmul2_rn(w2, over_255<0, 1>(t)), ba = __fmul2_rn(w2, over_255<2, 3>(t));
  o.x = first ? rg.x : __fadd_rn(o.x, rg.x);
  o.y = first ? rg.y : __fadd_rn(o.y, rg.y);
  o.z = first ? ba.x : __fadd_rn(o.z, ba.x);
  o.w = first ? ba.y : __fadd_rn(o.w, ba.y);
}

// read_linear_rgba8 with two channels per packed instruction: the bytes as
// 2^23 + b less 2^23, their quotients by 255, and the weighted texels, which
// are then added in the same order, one channel at a time: with a packed sum
// behind the packed product the results were those of one rounding, whatever
// --fmad says.  (A shared table of the 256 quotients took 16 lookups a tap, with
// bank conflicts, and bound the pass.)
__device__ __forceinline__ f4 read_linear_packed(const uint8_t* __restrict__ img, int W, int H, float cx, float cy) {
  const float u = cx - 0.5f, v = cy - 0.5f;
  const float fi = floorf(u), fj = floorf(v);
  const float a = u - fi, b = v - fj;
  const int i0 = (int)fi, j0 = (int)fj;
  const int xs[2] = {min(max(i0, 0), W - 1), min(max(i0 + 1, 0), W - 1)};
  const int ys[2] = {min(max(j0, 0), H - 1), min(max(j0 + 1, 0), H - 1)};
  const float ia = 1.0f - a, ib = 1.0f - b;
  const float wt[4] = {ia * ib, a * ib, ia * b, a * b};
  f4 o;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const uint32_t t = rgba8_word(img, (size_t)ys[k >> 1] * W + xs[k & 1]);
    add_texel(t, wt[k], k == 0, o);
  }
  return o;
}

// read_linear_packed at (cx + 0.5, cy + 0.5) for 1 <= cx <= W - 2, 1 <= cy <= H
// - 2, where nothing is clamped; the floors by addition of 2^23 rounded toward
// zero, whose low bits are the coordinates.
__device__ __forceinline__ f4 read_linear_inner(const uint8_t* __restrict__ img, int W, float cx, float cy) {
  const float u = (cx + 0.5f) - 0.5f, v = (cy + 0.5f) - 0.5f;
  const float zu = __fadd_rz(u, 8388608.0f), zv = __fadd_rz(v, 8388608.0f);
  const float a = u - (zu - 8388608.0f), b = v - (zv - 8388608.0f);
  const uint32_t magic = 0x4B000000u * (uint32_t)W + 0x4B000000u;
  const uint32_t* p = reinterpret_cast<const uint32_t*>(img) +
                      (__float_as_uint(zv) * (uint32_t)W + __float_as_uint(zu) - magic);
  const uint32_t* q = p + W;
  const uint32_t t0 = __ldg(p), t1 = __ldg(p + 1), t2 = __ldg(q), t3 = __ldg(q + 1);
  const float ia = 1.0f - a, ib = 1.0f - b;
  f4 o;
  add_texel(t0, ia * ib, true, o);
  add_texel(t1, a * ib, false, o);
  add_texel(t2, ia * b, false, o);
  add_texel(t3, a * b, false, o);
  return o;
}

// The pixel's surface point, in its object's frame, is carried through the
// object's pose of the previous frame (history slot 1 on even frame ids, 2 on
// odd) and projected with this frame's and the previous frame's camera; the
// blend of the two screen motions (camera_contribution), times strength and
// capped at 50 px, is averaged over that many bilinear taps centred on the
// pixel.  Objects with a pixel on screen are marked in seen[] for the history
// update.
struct MotionCam {
  f3 cpos, cc, cs, opos, oc, os;
  float fov, strength, cam_w;
  uint32_t frame_id;
};

__global__ void __launch_bounds__(256) k_motion_blur(const gbr_triangle* __restrict__ tris,
                                                     const gbr_obj_g_descriptor* __restrict__ descs,
                                                     const uint32_t* __restrict__ depth,
                                                     const uint32_t* __restrict__ ids, const uint8_t* __restrict__ in,
                                                     uint8_t* __restrict__ out, int W, int H, MotionCam a,
                                                     uint32_t* __restrict__ seen, uint32_t ntris) {
  const int x = blockIdx.x * 16 + (threadIdx.x & 15), y = blockIdx.y * 16 + (threadIdx.x >> 4);
  if (x >= W || y >= H) return;
  const size_t p = (size_t)y * W + x;
  const uint32_t d = depth[p], id = ids[p];
  const uint32_t own = __ldg(reinterpret_cast<const uint32_t*>(in) + p);  // (with the others: empty pixels wait once)
  uint32_t* o32 = reinterpret_cast<uint32_t*>(out);
  if (d == kDepthClear || id == kNoId || (id >> 1) >= ntris) {  // (an id past the triangles: left as it is)
    o32[p] = own;
    return;
  }
  const uint32_t obj = __ldg(&tris[id >> 1].vertices[0].object_id);
  if (!seen[obj]) seen[obj] = 1u;
  const gbr_obj_g_descriptor* G = descs + obj;
  const float dist = depth_to_dist(d);
  const f3 local = mk3(fdiv(((float)x - (float)W / 2.0f) * dist, a.fov), fdiv(((float)y - (float)H / 2.0f) * dist, a.fov),
                       dist);
  const f3 world = add3(back_rot_cs(local, mk3(0, 0, 0), a.cc, a.cs), a.cpos);
  const f3 objl = back_rot_quat(sub3(world, ld3(G->world_pos)), ld4(G->world_rot_quat));
  const bool even = (a.frame_id & 1u) == 0;
  const f3 opos = ld3(even ? G->old_world_pos_1 : G->old_world_pos_2);
  const f4 oq = ld4(even ? G->old_world_rot_quat_1 : G->old_world_rot_quat_2);
  const f3 last = add3(rot_quat(objl, oq), opos);
  const f3 nocam = depth_project1(rot_cs(last, a.cpos, a.cc, a.cs), (float)W, (float)H, a.fov);
  const f3 prev = depth_project1(rot_cs(last, a.opos, a.oc, a.os), (float)W, (float)H, a.fov);
  f4 acc;
  if (prev.z < 20.0f) {
    acc = read_linear_packed(in, W, H, (float)x + 0.5f, (float)y + 0.5f);
  } else {
    float mx = (float)x - prev.x, my = (float)y - prev.y;
    const float nx = (float)x - nocam.x, ny = (float)y - nocam.y;
    mx = a.cam_w * mx + (1.0f - a.cam_w) * nx;
    my = a.cam_w * my + (1.0f - a.cam_w) * ny;
    mx = mx * a.strength;
    my = my * a.strength;
    int n = f2i_sat(fmax_(fabsf(mx), fabsf(my)) + 1.0f);
    if (n > 50) {
      mx = fdiv(mx, (float)n) * 50.0f;
      my = fdiv(my, (float)n) * 50.0f;
      n = 50;
    }
    float sx = 0.0f, sy = 0.0f;
    if (n != 0) {
      sx = fdiv(mx, (float)n);
      sy = fdiv(my, (float)n);
    }
    float cx = (float)x - mx * 0.5f, cy = (float)y - my * 0.5f;  // mx / 2 exactly
    acc.x = acc.y = acc.z = acc.w = 0.0f;
    float cnt = 0.0f;
    // Taps that all keep a pixel and more inside the screen (they move
    // monotonically, and 50 additions stray by less than 0.01 px) need no
    // bounds tests or clamps.  (Every comparison fails on NaN.)  A warp takes
    // them so when all of its lanes can, else it would run its taps twice, once
    // each way: 284x175 under a moving camera 18 us, 25 with a choice per lane.
    const float ex = cx + sx * (float)n, ey = cy + sy * (float)n;
    const float xm = (float)W - 2.05f, ym = (float)H - 2.05f;
    int i = 0;
    const bool inner =
        cx >= 1.05f && ex >= 1.05f && cx <= xm && ex <= xm && cy >= 1.05f && ey >= 1.05f && cy <= ym && ey <= ym;
    if (__all_sync(__activemask(), inner)) {
      for (; i < n; i++, cx += sx, cy += sy) {
        const f4 c = read_linear_inner(in, W, cx, cy);
        acc.x += c.x; acc.y += c.y; acc.z += c.z; acc.w += c.w;
      }
      cnt = (float)n;
    }
    for (; i < n; i++, cx += sx, cy += sy) {
      if (cx < 0 || cx >= (float)W || cy < 0 || cy >= (float)H) continue;
      const f4 c = read_linear_packed(in, W, H, cx + 0.5f, cy + 0.5f);
      acc.x += c.x; acc.y += c.y; acc.z += c.z; acc.w += c.w;
      cnt += 1.0f;
    }
    if (cnt != 0.0f) {
      acc.x = fdiv(acc.x, cnt); acc.y = fdiv(acc.y, cnt); acc.z = fdiv(acc.z, cnt); acc.w = fdiv(acc.w, cnt);
    }
  }
  o32[p] = pack_rgba(acc.x, acc.y, acc.z, acc.w);
}

// The pose-history writes of do_motion_blur (cl2.cl:6771-6786): every object
// with a pixel on screen stores its current pose in the slot the next frame
// reads (2 on even frame ids, 1 on odd); the marks are cleared.
__global__ void k_motion_history(gbr_obj_g_descriptor* descs, uint32_t* seen, uint32_t n, uint32_t frame_id) {
  const uint32_t o = blockIdx.x * blockDim.x + threadIdx.x;
  if (o >= n || !seen[o]) return;
  seen[o] = 0;
  gbr_obj_g_descriptor* G = descs + o;
  float* pos = (frame_id & 1u) == 0 ? G->old_world_pos_2 : G->old_world_pos_1;
  float* q = (frame_id & 1u) == 0 ? G->old_world_rot_quat_2 : G->old_world_rot_quat_1;
  for (int k = 0; k < 3; k++) pos[k] = G->world_pos[k];
  for (int k = 0; k < 4; k++) q[k] = G->world_rot_quat[k];
}

cudaError_t launch_motion_blur(const gbr_triangle* tris, uint32_t ntris, gbr_obj_g_descriptor* descs, uint32_t ndescs,
                               const uint32_t* depth, const uint32_t* ids, const uint8_t* in, uint8_t* out, int W,
                               int H, float fov, const float cpos[3], const float cc[3], const float cs[3],
                               const float opos[3], const float oc[3], const float os[3], uint32_t frame_id,
                               float strength, float camera_contribution, uint32_t* seen, cudaStream_t st) {
  MotionCam a;
  a.cpos = mk3(cpos[0], cpos[1], cpos[2]);
  a.cc = mk3(cc[0], cc[1], cc[2]);
  a.cs = mk3(cs[0], cs[1], cs[2]);
  a.opos = mk3(opos[0], opos[1], opos[2]);
  a.oc = mk3(oc[0], oc[1], oc[2]);
  a.os = mk3(os[0], os[1], os[2]);
  a.fov = fov;
  a.strength = strength;
  a.cam_w = camera_contribution;
  a.frame_id = frame_id;
  dim3 grid((W + 15) / 16, (H + 15) / 16);
  k_motion_blur<<<grid, 256, 0, st>>>(tris, descs, depth, ids, in, out, W, H, a, seen, ntris);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess || !ndescs) return e;
  k_motion_history<<<(ndescs + 255) / 256, 256, 0, st>>>(descs, seen, ndescs, frame_id);
  return cudaGetLastError();
}

// ---- screenspace_reflections (cl2.cl:6862-7355) -----------------------------
// interpolate_single_line_depth (cl2.cl:6862-6873): the point at parameter a
// on the screen-space segment s -> f, depth interpolated in 1/z.
__device__ __forceinline__ f3 line_depth_point(f3 s, f3 f, float a) {
  s.z = rcp(s.z);
  f.z = rcp(f.z);
  const float b = 1.0f - a;
  const f3 r = mk3(fma_(s.x, b, f.x * a), fma_(s.y, b, f.y * a), fma_(s.z, b, f.z * a));
  return mk3(r.x, r.y, rcp(r.z));
}

struct ReflectCam {
  f3 cpos, cc, cs;
  float fov;
};

// A pixel of an object with FEATURE_FLAG_SS_REFLECTIVE: the eye ray mirrored
// in the interpolated normal is marched in screen space from a point 10.5
// units along it (at most 200 steps, until it passes more than 1 unit behind
// the depth buffer), refined in tenths of a step, and the colour there mixed
// in by a contact fade (400 units, fading towards the screen edge) times the
// object's reflection map (ssid) when it has one.  Returns 0 when the pixel
// keeps its colour.  Background pixels become 0.
__device__ int reflection_pixel(const SceneDev& sc, const ReflectCam& v, int x, int y, int W, int H,
                                const uint32_t* __restrict__ depth, const uint32_t* __restrict__ ids,
                                const uint8_t* __restrict__ in, f4* out) {
  const size_t p = (size_t)y * W + x;
  const uint32_t d = depth[p];
  if (d == kDepthClear) {
    out->x = out->y = out->z = out->w = 0.0f;
    return 1;
  }
  const uint32_t id = ids[p];
  if (id == kNoId || (id >> 1) >= sc.ntris) return 0;
  const uint32_t tri = id >> 1, sub = id & 1u;
  const gbr_triangle* T = sc.tris + tri;
  const uint32_t o_id = __ldg(&T->vertices[0].object_id);
  const gbr_obj_g_descriptor* G = sc.descs + o_id;
  if (!((__ldg(&G->feature_flag) & 1) > 0)) return 0;
  const float dist = depth_to_dist(d);
  const f3 local = mk3(fdiv(((float)x - (float)W / 2.0f) * dist, v.fov), fdiv(((float)y - (float)H / 2.0f) * dist, v.fov),
                       dist);
  const f3 zero = mk3(0, 0, 0);
  const f3 world = add3(back_rot_cs(local, zero, v.cc, v.cs), v.cpos);
  const f3 ray = sub3(world, v.cpos);
  const float scale = __ldg(&G->scale);
  f3 pv[3], nv[3];
  f2 tv[3];
#pragma unroll
  for (int k = 0; k < 3; k++) {
    pv[k] = mul3s(ld3(T->vertices[k].pos), scale);
    nv[k] = ld3(T->vertices[k].normal);
    tv[k] = mk2(__ldg(&T->vertices[k].vt[0]), __ldg(&T->vertices[k].vt[1]));
  }
  const f4 q = ld4(G->world_rot_quat);
  const f3 wpos = ld3(G->world_pos);
  const BaryFrame bf = bary_frame(pv[0], pv[1], pv[2]);
  float l1, l2, l3;
  bary_exact(bf, back_rot_quat(sub3(world, wpos), q), &l1, &l2, &l3);
  f3 normal = mk3(fma_(nv[0].x, l1, fma_(nv[1].x, l2, nv[2].x * l3)), fma_(nv[0].y, l1, fma_(nv[1].y, l2, nv[2].y * l3)),
                  fma_(nv[0].z, l1, fma_(nv[1].z, l2, nv[2].z * l3)));
  normal = fast_normalize3(rot_quat(normal, q));
  const f2 vt = mk2(fma_(tv[0].x, l1, fma_(tv[1].x, l2, tv[2].x * l3)), fma_(tv[0].y, l1, fma_(tv[1].y, l2, tv[2].y * l3)));
  float refl = 1.0f;
  const uint32_t ssid = __ldg(&G->ssid);
  if (ssid != 0xFFFFFFFFu) {
    // the pixel's clip output, as prearrange wrote it to cutdown_tris
    f3 w[3], tp[3];
    uint32_t oid;
    int flags;
    load_world(sc, tri, w, &oid, &flags);
    const int n = transform_clip(w, v.cpos, v.cc, v.cs, v.fov, (float)W, (float)H, (int)sub, tp);
    if ((int)sub >= n) return 0;
    const f3 xpv = mk3(roundf(tp[0].x), roundf(tp[1].x), roundf(tp[2].x));
    const f3 ypv = mk3(roundf(tp[0].y), roundf(tp[1].y), roundf(tp[2].y));
    const float rc = rconstant(xpv, ypv);
    // get_vtdiff (cl2.cl:5691-5760), per pixel
    const f3 depths = mk3(rcp(tp[0].z), rcp(tp[1].z), rcp(tp[2].z));
    float DA, DB, DC;
    plane_const(depths, xpv, ypv, rc, &DA, &DB, &DC);
    const float fx = (float)x, fy = (float)y;
    const float dmx = fma_(DA, fx + 1.0f, fma_(DB, fy, DC));
    const float dmy = fma_(DA, fx, fma_(DB, fy + 1.0f, DC));
    const float hw = (float)W / 2.0f, hh = (float)H / 2.0f;
    f3 lmx = mk3(fdiv((fx + 1.0f) - hw, v.fov), fdiv(fy - hh, v.fov), 1.0f);
    f3 lmy = mk3(fdiv(fx - hw, v.fov), fdiv((fy + 1.0f) - hh, v.fov), 1.0f);
    lmx = mk3(fdiv(lmx.x, dmx), fdiv(lmx.y, dmx), fdiv(lmx.z, dmx));
    lmy = mk3(fdiv(lmy.x, dmy), fdiv(lmy.y, dmy), fdiv(lmy.z, dmy));
    const f3 gmx = back_rot_quat(sub3(add3(back_rot_cs(lmx, zero, v.cc, v.cs), v.cpos), wpos), q);
    const f3 gmy = back_rot_quat(sub3(add3(back_rot_cs(lmy, zero, v.cc, v.cs), v.cpos), wpos), q);
    float lx1, lx2, lx3, ly1, ly2, ly3;
    bary_exact(bf, gmx, &lx1, &lx2, &lx3);
    bary_exact(bf, gmy, &ly1, &ly2, &ly3);
    const f2 vtx = mk2(fma_(tv[0].x, lx1, fma_(tv[1].x, lx2, tv[2].x * lx3)),
                       fma_(tv[0].y, lx1, fma_(tv[1].y, lx2, tv[2].y * lx3)));
    const f2 vty = mk2(fma_(tv[0].x, ly1, fma_(tv[1].x, ly2, tv[2].x * ly3)),
                       fma_(tv[0].y, ly1, fma_(tv[1].y, ly2, tv[2].y * ly3)));
    const float mip_bias = 1.0f / kMipBias;
    const f2 vtdiff = mk2((fabsf(vtx.x - vt.x) + fabsf(vty.x - vt.x)) * mip_bias,
                          (fabsf(vtx.y - vt.y) + fabsf(vty.y - vt.y)) * mip_bias);
    refl = texture_filter_diff<false>(sc, vt, vtdiff, (int)ssid).x;
    if (refl < 0.1f) return 0;
  }
  // reflect (cl2.cl:169-176) normalises the normal once more
  const f3 nn = fast_normalize3(normal);
  const float k2 = 2.0f * dot3(ray, nn);
  const f3 refd = fast_normalize3(sub3(ray, mul3s(nn, k2)));
  const f3 jit = add3(world, mul3s(refd, 10.5f));
  const f3 sj = depth_project1(rot_cs(jit, v.cpos, v.cc, v.cs), (float)W, (float)H, v.fov);
  const f3 ss = depth_project1(rot_cs(world, v.cpos, v.cc, v.cs), (float)W, (float)H, v.fov);
  const float dx = sj.x - ss.x, dy = sj.y - ss.y;
  const float sdist = fsqrt(dx * dx + dy * dy);
  const float back = 1.0f - fdiv(sdist - 3.0f, sdist);
  f3 vprev = mk3(ss.x * back + sj.x * (1.0f - back), ss.y * back + sj.y * (1.0f - back),
                 rcp(ss.z) * back + rcp(sj.z) * (1.0f - back));
  vprev.z = rcp(vprev.z);
  const f3 vstart = sj;
  const float fw = (float)W, fh = (float)H;
  if (sj.x < 0 || sj.y < 0 || sj.x >= fw || sj.y >= fh) return 0;
  // The march: step i at sj (i = 0) or line_depth_point(vprev, vstart, 1 + i),
  // i < 200, until the depth buffer is more than 1 unit in front of the ray;
  // a step off screen ends it unmet.  Step 0 first, then four steps at a
  // time: positions first (they do not depend on the loads), then their
  // depth loads in flight together, then the tests in order.
  const float ipz = rcp(vprev.z), isz = rcp(vstart.z);  // line_depth_point's reciprocals, loop-invariant
  // A step is on screen when 0 <= x < W and 0 <= y < H or a coordinate is NaN
  // (every comparison of the reference's test fails on NaN; it reads pixel 0
  // then): the conversion rounds down and turns NaN into 0, so that is one
  // unsigned comparison per coordinate.
  auto at = [](float c) { return (uint32_t)__float2int_rd(c); };
  float a = 1.0f, stop = 0.0f;
  bool found = false;
  {
    const float dd = depth_to_dist(__ldg(depth + (size_t)at(sj.y) * W + at(sj.x)));
    if (dd < sj.z - 1.0f) {
      found = true;
      stop = dd;  // the refinement reads the depth where the march stopped on every try
    }
  }
  for (int i0 = 1; i0 < 200 && !found; i0 += 4) {
    float w[4];  // 1 / z of the steps
    uint32_t px[4], py[4];
    int m = min(4, 200 - i0);  // the first step off screen, or past the last
    const float fi0 = (float)i0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      // ai = 1 + i and b = 1 - ai = -i, both exact (integers below 2^24)
      const float fi = fi0 + (float)k, ai = fi + 1.0f;
      px[k] = at(fma_(vprev.x, -fi, vstart.x * ai));
      py[k] = at(fma_(vprev.y, -fi, vstart.y * ai));
      w[k] = fma_(ipz, -fi, isz * ai);
    }
#pragma unroll
    for (int k = 3; k >= 0; k--)
      if (px[k] >= (uint32_t)W || py[k] >= (uint32_t)H) m = min(m, k);
    uint32_t dv[4];
#pragma unroll
    for (int k = 0; k < 4; k++) dv[k] = k < m ? __ldg(depth + (size_t)(py[k] * (uint32_t)W + px[k])) : 0u;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      if (found) break;
      if (k >= m) return 0;  // off screen (or past step 199) before the ray met anything
      // dd < 1 / w - 1: with the approximate reciprocal (2^-23 of it off, the
      // other roundings a few 2^-24) unless the two sides are too near to tell
      const float za = crcp(w[k]);
      const float gap = fma_(depth_scaled(dv[k]), -kInvMulInt, za - 1.0f);  // z - 1 - dd
      bool hit = gap > 0.0f;
      if (!(fabsf(gap) > fabsf(za) * 1e-6f + 1e-6f) || !(fabsf(za) < 1e30f))
        hit = depth_to_dist(dv[k]) < rcp(w[k]) - 1.0f;
      if (hit) {
        found = true;
        a = fi0 + (float)(k + 1);  // 1 + i
        stop = depth_to_dist(dv[k]);
      }
    }
  }
  if (!found) return 0;
  float ta = a;
  f3 hit = sj;
  bool ok = false;
  for (int i = 0; i < 10; i++) {
    // line_depth_point(vprev, vstart, ta) with its two reciprocals hoisted
    const float tb = 1.0f - ta;
    hit = mk3(fma_(vprev.x, tb, vstart.x * ta), fma_(vprev.y, tb, vstart.y * ta), rcp(fma_(ipz, tb, isz * ta)));
    if (stop < hit.z + 1.0f && stop > hit.z - 20.0f) {
      ok = true;
      break;
    }
    ta += 0.1f;  // fdiv(1.0f, 10.0f) = RN(0.1)
  }
  if (!ok) return 0;
  const f3 te = line_depth_point(vstart, hit, 1.35f);
  float fextra = 0.0f;
  if (te.x < 0) fextra += fabsf(te.x);
  if (te.y < 0) fextra += fabsf(te.y);
  if (te.x >= fw) fextra += te.x - fw;
  if (te.y >= fh) fextra += te.y - fh;
  fextra = clampf_(fdiv(fextra, 200.0f), 0.0f, 1.0f);
  f3 gl = mk3(fdiv((hit.x - fw / 2.0f) * hit.z, v.fov), fdiv((hit.y - fh / 2.0f) * hit.z, v.fov), hit.z);
  gl = add3(back_rot_cs(gl, zero, v.cc, v.cs), v.cpos);
  const float ray_len = fast_length3(sub3(gl, world));
  float fade = 1.0f - fdiv(ray_len, 400.0f);
  fade = fade - fextra;
  fade = clampf_(fade, 0.0f, 1.0f) * refl;
  const f4 fc = read_linear_rgba8(in, W, H, hit.x, hit.y);
  const uchar4 t = reinterpret_cast<const uchar4*>(in)[p];
  const float den = 1.0f + fade;
  out->x = fdiv(u8_over_255(t.x) + fc.x * fade, den);  // u8_over_255(t) = fdiv(t, 255.0f)
  out->y = fdiv(u8_over_255(t.y) + fc.y * fade, den);
  out->z = fdiv(u8_over_255(t.z) + fc.z * fade, den);
  out->w = 1.0f;
  return 1;
}

// engine::draw_screenspace_reflections (engine.cpp:1483-1511): one thread per pixel.
__global__ void __launch_bounds__(256, 4) k_reflections(SceneDev sc, ReflectCam v, const uint32_t* __restrict__ depth,
                                                     const uint32_t* __restrict__ ids, const uint8_t* __restrict__ in,
                                                     uint8_t* __restrict__ out, int W, int H) {
  const int x = blockIdx.x * 16 + (threadIdx.x & 15), y = blockIdx.y * 16 + (threadIdx.x >> 4);
  if (x >= W || y >= H) return;
  const size_t p = (size_t)y * W + x;
  f4 c;
  uint32_t* o32 = reinterpret_cast<uint32_t*>(out);
  if (reflection_pixel(sc, v, x, y, W, H, depth, ids, in, &c))
    o32[p] = pack_rgba(c.x, c.y, c.z, c.w);
  else
    o32[p] = reinterpret_cast<const uint32_t*>(in)[p];
}

cudaError_t launch_reflections(const SceneDev& sc, const uint32_t* depth, const uint32_t* ids, const uint8_t* in,
                               uint8_t* out, int W, int H, float fov, const float cpos[3], const float cc[3],
                               const float cs[3], cudaStream_t st) {
  ReflectCam v;
  v.cpos = mk3(cpos[0], cpos[1], cpos[2]);
  v.cc = mk3(cc[0], cc[1], cc[2]);
  v.cs = mk3(cs[0], cs[1], cs[2]);
  v.fov = fov;
  dim3 grid((W + 15) / 16, (H + 15) / 16);
  k_reflections<<<grid, 256, 0, st>>>(sc, v, depth, ids, in, out, W, H);
  return cudaGetLastError();
}

}  // namespace gbr
