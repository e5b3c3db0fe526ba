// kernels.cuh -- CUDA kernels of the rasterizer hot path (sm_100a).
//
// Frame = visibility then shading:
//   k_init_keys    one 64-bit visibility word per pixel from the depth buffer
//   k_setup        per triangle: projection, rejection, small/large split
//                  (trisetup.c), warp-ballot compaction into two lists
//   k_raster_small persistent; warps take 32 small triangles, each lane walks
//                  its rows (drawSmall, Templates.py:250-323) and the warp
//                  fills the queued spans pixel-parallel; fragment = 64-bit
//                  atomicMin(depth key | ~order) in the L2-resident buffer.
//                  Opaque and alpha-tested materials run as separate
//                  specialisations (the opaque one needs far fewer registers)
//   k_coarse       per large triangle: tile binning of coarse.c, written as
//                  (triangle, tile) units with warp-scan offsets
//   k_raster_tiled persistent over units: per-tile restart of the tiled
//                  `draw` (Templates.py:93-185), same span queue
//   k_shade        per 16 x 16 tile: decode the winners, replay their row interpolants
//                  and shade once (bilinear/trilinear, alpha, shadow)
// The packed key makes the result independent of scheduling: smallest depth
// wins, equal depths go to the later fragment of the reference's serial
// order (small pass < large pass, material, triangle, bottom < top half).
#pragma once
#include "raster.cuh"

namespace axr {

struct DrawParams {
  const GroupDev *groups;
  int ngroups;
  int total_tris;
  ViewDev view;
  LightDev light;
  ShadowDev sh[2];
  int nsh;
  uint64_t *keys;
  uint16_t *ro, *go, *bo;
  float *db;
  uint32_t *small_list;  // opaque small triangles from the front, alpha-tested from the back
  uint32_t *items;       // row chunks of small triangles: (list position << 2 | chunk), same two ends
  uint32_t *large_list;
  uint2 *units;          // opaque (triangle, tile) units from the front, alpha-tested from the back
  uint32_t *ctr;         // see CTR_*
  uint32_t cap_list, cap_units;
  int min_chunk;         // rows per small-triangle work item (at least; tuning knob)
  int claim_k;           // claim_size's k for the short queues (0: 32 items per claim)
  uint32_t *host_ctr;    // pinned host copy of the counters, written by the shade; null: none
};

enum {
  CTR_SMALL = 0, CTR_SMALL_A, CTR_LARGE, CTR_UNITS, CTR_UNITS_A, CTR_WORK_SMALL, CTR_WORK_SMALL_A, CTR_WORK_LARGE,
  CTR_WORK_UNITS, CTR_WORK_UNITS_A, CTR_OVERFLOW, CTR_SH_LIST, CTR_SH_LIST_A, CTR_SH_WORK, CTR_SH_WORK_A,
  CTR_UNITS_RESERVED, CTR_LIMIT, CTR_ITEMS, CTR_ITEMS_A, CTR_SH_ITEMS, CTR_SH_ITEMS_A,
  // tiled shadow pass: unit queue overflowed (the per-caster path drew the
  // map), units the map needed, non-empty tiles, tiles claimed (opaque, alpha)
  CTR_SH_OVERFLOW, CTR_SH_UNITS_NEED, CTR_SH_TILES, CTR_SH_TILE_WORK, CTR_SH_TILE_WORK_A, CTR_SH_ITEMS_TILED,
  CTR_N = 32
};

// Every data-dependent loop is bounded by construction (rows of a small
// triangle < 2*96, of a tile unit <= 2*16, of a shadow triangle <= 2*(dim+240)
// because of the setup rejections).  As a second line of defence each one
// also stops after LOOP_LIMIT rounds and records that in ctr[CTR_LIMIT],
// which the host reports as an error.
constexpr int LOOP_LIMIT = 1 << 16;


// ------------------------------------------------------------ helpers

__device__ __forceinline__ int find_group(const GroupDev *__restrict__ gs, int ng, uint32_t gtri) {
  int lo = 0, hi = ng - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if ((uint32_t)gs[mid].tri_base <= gtri) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// count of x in [ax0, ...] with (float)x <= bound, clipped to [0, w)
__device__ __forceinline__ void span_clip(int ax0, float bound, int w, int &lo, int &cnt) {
  lo = ax0 < 0 ? 0 : ax0;
  if (bound != bound) { cnt = 0; return; }
  float fb = floorf(bound);
  int hi = fb >= (float)(w - 1) ? w - 1 : f2i(fb);
  cnt = hi >= lo ? hi - lo + 1 : 0;
}

// A small triangle's rows (bottom half y1..y2, then top half y3..y2, both
// inclusive) are cut into at most MAX_CHUNKS chunks of at least MIN_CHUNK
// rows, so that large "small" triangles spread over several lanes; a lane
// replays the row accumulation up to its chunk, which keeps every
// interpolant bit-identical to the serial walk.
constexpr int MIN_CHUNK = 12;   // DrawParams::min_chunk of smaller scenes and of batches where no tuning is set
constexpr int CHUNK_BITS = 3;   // work item = list position << CHUNK_BITS | chunk
constexpr int MAX_CHUNKS = 1 << CHUNK_BITS;
__device__ __forceinline__ int small_rows(int y1, int y3) { return y3 - y1 + 2; }
// Items a warp claims at a time in a persistent loop over n work items: one
// per lane, unless that leaves warps of the launch without work (short
// queues); then fewer, so that every warp gets about one claim (k = 1), but at
// least `least`.  The value is the same for every warp.  Fewer items a claim
// idle lanes in the row phase, which costs issue slots that other kernels on
// the GPU could use; more items make one warp's chain of rows and pixels the
// length of the kernel.  One claim a warp and 8 items, against two claims and
// any number (alpha-tested queues, casters) or always 32 (opaque): 640x480 /
// 24k triangles alone 225 -> 183 us, 88 -> 77 us among other frames; 720p /
// 300k 336 -> 316 and 1080p / 1.04M 886 -> 869 among others (alone 970 -> 990).
// A queue of fewer items than warps leaves most of the GPU idle whatever the claim,
// so `least` falls with n / nw there (376 triangles at 320x192, the view alone, 135
// -> 120 us; 1,552 at 1280x720 204 -> 189).
// k = 0: always 32 -- the batched launches, whose warps move on to the
// next view's queue when one runs dry, so no warp idles.
__device__ __forceinline__ uint32_t claim_size(uint32_t n, uint32_t k, uint32_t least) {
  if (k == 0) return 32u;
  uint32_t nw = gridDim.x * (blockDim.x >> 5) * k;
  uint32_t per = (n + nw - 1) / nw;
  if (n < nw) least = max((least * n + nw - 1) / nw, 1u);
  return per < least ? least : (per > 32u ? 32u : per);
}
constexpr uint32_t CLAIM_LEAST = 8;   // of the rasterizers

__device__ __forceinline__ int chunk_len(int rows, int min_chunk) {
  int c = (rows + MAX_CHUNKS - 1) / MAX_CHUNKS;
  return c < min_chunk ? min_chunk : c;
}

// ------------------------------------------------------------ keys / clear

// A draw's or pass's group table as a kernel argument: the first kernel of the
// chain writes it to the device table that the later ones read, so that no
// host-to-device copy (and no staging buffer to wait for) stands before them.
template <int N>
struct GroupTab {
  GroupDev g[N];
};
template <int N>
__device__ __forceinline__ void store_table(const GroupTab<N> &tab, GroupDev *dst, int ngroups) {
  const uint32_t *src = reinterpret_cast<const uint32_t *>(tab.g);
  uint32_t *d = reinterpret_cast<uint32_t *>(dst);
  for (int i = threadIdx.x; i < ngroups * (int)(sizeof(GroupDev) / 4); i += blockDim.x) d[i] = src[i];
}

template <int N>
__global__ void k_init_keys(const float *__restrict__ db, uint64_t *__restrict__ keys, int n, uint32_t *ctr,
                            const __grid_constant__ GroupTab<N> tab, GroupDev *dst, int ngroups) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < CTR_N && blockIdx.x == 0) ctr[i] = 0;
  if (blockIdx.x == 0) store_table(tab, dst, ngroups);
  for (; i < n; i += gridDim.x * blockDim.x) keys[i] = ((uint64_t)depth_key(db[i]) << 32) | 0xffffffffull;
}

// clearzb.c:10-22 over lenP x lenP work-items of (w/lenP) x (h/lenP)
// blocks: columns [0, bw) of rows [0, bh) := 65535.  When bw == w those rows
// are one contiguous range, written with 16-byte stores.
__global__ void k_clear_depth(float *__restrict__ f, int w, int h, int lenP) {
  int bw = (w / lenP) * lenP, bh = (h / lenP) * lenP;
  size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (size_t)gridDim.x * blockDim.x;
  if (bw == w && ((uintptr_t)f & 15) == 0) {
    size_t n = (size_t)w * bh, n4 = n >> 2;
    const float4 v = make_float4(65535.f, 65535.f, 65535.f, 65535.f);
    for (size_t i = tid; i < n4; i += stride) reinterpret_cast<float4 *>(f)[i] = v;
    for (size_t i = (n4 << 2) + tid; i < n; i += stride) f[i] = 65535.f;
    return;
  }
  int n = bw * bh;
  for (int i = (int)tid; i < n; i += (int)stride) {
    int y = i / bw, x = i - y * bw;
    f[(size_t)w * y + x] = 65535.f;
  }
}

// Colour half of the current reference's clearZBuffer (Ops.py:939-946):
// every pixel of the three colour planes := (r, g, b); 16-byte stores when
// the planes are 16-byte aligned.
__global__ void k_fill_rgb(uint16_t *__restrict__ ro, uint16_t *__restrict__ go, uint16_t *__restrict__ bo, int n,
                           uint16_t r, uint16_t g, uint16_t b) {
  size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (size_t)gridDim.x * blockDim.x;
  size_t done = 0;
  if ((((uintptr_t)ro | (uintptr_t)go | (uintptr_t)bo) & 15) == 0) {
    size_t n8 = (size_t)n >> 3;
    uint32_t rr = r * 0x10001u, gg = g * 0x10001u, bb = b * 0x10001u;
    const uint4 vr = make_uint4(rr, rr, rr, rr), vg = make_uint4(gg, gg, gg, gg), vb = make_uint4(bb, bb, bb, bb);
    for (size_t i = tid; i < n8; i += stride) {
      reinterpret_cast<uint4 *>(ro)[i] = vr;
      reinterpret_cast<uint4 *>(go)[i] = vg;
      reinterpret_cast<uint4 *>(bo)[i] = vb;
    }
    done = n8 << 3;
  }
  for (size_t i = done + tid; i < (size_t)n; i += stride) {
    ro[i] = r;
    go[i] = g;
    bo[i] = b;
  }
}

// Conversions without the conversion unit (16 a cycle and SM, the limit of
// these kernels): a whole number below 2^23 sits in the low bits of 2^23 + it.
__device__ __forceinline__ float u16f(uint32_t x) { return __uint_as_float(0x4b000000u | x) - 8388608.f; }
// truncation of 0 <= x < 2^16 (addition rounded towards zero)
__device__ __forceinline__ uint32_t trunc16(float x) { return __float_as_uint(__fadd_rz(x, 8388608.f)) & 0xffffu; }

// Post/gamma.c:38-52 (quotients that share a divisor through its reciprocal:
// the IEEE quotient, see quot_by_recip)
__device__ __forceinline__ void gamma_px(uint32_t r, uint32_t g, uint32_t b, float e8, uint32_t &ro, uint32_t &go,
                                         uint32_t &bo) {
  const float y11 = 1.0f / 1.1f, y255 = 1.0f / 255.f;
  float jx = quot_by_recip(sqrtf(e8 * u16f(r)), 1.1f, y11);
  float jy = quot_by_recip(sqrtf(e8 * u16f(g)), 1.1f, y11);
  float jz = quot_by_recip(sqrtf(e8 * u16f(b)), 1.1f, y11);
  float m = quot_by_recip(fmaxf(jx, fmaxf(jy, jz)), 255.f, y255);
  if (m > 1.f) {
    float sm = sqrtf(m), y = span_recip(sm);
    jx = quot_by_recip(jx, sm, y); jy = quot_by_recip(jy, sm, y); jz = quot_by_recip(jz, sm, y);
  }
  ro = trunc16(fminf(255.f, jx));
  go = trunc16(fminf(255.f, jy));
  bo = trunc16(fminf(255.f, jz));
}

// Two pixels a thread (the width is a multiple of 16): one 4-byte load and store
// a plane.  Bound by issue and the square roots.  With events, one pixel and three
// divisions a pixel, eight pixels, two: 64x64 6.5, 8.6, 6.6 us; 1280x720 10.7,
// 10.7, 8.9; 1920x1080 14.8, 14.8, 12.9; 3840x2160 39.4, 37.2, 33.2.  More pixels a
// thread are a longer chain for small frames, and save nothing in large ones.
__global__ void __launch_bounds__(256, 8) k_gamma(uint16_t *r, uint16_t *g, uint16_t *b, int n, float exposure) {
  const float e8 = 8 * exposure;
  uint32_t *pr = reinterpret_cast<uint32_t *>(r), *pg = reinterpret_cast<uint32_t *>(g), *pb = reinterpret_cast<uint32_t *>(b);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n / 2; i += gridDim.x * blockDim.x) {
    const uint32_t R = pr[i], G = pg[i], B = pb[i];
    uint32_t x0, y0, z0, x1, y1, z1;
    gamma_px(R & 0xffffu, G & 0xffffu, B & 0xffffu, e8, x0, y0, z0);
    gamma_px(R >> 16, G >> 16, B >> 16, e8, x1, y1, z1);
    pr[i] = x0 | x1 << 16; pg[i] = y0 | y1 << 16; pb[i] = z0 | z1 << 16;
  }
}

// Post/gamma.c's mapping packed as interleaved 8-bit RGB for display (the
// planes are left as they are): 3 bytes per pixel instead of 6 + 4.  Two pixels
// a thread, three half-words out: 128x96 8.3 us (one pixel 8.1, four 8.9),
// 1920x1080 17.7 (18.4, 18.0; with three divisions a pixel 19.2).
__global__ void k_pack_rgb8(const uint16_t *__restrict__ r, const uint16_t *__restrict__ g,
                            const uint16_t *__restrict__ b, int n, float exposure, uint8_t *__restrict__ out) {
  const float e8 = 8 * exposure;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n / 2; i += gridDim.x * blockDim.x) {
    const uint32_t R = reinterpret_cast<const uint32_t *>(r)[i], G = reinterpret_cast<const uint32_t *>(g)[i],
                   B = reinterpret_cast<const uint32_t *>(b)[i];
    uint32_t x0, y0, z0, x1, y1, z1;
    gamma_px(R & 0xffffu, G & 0xffffu, B & 0xffffu, e8, x0, y0, z0);
    gamma_px(R >> 16, G >> 16, B >> 16, e8, x1, y1, z1);
    uint16_t *o = reinterpret_cast<uint16_t *>(out) + 3 * (size_t)i;
    o[0] = (uint16_t)(x0 | y0 << 8);
    o[1] = (uint16_t)(z0 | x1 << 8);
    o[2] = (uint16_t)(y1 | z1 << 8);
  }
}

// ------------------------------------------------------------ post effects
//
// Post/ssao.c and Post/dof.c over the (w/16*16) x (h/16*16) region their
// 16 x 16 work-groups cover (Ops.py:973-995); one thread a pixel, a block a
// 16 x 16 tile.  Arithmetic in source order, one IEEE rounding an operation.

struct SsaoParams {
  float rnd[32];      // the random table (entries 0..31 of the reference's 48)
  float sscale;
};

__device__ __forceinline__ V3 cross3(V3 a, V3 b) {
  return V3{a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}

// The occlusion that a pixel's 16 samples add up to.  TAME: the sample's depth
// is in [0.46, 2^14], its x and y below 2^35, ss in [1, 2^20] and w, h in
// [16, 2^20].  Then the shared reciprocal gives the IEEE quotients without a
// look at each sample: a numerator below 2^-60, for which it need not, ends as
// exactly w2 or h2 (>= 8) either way.  floor() of a coordinate, taken as unsigned,
// compares with w and h as the coordinate itself with 0 and w, h.
template <bool TAME>
__device__ __forceinline__ float ssao_samples(const float4 *T, const float *__restrict__ F, V3 pos, V3 norm, V3 norm2,
                                              float d, float ss, float w2, float h2, int w, int h, uint32_t pix) {
  const float bias = 0.002f, fw = (float)w, fh = (float)h;
  float ao = 0.f;
  for (int i = 0; i < 16; i += 8) {          // eight samples at a time: their depth reads overlap
    float sampd[8], zb[8];
    bool in[8];
#pragma unroll
    for (int k = 0; k < 8; k++) {
      float4 q = T[i + k];
      V3 sv{q.x, q.y, q.z};
      float dt = dot3(sv, norm);
      if (dt < 0) sv = sub3(sv, mul3(norm2, dt));
      sv = add3(mul3(sv, q.w), pos);
      float sz = sv.z, qx, qy;
      if (TAME) {
        float y = recip_rn(sz);
        qx = quot_fast(sv.x, sz, y);
        qy = quot_fast(-sv.y, sz, y);
      } else {
        float ax = fabsf(sv.x), ay = fabsf(sv.y), az = fabsf(sz);
        if (ax >= 0x1p-60f && ax <= 0x1p60f && ay >= 0x1p-60f && ay <= 0x1p60f && az >= 0x1p-60f && az <= 0x1p60f) {
          float y = recip_rn(sz);
          qx = quot_fast(sv.x, sz, y);
          qy = quot_fast(-sv.y, sz, y);
        } else {
          qx = sv.x / sz;
          qy = -sv.y / sz;
        }
      }
      float sx = (qx * ss) + w2;
      float sy = (qy * ss) + h2;
      int ix, iy;
      if (TAME) {
        ix = __float2int_rd(sx); iy = __float2int_rd(sy);
        in[k] = (uint32_t)ix < (uint32_t)w && (uint32_t)iy < (uint32_t)h;
      } else {
        ix = f2i(sx); iy = f2i(sy);
        in[k] = sx >= 0 && sx < fw && sy >= 0 && sy < fh;
      }
      sampd[k] = __ldg(F + (in[k] ? (uint32_t)(w * iy + ix) : pix));
      zb[k] = sz - bias;
    }
#pragma unroll
    for (int k = 0; k < 8; k++)
      if (in[k] && sampd[k] < zb[k]) ao += __saturatef(2.f - (d - sampd[k]));
  }
  return ao;
}

// ssao.c:6-97 in place on the colour planes; the depth row past the buffer
// (read on the last row when h is a multiple of 16) reads 65535.  A pixel's
// 16 sample directions depend on it only through cx mod 8 and cy mod 8, so
// a block first builds the 64 x 16 normalised directions and length
// factors (stride 17 float4 per (cx, cy) class: conflict-free reads), with
// the same arithmetic as the per-pixel loop, and then takes tile after tile:
// the grid is one wave, so the table is built once for about nine tiles of a
// 1080p frame.  Pixels beyond depth 6000 keep their colour (ao = 0) and take no
// samples.  The two quotients by the sample depth share one reciprocal; the ranges
// in which it gives the IEEE quotient are checked once a pixel, from its depth, its
// normal and the block's table (ssao_samples), and by sample only in warps where that
// fails: nearer than 1.5, degenerate normals, unusual tables and scales.  Eight samples'
// depth reads are in flight at a time.  Bound by instruction issue
// (2.8 of 4 a cycle): 76 us of a 1080p frame; 91 with the range checks by sample and
// four reads in flight, 133 with a table for every tile and samples one by one as
// well.  The four effects of the frame: 124 us with four reads in flight, 122 with
// eight (132 before).
__global__ void __launch_bounds__(256) k_ssao(uint16_t *__restrict__ ro, uint16_t *__restrict__ go,
                                              uint16_t *__restrict__ bo, const float *__restrict__ F, int w, int h,
                                              SsaoParams S) {
  const float radius = 1.f;
  __shared__ float rnd[32];                  // indexed per lane: staged out of the parameter space
  __shared__ float4 tab[64 * 17];
  if (threadIdx.x < 32) rnd[threadIdx.x] = S.rnd[threadIdx.x];
  __syncthreads();
  bool tab_tame = true;                      // directions of length <= 1.005, scaled by at most 1.005
  for (int e = threadIdx.x; e < 64 * 16; e += blockDim.x) {
    int i = e & 15, mx = (e >> 4) & 7, my = e >> 7;
    int c3 = 13 * ((mx * 3) & 7), c7 = 13 * ((mx * 7) & 7), c5 = 13 * ((mx * 5) & 7);
    int y7 = 17 * ((my * 7) & 7), y5 = 17 * ((my * 5) & 7), y3 = 17 * ((my * 3) & 7);
    V3 sv{rnd[(7 * i + c3 + y7) & 31], rnd[(7 * i + 1 + c7 + y5) & 31], rnd[(7 * i + 2 + c5 + y3) & 31]};
    sv = fast_normalize(sub3(mul3(sv, 2.f), V3{1.f, 1.f, 1.f}));
    float rlen = rnd[(7 * i + 3 + c3 + y3) & 31];
    float len2 = rlen * rlen * radius;
    tab[(my * 8 + mx) * 17 + i] = make_float4(sv.x, sv.y, sv.z, len2);
    tab_tame &= dot3(sv, sv) <= 1.01f && len2 <= 1.005f;
  }
  const bool block_tame = __syncthreads_and(tab_tame) && S.sscale >= 1.f && S.sscale <= 0x1p20f && w <= 1 << 20 &&
                          h <= 1 << 20;
  const int tw = w / 16, nt = tw * (h / 16), lx = threadIdx.x & 15, ly = threadIdx.x >> 4;
  const size_t n = (size_t)w * h;
  const float w2 = (float)(w / 2), h2 = (float)(h / 2), ss = S.sscale;
  const float yss = span_recip(ss);
  const float4 *T = tab + ((ly & 7) * 8 + (lx & 7)) * 17;
  for (int t = blockIdx.x; t < nt; t += gridDim.x) {
    const int ty = t / tw, cx = (t - ty * tw) * 16 + lx, cy = ty * 16 + ly;
    const size_t pix = (size_t)w * cy + cx;
    const float d = F[pix];
    if (d > 6000) continue;                  // ao = 0: (1 - 0) c = c
    const float fx = (float)cx + 0.5f, fy = (float)cy + 0.5f;
    const float vx = quot_by_recip(fx - w2, ss, yss), vy = quot_by_recip(-(fy - h2), ss, yss);
    V3 pos = smul3(d, V3{vx, vy, 1.f});
    float dx = pix + 1 < n ? F[pix + 1] : 65535.f;
    float dy = pix + w < n ? F[pix + w] : 65535.f;
    V3 px = smul3(dx, V3{quot_by_recip(fx + 1.f - w2, ss, yss), vy, 1.f});
    V3 py = smul3(dy, V3{vx, quot_by_recip(-(fy + 1.f - h2), ss, yss), 1.f});
    V3 norm = fast_normalize(cross3(sub3(pos, px), sub3(pos, py)));   // rx * ry = 1
    V3 norm2 = smul3(2.f, norm);
    // A reflection about norm takes |sv|^2 to |sv|^2 + 4 dt^2 (|norm|^2 - 1): with the table's
    // lengths a sample stays within 1.04 of pos, so its z is at least 0.46.  By warp, as one
    // that ran both loops would take 161 us where 132 had done (near and far pixels mixed).
    const bool tame = __all_sync(__activemask(), block_tame && d >= 1.5f && dot3(norm, norm) <= 1.01f);
    float ao = tame ? ssao_samples<true>(T, F, pos, norm, norm2, d, ss, w2, h2, w, h, (uint32_t)pix)
                    : ssao_samples<false>(T, F, pos, norm, norm2, d, ss, w2, h2, w, h, (uint32_t)pix);
    ao /= 16.f;
    ao = fminf(fmaxf(ao * 2.f, 0.f), 1.f);
    ro[pix] = u16sat((1 - ao) * (float)ro[pix]);
    go[pix] = u16sat((1 - ao) * (float)go[pix]);
    bo[pix] = u16sat((1 - ao) * (float)bo[pix]);
  }
}

// dof.c:4-69: the circle-of-confusion gather into (r2, g2, b2).  The tile and
// a 4-pixel halo (the largest radius) are staged in shared memory as floats
// with each source pixel's own circle of confusion (NaN outside the frame,
// which no source pixel has), so that a tap is one 16-byte read without
// conversions; the quotients by the radius share its reciprocal.
// 35 us of a 1080p frame (37 with 16-bit staging), plus 7 for k_copy3 in the place
// of three copies.
constexpr int DOF_HALO = 4, DOF_SIDE = 16 + 2 * DOF_HALO;
__global__ void __launch_bounds__(256) k_dof(const uint16_t *__restrict__ ro, const uint16_t *__restrict__ go,
                                             const uint16_t *__restrict__ bo, const float *__restrict__ F, int w,
                                             int h, float focus, uint16_t *__restrict__ r2, uint16_t *__restrict__ g2,
                                             uint16_t *__restrict__ b2) {
  const float maxcoc = 4.f, aperture = 4.f;
  __shared__ float4 cs[DOF_SIDE * DOF_SIDE];
  const float yf = span_recip(focus);
  int x0 = blockIdx.x * 16 - DOF_HALO, y0 = blockIdx.y * 16 - DOF_HALO;
  for (int k = threadIdx.x; k < DOF_SIDE * DOF_SIDE; k += blockDim.x) {
    int sx = x0 + k % DOF_SIDE, sy = y0 + k / DOF_SIDE;
    float4 c = make_float4(0.f, 0.f, 0.f, __int_as_float(0x7fc00000));
    if (sx >= 0 && sx < w && sy >= 0 && sy < h) {
      size_t q = (size_t)w * sy + sx;
      float f = F[q];
      c = make_float4(u16f(ro[q]), u16f(go[q]), u16f(bo[q]),
                      fminf(maxcoc, quot_by_recip(aperture * fabsf(f - focus), focus, yf) / f));
    }
    cs[k] = c;
  }
  __syncthreads();
  int lx = threadIdx.x & 15, ly = threadIdx.x >> 4, ix = blockIdx.x * 16 + lx, iy = blockIdx.y * 16 + ly;
  float cx = (float)ix + 0.5f, cy = (float)iy + 0.5f;
  float dofR = 0, dofG = 0, dofB = 0, nsamples = 0;
  float radius = cs[(ly + DOF_HALO) * DOF_SIDE + lx + DOF_HALO].w, yr = span_recip(radius);   // min(maxcoc, its own)
  float ylim = ceilf(cy + radius), xlim = ceilf(cx + radius);
  float fx0 = floorf(cx - radius), fy0 = floorf(cy - radius);
  const float4 *row = cs + (f2i(fy0) - y0) * DOF_SIDE + (f2i(fx0) - x0);
  for (float fy = fy0; fy < ylim; fy += 1.f, row += DOF_SIDE) {
    float wy0 = 1.f - fmaxf(cy - radius - fy, 0.f), wy1 = fminf(cy + radius - fy, 1.f);
    const float4 *p = row;
    for (float fx = fx0; fx < xlim; fx += 1.f) {
      float4 c = *p++;
      float cover = (1.f - fmaxf(cx - radius - fx, 0.f)) * wy0;
      cover *= fminf(cx + radius - fx, 1.f) * wy1;
      if (c.w != c.w) continue;
      if (radius > c.w) cover *= quot_by_recip(c.w, radius, yr);
      dofR += c.x * cover;
      dofG += c.y * cover;
      dofB += c.z * cover;
      nsamples += cover;
    }
  }
  dofR /= nsamples; dofG /= nsamples; dofB /= nsamples;
  size_t pix = (size_t)w * iy + ix;
  r2[pix] = u16sat(dofR); g2[pix] = u16sat(dofG); b2[pix] = u16sat(dofB);
}

// The gathered planes back over the frame's (Ops.py:993-995), 8 pixels at a time
__global__ void k_copy3(uint4 *__restrict__ r, uint4 *__restrict__ g, uint4 *__restrict__ b,
                        const uint4 *__restrict__ r2, const uint4 *__restrict__ g2, const uint4 *__restrict__ b2, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    r[i] = r2[i];
    g[i] = g2[i];
    b[i] = b2[i];
  }
}

// Post/blur.c + Post/blur2.c (CLDraw.blur): the bloom, each pass over the
// whole image before the next that reads its neighbours (the reference's
// barrier orders only its work-group; the launch-wide order is the one its
// phases are written for), in two launches: the bright pass with the
// horizontal blur, and the vertical blur with the upsampled addition to the
// frame.  A block keeps its tile of the earlier pass in shared memory as
// floats, so no tap converts or leaves the SM.  The half-resolution planes are wf x hf
// with wf = w/2, hf = h/2; rows no pass writes, and taps outside, are 0 (a sum
// of the non-negative terms does not change by adding 0).  32 us of a 1080p
// frame (12 + 20) against 62 as four launches through planes in memory.
struct BloomPlanes {
  uint16_t *hb[3];   // horizontal blur, rows [0, hf - 1)
};

__constant__ float c_bloom_w[9] = {0.00816f, 0.01384f, 0.02207f, 0.03306f, 0.04654f,
                                   0.06157f, 0.07654f, 0.08941f, 0.09815f};   // taps 9..1

// the 19 taps centred at v[9] (blur.c:46-66's order), as stored: / 0.9, u16
__device__ __forceinline__ uint16_t bloom_taps(const float *v, int step) {
  float a = 0.f;
#pragma unroll
  for (int d = 9; d >= 1; d--) a = a + c_bloom_w[9 - d] * v[(9 - d) * step];
  a += 0.10125f * v[9 * step];
#pragma unroll
  for (int d = 1; d <= 9; d++) a = a + c_bloom_w[9 - d] * v[(9 + d) * step];
  const float y = 1.0f / 0.9f;
  return u16sat(quot_fast(a, 0.9f, y));   // a is 0 or at least 0.008
}

constexpr int BLOOM_W = 128;
// blur.c:22-34 (bright pass, rows [0, hf - 2)) and :38-66 (rows [0, hf - 1))
__global__ void __launch_bounds__(BLOOM_W) k_bloom_h(const uint16_t *__restrict__ ro, const uint16_t *__restrict__ go,
                                                     const uint16_t *__restrict__ bo, int wf, int hf, BloomPlanes B) {
  __shared__ float v[3][BLOOM_W + 18];
  const int x0 = blockIdx.x * BLOOM_W, cy = blockIdx.y;
  const uint16_t *f[3] = {ro, go, bo};
  for (int i = threadIdx.x; i < BLOOM_W + 18; i += BLOOM_W) {
    int cx = x0 + i - 9;
    float br[3] = {0.f, 0.f, 0.f};
    if (cx >= 0 && cx < wf && cy < hf - 2) {
      int y1 = min(wf * (hf - 1) * 4, wf * cy * 4 + 1);
      int x1 = min(wf * 2 - 1, cx * 2 + 1);
      int i0 = wf * cy * 4 + cx * 2, i1 = y1 + cx * 2, i2 = wf * cy * 4 + x1, i3 = y1 + x1;
      float c[3];
#pragma unroll
      for (int k = 0; k < 3; k++)
        c[k] = (float)((int)f[k][i0] / 4 + (int)f[k][i1] / 4 + (int)f[k][i2] / 4 + (int)f[k][i3] / 4);
      float lum = (float)(0.3626 * (double)c[0] + 0.5152 * (double)c[1] + 0.1222 * (double)c[2]);
#pragma unroll
      for (int k = 0; k < 3; k++) br[k] = (float)u16sat(c[k] * lum / 256.f / 256.f);
    }
#pragma unroll
    for (int k = 0; k < 3; k++) v[k][i] = br[k];
  }
  __syncthreads();
  const int cx = x0 + threadIdx.x;
  if (cx >= wf) return;
#pragma unroll
  for (int k = 0; k < 3; k++) B.hb[k][(size_t)wf * cy + cx] = bloom_taps(&v[k][threadIdx.x], 1);
}

// blur2.c:22-50 (the vertical blur of rows [0, hf - 1), whose lower taps are
// bounded by the half width, as blur2.c writes it) and :54-79 (upsampled
// bilinearly and added to the frame's rows [0, 2 hf) and columns [0, 2 wf)),
// one plane a block (blockIdx.z): 62 x 31 half-resolution pixels and one more
// column and row for the upsampling; a thread blurs four rows of a column and
// adds to 2 x 2 pixels of the frame at a time.
constexpr int BLOOM_TW = 62, BLOOM_TH = 31, BLOOM_V_THREADS = 512;
__global__ void __launch_bounds__(BLOOM_V_THREADS) k_bloom_v(uint16_t *__restrict__ ro, uint16_t *__restrict__ go,
                                                             uint16_t *__restrict__ bo, int w, int wf, int hf,
                                                             BloomPlanes B) {
  constexpr int TW = 64, TH = BLOOM_TH + 1;
  static_assert(TW * TH == 4 * BLOOM_V_THREADS, "four rows of a column a thread");
  __shared__ float hb[(TH + 18) * TW];
  __shared__ float vb[TH * TW];
  const int plane = blockIdx.z, x0 = blockIdx.x * BLOOM_TW, first = blockIdx.y * BLOOM_TH;
  const int y0 = min(first, hf - 2);         // row hf - 1 also reads row hf - 2
  const uint16_t *src = B.hb[plane];
  for (int i = threadIdx.x; i < (TH + 18) * (TW / 2); i += BLOOM_V_THREADS) {   // wf and x0 are even
    int r = y0 - 9 + i / (TW / 2), cx = x0 + 2 * (i % (TW / 2));
    uint32_t c = 0;
    if (r >= 0 && r < hf - 1 && cx < wf) c = *reinterpret_cast<const uint32_t *>(src + (size_t)wf * r + cx);
    hb[2 * i] = u16f(c & 0xffffu);
    hb[2 * i + 1] = u16f(c >> 16);
  }
  __syncthreads();
  {
    const int x = threadIdx.x % TW, strip = threadIdx.x / TW * 4;
    float v[22];
#pragma unroll
    for (int i = 0; i < 22; i++) v[i] = hb[(strip + i) * TW + x];
    const bool bounded = y0 + strip + 3 + 9 >= wf;      // some lower tap ends at the half width
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const int cy = y0 + strip + k;
      uint16_t out;
      if (bounded) {
        float t[19];
#pragma unroll
        for (int i = 0; i < 19; i++) t[i] = (i < 10 || cy + i - 9 < wf) ? v[k + i] : 0.f;
        out = bloom_taps(t, 1);
      } else {
        out = bloom_taps(v + k, 1);
      }
      vb[(strip + k) * TW + x] = cy < hf - 1 ? u16f(out) : 0.f;
    }
  }
  __syncthreads();
  uint16_t *dst = plane == 0 ? ro : plane == 1 ? go : bo;
  const int x = threadIdx.x % TW, tex1 = x0 + x, last = min(first + BLOOM_TH, hf);
  if (x >= BLOOM_TW || tex1 >= wf) return;
  const int t1n = min(tex1 + 1, wf - 1) - x0;
  for (int tex2 = first + threadIdx.x / TW; tex2 < last; tex2 += BLOOM_V_THREADS / TW) {
    const float *T0 = vb + (tex2 - y0) * TW, *T1 = vb + (min(tex2 + 1, hf - 2) - y0) * TW;
    const float t00 = T0[x], t10 = T0[t1n], t01 = T1[x], t11 = T1[t1n];
    // fractions 0 (weights 1 and 0) and 1/2 along each axis
    uint32_t *p = reinterpret_cast<uint32_t *>(dst + (size_t)w * 2 * tex2 + 2 * tex1), *q = p + w / 2;
    const uint32_t c = *p, e = *q;
    *p = (uint32_t)u16sat(u16f(c & 0xffffu) + t00) | (uint32_t)u16sat(u16f(c >> 16) + (0.5f * t00 + 0.5f * t10)) << 16;
    *q = (uint32_t)u16sat(u16f(e & 0xffffu) + (0.5f * t00 + 0.5f * t01)) |
         (uint32_t)u16sat(u16f(e >> 16) + (0.25f * t00 + 0.25f * t10 + 0.25f * t01 + 0.25f * t11)) << 16;
  }
}

// ------------------------------------------------------------ vertex stage
//
// Pipe/vert.c over a group's packed vertex arrays (3 floats a vertex).  A
// thread takes a quad of 4 consecutive vertices -- three aligned 16-byte
// words of each array (the arrays start 256-byte aligned, so vertex 4k
// starts a word) -- when the whole quad lies in [v0, v1); the partial quads
// at both ends go vertex by vertex.  The arithmetic is vert.c's, one IEEE
// rounding an operation in source order (no contraction).

struct VertXform {
  float oldr[9];   // rows of oldRM
  float rr[9];     // rows of rotMat transposed (CLDraw.rotate uploads rotMat.T)
  float o[3];      // origin (transform) or offset (Ttranslate)
};

struct VertLights {
  const float *dint, *ddir;           // directional lights; light 0 is shaded per pixel
  const float *pint, *ppos;           // point lights
  const float *sint, *sdir, *spos;    // spot lights
  int nd, np, ns;
  float amb;
};

__device__ __forceinline__ V3 rows3(const float *m, V3 v) {
  return V3{dot3(v, V3{m[0], m[1], m[2]}), dot3(v, V3{m[3], m[4], m[5]}), dot3(v, V3{m[6], m[7], m[8]})};
}

// vert.c:3-28 (transform)
__device__ __forceinline__ void xform_rotate(const VertXform &X, V3 &p, V3 &n) {
  V3 o{X.o[0], X.o[1], X.o[2]};
  p = add3(rows3(X.rr, rows3(X.oldr, sub3(p, o))), o);
  n = rows3(X.rr, rows3(X.oldr, n));
}

// vert.c:29-36 (Ttranslate)
__device__ __forceinline__ void xform_translate(const VertXform &X, V3 &p) { p = add3(p, V3{X.o[0], X.o[1], X.o[2]}); }

__device__ __forceinline__ V3 ldg3(const float *p, int i) { return ld3(p + 3 * i); }

__device__ __forceinline__ float fast_length(V3 v) { return sqrtf(dot3(v, v)); }

__device__ __forceinline__ void quad_ld(const float *a, int q, V3 v[4]) {
  const float4 *w = reinterpret_cast<const float4 *>(a) + 3 * (size_t)q;
  float4 w0 = w[0], w1 = w[1], w2 = w[2];
  v[0] = V3{w0.x, w0.y, w0.z}; v[1] = V3{w0.w, w1.x, w1.y};
  v[2] = V3{w1.z, w1.w, w2.x}; v[3] = V3{w2.y, w2.z, w2.w};
}

__device__ __forceinline__ void quad_st(float *a, int q, const V3 v[4]) {
  float4 *w = reinterpret_cast<float4 *>(a) + 3 * (size_t)q;
  w[0] = make_float4(v[0].x, v[0].y, v[0].z, v[1].x);
  w[1] = make_float4(v[1].y, v[1].z, v[2].x, v[2].y);
  w[2] = make_float4(v[2].z, v[3].x, v[3].y, v[3].z);
}

__device__ __forceinline__ V3 v_ld(const float *a, int v) { return V3{a[3 * (size_t)v], a[3 * (size_t)v + 1], a[3 * (size_t)v + 2]}; }
__device__ __forceinline__ void v_st(float *a, int v, V3 x) {
  a[3 * (size_t)v] = x.x; a[3 * (size_t)v + 1] = x.y; a[3 * (size_t)v + 2] = x.z;
}

// CLDraw.rotate (ROT) / CLDraw.translate over vertices [v0, v1)
template <bool ROT>
__global__ void k_vert_xform(float *__restrict__ xyz, float *__restrict__ vn, int v0, int v1, VertXform X) {
  int q1 = (v1 + 3) >> 2;
  for (int q = (v0 >> 2) + blockIdx.x * blockDim.x + threadIdx.x; q < q1; q += gridDim.x * blockDim.x) {
    int a = q << 2;
    if (a >= v0 && a + 4 <= v1) {
      V3 p[4], n[4];
      quad_ld(xyz, q, p);
      if (ROT) quad_ld(vn, q, n);
#pragma unroll
      for (int k = 0; k < 4; k++) {
        if (ROT) xform_rotate(X, p[k], n[k]);
        else xform_translate(X, p[k]);
      }
      quad_st(xyz, q, p);
      if (ROT) quad_st(vn, q, n);
    } else {
      for (int v = max(a, v0); v < min(a + 4, v1); v++) {
        V3 p = v_ld(xyz, v), n;
        if (ROT) {
          n = v_ld(vn, v);
          xform_rotate(X, p, n);
          v_st(vn, v, n);
        } else {
          xform_translate(X, p);
        }
        v_st(xyz, v, p);
      }
    }
  }
}

// a / d for d in [1, 2^61): through the reciprocal where that gives the IEEE
// quotient (a not too small or large), else the division
__device__ __forceinline__ float quot_light(float a, float d) {
  return a >= 0x1p-60f && a <= 0x1p60f ? quot_fast(a, d, recip_rn(d)) : a / d;
}

// A vertex's light from a point (SPOT = false) or spot light at offset pl:
// vert.c:60-69 / :71-84, added where the light reaches the vertex.  Offsets of
// a length within [2^-30, 2^30] take the reciprocal of their length, and the
// falloff its divisor's, without the divisions' special cases.
template <bool SPOT>
__device__ __forceinline__ void light_at(V3 pl, V3 n, V3 sd, V3 intensity, V3 &light) {
  if (SPOT && !(dot3(sd, pl) > 0.f)) return;
  if (!(dot3(n, pl) > 0.f)) return;
  const float dd = dot3(pl, pl), fl = sqrtf(dd);
  V3 u;
  float s;
  if (dd >= 0x1p-60f && dd <= 0x1p60f) {
    u = mul3(pl, recip_rn(fl));
    s = SPOT ? quot_light(dot3(n, u) * dot3(u, sd), 1.5f + fl * fl) : quot_light(dot3(n, u), 1.f + fl * fl);
  } else {
    u = fast_normalize(pl);
    s = SPOT ? dot3(n, u) * dot3(u, sd) / (1.5f + fl * fl) : dot3(n, u) / (1.f + fl * fl);
  }
  light = add3(light, smul3(s, intensity));
}

// vert.c:49-86 (vertL) for N vertices: the lights outermost, so that each is
// loaded once for all of them
template <int N>
__device__ __forceinline__ void vert_light_n(const VertLights &L, const V3 x[N], const V3 n[N], V3 light[N]) {
#pragma unroll
  for (int k = 0; k < N; k++) light[k] = V3{0.f, 0.f, 0.f};
  for (int i = 1; i < L.nd; i++) {
    const V3 d = ldg3(L.ddir, i), c = ldg3(L.dint, i);
#pragma unroll
    for (int k = 0; k < N; k++) light[k] = add3(light[k], smul3(fmaxf(0.f, dot3(n[k], d) + 0.5f) * 0.66f, c));
  }
  for (int i = 0; i < L.np; i++) {
    const V3 p = ldg3(L.ppos, i), c = ldg3(L.pint, i);
#pragma unroll
    for (int k = 0; k < N; k++) light_at<false>(sub3(x[k], p), n[k], n[k], c, light[k]);
  }
  for (int i = 0; i < L.ns; i++) {
    const V3 p = ldg3(L.spos, i), d = ldg3(L.sdir, i), c = ldg3(L.sint, i);
#pragma unroll
    for (int k = 0; k < N; k++) light_at<true>(sub3(x[k], p), n[k], d, c, light[k]);
  }
#pragma unroll
  for (int k = 0; k < N; k++)
    light[k] = V3{fmaxf(light[k].x, L.amb), fmaxf(light[k].y, L.amb), fmaxf(light[k].z, L.amb)};
}

// CLDraw.vertLight for every masked group in one launch (blockIdx.y: the
// group), four consecutive vertices a thread as in k_vert_xform; positions are
// read only when point or spot lights exist.  Bound by instruction issue (the
// square root and quotients of each light and vertex): 1.5M vertices in four
// groups under 2 directional, 8 point and 4 spot lights take 55 us, against 88 us
// with a launch a group, a vertex a thread and IEEE divisions throughout.
struct VertJob { const float *xyz, *vn; float *li; int nv; };
template <int G>
struct VertJobs { VertJob g[G]; };
// N = 1, one vertex a thread, for calls that would not fill the GPU with four:
// the time is then one thread's chain over the lights.  40 registers, as the quads'
// code is not compiled in: 1,536 threads an SM.  One group under the same lights,
// with events, one a thread and four: 3,840 vertices 11.8 and 17.4 us, 160,000
// 14.9 and 19.9, 300,000 18.2 and 19.1, 450,000 22.8 and 20.8; 16 groups of
// 50,000 33.3 and 33.2, 64 of 50,000 109 and 97.  So the line is at 2,048 vertices an
// SM, of all groups of the call (axr_vert_light).  G: groups in the argument; a
// short one costs a small call less.
constexpr int light_threads(int n) { return n == 4 ? 256 : 128; }
template <int N, int G>
__global__ void __launch_bounds__(light_threads(N), N == 4 ? 4 : 12)
    k_vert_light(const __grid_constant__ VertJobs<G> J, VertLights L) {
  const VertJob &g = J.g[blockIdx.y];
  const bool pos = L.np + L.ns > 0;
  const uint32_t nv = g.nv, first = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
  uint32_t done = 0;
  if constexpr (N == 4) {
    for (int q = first; q < (int)(nv >> 2); q += step) {
      V3 x[4] = {}, n[4], light[4];
      if (pos) quad_ld(g.xyz, q, x);
      quad_ld(g.vn, q, n);
      vert_light_n<4>(L, x, n, light);
      quad_st(g.li, q, light);
    }
    done = nv & ~3u;
  }
  for (uint32_t v = done + first; v < nv; v += step) {
    V3 x[1] = {}, n[1] = {ld3(g.vn + 3 * (size_t)v)}, light[1];
    if (pos) x[0] = ld3(g.xyz + 3 * (size_t)v);
    vert_light_n<1>(L, x, n, light);
    v_st(g.li, v, light[0]);
  }
}

// ------------------------------------------------------------ setup

// one thread per triangle of every enabled group; lists hold global ids.
// `first`/`step` give the block's grid-stride over the triangles.
// One reservation per block and counter in a grid-stride loop that every
// thread of the block runs in step: warp w's totals v[k] (the same in all
// its lanes) become offsets out[k] into the counters ctr[idx[k]].  The
// counters are the same few addresses for the whole launch, so one
// atomicAdd per block instead of one per warp keeps them from serialising.
template <int K>
__device__ __forceinline__ void block_reserve(const uint32_t (&v)[K], const int (&idx)[K], uint32_t *ctr,
                                              uint32_t (&out)[K]) {
  __shared__ uint32_t part[32][K];
  __shared__ uint32_t base[K];
  const int w = threadIdx.x >> 5, nw = (int)(blockDim.x >> 5);
  if ((threadIdx.x & 31) == 0)
#pragma unroll
    for (int k = 0; k < K; k++) part[w][k] = v[k];
  __syncthreads();
  if (threadIdx.x < K) {
    const int k = threadIdx.x;
    uint32_t run = 0;
    for (int i = 0; i < nw; i++) {
      uint32_t x = part[i][k];
      part[i][k] = run;
      run += x;
    }
    base[k] = run ? atomicAdd(&ctr[idx[k]], run) : 0u;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < K; k++) out[k] = base[k] + part[w][k];
}

// Writes the row-chunk work items of a block's triangles (or casters),
// sorted by their row count, longest first (15 rows and more share a bucket and
// are not ordered among themselves), into one region per kind and
// block (opaque items from the front of `items`, alpha-tested ones from the
// back).  A warp of the raster claims 32 consecutive items, so sorted items
// give it rows of about the same count, and fewer lanes idle while the
// longest item of the claim finishes.  The raster's results do not depend
// on the order.  Every thread of the block calls it in step; a thread adds
// the nch items of its list entry `pos` (chunk c has min(cl, rows - c cl)
// rows).
constexpr int LEN_BUCKETS = 16;
__device__ __forceinline__ void block_items(uint32_t *items, uint32_t cap_items, uint32_t *ctr, int ctr_o, int ctr_a,
                                            uint32_t pos, bool alpha, int rows, int cl, int nch) {
  __shared__ uint32_t hist[2][LEN_BUCKETS];
  __shared__ uint32_t bbase[2];
  for (int i = threadIdx.x; i < 2 * LEN_BUCKETS; i += blockDim.x) hist[i / LEN_BUCKETS][i % LEN_BUCKETS] = 0;
  __syncthreads();
  const int k = alpha ? 1 : 0;
  // its chunks are cl rows long but for the last: bucket 0 holds the longest
  const int bf = LEN_BUCKETS - 1 - min(cl, LEN_BUCKETS - 1);
  const int bl = LEN_BUCKETS - 1 - min(rows - (nch - 1) * cl, LEN_BUCKETS - 1);
  uint32_t rf = 0, rl = 0;
  if (nch > 1) rf = atomicAdd(&hist[k][bf], (uint32_t)(nch - 1));
  if (nch > 0) rl = atomicAdd(&hist[k][bl], 1u);
  __syncthreads();
  if (threadIdx.x < 2) {
    uint32_t run = 0;
    for (int b = 0; b < LEN_BUCKETS; b++) {
      uint32_t x = hist[threadIdx.x][b];
      hist[threadIdx.x][b] = run;
      run += x;
    }
    bbase[threadIdx.x] = run ? atomicAdd(&ctr[threadIdx.x ? ctr_a : ctr_o], run) : 0u;
  }
  __syncthreads();
  for (int c = 0; c < nch; c++) {
    uint32_t p = bbase[k] + (c < nch - 1 ? hist[k][bf] + rf + c : hist[k][bl] + rl);
    uint32_t item = (pos << CHUNK_BITS) | (uint32_t)c;
    if (!alpha) items[p] = item;
    else items[cap_items - 1 - p] = item;
  }
  __syncthreads();   // the next call reuses hist and bbase
}

__device__ __forceinline__ void setup_phase(const DrawParams &P, const GroupDev *sg, int first, int step) {
  int lane = threadIdx.x & 31;
  for (int base = first; base < P.total_tris; base += step) {
    int t = base + threadIdx.x;
    int cls = 0;
    bool alpha = false;
    int iy0 = 0, iy1 = 0, iy2 = 0;
    if (t < P.total_tris) {
      int g = find_group(sg, P.ngroups, (uint32_t)t);
      const GroupDev &G = sg[g];
      if (G.enabled) {
        float sx[3], sy[3], sz[3];
        cls = project_persp(G, t - G.tri_base, P.view, sx, sy, sz);
        alpha = (G.flags & F_ALPHA) != 0;
        iy0 = f2i(sy[0]); iy1 = f2i(sy[1]); iy2 = f2i(sy[2]);
      }
    }
    unsigned ms = __ballot_sync(FULL, cls == 1 && !alpha), ma = __ballot_sync(FULL, cls == 1 && alpha);
    unsigned ml = __ballot_sync(FULL, cls == 2);
    const uint32_t want[3] = {(uint32_t)__popc(ms), (uint32_t)__popc(ma), (uint32_t)__popc(ml)};
    const int idx[3] = {CTR_SMALL, CTR_SMALL_A, CTR_LARGE};
    uint32_t got[3];
    block_reserve<3>(want, idx, P.ctr, got);
    unsigned lt = (1u << lane) - 1;
    uint32_t pos = 0;
    if (cls == 1 && !alpha) { pos = got[0] + __popc(ms & lt); P.small_list[pos] = (uint32_t)t; }
    if (cls == 1 && alpha) { pos = got[1] + __popc(ma & lt); P.small_list[P.cap_list - 1 - pos] = (uint32_t)t; }
    if (cls == 2) P.large_list[got[2] + __popc(ml & lt)] = (uint32_t)t;
    // row chunks of the small triangles
    int rows = 0, cl = 1, nch = 0;
    if (cls == 1) {
      int y0 = min(iy0, min(iy1, iy2)), y3 = max(iy0, max(iy1, iy2));
      rows = small_rows(y0, y3);
      cl = chunk_len(rows, P.min_chunk);
      nch = (rows + cl - 1) / cl;
    }
    block_items(P.items, P.cap_list * MAX_CHUNKS, P.ctr, CTR_ITEMS, CTR_ITEMS_A, pos, alpha, rows, cl, nch);
  }
}

// 512 threads: block_items sorts the row-chunk items of 512 triangles at a
// time (small raster 242 -> 234 us on the 1080p frame against 256 threads,
// same setup time; the casters' setup is faster at 256).
constexpr int SETUP_THREADS = 512;
__global__ void __launch_bounds__(SETUP_THREADS) k_setup(DrawParams P) {
  __shared__ GroupDev sg[64];
  for (int i = threadIdx.x; i < P.ngroups; i += blockDim.x) sg[i] = P.groups[i];
  __syncthreads();
  setup_phase(P, sg, blockIdx.x * blockDim.x, gridDim.x * blockDim.x);
}

// ------------------------------------------------------------ span queue

// One round of a warp: every lane queues the spans of its item's next two
// rows (row k of lane l in slot l + SLOT2 k), structure of arrays in shared
// memory, and the warp then fills their pixels cooperatively.  Two rows a
// round, not one: numbering a round's pixels costs the same for both, and
// the last, partly empty window of 32 pixels comes half as often.  Spans of
// tall thin triangles (two pixels a row) cost the most per row, and gain most.
// What bounds it is instruction issue: with the pixel body that span_put's
// ranges allow (no division, no NaN or sign case), warp instructions of the
// 1080p / 1.04M-triangle frame went 208 -> 145M and 123 -> 82M (opaque casters
// of the two cascades), 125 -> 82M (opaque small triangles), 92 -> 72M
// (alpha-tested), 49 -> 40M and 29 -> 18M (tile units), frame 1051 -> 900 us.
// A lane's second slot lies 64 bytes off its first in the banks, so that a
// window's reads (both rows of about four neighbouring lanes) do not collide.
constexpr int SLOT2 = 36, SLOTS = SLOT2 + 32;
template <bool ALPHA>
struct SpanQ {
  float4 a[SLOTS];               // cx2, d = cx1 - cx2, RN(1 / d), cz1
  float4 b[SLOTS];               // cz2, ~order (views), address and x of pixel number 0
  float4 c[ALPHA ? SLOTS : 1];   // u, v (times z) of the first end, of the second
  int g[ALPHA ? SLOTS : 1];
  int at[64];                    // rank among the round's non-empty spans -> byte offset of its a and b
};

// A lane's two rows of a round: pixel counts, address and x of the first pixel
struct RowPair {
  int cnt[2], addr[2], x[2];
};

// Interpolants (1 / depth) of an item whose vertices' z pass this stay in
// [2^-32, 2^59] on every row, so pixels need no sign or range case, and
// differences of such z are 0 or at least 2^-55, so slopes can take the
// reciprocal path.  A walk of up to `rows` = y3 - y1 additions of a slope starts
// at a vertex.  Each addition rounds by at most 2^-24 of the largest z, the slope
// (difference, quotient or reciprocal, product) by 3 x 2^-24 of it over the whole
// walk, and the split vertex's z by 4 x 2^-24, all but for factors 1 + rows 2^-24:
// together (rows + 8) 2^-24 of the largest.  That moves the SMALLEST value too, so
// it has to be at least twice that: the walk then stays above about half of it.
__device__ __forceinline__ bool z_safe(float z1, float z2, float z3, float rows) {
  const float hi = fmaxf(z1, fmaxf(z2, z3)), lo = fmaxf(0x1p-30f, hi * ((rows + 8.f) * 0x1p-23f));
  return z1 >= lo && z2 >= lo && z3 >= lo && hi <= 0x1p58f;
}

// Writes a span's ends to `slot`: first pixel lo, edges cx1 / cx2 with 1/depth
// cz1 / cz2.  `safe`: cz1, cz2 lie in [2^-60, 2^60] and |cx2|, |d| below 2^59.
// Every pixel x then takes t = span_t(x - cx2, d, RN(1/d)) -- exact when the
// operands are also not too small: |d| >= 2^-60, and |cx2| >= 2^-36 or lo > 0
// (x - cx2 is 0 or a multiple of ulp(cx2) >= 2^-59, or at least 1 - 2^-36).
// d = +-0 means the span is the one pixel lo: its n / d is an infinity of
// sign(n) xor sign(d), clamped to 1 or 0, or NaN for n = 0, clamped to 1; that
// t is fixed as cx2 = lo - 1 (t = 1) or lo + 1 (t = 0) with d = 1.
// Returns false for a span outside these ranges (real scenes almost never
// have one); the lane then draws it alone with true divisions, and the slot
// holds the true cx2 and d.
template <bool ALPHA>
__device__ __forceinline__ bool span_put(SpanQ<ALPHA> &q, int slot, bool safe, int lo, uint32_t key, float cx1,
                                         float cx2, float cz1, float cz2, V2 cu1, V2 cu2, int g) {
  const float d = cx1 - cx2, fl = (float)lo;
  const bool point = d == 0.f;
  const float n = fl - cx2;
  const bool one = n == 0.f || (int)(__float_as_uint(n) ^ __float_as_uint(d)) >= 0;
  const bool ok = safe && (point || (fabsf(d) >= 0x1p-60f && (fabsf(cx2) >= 0x1p-36f || lo > 0)));
  const float qx = ok && point ? (one ? fl - 1.f : fl + 1.f) : cx2;
  const float qd = ok && point ? 1.f : d;
  q.a[slot] = make_float4(qx, qd, recip_rn(qd), cz1);
  *reinterpret_cast<float2 *>(&q.b[slot]) = make_float2(cz2, __uint_as_float(key));
  if (ALPHA) {
    q.c[slot] = make_float4(cu1.x, cu1.y, cu2.x, cu2.y);
    q.g[slot] = g;
  }
  return ok;
}

// The second half of a slot's b: address and x of pixel number 0.
template <class Q>
__device__ __forceinline__ void span_base(Q &q, int slot, int addr, int x) {
  reinterpret_cast<int2 *>(&q.b[slot])[1] = make_int2(addr, x);
}

__device__ __forceinline__ unsigned bit_at(uint32_t k) {   // 1 << k, 0 for k >= 32
  unsigned r;
  asm("shl.b32 %0, 1, %1;" : "=r"(r) : "r"(k));
  return r;
}

// Numbers a round's pixels (lane by lane, a lane's first row before its
// second), completes the slots and calls pix(offset, p) for every pixel number
// p, lane j taking pixels j, j + 32, ...  A pixel's span is the last non-empty
// one starting at or before it: its rank is the starts before the window
// (carried along) plus those inside up to this lane (one OR-reduction of the
// start bits).  STAGED: pix returns a state whose dependent load is in
// flight, and `then(state)` consumes it after the next window's pix, so that
// the load overlaps that window's lookup and arithmetic.
template <bool STAGED, class Q, class F, class G>
__device__ __forceinline__ void fill_rows(Q &q, int lane, const RowPair &r, F &&pix, G &&then) {
  const int c0 = r.cnt[0], c1 = r.cnt[1];
  int incl = c0 + c1;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int v = __shfl_up_sync(FULL, incl, o);
    if (lane >= o) incl += v;
  }
  const int total = __shfl_sync(FULL, incl, 31);
  if (total == 0) return;
  const int pre1 = incl - c1, pre0 = pre1 - c0;
  const unsigned n0 = __ballot_sync(FULL, c0 > 0), n1 = __ballot_sync(FULL, c1 > 0), lt = (1u << lane) - 1u;
  int rank = __popc(n0 & lt) + __popc(n1 & lt);
  if (c0) {
    span_base(q, lane, r.addr[0] - pre0, r.x[0] - pre0);
    q.at[rank++] = lane * 16;
  }
  if (c1) {
    span_base(q, lane + SLOT2, r.addr[1] - pre1, r.x[1] - pre1);
    q.at[rank] = (lane + SLOT2) * 16;
  }
  __syncwarp();
  uint32_t s0 = c0 ? (uint32_t)pre0 : 0x80000000u, s1 = c1 ? (uint32_t)pre1 : 0x80000000u;
  const unsigned upto = 0xffffffffu >> (31 - lane);
  int before = -1;
  if constexpr (STAGED) {
    decltype(pix(0, 0)) cur;
    bool have = false;
    for (int p = lane; p - lane < total; p += 32, s0 -= 32, s1 -= 32) {
      unsigned starts = __reduce_or_sync(FULL, bit_at(s0) | bit_at(s1));
      int k = before + __popc(starts & upto);
      before += __popc(starts);
      decltype(pix(0, 0)) nxt;
      const bool hn = p < total;
      if (hn) nxt = pix(q.at[k], p);
      if (have) then(cur);
      cur = nxt;
      have = hn;
    }
    if (have) then(cur);
  } else {
    for (int p = lane; p - lane < total; p += 32, s0 -= 32, s1 -= 32) {
      unsigned starts = __reduce_or_sync(FULL, bit_at(s0) | bit_at(s1));
      int k = before + __popc(starts & upto);
      before += __popc(starts);
      if (p < total) pix(q.at[k], p);
    }
  }
  __syncwarp();
}

template <class T>
__device__ __forceinline__ const T &span_at(const T *base, int off) {
  return *reinterpret_cast<const T *>(reinterpret_cast<const char *>(base) + off);
}

// Per-fragment visibility: the depth 1 / (interpolated 1/z), the alpha test
// (av_draw_alpha.c:80-97), then the packed depth/order atomicMin.
// Pixel number p of the span at byte offset `off` (x = p + b.w, address =
// p + b.z); the depth is positive and finite there, so its key is its bits
// with the sign set (frag_key).
template <bool ALPHA>
__device__ __forceinline__ void vis_pixel(const DrawParams &P, const GroupDev *sg, const SpanQ<ALPHA> &q, int off,
                                          int p) {
  const float4 a = span_at(q.a, off), b = span_at(q.b, off);
  float t = span_t((float)(p + __float_as_int(b.w)) - a.x, a.y, a.z), omt = 1 - t;
  float tz = recip_rn(omt * b.x + t * a.w);
  if (ALPHA) {
    const float4 c = span_at(q.c, off);
    const GroupDev &G = sg[span_at(q.g, off >> 2)];
    V2 uvi{omt * c.z + t * c.x, omt * c.w + t * c.y};
    Taps tp = make_taps(uvi, tz, G.alen, 0);
    if (!(bilerp_quad(tp, G.aquad) > 0.5f)) return;
  }
  atomicMin((unsigned long long *)&P.keys[(uint32_t)(p + __float_as_int(b.z))],
            (unsigned long long)(__float_as_uint(tz) | 0x80000000u) << 32 | __float_as_uint(b.y));
}

// The span in `slot`, drawn by its lane alone with true divisions.
template <bool ALPHA>
__device__ __noinline__ void vis_serial(uint64_t *keys, const GroupDev *sg, const SpanQ<ALPHA> &q, int slot,
                                        int cnt, int addr, int x) {
  const float4 a = q.a[slot], b = q.b[slot];
  for (int j = 0; j < cnt; j++) {
    float t = clamp_t(((float)(x + j) - a.x) / a.y);
    float tz = 1.0f / ((1 - t) * b.x + t * a.w);
    if (tz != tz) continue;
    if (ALPHA) {
      const float4 c = q.c[slot];
      const GroupDev &G = sg[q.g[slot]];
      float omt = 1 - t;
      V2 uvi{omt * c.z + t * c.x, omt * c.w + t * c.y};
      Taps tp = make_taps(uvi, tz, G.alen, 0);
      if (!(bilerp_quad(tp, G.aquad) > 0.5f)) continue;
    }
    atomicMin((unsigned long long *)&keys[(size_t)(addr + j)],
              (unsigned long long)frag_key(tz, ~__float_as_uint(b.y)));
  }
}

// vis_pixel<true> in two stages: the first takes the depth, the alpha
// footprint's weights and the order key, and issues the load of the packed
// mask quad; the second tests the bilinear alpha and resolves the word.
struct AlphaFrag {
  unsigned long long key;
  uint32_t addr;
  unsigned m;          // the packed 2 x 2 mask quad (loaded in stage one)
  float r1, r2;        // bilinear fractions
};
__device__ __forceinline__ AlphaFrag vis_alpha_first(const DrawParams &P, const GroupDev *sg, const SpanQ<true> &q,
                                                     int off, int p) {
  AlphaFrag f;
  const float4 a = span_at(q.a, off), b = span_at(q.b, off), c = span_at(q.c, off);
  float t = span_t((float)(p + __float_as_int(b.w)) - a.x, a.y, a.z), omt = 1 - t;
  float tz = recip_rn(omt * b.x + t * a.w);
  const GroupDev &G = sg[span_at(q.g, off >> 2)];
  V2 uvi{omt * c.z + t * c.x, omt * c.w + t * c.y};
  Taps tp = make_taps(uvi, tz, G.alen, 0);
  f.m = (unsigned)__ldg(G.aquad + tp.tex);
  f.r1 = tp.texr1;
  f.r2 = tp.texr2;
  f.key = (unsigned long long)(__float_as_uint(tz) | 0x80000000u) << 32 | __float_as_uint(b.y);
  f.addr = (uint32_t)(p + __float_as_int(b.z));
  return f;
}
__device__ __forceinline__ void vis_alpha_second(const DrawParams &P, const AlphaFrag &f) {
  float i1 = 1 - f.r1, i2 = 1 - f.r2;
  float ca = i1 * i2 * (float)(f.m & 1) + f.r1 * i2 * (float)((f.m >> 1) & 1) + i1 * f.r2 * (float)((f.m >> 2) & 1) +
             f.r1 * f.r2 * (float)((f.m >> 3) & 1);
  if (!(ca > 0.5f)) return;
  atomicMin((unsigned long long *)&P.keys[f.addr], f.key);
}

// STAGED: alpha-tested fragments through the two-stage pipeline (the small
// triangles' raster: 407 -> 390 us in the 1080p frame; the tiled raster,
// whose spans are at most 16 pixels, was 3 us slower with it).
template <bool ALPHA, bool STAGED = false>
__device__ __forceinline__ void vis_fill(const DrawParams &P, const GroupDev *sg, SpanQ<ALPHA> &q, int lane,
                                         const RowPair &r) {
  if constexpr (ALPHA && STAGED)
    fill_rows<true>(q, lane, r, [&](int off, int p) { return vis_alpha_first(P, sg, q, off, p); },
                    [&](const AlphaFrag &f) { vis_alpha_second(P, f); });
  else
    fill_rows<false>(q, lane, r, [&](int off, int p) { vis_pixel<ALPHA>(P, sg, q, off, p); }, [](int) {});
}

// ------------------------------------------------------------ small triangles

template <bool ALPHA>
struct SmallLane {
  int g;
  bool safe;       // z_safe of its vertices and rows
  uint32_t gtri;
  int x1, x2, x3, y1, y2, y3;
  float z1, z2, z3, x4, z4;
  V2 uv1, uv2, uv3, uv4;
  int half, cy;
  float s1, s2, sz1, sz2, cx1, cx2, cz1, cz2;
  V2 su1, su2, cu1, cu2;

  __device__ __forceinline__ void start_half0() {
    half = 0;
    float yd = recip_rn((float)(y2 - y1));   // (y2 == y1: the half is one row, its slopes are not used)
    s1 = (float)(x2 - x1) * yd;
    s2 = (x4 - (float)x1) * yd;
    sz1 = (z2 - z1) * yd;
    sz2 = (z4 - z1) * yd;
    cx1 = cx2 = (float)x1;
    cz1 = cz2 = z1;
    if (ALPHA) {
      su1 = mul2(sub2(uv2, uv1), yd);
      su2 = mul2(sub2(uv4, uv1), yd);
      cu1 = cu2 = uv1;
    }
    if (s1 < s2) {
      float t = s1; s1 = s2; s2 = t;
      t = sz1; sz1 = sz2; sz2 = t;
      if (ALPHA) { V2 tv = su1; su1 = su2; su2 = tv; }
    }
    cy = y1;
  }
  // The second half's slopes are computed at set-up (see ShadowLane), so
  // that reaching the middle row during the walk costs a few copies.
  float hs1, hs2, hsz1, hsz2;
  V2 hsu1, hsu2;
  __device__ __forceinline__ void half1_slopes() {
    float yd = recip_rn((float)(y3 - y2));
    hs1 = (float)(x3 - x2) * yd;
    hs2 = ((float)x3 - x4) * yd;
    hsz1 = (z3 - z2) * yd;
    hsz2 = (z3 - z4) * yd;
    if (ALPHA) {
      hsu1 = mul2(neg2(sub2(uv2, uv3)), yd);
      hsu2 = mul2(neg2(sub2(uv4, uv3)), yd);
    }
    if (hs1 < hs2) {
      float t = hs1; hs1 = hs2; hs2 = t;
      t = hsz1; hsz1 = hsz2; hsz2 = t;
      if (ALPHA) { V2 tv = hsu1; hsu1 = hsu2; hsu2 = tv; }
    }
    // the second half walks upwards and subtracts its slopes: a - b is
    // a + (-b) exactly, so both halves advance by the same additions
    hs1 = -hs1; hs2 = -hs2; hsz1 = -hsz1; hsz2 = -hsz2;
    if (ALPHA) { hsu1 = neg2(hsu1); hsu2 = neg2(hsu2); }
  }
  __device__ __forceinline__ void start_half1() {
    half = 1;
    s1 = hs1; s2 = hs2; sz1 = hsz1; sz2 = hsz2;
    cx1 = cx2 = (float)x3;
    cz1 = cz2 = z3;
    if (ALPHA) {
      su1 = hsu1; su2 = hsu2;
      cu1 = cu2 = uv3;
    }
    cy = y3;
  }

  int left;   // rows left in this lane's chunk

  // advances one row of the current half
  __device__ __forceinline__ void step() {
    cx1 += s1; cx2 += s2; cz1 += sz1; cz2 += sz2;
    if (ALPHA) { cu1 = add2(cu1, su1); cu2 = add2(cu2, su2); }
  }
  __device__ __forceinline__ void next_row() {
    step();
    cy += half == 0 ? 1 : -1;
    if (half == 0 && cy > y2) start_half1();
  }
  // To row `first` of the walk: the additions of the half it lies in (the
  // second half starts from its own vertex, so the first one's are not needed).
  // A warp pays for its deepest chunk, so this loop holds the additions alone:
  // the caster raster of the 1080p / 1.04M-triangle scene issued 222 -> 208M
  // warp instructions, the small raster 141 -> 125M, frame 1086 -> 1051 us.
  __device__ __forceinline__ void seek(int first) {
    int n0 = y2 - y1 + 1;
    if (first >= n0) {
      start_half1();
      first -= n0;
    }
    for (int r = 0; r < first; r++) step();
    cy += half == 0 ? first : -first;
  }

  __device__ __forceinline__ void init_chunk(const DrawParams &P, const GroupDev *sg, uint32_t t, int chunk) {
    init(P, sg, t);
    int rows = small_rows(y1, y3);
    int cl = chunk_len(rows, P.min_chunk);
    int first = chunk * cl;
    left = min(cl, rows - first);
    seek(first);
  }

  __device__ __forceinline__ void init(const DrawParams &P, const GroupDev *sg, uint32_t t) {
    gtri = t;
    g = find_group(sg, P.ngroups, t);
    const GroupDev &G = sg[g];
    int tri = (int)(t - G.tri_base);
    float sx[3], sy[3], sz[3];
    project_persp(G, tri, P.view, sx, sy, sz);
    int ix[3], iy[3];
    float z[3];
    Attr<false> a[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
      ix[k] = f2i(sx[k]); iy[k] = f2i(sy[k]); z[k] = sz[k];
      if (ALPHA) a[k] = a_load<false>(G, tri, k, sz[k]);
    }
#define SW(i, j) { int ti = iy[i]; iy[i] = iy[j]; iy[j] = ti; ti = ix[i]; ix[i] = ix[j]; ix[j] = ti; \
                   float tf = z[i]; z[i] = z[j]; z[j] = tf; if (ALPHA) { Attr<false> ta = a[i]; a[i] = a[j]; a[j] = ta; } }
    if (iy[0] > iy[1]) SW(0, 1);
    if (iy[1] > iy[2]) SW(1, 2);
    if (iy[0] > iy[1]) SW(0, 1);
#undef SW
    x1 = ix[0]; x2 = ix[1]; x3 = ix[2]; y1 = iy[0]; y2 = iy[1]; y3 = iy[2];
    z1 = z[0]; z2 = z[1]; z3 = z[2];
    float hgt = (float)(y3 - y1);
    float yd = quot_fast((float)(y2 - y1), hgt, recip_rn(hgt));
    x4 = (float)x1 + yd * (float)(x3 - x1);
    z4 = z1 + yd * (z3 - z1);
    safe = z_safe(z1, z2, z3, hgt);
    if (ALPHA) {
      uv4 = add2(a[0].uv, smul2(yd, sub2(a[2].uv, a[0].uv)));
      if (G.flags & F_MIP) mip_setup<false>(a, z, true, ix, iy, nullptr, nullptr, G.tex_size, G.mip_bias);
      uv1 = a[0].uv; uv2 = a[1].uv; uv3 = a[2].uv;
    }
    half1_slopes();
    start_half0();
  }

  // writes the current row's span into `slot`, advances; returns the span's
  // pixel count and sets `live` false after the last row
  __device__ __forceinline__ int emit(const DrawParams &P, const GroupDev *sg, SpanQ<ALPHA> &q, int slot, int &addr,
                                      int &x, bool &live) {
    int cnt = 0;
    if (cy >= 0 && cy < P.view.h) {
      // the vertices are integers, so the edges are finite on every row
      int lo = max(f2i(half == 0 ? cx2 : cx1), 0);
      int hi = min(__float2int_rd(half == 0 ? cx1 : cx2), P.view.w - 1);
      cnt = hi >= lo ? hi - lo + 1 : 0;
      x = lo;
      addr = cy * P.view.w + lo;
      if (cnt && !span_put<ALPHA>(q, slot, safe, lo, ~make_order(0, gtri, half), cx1, cx2, cz1, cz2, cu1, cu2, g)) {
        vis_serial<ALPHA>(P.keys, sg, q, slot, cnt, addr, x);
        cnt = 0;
      }
    }
    next_row();
    live = --left > 0;
    return cnt;
  }
};

template <bool ALPHA>
__device__ __forceinline__ void raster_small_loop(const DrawParams &P, const GroupDev *sg, SpanQ<ALPHA> &q, int lane) {
  uint32_t n = P.ctr[ALPHA ? CTR_ITEMS_A : CTR_ITEMS];
  uint32_t cap_items = P.cap_list * MAX_CHUNKS;
  const uint32_t per = claim_size(n, (uint32_t)P.claim_k, CLAIM_LEAST);
  while (true) {
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(&P.ctr[ALPHA ? CTR_WORK_SMALL_A : CTR_WORK_SMALL], per);
    base = __shfl_sync(FULL, base, 0);
    if (base >= n) break;
    SmallLane<ALPHA> L;
    bool live = (uint32_t)lane < per && base + lane < n;
    if (live) {
      uint32_t idx = base + lane;
      uint32_t item = P.items[ALPHA ? cap_items - 1 - idx : idx];
      uint32_t pos = item >> CHUNK_BITS;
      L.init_chunk(P, sg, P.small_list[ALPHA ? P.cap_list - 1 - pos : pos], (int)(item & (MAX_CHUNKS - 1)));
    }
    for (int round = 0; __any_sync(FULL, live); round++) {
      if (round == LOOP_LIMIT) {
        if (lane == 0) atomicOr(&P.ctr[CTR_LIMIT], 1u);
        break;
      }
      RowPair r = {};
      if (live) r.cnt[0] = L.emit(P, sg, q, lane, r.addr[0], r.x[0], live);
      if (live) r.cnt[1] = L.emit(P, sg, q, lane + SLOT2, r.addr[1], r.x[1], live);
      vis_fill<ALPHA, true>(P, sg, q, lane, r);
    }
  }
}

template <bool ALPHA>
__global__ void __launch_bounds__(128, ALPHA ? 6 : 8) k_raster_small(DrawParams P) {
  __shared__ GroupDev sg[64];
  __shared__ SpanQ<ALPHA> qs[4];
  for (int i = threadIdx.x; i < P.ngroups; i += blockDim.x) sg[i] = P.groups[i];
  __syncthreads();
  raster_small_loop<ALPHA>(P, sg, qs[threadIdx.x >> 5], threadIdx.x & 31);
}

// ------------------------------------------------------------ coarse binning

// coarse.c:17-125 in tile units, one tile row at a time: the bottom half's
// rows upwards, then the top half's downwards.
struct CoarseWalk {
  float x2, x3, y2, y3, x4, wcm1;
  float s1, s2, cx1, cx2, sbias, bound;
  int cy, half, guard, wc, hc;

  __device__ __forceinline__ void init(const float sx[3], const float sy[3], int wc_, int hc_) {
    float x1 = sx[0] / 16.f - 0.5f, y1 = sy[0] / 16.f - 0.5f;
    x2 = sx[1] / 16.f - 0.5f; x3 = sx[2] / 16.f - 0.5f;
    y2 = sy[1] / 16.f - 0.5f; y3 = sy[2] / 16.f - 0.5f;
    if (y1 > y2) { swap_(y1, y2); swap_(x1, x2); }
    if (y2 > y3) { swap_(y2, y3); swap_(x2, x3); }
    if (y1 > y2) { swap_(y1, y2); swap_(x1, x2); }
    x4 = (x1 + ((y2 - y1) / (y3 - y1)) * (x3 - x1));
    s1 = (x2 - x1) / (y2 - y1);
    s2 = (x4 - x1) / (y2 - y1);
    cx1 = x1; cx2 = x1;
    if (s1 < s2) swap_(s1, s2);
    sbias = 1.f + floorf(y1) - y1;
    wc = wc_; hc = hc_; wcm1 = (float)wc - 1;
    half = 0;
    guard = 0;
    cy = f2i(floorf(y1));
    bound = ceilf(y2);
    if (y1 == y2 || !((float)cy <= bound)) top();
  }
  __device__ __forceinline__ void top() {
    half = 1;
    s1 = (x3 - x2) / (y3 - y2);
    s2 = (x3 - x4) / (y3 - y2);
    cx1 = x3; cx2 = x3;
    if (s1 < s2) swap_(s1, s2);
    sbias = y3 - floorf(y3);
    cy = f2i(ceilf(y3));
    bound = floorf(y2);
    if (y2 == y3 || !((float)cy >= bound) || guard >= 2 * LOOP_LIMIT) half = 2;
  }
  __device__ __forceinline__ bool done() const { return half == 2; }
  // the current row's tiles [first, first + n); then to the next row
  __device__ __forceinline__ void row(int &first, int &n) {
    const float dir = half == 0 ? 1.f : -1.f;          // products with -1 and a + (-b) are exact
    float mx1 = cx1 + dir * (sbias * s1), mx2 = cx2 + dir * (sbias * s2);
    if (s1 < 0) mx1 -= dir * s1;
    if (s2 > 0) mx2 -= dir * s2;
    const float hi = fminf(half == 0 ? mx1 : mx2, wcm1), lo = fmaxf(half == 0 ? mx2 : mx1, 0.f);
    n = 0;
    first = 0;
    if (cy >= 0 && cy < hc) {
      int a1 = f2i(floorf(lo));
      float hb = ceilf(hi);                            // at most wc - 1
      if ((float)a1 <= hb) n = f2i(hb) - a1 + 1;
      first = wc * cy + a1;
    }
    cx1 += dir * s1;
    cx2 += dir * s2;
    guard++;
    if (half == 0) {
      cy++;
      if (!((float)cy <= bound) || guard >= LOOP_LIMIT) top();
    } else {
      cy--;
      if (!((float)cy >= bound) || guard >= 2 * LOOP_LIMIT) half = 2;
    }
  }
};
// calls emit(tile) for every bin entry
template <class F>
__device__ __forceinline__ void coarse_walk(const float sx[3], const float sy[3], int wc, int hc, F emit) {
  CoarseWalk W;
  W.init(sx, sy, wc, hc);
  while (!W.done()) {
    int first, n;
    W.row(first, n);
    for (int k = 0; k < n; k++) emit(first + k);
  }
}

// Opaque units fill the queue from the front, alpha-tested ones from the
// back.  A lane walks its triangle's tile rows twice: to count its units (a row's
// number is known without walking its tiles), and, once the queue's room is
// reserved, row by row with the others, the warp writing each row's units
// together.  Walking every tile twice on its own lane took 30 us for the 4,329
// large triangles of the 1080p frame, this 23 us; 4 lanes a claim instead of as few
// as one saves instructions and not time.
__device__ __forceinline__ void coarse_loop(const DrawParams &P, const GroupDev *sg, int lane) {
  uint32_t n = P.ctr[CTR_LARGE];
  int wc = P.view.w / TILE, hc = P.view.h / TILE;
  const uint32_t per = claim_size(n, (uint32_t)P.claim_k, 1u);
  while (true) {
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(&P.ctr[CTR_WORK_LARGE], per);
    base = __shfl_sync(FULL, base, 0);
    if (base >= n) break;
    bool live = (uint32_t)lane < per && base + lane < n;
    CoarseWalk start;
    start.half = 2;
    uint32_t gt = 0;
    int cnt = 0;
    bool alpha = false;
    if (live) {
      float sx[3], sy[3], sz[3];
      gt = P.large_list[base + lane];
      const GroupDev &G = sg[find_group(sg, P.ngroups, gt)];
      alpha = (G.flags & F_ALPHA) != 0;
      project_persp(G, (int)(gt - G.tri_base), P.view, sx, sy, sz);
      start.init(sx, sy, wc, hc);
      CoarseWalk W = start;
      while (!W.done()) {
        int first, m;
        W.row(first, m);
        cnt += m;
      }
    }
    int co = alpha ? 0 : cnt, ca = alpha ? cnt : 0;
    int io = co, ia = ca;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int v = __shfl_up_sync(FULL, io, o);
      int va = __shfl_up_sync(FULL, ia, o);
      if (lane >= o) { io += v; ia += va; }
    }
    uint32_t to = (uint32_t)__shfl_sync(FULL, io, 31), ta = (uint32_t)__shfl_sync(FULL, ia, 31);
    // Capacity is reserved for both kinds together, so the opaque units
    // (growing from the front) and the alpha units (from the back) never
    // meet; after an overflow the fallback kernel draws every large triangle.
    uint32_t oo = 0, oa = 0, fits = 1;
    if (lane == 31 && to + ta) {
      uint32_t r = atomicAdd(&P.ctr[CTR_UNITS_RESERVED], to + ta);
      if ((uint64_t)r + to + ta > (uint64_t)P.cap_units) {
        fits = 0;
        atomicOr(&P.ctr[CTR_OVERFLOW], 1u);
      } else {
        if (to) oo = atomicAdd(&P.ctr[CTR_UNITS], to);
        if (ta) oa = atomicAdd(&P.ctr[CTR_UNITS_A], ta);
      }
    }
    fits = __shfl_sync(FULL, fits, 31);
    if (!fits) continue;
    oo = __shfl_sync(FULL, oo, 31) + (uint32_t)(io - co);
    oa = __shfl_sync(FULL, oa, 31) + (uint32_t)(ia - ca);
    // position of the lane's next unit, and whether positions run downwards
    uint32_t at = alpha ? P.cap_units - 1 - oa : oo;
    while (__any_sync(FULL, !start.done())) {
      int first = 0, m = 0;
      if (!start.done()) start.row(first, m);
      for (unsigned todo = __ballot_sync(FULL, m > 0); todo; todo &= todo - 1) {
        const int src = __ffs(todo) - 1;
        const int f = __shfl_sync(FULL, first, src), c = __shfl_sync(FULL, m, src);
        const uint32_t p = __shfl_sync(FULL, at, src), g = __shfl_sync(FULL, gt, src);
        const bool down = __shfl_sync(FULL, (int)alpha, src) != 0;
        for (int k = lane; k < c; k += 32) P.units[down ? p - k : p + k] = make_uint2(g, (uint32_t)(f + k));
      }
      at = alpha ? at - m : at + m;
    }
  }
}

__global__ void __launch_bounds__(128) k_coarse(DrawParams P) {
  __shared__ GroupDev sg[64];
  for (int i = threadIdx.x; i < P.ngroups; i += blockDim.x) sg[i] = P.groups[i];
  __syncthreads();
  coarse_loop(P, sg, threadIdx.x & 31);
}

// ------------------------------------------------------------ tiled (large) raster

template <bool ALPHA>
struct TileLane {
  int g;
  uint32_t gtri;
  float x1, x2, x3, y1, y2, y3, z1, z2, z3, x4, z4;
  V2 uv1, uv2, uv3, uv4;
  float xMin, xMax, yMin, yMax;
  int half, cy;
  bool live_half;
  float ybound;
  float s1, s2, sz1, sz2, cx1, cx2, cz1, cz2;
  V2 su1, su2, cu1, cu2;

  __device__ __forceinline__ void start_half0() {
    half = 0;
    float yd = 1.0f / (y2 - y1);
    s1 = (x2 - x1) * yd;
    s2 = (x4 - x1) * yd;
    sz1 = (z2 - z1) * yd;
    sz2 = (z4 - z1) * yd;
    if (ALPHA) { su1 = mul2(sub2(uv2, uv1), yd); su2 = mul2(sub2(uv4, uv1), yd); }
    if (s1 < s2) {
      float t = s1; s1 = s2; s2 = t;
      t = sz1; sz1 = sz2; sz2 = t;
      if (ALPHA) { V2 tv = su1; su1 = su2; su2 = tv; }
    }
    cy = f2i(clampf_(y1, yMin, yMax));
    float dy = (float)cy - y1;
    cx1 = x1 + dy * s1; cx2 = x1 + dy * s2;
    cz1 = z1 + dy * sz1; cz2 = z1 + dy * sz2;
    if (ALPHA) { cu1 = add2(uv1, smul2(dy, su1)); cu2 = add2(uv1, smul2(dy, su2)); }
    ybound = clampf_(y2, yMin, yMax);
    live_half = (y2 > yMin) && ((float)cy <= ybound);
  }
  // The second half's slopes are computed at set-up (see ShadowLane), so
  // that the lanes reaching the middle row during the walk do less while
  // the others wait.
  float hs1, hs2, hsz1, hsz2;
  V2 hsu1, hsu2;
  __device__ __forceinline__ void half1_slopes() {
    float yd = 1.0f / (y3 - y2);
    hs1 = (x3 - x2) * yd;
    hs2 = (x3 - x4) * yd;
    hsz1 = (z3 - z2) * yd;
    hsz2 = (z3 - z4) * yd;
    if (ALPHA) { hsu1 = mul2(neg2(sub2(uv2, uv3)), yd); hsu2 = mul2(neg2(sub2(uv4, uv3)), yd); }
    if (hs1 < hs2) {
      float t = hs1; hs1 = hs2; hs2 = t;
      t = hsz1; hsz1 = hsz2; hsz2 = t;
      if (ALPHA) { V2 tv = hsu1; hsu1 = hsu2; hsu2 = tv; }
    }
  }
  __device__ __forceinline__ void start_half1() {
    half = 1;
    s1 = hs1; s2 = hs2; sz1 = hsz1; sz2 = hsz2;
    if (ALPHA) { su1 = hsu1; su2 = hsu2; }
    cy = f2i(clampf_(y3, yMin, yMax));
    float dy = (float)cy - y3;
    cx1 = x3 + dy * s1; cx2 = x3 + dy * s2;
    cz1 = z3 + dy * sz1; cz2 = z3 + dy * sz2;
    if (ALPHA) { cu1 = add2(uv3, smul2(dy, su1)); cu2 = add2(uv3, smul2(dy, su2)); }
    s1 = -s1; s2 = -s2; sz1 = -sz1; sz2 = -sz2;      // upwards: a - b is a + (-b) exactly
    if (ALPHA) { su1 = neg2(su1); su2 = neg2(su2); }
    ybound = clampf_(y2, yMin, yMax);
    live_half = (y2 < yMax) && ((float)cy >= ybound);
  }

  // returns false if the unit has no rows at all
  __device__ __forceinline__ bool init(const DrawParams &P, const GroupDev *sg, uint2 unit) {
    gtri = unit.x;
    int bx = (int)unit.y;
    g = find_group(sg, P.ngroups, gtri);
    const GroupDev &G = sg[g];
    int tri = (int)(gtri - G.tri_base);
    float sx[3], sy[3], sz[3];
    project_persp(G, tri, P.view, sx, sy, sz);
    Attr<false> a[3];
    float x[3], y[3], z[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
      x[k] = sx[k]; y[k] = sy[k]; z[k] = sz[k];
      if (ALPHA) a[k] = a_load<false>(G, tri, k, sz[k]);
    }
#define SW(i, j) { float tf = y[i]; y[i] = y[j]; y[j] = tf; tf = x[i]; x[i] = x[j]; x[j] = tf; \
                   tf = z[i]; z[i] = z[j]; z[j] = tf; if (ALPHA) { Attr<false> ta = a[i]; a[i] = a[j]; a[j] = ta; } }
    if (y[0] > y[1]) SW(0, 1);
    if (y[1] > y[2]) SW(1, 2);
    if (y[0] > y[1]) SW(0, 1);
#undef SW
    x1 = x[0]; x2 = x[1]; x3 = x[2]; y1 = y[0]; y2 = y[1]; y3 = y[2];
    z1 = z[0]; z2 = z[1]; z3 = z[2];
    float yd = (y2 - y1) / (y3 - y1);
    x4 = x1 + yd * (x3 - x1);
    z4 = z1 + yd * (z3 - z1);
    if (ALPHA) {
      uv4 = add2(a[0].uv, smul2(yd, sub2(a[2].uv, a[0].uv)));
      if (G.flags & F_MIP) mip_setup<false>(a, z, false, nullptr, nullptr, x, y, G.tex_size, G.mip_bias);
      uv1 = a[0].uv; uv2 = a[1].uv; uv3 = a[2].uv;
    }
    int wc = P.view.w / TILE;
    int tileX = bx % wc;
    int tileY = f2i((float)bx / ((float)P.view.w / 16.f));
    xMin = (float)tileX * 16.f;
    xMax = ((float)tileX + 1.f) * 16.f - 1.f;
    yMin = (float)tileY * 16.f;
    yMax = ((float)tileY + 1.f) * 16.f - 1.f;
    half1_slopes();
    start_half0();
    if (!live_half) start_half1();
    return live_half;
  }

  // queues the row's span, or draws it with the lane alone; returns the
  // pixels queued.  The vertices are not integers here and a row may start
  // up to one row outside the triangle, so the ranges are checked by row.
  __device__ __forceinline__ int put(const DrawParams &P, const GroupDev *sg, SpanQ<ALPHA> &q, int slot, int lo,
                                     int cnt, int &addr, int &x) {
    x = lo;
    addr = cy * P.view.w + lo;
    bool safe = cz1 >= 0x1p-60f && cz2 >= 0x1p-60f && cz1 <= 0x1p60f && cz2 <= 0x1p60f && fabsf(cx2) <= 0x1p59f &&
                fabsf(cx1 - cx2) <= 0x1p59f;
    if (span_put<ALPHA>(q, slot, safe, lo, ~make_order(1, gtri, half), cx1, cx2, cz1, cz2, cu1, cu2, g)) return cnt;
    vis_serial<ALPHA>(P.keys, sg, q, slot, cnt, addr, x);
    return 0;
  }

  __device__ __forceinline__ int emit(const DrawParams &P, const GroupDev *sg, SpanQ<ALPHA> &q, int slot, int &addr,
                                      int &x, bool &live) {
    int cnt = 0;
    // the half's left and right edge; both halves advance alike (start_half1
    // negates the slopes)
    const float l = half == 0 ? cx2 : cx1, r = half == 0 ? cx1 : cx2;
    if (l < xMax && r > xMin) {
      int lo = f2i(clampf_(l, xMin, xMax));
      int hi = f2i(floorf(clampf_(r, xMin, xMax)));
      cnt = hi >= lo ? hi - lo + 1 : 0;
      if (cnt) cnt = put(P, sg, q, slot, lo, cnt, addr, x);
    }
    cx1 += s1; cx2 += s2; cz1 += sz1; cz2 += sz2;
    if (ALPHA) { cu1 = add2(cu1, su1); cu2 = add2(cu2, su2); }
    if (half == 0) {
      cy++;
      if ((float)cy > ybound) {
        start_half1();
        live = live_half;
      }
    } else {
      cy--;
      live = (float)cy >= ybound;
    }
    return cnt;
  }
};

template <bool ALPHA>
__device__ __forceinline__ void raster_tiled_loop(const DrawParams &P, const GroupDev *sg, SpanQ<ALPHA> &q, int lane) {
  if (P.ctr[CTR_OVERFLOW]) return;
  uint32_t n = P.ctr[ALPHA ? CTR_UNITS_A : CTR_UNITS];
  const uint32_t per = claim_size(n, (uint32_t)P.claim_k, CLAIM_LEAST);
  while (true) {
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(&P.ctr[ALPHA ? CTR_WORK_UNITS_A : CTR_WORK_UNITS], per);
    base = __shfl_sync(FULL, base, 0);
    if (base >= n) break;
    TileLane<ALPHA> L;
    bool live = false;
    if ((uint32_t)lane < per && base + lane < n) {
      uint32_t idx = base + lane;
      live = L.init(P, sg, P.units[ALPHA ? P.cap_units - 1 - idx : idx]);
    }
    for (int round = 0; __any_sync(FULL, live); round++) {
      if (round == LOOP_LIMIT) {
        if (lane == 0) atomicOr(&P.ctr[CTR_LIMIT], 1u);
        break;
      }
      RowPair r = {};
      if (live) r.cnt[0] = L.emit(P, sg, q, lane, r.addr[0], r.x[0], live);
      if (live) r.cnt[1] = L.emit(P, sg, q, lane + SLOT2, r.addr[1], r.x[1], live);
      vis_fill<ALPHA>(P, sg, q, lane, r);
    }
  }
}

template <bool ALPHA>
__global__ void __launch_bounds__(128, ALPHA ? 6 : 8) k_raster_tiled(DrawParams P) {
  __shared__ GroupDev sg[64];
  __shared__ SpanQ<ALPHA> qs[4];
  for (int i = threadIdx.x; i < P.ngroups; i += blockDim.x) sg[i] = P.groups[i];
  __syncthreads();
  raster_tiled_loop<ALPHA>(P, sg, qs[threadIdx.x >> 5], threadIdx.x & 31);
}

// Tile-unit queue overflow: every large triangle is rasterized here instead,
// one triangle per warp, its coarse tiles dealt round-robin to the lanes and
// each lane filling its tiles on its own (slow, same fragments).
template <bool ALPHA>
__device__ __forceinline__ void fallback_unit(const DrawParams &P, const GroupDev *sg, SpanQ<ALPHA> &q, int lane,
                                              uint32_t gt, int tile) {
  TileLane<ALPHA> L;
  bool live = L.init(P, sg, make_uint2(gt, (uint32_t)tile));
  for (int round = 0; live && round < LOOP_LIMIT; round++) {
    int addr = 0, x = 0, cnt = L.emit(P, sg, q, lane, addr, x, live);   // the lane's own slot: pixel j is x + j
    if (cnt) span_base(q, lane, addr, x);
    for (int j = 0; j < cnt; j++) vis_pixel<ALPHA>(P, sg, q, lane * 16, j);
  }
}

__device__ __forceinline__ void fallback_loop(const DrawParams &P, const GroupDev *sg, SpanQ<false> &qo, SpanQ<true> &qa,
                                              int lane, int gw, int nw) {
  if (!P.ctr[CTR_OVERFLOW]) return;
  uint32_t n = P.ctr[CTR_LARGE];
  int wc = P.view.w / TILE, hc = P.view.h / TILE;
  for (uint32_t i = gw; i < n; i += nw) {
    uint32_t gt = P.large_list[i];
    const GroupDev &G = sg[find_group(sg, P.ngroups, gt)];
    bool alpha = (G.flags & F_ALPHA) != 0;
    float sx[3], sy[3], sz[3];
    project_persp(G, (int)(gt - G.tri_base), P.view, sx, sy, sz);
    int k = 0;
    coarse_walk(sx, sy, wc, hc, [&](int tile) {
      if ((k++ & 31) != lane) return;
      if (alpha) fallback_unit<true>(P, sg, qa, lane, gt, tile);
      else fallback_unit<false>(P, sg, qo, lane, gt, tile);
    });
  }
}

__global__ void __launch_bounds__(128) k_raster_tiled_fallback(DrawParams P) {
  __shared__ GroupDev sg[64];
  __shared__ SpanQ<false> qo[4];
  __shared__ SpanQ<true> qa[4];
  for (int i = threadIdx.x; i < P.ngroups; i += blockDim.x) sg[i] = P.groups[i];
  __syncthreads();
  int w = threadIdx.x >> 5;
  fallback_loop(P, sg, qo[w], qa[w], threadIdx.x & 31, (blockIdx.x * blockDim.x + threadIdx.x) >> 5,
                (gridDim.x * blockDim.x) >> 5);
}

// ------------------------------------------------------------ shade

// double-cascade 5-tap count: av_alpha_max.c:53-84 (shDist 2)
__device__ __forceinline__ float shadow_light(const DrawParams &P, V3 p) {
  int shadow = 0;
  for (int k = 0; k < P.nsh; k++) {
    const ShadowDev &s = P.sh[k];
    int wS = s.dim / 2;
    V3 pos = sub3(p, V3{s.pos[0], s.pos[1], s.pos[2]});
    float depth = dot3(pos, V3{s.vv[0], s.vv[1], s.vv[2]});
    int sx = f2i(dot3(pos, V3{s.vv[3], s.vv[4], s.vv[5]}) * s.scale) + wS;
    int sy = f2i(dot3(pos, V3{s.vv[6], s.vv[7], s.vv[8]}) * -s.scale) + wS;
    if (sx >= 2 && sx < 2 * wS - 2 && sy >= 2 && sy < 2 * wS - 2) {
      const float *SD = s.map;
      int r = 2 * wS;
      if (__ldg(SD + r * sy + sx) < depth) shadow += 1;
      if (__ldg(SD + r * (sy + 2) + sx) < depth) shadow += 1;
      if (__ldg(SD + r * (sy - 2) + sx) < depth) shadow += 1;
      if (__ldg(SD + r * sy + (sx + 2)) < depth) shadow += 1;
      if (__ldg(SD + r * sy + (sx - 2)) < depth) shadow += 1;
    }
  }
  shadow = min(5, shadow);
  float light = (float)shadow * P.light.amb + (float)(5 - shadow);
  return light * 0.2f;
}

// One edge chain of a triangle half on some row: x, 1/depth and the attributes
// (times 1/depth).
struct EdgeState {
  float cx, cz;
  Attr<true> c;
};
constexpr int EDGE_WORDS = sizeof(EdgeState) / 4;
// A (winner, row) pair's two edge chains (an odd number of words: pairs in
// different banks)
struct RowState {
  EdgeState e[2];
  float pad_;
};
// A winner (triangle half) in one tile: its edge chains' first states there,
// their steps a row (negated for the half walked upwards: a - b is a + (-b)
// exactly), and the row they start from.
struct WinnerState {
  EdgeState start[2], step[2];
  int y0;
};
// What its pixels need of the winner itself
struct WinnerBase {
  float fmip;
  int mip, g;
};
template <bool NRM>
struct WinnerConst : WinnerBase {};
template <>
struct WinnerConst<true> : WinnerBase {
  V3 tan, bit;   // F_NORMAL: the triangle's tangent frame
};

// shader_setup of the normal-mapped sources (av_draw_normmap.c:24-38): the
// tangent frame from the sorted vertices' uv and position (times z) divided by z
// (before the round trip multiplies them back)
__device__ __forceinline__ void normal_frame(const Attr<false> a[3], const V3 p[3], const float z[3], V3 &tan,
                                             V3 &bit) {
  V2 uv1 = div2(a[0].uv, z[0]), uv2 = div2(a[1].uv, z[1]), uv3 = div2(a[2].uv, z[2]);
  V3 p1 = div3(p[0], z[0]), p2 = div3(p[1], z[1]), p3 = div3(p[2], z[2]);
  V2 dUV1 = sub2(uv2, uv1), dUV2 = sub2(uv3, uv1);
  V3 dPos1 = sub3(p2, p1), dPos2 = sub3(p3, p1);
  float rdet = 1.f / (dUV1.x * dUV2.y - dUV1.y * dUV2.x);
  tan = fast_normalize(mul3(sub3(mul3(dPos1, dUV2.y), mul3(dPos2, dUV1.y)), rdet));
  bit = fast_normalize(mul3(sub3(mul3(dPos2, dUV1.x), mul3(dPos1, dUV2.x)), rdet));
}

// Eight threads set winner `ord` up for the tile of row cy, once for all its
// rows and pixels there.  Each projects and orders the vertices; thread j
// then takes one attribute (j >> 1: uv with the edge itself, light, normal,
// position) along one edge (j & 1: to the middle vertex or to the split
// vertex), as the rasterizer's walk has it: the difference of the ends scaled
// by 1 / rows, for the half walked upwards with the vertices exchanged.  Thread
// 0 also takes the mip level, the group and (NRM, F_NORMAL groups) the tangent
// frame.  NRM = false: draws without normal-mapped groups, whose shade then
// carries none of that code.  PAIR: two threads set up the (winner, row) pair of
// row cy instead, each all attributes along one edge, and make the additions up
// to that row themselves.
template <bool NRM, bool PAIR>
__device__ __forceinline__ void winner_setup(const DrawParams &P, const GroupDev *sg, uint32_t ord, int cy, int j,
                                             WinnerState &w, RowState &rs, WinnerConst<NRM> &wc) {
  const int k = j & 1;
  int role = j >> 1;
  const uint32_t o = ord - 1;
  const bool tiled = (o >> 31) != 0, up = (o & 1) != 0;
  const uint32_t gtri = (o >> 1) & 0x3fffffffu;
  const int g = find_group(sg, P.ngroups, gtri);
  const GroupDev &G = sg[g];
  const int tri = (int)(gtri - G.tri_base);
  // a role's attribute of vertices p0, p1, p2
  auto load = [&](V3 a[3], int role, int p0, int p1, int p2) {
    const float *src = role == 0 ? G.uv : role == 1 ? G.li : role == 2 ? G.vn : G.xyz;
    const int n = role == 0 ? 2 : 3, p[3] = {p0, p1, p2};
    src += (size_t)tri * 3 * n;
#pragma unroll
    for (int i = 0; i < 3; i++)
      a[i] = V3{__ldg(src + p[i] * n), __ldg(src + p[i] * n + 1), role == 0 ? 0.f : __ldg(src + p[i] * n + 2)};
  };
  V3 a[3];                       // the thread's attribute, in vertex order below
  load(a, role, 0, 1, 2);
  float x[3], y[3], z[3];
  project_persp(G, tri, P.view, x, y, z);
  int ix[3] = {0, 0, 0}, iy[3] = {0, 0, 0}, v0[3] = {0, 1, 2};   // v0: the vertices
  if (!tiled) {
    // untiled path: integer vertices (Templates.py:230-231)
#pragma unroll
    for (int i = 0; i < 3; i++) { ix[i] = f2i(x[i]); iy[i] = f2i(y[i]); }
  }
#define SW(i, l) \
  if (tiled ? y[i] > y[l] : iy[i] > iy[l]) { swap_(x[i], x[l]); swap_(y[i], y[l]); swap_(z[i], z[l]); swap_(ix[i], ix[l]); \
                                             swap_(iy[i], iy[l]); swap_(a[i], a[l]); swap_(v0[i], v0[l]); }
  SW(0, 1)
  SW(1, 2)
  SW(0, 1)
#undef SW
#pragma unroll
  for (int i = 0; i < 3; i++) {
    a[i] = mul3(a[i], z[i]);
    if (!tiled) x[i] = (float)ix[i];
  }
  // heights and x differences: of the integers on the untiled path
  float h21, h32, h31, x21, x32, x31;
  if (tiled) {
    h21 = y[1] - y[0]; h32 = y[2] - y[1]; h31 = y[2] - y[0];
    x21 = x[1] - x[0]; x32 = x[2] - x[1]; x31 = x[2] - x[0];
  } else {
    h21 = (float)(iy[1] - iy[0]); h32 = (float)(iy[2] - iy[1]); h31 = (float)(iy[2] - iy[0]);
    x21 = (float)(ix[1] - ix[0]); x32 = (float)(ix[2] - ix[1]); x31 = (float)(ix[2] - ix[0]);
  }
  const float yd = h21 / h31;
  const float x4 = x[0] + yd * x31, z4 = z[0] + yd * (z[2] - z[0]);
  const bool mip = (G.flags & F_MIP) != 0, normal = NRM && (G.flags & F_NORMAL) != 0;
  if (j == 0) {
    wc.g = g;
    wc.fmip = 0.f;
    wc.mip = 0;
    Attr<false> uv[3];
#pragma unroll
    for (int i = 0; i < 3; i++) uv[i].uv = V2{a[i].x, a[i].y};
    if constexpr (NRM)
      if (normal) {
        const float *xyz = G.xyz + (size_t)tri * 9;
        V3 p[3] = {mul3(ld3(xyz + 3 * v0[0]), z[0]), mul3(ld3(xyz + 3 * v0[1]), z[1]), mul3(ld3(xyz + 3 * v0[2]), z[2])};
        normal_frame(uv, p, z, wc.tan, wc.bit);
      }
    if (mip) {
      MipSel ms = mip_setup<false>(uv, z, !tiled, ix, iy, x, y, G.tex_size, G.mip_bias);
      wc.fmip = ms.fmip;
      wc.mip = ms.mip;
    }
  }
  // the half's first vertex, its slopes to the middle and to the split vertex
  const float d = 1.0f / (up ? h32 : h21);
  const float xs = up ? x[2] : x[0], ys = up ? y[2] : y[0], zs = up ? z[2] : z[0];
  const float s1 = (up ? x32 : x21) * d, s2 = (up ? x[2] - x4 : x4 - x[0]) * d;
  const float sz = (k ? (up ? z[2] - z4 : z4 - z[0]) : (up ? z[2] - z[1] : z[1] - z[0])) * d, s = k ? s2 : s1;
  const float yMin = (float)(cy / TILE) * 16.f;
  const int cy0 = tiled ? f2i(clampf_(ys, yMin, yMin + 15.f)) : (up ? iy[2] : iy[0]);
  const float dy = (float)cy0 - ys;          // tiled path: restarted at the tile's first row
  const int e = (s1 < s2) ? 1 - k : k;       // the larger slope is the first chain's
  const int rows = iabs_(cy - cy0);
  float *st = reinterpret_cast<float *>(PAIR ? &rs.e[e] : &w.start[e]), *sp = reinterpret_cast<float *>(&w.step[e]);
  if (role == 0) {
    float cx = tiled ? xs + dy * s : xs, cz = tiled ? zs + dy * sz : zs;
    const float sx = up ? -s : s, sw = up ? -sz : sz;
    if (PAIR) {
      for (int r = rows; r > 0; r--) { cx += sx; cz += sw; }
    } else {
      sp[0] = sx;
      sp[1] = sw;
      if (k == 0) w.y0 = cy0;
    }
    st[0] = cx;
    st[1] = cz;
  }
#pragma unroll 1
  while (true) {
    if ((mip || normal) && (role == 0 || role == 3)) {   // the round trip of uv and position (mip_setup)
#pragma unroll
      for (int i = 0; i < 3; i++) a[i] = mul3(div3(a[i], z[i]), z[i]);
    }
    const V3 from = up ? a[2] : a[0], a4 = add3(a[0], smul3(yd, sub3(a[2], a[0])));
    V3 sa = sub3(k ? a4 : a[1], from);
    sa = mul3(up ? neg3(sa) : sa, d);
    V3 c = tiled ? add3(from, smul3(dy, sa)) : from;
    if (up) sa = neg3(sa);
    const int at = role == 0 ? 2 : 1 + 3 * role;
    if (PAIR) {
      for (int r = rows; r > 0; r--) c = add3(c, sa);
    } else {
      sp[at] = sa.x; sp[at + 1] = sa.y;
      if (role) sp[at + 2] = sa.z;
    }
    st[at] = c.x; st[at + 1] = c.y;
    if (role) st[at + 2] = c.z;
    if (!PAIR || ++role == 4) break;
    load(a, role, v0[0], v0[1], v0[2]);
#pragma unroll
    for (int i = 0; i < 3; i++) a[i] = mul3(a[i], z[i]);
  }
}

// The chain e of winner w on row cy: the rasterizer's additions.
__device__ __forceinline__ void replay_edge(const WinnerState &w, int e, int cy, EdgeState &out) {
  EdgeState c = w.start[e];
  const EdgeState s = w.step[e];
  for (int r = iabs_(cy - w.y0); r > 0; r--) {
    c.cx += s.cx; c.cz += s.cz;
    c.c = a_add(c.c, s.c);
  }
  out = c;
}

// av_draw_multi.c:30-105: the 4-way terrain blend of a F_MULTI group.  Its
// texture and the next three groups' (Ops0.py:533-545 binds TR[tn+1..tn+3])
// are sampled at the same bilinear taps; blend weights come from the world
// height and the normal; no shadow lookup.  The blended texel is converted
// to u16 before the lighting product, as the source does.
__device__ __forceinline__ void shade_multi(const DrawParams &P, const GroupDev *G, size_t pix, float t, float tz,
                                            V2 uvi, const RowState &st) {
  float omt = 1 - t;
  const Attr<true> &c1 = st.e[0].c, &c2 = st.e[1].c;
  Taps q = make_taps(uvi, tz, G[0].tex_size, 0);
  V3 tx[4];
#pragma unroll
  for (int k = 0; k < 4; k++) tx[k] = bilerp_rgb(q, G[k].tex);
  V3 col = mul3(add3(smul3(omt, c2.li), smul3(t, c1.li)), tz);
  V3 nrm = fast_normalize(mul3(add3(smul3(omt, c2.n), smul3(t, c1.n)), tz));
  V3 ldir{P.light.ldir[0], P.light.ldir[1], P.light.ldir[2]};
  V3 lint{P.light.lint[0], P.light.lint[1], P.light.lint[2]};
  V3 dc = smul3(fmaxf(0.f, dot3(nrm, ldir)), lint);
  V3 cpos = mul3(add3(smul3(omt, c2.p), smul3(t, c1.p)), tz);
  float m = (cpos.y - 15.f) / 4.f;
  m = fminf(fmaxf(m, 0.f), 1.f);
  float ny = fmaxf(0.f, fabsf(nrm.y) - 0.33f) * 1.5f;
  m -= 1.5f * (ny * ny - 0.4f);
  m = fminf(fmaxf(m, 0.f), 1.f);
  V3 qv = div3(cpos, 3.f);
  float threshy = 16.f + 2.f * fabsf(qv.x - roundf(qv.x)) + 2.f * fabsf(qv.z - roundf(qv.z));
  float n = fminf(fmaxf((cpos.y - threshy) / 2.f, 0.f), 4.f);
  n = n * n * n;
  n += 1.5f * (ny * ny - 0.4f);
  n = fminf(fmaxf(n, 0.f), 32.f);
  float o = fminf(fmaxf((5.f - cpos.y) / 4.f, 0.f), 1.f);
  if (m + n + o > 1.f) {   // each weight divides by the sum of the updated ones
    n = n / (n + m + o);
    m = m / (n + m + o);
    o = o / (n + m + o);
  }
  float w1 = 1 - m - n - o;
  const float light = 1;
  P.ro[pix] = u16sat((float)u16sat(m * tx[1].x + n * tx[2].x + o * tx[3].x + w1 * tx[0].x) * (light * dc.x + col.x));
  P.go[pix] = u16sat((float)u16sat(m * tx[1].y + n * tx[2].y + o * tx[3].y + w1 * tx[0].y) * (light * dc.y + col.y));
  P.bo[pix] = u16sat((float)u16sat(m * tx[1].z + n * tx[2].z + o * tx[3].z + w1 * tx[0].z) * (light * dc.z + col.z));
  P.db[pix] = tz;
}

// pown(x, n), n >= 0, by repeated squaring (the convention pinned for
// OpenCL's pown, whose rounding the device chooses)
__device__ __forceinline__ float pown_rs(float x, int n) {
  unsigned k = n < 0 ? 0u - (unsigned)n : (unsigned)n;
  float r = 1.0f, b = x;
  while (k) {
    if (k & 1u) r *= b;
    b *= b;
    k >>= 1;
  }
  return n < 0 ? 1.0f / r : r;
}

// sampleShadow of the normal-mapped sources, which the reference calls but
// defines nowhere, as this library defines it: the five taps of one cascade
// (centre, +-2 texels in x and y) at the truncated map position, counted
// where the map is nearer than `depth`, only when the centre lies in
// [2, 2 wS - 2) on both axes; the shadowed fraction is count * 0.2.
__device__ __forceinline__ float sample_shadow5(const ShadowDev &s, float depth, float sfx, float sfy) {
  int wS = s.dim / 2;
  int sx = f2i(sfx), sy = f2i(sfy), n = 0;
  if (sx >= 2 && sx < 2 * wS - 2 && sy >= 2 && sy < 2 * wS - 2) {
    const float *SD = s.map;
    int r = 2 * wS;
    if (__ldg(SD + r * sy + sx) < depth) n += 1;
    if (__ldg(SD + r * (sy + 2) + sx) < depth) n += 1;
    if (__ldg(SD + r * (sy - 2) + sx) < depth) n += 1;
    if (__ldg(SD + r * sy + (sx + 2)) < depth) n += 1;
    if (__ldg(SD + r * sy + (sx - 2)) < depth) n += 1;
  }
  return (float)n * 0.2f;
}

// bilinear normal-map texel at the taps (texi1*texi2*convert_float3(NM[tex]) + ...)
__device__ __forceinline__ V3 bilerp_nm(const Taps &q, const uchar4 *__restrict__ NM) {
  uchar4 a = __ldg(NM + q.tex), b = __ldg(NM + q.tex10), c = __ldg(NM + q.tex01), d = __ldg(NM + q.tex11);
  float w00 = q.texi1 * q.texi2, w10 = q.texr1 * q.texi2, w01 = q.texi1 * q.texr2, w11 = q.texr1 * q.texr2;
  V3 r;
  r.x = w00 * (float)a.x + w10 * (float)b.x + w01 * (float)c.x + w11 * (float)d.x;
  r.y = w00 * (float)a.y + w10 * (float)b.y + w01 * (float)c.y + w11 * (float)d.y;
  r.z = w00 * (float)a.z + w10 * (float)b.z + w01 * (float)c.z + w11 * (float)d.z;
  return r;
}

// The normal-mapped fragment cores: av_draw_normmap.c:47-149 (its alpha
// variant after the visibility pass's alpha test) and, with F_MIP,
// av_draw_normmap_mip.c:73-160.  The light comes from the draw's first
// cascade (sample_shadow5), 1 without one.  Inlined, as its arguments went
// through local memory otherwise; draws without such a material launch a shade
// without this code.
__device__ __forceinline__ void shade_normal(const DrawParams &P, const GroupDev &G, size_t pix, float t, float tz,
                                          V2 uvi, const RowState &st, const WinnerConst<true> &wc, MipSel ms) {
  const Attr<true> &c1 = st.e[0].c, &c2 = st.e[1].c;
  const bool mip = (G.flags & F_MIP) != 0;
  float omt = 1 - t;
  Taps q = make_taps(uvi, tz, mip ? ms.len_mip : G.tex_size, mip ? ms.start_mip : 0);
  V3 c = bilerp_rgb(q, G.tex);
  float outR = c.x, outG = c.y, outB = c.z;
  V3 tg = bilerp_nm(q, G.nm);
  if (mip) {
    Taps q2 = make_taps(uvi, tz, ms.len_mip2, ms.start_mip2);
    float ofm = 1 - ms.fmip;
    V3 cb = bilerp_rgb(q2, G.tex);
    outR = ofm * outR + ms.fmip * cb.x;
    outG = ofm * outG + ms.fmip * cb.y;
    outB = ofm * outB + ms.fmip * cb.z;
    tg = add3(smul3(ofm, tg), smul3(ms.fmip, bilerp_nm(q2, G.nm)));
  }
  float light = 1;
  if (P.nsh > 0) {
    const ShadowDev &sh = P.sh[0];
    V3 pos = sub3(mul3(add3(smul3(omt, c2.p), smul3(t, c1.p)), tz), V3{sh.pos[0], sh.pos[1], sh.pos[2]});
    float depth = dot3(pos, V3{sh.vv[0], sh.vv[1], sh.vv[2]});
    float wS = (float)(sh.dim / 2);
    float sfx = (dot3(pos, V3{sh.vv[3], sh.vv[4], sh.vv[5]}) * sh.scale) + wS;
    float sfy = (dot3(pos, V3{sh.vv[6], sh.vv[7], sh.vv[8]}) * -sh.scale) + wS;
    light = 1 - sample_shadow5(sh, depth, sfx, sfy);
  } else {
    light = 1 - 0.f;
  }
  V3 col = mul3(add3(smul3(omt, c2.li), smul3(t, c1.li)), tz);
  V3 norm = fast_normalize(mul3(add3(smul3(omt, c2.n), smul3(t, c1.n)), tz));
  tg = sub3(mul3(div3(tg, 255.f), 2.f), V3{1.f, 1.f, 1.f});
  tg = fast_normalize(tg);
  norm = fast_normalize(add3(add3(smul3(tg.z, norm), smul3(-tg.y, wc.tan)), smul3(-tg.x, wc.bit)));
  V3 vp{P.view.pos[0], P.view.pos[1], P.view.pos[2]};
  V3 lint{P.light.lint[0], P.light.lint[1], P.light.lint[2]};
  V3 ldir{P.light.ldir[0], P.light.ldir[1], P.light.ldir[2]};
  V3 pos = mul3(add3(smul3(omt, c2.p), smul3(t, c1.p)), tz);
  V3 spec;
  if (mip) {
    V3 a = sub3(pos, vp);
    V3 h = fast_normalize(add3(fast_normalize(a), ldir));
    float theta = fmaxf(0.f, dot3(h, norm));
    float mf = (float)ms.mip + ms.fmip;
    int sp = f2i(1.f * (mf * mf));
    spec = smul3(((pown_rs(theta, sp) * 256.f) * light) * 2.f, lint);
    spec = mul3(spec, (float)(sp + 1) / (2.f * 3.1416f));
  } else {
    V3 a = fast_normalize(sub3(pos, vp));
    V3 h = fast_normalize(add3(a, ldir));
    float theta = fmaxf(0.f, dot3(h, norm));
    int sp = G.spec_pow;
    spec = smul3(((pown_rs(theta, sp) * 256.f) * 4.f) * light, lint);
    spec = mul3(spec, (float)(sp + 2) / (8.f * 3.1416f));
    a = sub3(pos, vp);
    float nd = dot3(a, norm);
    V3 refl = fast_normalize(sub3(a, smul3(2.f * nd, norm)));
    theta = fmaxf(0.f, dot3(refl, V3{0.f, 1.f, 0.f}));
    spec = add3(spec, smul3((pown_rs(theta, 2) * 128.f) * (float)(1 + G.is_metal), V3{0.1f, 0.3f, 0.5f}));
    theta = fmaxf(0.f, dot3(fast_normalize(a), refl));
    spec = add3(spec, smul3(pown_rs(theta, G.spec_pow2) * 256.f, V3{0.2f, 0.2f, 0.2f}));
    if (G.is_metal) {
      ushort4 tx = __ldg(G.tex + q.tex);
      spec.x *= (float)tx.x / 1024.f;
      spec.y *= (float)tx.y / 1024.f;
      spec.z *= (float)tx.z / 1024.f;
      light = 0.f;
      col = V3{0.f, 0.f, 0.f};
    }
  }
  V3 dc = smul3(fmaxf(0.f, dot3(norm, ldir)), lint);
  P.ro[pix] = u16sat(spec.x + outR * (light * dc.x + col.x));
  P.go[pix] = u16sat(spec.y + outG * (light * dc.y + col.y));
  P.bo[pix] = u16sat(spec.z + outB * (light * dc.z + col.z));
  P.db[pix] = tz;
}

// Shades pixel ax of row cy from its winner's row state.
template <bool NRM = true>
__device__ __forceinline__ void shade_from_row(const DrawParams &P, const GroupDev *sg, int ax, int cy,
                                               const RowState &st, const WinnerConst<NRM> &wc) {
  const GroupDev &G = sg[wc.g];
  const bool mip = (G.flags & F_MIP) != 0;
  MipSel ms;
  ms.fmip = wc.fmip; ms.mip = wc.mip;
  ms.len_mip = 1 << ms.mip; ms.len_mip2 = ms.len_mip << 1;
  ms.start_mip = ((1 << (2 * ms.mip)) - 1) / 3;            // sum of 4^i for i < mip
  ms.start_mip2 = ms.start_mip + ms.len_mip * ms.len_mip;
  const float cx1 = st.e[0].cx, cx2 = st.e[1].cx, cz1 = st.e[0].cz, cz2 = st.e[1].cz;
  const Attr<true> &c1 = st.e[0].c, &c2 = st.e[1].c;
  float t = ((float)ax - cx2) / (cx1 - cx2);
  t = clamp_t(t);
  float tz = 1.0f / ((1 - t) * cz2 + t * cz1);
  float omt = 1 - t;
  V2 uvi = add2(smul2(omt, c2.uv), smul2(t, c1.uv));
  if (G.flags & F_MULTI) {                 // the group table clears F_MULTI on alpha-tested groups
    shade_multi(P, &G, (size_t)P.view.w * cy + ax, t, tz, uvi, st);
    return;
  }
  if constexpr (NRM)
    if (G.flags & F_NORMAL) {
      shade_normal(P, G, (size_t)P.view.w * cy + ax, t, tz, uvi, st, wc, ms);
      return;
    }
  float outR, outG, outB;
  if (mip) {
    // av_draw_normmap_mip.c:73-123
    Taps q1 = make_taps(uvi, tz, ms.len_mip, ms.start_mip);
    V3 c1v = bilerp_rgb(q1, G.tex);
    outR = c1v.x; outG = c1v.y; outB = c1v.z;
    Taps q2 = make_taps(uvi, tz, ms.len_mip2, ms.start_mip2);
    float ofm = 1 - ms.fmip;
    V3 c2v = bilerp_rgb(q2, G.tex);
    outR = ofm * outR + ms.fmip * c2v.x;
    outG = ofm * outG + ms.fmip * c2v.y;
    outB = ofm * outB + ms.fmip * c2v.z;
  } else {
    Taps q = make_taps(uvi, tz, G.tex_size, 0);
    V3 cv = bilerp_rgb(q, G.tex);
    outR = cv.x; outG = cv.y; outB = cv.z;
  }
  float light = 1;
  if (G.flags & F_SHADOW) {
    V3 p = mul3(add3(smul3(omt, c2.p), smul3(t, c1.p)), tz);
    light = shadow_light(P, p);
  }
  V3 col = mul3(add3(smul3(omt, c2.li), smul3(t, c1.li)), tz);
  V3 nrm = fast_normalize(mul3(add3(smul3(omt, c2.n), smul3(t, c1.n)), tz));
  V3 ldir{P.light.ldir[0], P.light.ldir[1], P.light.ldir[2]};
  V3 lint{P.light.lint[0], P.light.lint[1], P.light.lint[2]};
  V3 dc = smul3(fmaxf(0.f, dot3(nrm, ldir)), lint);
  float oml = 1 - light;
  size_t pix = (size_t)P.view.w * cy + ax;
  P.ro[pix] = u16sat(outR * (light * (dc.x + col.x) + oml * col.x));
  P.go[pix] = u16sat(outG * (light * (dc.y + col.y) + oml * col.y));
  P.bo[pix] = u16sat(outB * (light * (dc.z + col.z) + oml * col.z));
  P.db[pix] = tz;
}

// Shared memory of shade_tile for a block of NT threads (16 x NT/16 pixels).
constexpr int WINNERS = 32;        // winners set up at a time
// DENSE: tiles with many winners of a row or two are set up by pair.
template <int NT, bool NRM, bool DENSE>
struct ShadeSmem {
  // entries (winners, or pairs) shaded at a time: all, or with tangent frames what 48 KB hold
  static constexpr int AT_ONCE = !NRM || NT <= 128 ? NT : DENSE ? 96 : WINNERS;
  uint32_t hkey[NT];               // open-addressing table of the tile's winners (order keys)
  uint16_t hent[NT];               // its entry numbers
  uint32_t ekey[NT];               // entry -> order key
  int nent, npair;
  uint16_t pair[NT];               // (winner, row) pairs: table slot << 4 | row
  WinnerConst<NRM> wc[AT_ONCE];
  WinnerState ws[WINNERS];
  RowState rs[NT];                 // their edge chains, indexed alike
};

// Shades the 16 x (NT/16) pixels at (x0, y0) in three steps.  The block finds
// the distinct winners (triangle halves) among its pixels, through a bounded
// open-addressing table in shared memory, and their (winner, row) pairs;
// eight threads a winner set it up for the tile; two threads a pair replay its
// edge chains; then every pixel shades from its pair.  The arithmetic is the
// rasterizer's walk, the set-up done once a winner, the additions once a pair.
//
// A tile of the 1080p / 1.04M-triangle frame has 5.5 winners and 41 pairs (of
// 256 pixels).  With every pair set up by itself (projection, mip level, slopes:
// most of the kernel's instructions, on three of the block's eight warps) the
// kernel took 177 us of that frame and 95M warp instructions; set up by winner
// 149 us, with the pairs of the whole block replayed together 142 us and 71M,
// with eight threads a winner instead of two 137 us.  What is left is waiting at
// the barriers between the steps (6.9 of 14 cycles an instruction) with four
// blocks of 64 registers an SM.  8-row tiles (half the threads a block) take 12%
// longer; two or three blocks an SM 3-10%.
//
// Every pixel shades in one pass after the last winners' set-up: with a pass after
// each 32 winners a warp of a tile with many of them shaded up to eight times.  And
// where winners are nearly as many as pairs (fine meshes in small views), two
// threads a pair take fewer rounds than eight a winner (DENSE, by_pair).  k_shade with
// every pair set up by itself, by winner with a pass after each 32, now: 1.04M
// triangles at 64x48 31, 74, 33 us; at 320x192 from above 37, 81, 35; 2.9M at 640x480
// from above 75, 142, 75; 300,000 at 720p from above 109, 137, 122; from the side
// 99, 80, 78.
template <int NT, bool NRM, bool DENSE>
__device__ __forceinline__ void shade_tile(const DrawParams &P, const GroupDev *sg, int x0, int y0,
                                           ShadeSmem<NT, NRM, DENSE> &sm) {
  const int tid = threadIdx.x, lane = tid & 31;
  const int ax = x0 + (tid & 15), cy = y0 + (tid >> 4);
  const bool in = ax < P.view.w && cy < P.view.h;
  const uint32_t ord = in ? 0xffffffffu - (uint32_t)P.keys[(size_t)P.view.w * cy + ax] : 0u;
  sm.hkey[tid] = 0u;                     // 0: no winner has order 0
  if (tid == 0) sm.nent = sm.npair = 0;
  __syncthreads();
  // a row of the tile lies in one warp, so the first lane of each (winner,
  // row) is the pair's only one in the block
  const unsigned row = __match_any_sync(FULL, ord) & (lane < 16 ? 0xffffu : 0xffff0000u);
  const int leader = __ffs(row) - 1;
  const bool leads = ord != 0 && lane == leader;
  int slot = 0;
  if (leads) {
    uint32_t h = (ord * 2654435761u >> 16) % NT;
    for (int i = 0; i < NT; i++) {       // at most NT keys: always finds a slot
      uint32_t prev = atomicCAS(&sm.hkey[h], 0u, ord);
      if (prev == 0u) {
        int e = atomicAdd(&sm.nent, 1);
        sm.hent[h] = (uint16_t)e;
        sm.ekey[e] = ord;
      }
      if (prev == 0u || prev == ord) { slot = (int)h; break; }
      h = (h + 1) % NT;
    }
  }
  const unsigned leaders = __ballot_sync(FULL, leads);
  int first = 0;
  if (lane == 0) first = atomicAdd(&sm.npair, __popc(leaders));
  const int pair = __shfl_sync(FULL, first, 0) + __popc(leaders & ((1u << leader) - 1u));   // of this lane's pixel
  if (leads) sm.pair[pair] = (uint16_t)(slot << 4 | tid >> 4);
  __syncthreads();
  const int nw = sm.nent, npairs = sm.npair;
  sm.hkey[tid] = ord ? pair + 1u : 0u;   // (the keys are not read again) kept there, not in a register
  constexpr int AT_ONCE = ShadeSmem<NT, NRM, DENSE>::AT_ONCE;
  constexpr bool ALL = AT_ONCE == NT;    // one pass of the outer loop
  // a round of pairs costs about twice one of winners
  const bool by_pair = DENSE && (nw + WINNERS - 1) / WINNERS > 2 * ((2 * npairs + NT - 1) / NT);
  const int total = by_pair ? npairs : nw;
  for (int c0 = 0; c0 < (ALL ? 1 : total); c0 += AT_ONCE) {
    const int n = ALL ? total : min(AT_ONCE, total - c0);
    if (by_pair) {
      for (int j = tid; j < 2 * n; j += NT) {
        const int i = c0 + (j >> 1), info = sm.pair[i];
        winner_setup<NRM, true>(P, sg, sm.ekey[sm.hent[info >> 4]], y0 + (info & 15), j & 1, sm.ws[0], sm.rs[i], sm.wc[j >> 1]);
      }
      __syncthreads();
    } else {
      for (int base = c0; base < c0 + n; base += WINNERS) {
        const int m = min(WINNERS, c0 + n - base);
        for (int j = tid; j < 8 * m; j += NT)
          winner_setup<NRM, false>(P, sg, sm.ekey[base + (j >> 3)], y0, j & 7, sm.ws[j >> 3], sm.rs[0], sm.wc[base - c0 + (j >> 3)]);
        __syncthreads();
        for (int j = tid; j < 2 * npairs; j += NT) {
          const int info = sm.pair[j >> 1], w = (int)sm.hent[info >> 4] - base;
          if ((unsigned)w < (unsigned)m) replay_edge(sm.ws[w], j & 1, y0 + (info & 15), sm.rs[j >> 1].e[j & 1]);
        }
        __syncthreads();
      }
    }
    const int mine = (int)sm.hkey[tid] - 1;
    if (mine >= 0) {
      const int w = (by_pair ? mine : (int)sm.hent[sm.pair[mine] >> 4]) - c0;
      if (ALL || (unsigned)w < (unsigned)n)
        shade_from_row<NRM>(P, sg, x0 + (tid & 15), y0 + (tid >> 4), sm.rs[mine], sm.wc[w]);
    }
    __syncthreads();                     // the next entries (or the next tile) reuse the shared memory
  }
}

// one 256-thread block per 16x16 tile
// NRM: the draw has normal-mapped groups
template <bool NRM, bool DENSE>
__global__ void __launch_bounds__(256, 4) k_shade(DrawParams P) {   // 64 registers: 4 blocks per SM
  __shared__ GroupDev sg[64];
  __shared__ ShadeSmem<256, NRM, DENSE> sm;
  for (int i = threadIdx.x; i < P.ngroups; i += blockDim.x) sg[i] = P.groups[i];
  if (P.host_ctr && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x < CTR_N)
    P.host_ctr[threadIdx.x] = P.ctr[threadIdx.x];     // final: every kernel that counts has finished
  __syncthreads();
  shade_tile<256, NRM, DENSE>(P, sg, blockIdx.x * TILE, blockIdx.y * TILE, sm);
}

__global__ void k_ids(const uint64_t *__restrict__ keys, int n, int32_t *tri_id, uint8_t *cov) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    uint32_t ord = 0xffffffffu - (uint32_t)keys[i];
    int32_t id = ord == 0 ? -1 : (int32_t)(((ord - 1) >> 1) & 0x3fffffffu);
    if (tri_id) tri_id[i] = id;
    if (cov) cov[i] = ord != 0;
  }
}

// ------------------------------------------------------------ shadow depth pass

struct ShadowParams {
  const GroupDev *groups;
  int ngroups;
  int total_tris;
  ShadowDev sh;
  float *map;
  float bias;
  uint32_t *list;      // opaque casters from the front, alpha-tested from the back
  uint32_t cap_list;
  uint32_t *ctr;
  uint32_t *zero;      // the next pass's counters, cleared by this one's setup; null: none
  uint32_t *items;     // row chunks of the casters, same two ends (cap_list * MAX_CHUNKS);
                       // null: one work item per caster
  int min_chunk;       // rows per chunk (at least)
  int claim_k;         // claim_size's k (0: 32 items per claim)
  // tiled pass (rec != null): one record per caster at its list position,
  // per-tile unit counts (opaque [0, ntiles), alpha [ntiles, 2 ntiles)),
  // offsets, scatter cursors and claim counters (opaque, alpha per tile),
  // the non-empty tiles in order with the prefix of their block counts, units
  uint4 *rec;          // 2 per caster: sorted vertices, z, triangle, vertex order
  uint32_t *tcnt, *toff, *tcur, *tclaim, *tord, *hpre, *units;
  uint32_t cap_units;
  int ntx, ntiles;     // tiles per side, tiles
  int slice;           // units per block of a tile: a tile with n units gets ceil(n / slice) blocks
  int sort;            // 1: each tile's units front (nearest the light) first
};

// Rows per work item of a caster (at least).  Alpha-tested casters take half:
// their fragments cost more (the mask), so they balance better over shorter
// items (an earlier build took 86 us for the 1080p scene's cascades with 6 rows
// and 102 with 12; it is 10 and 20 rows now, see LONG_ITEM).
__device__ __forceinline__ int shadow_min_chunk(const ShadowParams &S, bool alpha) {
  return alpha ? max(1, S.min_chunk >> 1) : S.min_chunk;
}

// rows = the caster's row count in the map (drawmin.c: y1..y2 up, y3..y2+1 down);
// g, ix, iy, z = its group and projected vertices (trisetupOrtho.c)
__device__ __forceinline__ void shadow_classify(const GroupDev *sg, const ShadowParams &S, int t, bool &ok, bool &alpha,
                                                int &rows, int &g, int ix[3], int iy[3], float z[3]) {
  ok = false;
  alpha = false;
  rows = 0;
  g = 0;
  if (t < S.total_tris) {
    g = find_group(sg, S.ngroups, (uint32_t)t);
    const GroupDev &G = sg[g];
    if (G.enabled) {
      ok = project_ortho(G, t - G.tri_base, S.sh, S.bias, ix, iy, z);
      alpha = (G.flags & F_ALPHA) != 0;
      rows = max(iy[0], max(iy[1], iy[2])) - min(iy[0], min(iy[1], iy[2])) + 1;
    }
  }
}

// Appends the casters of a warp to the list (opaque from the front,
// alpha-tested from the back) and their row chunks to the work items;
// returns the caster's list slot.
__device__ __forceinline__ uint32_t shadow_append(const ShadowParams &S, int t, bool ok, bool alpha, int rows,
                                                  int lane) {
  unsigned mo = __ballot_sync(FULL, ok && !alpha), ma = __ballot_sync(FULL, ok && alpha);
  const uint32_t want[2] = {(uint32_t)__popc(mo), (uint32_t)__popc(ma)};
  const int idx[2] = {CTR_SH_LIST, CTR_SH_LIST_A};
  uint32_t got[2];
  block_reserve<2>(want, idx, S.ctr, got);
  unsigned lt = (1u << lane) - 1;
  uint32_t pos = 0;
  if (ok && !alpha) { pos = got[0] + __popc(mo & lt); S.list[pos] = (uint32_t)t; }
  if (ok && alpha) { pos = got[1] + __popc(ma & lt); S.list[S.cap_list - 1 - pos] = (uint32_t)t; }
  uint32_t slot = alpha ? S.cap_list - 1 - pos : pos;
  if (!S.items) return slot;
  // row chunks of the casters, as for the small triangles of the view
  int cl = 1, nch = 0;
  if (ok) {
    cl = chunk_len(rows, shadow_min_chunk(S, alpha));
    nch = (rows + cl - 1) / cl;
  }
  block_items(S.items, S.cap_list * MAX_CHUNKS, S.ctr, CTR_SH_ITEMS, CTR_SH_ITEMS_A, pos, alpha, rows, cl, nch);
  return slot;
}

// ---- tiled shadow pass: caster records and tile binning

constexpr int STILE_LOG = 5;
constexpr int STILE = 1 << STILE_LOG;   // a map tile is STILE x STILE texels
constexpr int TROW = STILE + 1;         // row stride of a tile in shared memory (rows in different banks)
constexpr int SUB_LOG = 3;              // the tile's texel maxima are kept per 8 x 8 sub-block
constexpr int SUBS = STILE >> SUB_LOG;  // sub-blocks per tile side

// drawmin.c's vertex order: sorted by y with its three compare-and-swaps;
// perm packs which of the triangle's vertices became vertex k (2 bits each)
__device__ __forceinline__ int caster_sort(int ix[3], int iy[3], float z[3]) {
  int p0 = 0, p1 = 1, p2 = 2;
  if (iy[0] > iy[1]) { swap_(iy[0], iy[1]); swap_(ix[0], ix[1]); swap_(z[0], z[1]); swap_(p0, p1); }
  if (iy[1] > iy[2]) { swap_(iy[1], iy[2]); swap_(ix[1], ix[2]); swap_(z[1], z[2]); swap_(p1, p2); }
  if (iy[0] > iy[1]) { swap_(iy[0], iy[1]); swap_(ix[0], ix[1]); swap_(z[0], z[1]); swap_(p0, p1); }
  return p0 | (p1 << 2) | (p2 << 4);
}

__device__ __forceinline__ uint32_t pack_xy(int x, int y) { return ((uint32_t)x & 0xffffu) | ((uint32_t)y << 16); }
__device__ __forceinline__ int unpack_x(uint32_t w) { return (int)(int16_t)(w & 0xffffu); }
__device__ __forceinline__ int unpack_y(uint32_t w) { return (int)w >> 16; }

// The tiles a caster (sorted vertices) can write: rows y1..y3, and columns
// x_min..x_max widened by the drift of the accumulated edge positions (an
// addition rounds by at most |x| 2^-24, so `rows` of them stay below
// rows * X * 2^-23) and by one for the truncated split vertex x4; all
// clipped to the map.  False when nothing of the caster lies on the map.
__device__ __forceinline__ bool caster_tiles(const int x[3], int y1, int y3, int dim, int &tx0, int &tx1, int &ty0,
                                             int &ty1) {
  if (!(y1 < dim && y3 >= 0)) return false;
  int mn = min(x[0], min(x[1], x[2])), mx = max(x[0], max(x[1], x[2]));
  long long X = (long long)max(iabs_(mn), iabs_(mx)) + 2;
  long long rows = (long long)y3 - y1 + 1;
  int m = 1 + (int)((rows * X) >> 22);
  int c0 = mn - m, c1 = mx + m;
  if (c1 < 0 || c0 > dim - 1) return false;
  c0 = max(c0, 0);
  c1 = min(c1, dim - 1);
  tx0 = c0 >> STILE_LOG;
  tx1 = c1 >> STILE_LOG;
  ty0 = max(y1, 0) >> STILE_LOG;
  ty1 = min(y3, dim - 1) >> STILE_LOG;
  return true;
}

// Writes caster t's record at its list slot and, in the tiled pass, counts
// it in every tile it can write (opaque counts first, alpha-tested after them).
__device__ __forceinline__ void shadow_record(const ShadowParams &S, int t, int g, bool alpha, int ix[3], int iy[3],
                                              float z[3], uint32_t slot) {
  int perm = caster_sort(ix, iy, z);
  S.rec[2 * (size_t)slot] = make_uint4(pack_xy(ix[0], iy[0]), pack_xy(ix[1], iy[1]), pack_xy(ix[2], iy[2]),
                                       __float_as_uint(z[0]));
  S.rec[2 * (size_t)slot + 1] = make_uint4(__float_as_uint(z[1]), __float_as_uint(z[2]), (uint32_t)t,
                                           (uint32_t)perm | ((uint32_t)g << 8));
  int tx0, tx1, ty0, ty1;
  if (!S.tcnt || !caster_tiles(ix, iy[0], iy[2], S.sh.dim, tx0, tx1, ty0, ty1)) return;
  const uint32_t base = alpha ? (uint32_t)S.ntiles : 0u;
  for (int ty = ty0; ty <= ty1; ty++)
    for (int tx = tx0; tx <= tx1; tx++) {
      // lanes counting into the same tile add once (casters crowd into few tiles)
      uint32_t key = base + (uint32_t)(ty * S.ntx + tx);
      unsigned peers = __match_any_sync(__activemask(), key);
      if ((threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&S.tcnt[key], (uint32_t)__popc(peers));
    }
}

__device__ __forceinline__ void shadow_setup_phase(const ShadowParams &S, const GroupDev *sg, int first, int step) {
  int lane = threadIdx.x & 31;
  for (int base = first; base < S.total_tris; base += step) {
    int t = base + threadIdx.x;
    bool ok, alpha;
    int rows, g, ix[3], iy[3];
    float z[3];
    shadow_classify(sg, S, t, ok, alpha, rows, g, ix, iy, z);
    uint32_t slot = shadow_append(S, t, ok, alpha, rows, lane);
    if (S.rec && ok) shadow_record(S, t, g, alpha, ix, iy, z, slot);
  }
}

template <int N>
__global__ void __launch_bounds__(256, 6) k_shadow_setup(ShadowParams S, const __grid_constant__ GroupTab<N> tab,
                                                      GroupDev *dst) {
  __shared__ GroupDev sg[N];
  for (int i = threadIdx.x; i < S.ngroups; i += blockDim.x) sg[i] = tab.g[i];
  if (blockIdx.x == 0) {
    store_table(tab, dst, S.ngroups);
    if (S.zero && threadIdx.x < CTR_N) S.zero[threadIdx.x] = 0;
  }
  __syncthreads();
  shadow_setup_phase(S, sg, blockIdx.x * blockDim.x, gridDim.x * blockDim.x);
}

__device__ __forceinline__ void atomic_min_depth(float *addr, float v) {
  if (v >= 0.f) atomicMin((int *)addr, __float_as_int(v));
  else atomicMax((unsigned int *)addr, __float_as_uint(v));
}

// The texel test of the tiled pass.  Every pixel of a span stores
// tz = RN(1 / v), v = RN(RN((1 - t) cz2) + RN(t cz1)), t in [0, 1]; when cz1
// and cz2 are positive, v <= max(cz1, cz2) (1 + 2^-24)^3, so tz stays above
// (1 / max) (1 - 2^-22).  The returned threshold is one more than the bits
// of a float below that (an approximate reciprocal, within 2 ulp, taken
// down by 2^-18): a texel whose bits are smaller already holds a depth no
// pixel of the span undercuts, so its min update would change nothing.
// Spans whose ends are not positive and within [2^-60, 2^60] get INT_MIN,
// which no texel is below.  (A NaN end makes every pixel's depth NaN, which
// is never stored.)
__device__ __forceinline__ int depth_floor_bits(float cz1, float cz2) {
  float hi = fmaxf(cz1, cz2), lo = fminf(cz1, cz2);
  if (!(lo > 0.f) || !(hi >= 0x1p-60f) || !(hi <= 0x1p60f)) return INT_MIN;
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(hi));
  return __float_as_int(__fmul_rn(r, 1.0f - 0x1p-18f)) + 1;
}

// The mask texel of drawminalpha.c:86-96 at a pixel's uv (times z) and depth.
__device__ __forceinline__ bool mask_texel(const GroupDev &G, float u, float v, float tz) {
  int len = G.alen;
  float lm1 = (float)(len - 1);
  int t1 = f2i((u * tz) * lm1);
  t1 = iabs_(t1) & (len - 1);
  int t2 = f2i((lm1 * v) * tz);
  t2 = iabs_(t2) & (len - 1);
  return __ldg(G.amask + t1 + t2 * len) != 0;
}

// drawmin.c:71-76 for pixel number p of the span at byte offset `off`; its
// depth is positive and finite, so it orders as its bits.
__device__ __forceinline__ void shadow_pixel(float *map, const SpanQ<false> &q, int off, int p) {
  const float4 a = span_at(q.a, off), b = span_at(q.b, off);
  float t = span_t((float)(p + __float_as_int(b.w)) - a.x, a.y, a.z);
  float tz = recip_rn((1 - t) * b.x + t * a.w);
  atomicMin((int *)map + (uint32_t)(p + __float_as_int(b.z)), __float_as_int(tz));
}

// drawminalpha.c:83-97 in two stages: the first reads the texel, the second
// drops the pixel when the texel already holds a depth <= its own (most of
// them, behind the opaque casters) and looks the mask up otherwise.  Texels only
// decrease, so any value read bounds the final one.  Staged, since the read
// was what the kernel waited for (5.8 long-scoreboard cycles per issue): the
// 4K / 2.9M-triangle frame 2267 -> 2245 us, 1080p / 1.04M 887 -> 881 us.
struct CasterFrag {
  float tz, cur, t;
  int off;
  uint32_t addr;
};
__device__ __forceinline__ CasterFrag caster_first(const float *map, const SpanQ<true> &q, int off, int p) {
  const float4 a = span_at(q.a, off), b = span_at(q.b, off);
  CasterFrag f;
  f.addr = (uint32_t)(p + __float_as_int(b.z));
  f.cur = __ldcg(map + f.addr);
  f.t = span_t((float)(p + __float_as_int(b.w)) - a.x, a.y, a.z);
  f.tz = recip_rn((1 - f.t) * b.x + f.t * a.w);
  f.off = off;
  return f;
}
__device__ __forceinline__ void caster_second(float *map, const GroupDev *sg, const SpanQ<true> &q,
                                              const CasterFrag &f) {
  if (!(f.cur > f.tz)) return;
  const float4 c = span_at(q.c, f.off);
  float omt = 1 - f.t;
  if (!mask_texel(sg[span_at(q.g, f.off >> 2)], omt * c.z + f.t * c.x, omt * c.w + f.t * c.y, f.tz)) return;
  atomicMin((int *)map + f.addr, __float_as_int(f.tz));
}

// The span in `slot`, drawn by its lane alone with true divisions.
template <bool ALPHA>
__device__ __noinline__ void shadow_serial(float *map, const GroupDev *sg, const SpanQ<ALPHA> &q, int slot, int cnt,
                                           int addr, int x) {
  const float4 a = q.a[slot], b = q.b[slot];
  for (int j = 0; j < cnt; j++) {
    float t = clamp_t(((float)(x + j) - a.x) / a.y), omt = 1 - t;
    float tz = 1.0f / (omt * b.x + t * a.w);
    if (tz != tz) continue;
    if (ALPHA) {
      const float4 c = q.c[slot];
      if (!mask_texel(sg[q.g[slot]], omt * c.z + t * c.x, omt * c.w + t * c.y, tz)) continue;
    }
    atomic_min_depth(map + (size_t)(addr + j), tz);
  }
}

template <bool ALPHA>
struct ShadowLane {
  bool safe;     // z_safe of its vertices and rows
  int x1, x2, x3, y1, y2, y3, x4;
  float z1, z2, z3, z4, u1, u2, u3, u4, v1, v2, v3, v4;
  int half, cy, g;
  float s1, s2, sz1, sz2, su1, su2, sv1, sv2;
  float cx1, cx2, cz1, cz2, cu1, cu2, cv1, cv2;

  // drawmin.c divides each slope by the row count; one reciprocal serves
  // them all (the correctly rounded quotients: whole numbers for x, safe z's
  // differences, see z_safe; u and v checked one by one).  The second half's
  // slopes are computed with the first's: a lane that reaches its caster's
  // middle row during the walk then only copies them, instead of stalling the
  // warp's other lanes for the divisions.
  float hs1, hs2, hsz1, hsz2, hsu1, hsv1, hsu2, hsv2;
  __device__ __forceinline__ void slopes() {
    float d = (float)(y2 - y1), e = (float)(y3 - y2);
    if (safe) {
      float y = recip_rn(d), w = recip_rn(e);   // (d or e = 0: that half's slopes are not used)
      s1 = quot_fast((float)(x2 - x1), d, y); s2 = quot_fast((float)(x4 - x1), d, y);
      sz1 = quot_fast(z2 - z1, d, y); sz2 = quot_fast(z4 - z1, d, y);
      hs1 = quot_fast((float)(x3 - x2), e, w); hs2 = quot_fast((float)(x3 - x4), e, w);
      hsz1 = quot_fast(z3 - z2, e, w); hsz2 = quot_fast(z3 - z4, e, w);
    } else {
      s1 = (float)(x2 - x1) / d; s2 = (float)(x4 - x1) / d;
      sz1 = (z2 - z1) / d; sz2 = (z4 - z1) / d;
      hs1 = (float)(x3 - x2) / e; hs2 = (float)(x3 - x4) / e;
      hsz1 = (z3 - z2) / e; hsz2 = (z3 - z4) / e;
    }
    if (ALPHA) {
      float y = span_recip(d), w = span_recip(e);
      su1 = quot_by_recip(u2 - u1, d, y); sv1 = quot_by_recip(v2 - v1, d, y);
      su2 = quot_by_recip(u4 - u1, d, y); sv2 = quot_by_recip(v4 - v1, d, y);
      hsu1 = quot_by_recip(u3 - u2, e, w); hsv1 = quot_by_recip(v3 - v2, e, w);
      hsu2 = quot_by_recip(u3 - u4, e, w); hsv2 = quot_by_recip(v3 - v4, e, w);
    }
    if (s1 < s2) {
      swap_(s1, s2); swap_(sz1, sz2);
      if (ALPHA) { swap_(su1, su2); swap_(sv1, sv2); }
    }
    if (hs1 < hs2) {
      swap_(hs1, hs2); swap_(hsz1, hsz2);
      if (ALPHA) { swap_(hsu1, hsu2); swap_(hsv1, hsv2); }
    }
    // walked upwards by additions of the negated slopes (see SmallLane)
    hs1 = -hs1; hs2 = -hs2; hsz1 = -hsz1; hsz2 = -hsz2;
    if (ALPHA) { hsu1 = -hsu1; hsv1 = -hsv1; hsu2 = -hsu2; hsv2 = -hsv2; }
  }
  __device__ __forceinline__ void start_half0() {
    half = 0;
    cx1 = cx2 = (float)x1; cz1 = cz2 = z1;
    if (ALPHA) { cu1 = cu2 = u1; cv1 = cv2 = v1; }
    cy = y1;
  }
  __device__ __forceinline__ void start_half1() {
    half = 1;
    s1 = hs1; s2 = hs2; sz1 = hsz1; sz2 = hsz2;
    if (ALPHA) { su1 = hsu1; sv1 = hsv1; su2 = hsu2; sv2 = hsv2; }
    cx1 = cx2 = (float)x3; cz1 = cz2 = z3;
    if (ALPHA) { cu1 = cu2 = u3; cv1 = cv2 = v3; }
    cy = y3;
  }

  __device__ __forceinline__ bool init(const ShadowParams &S, const GroupDev *sg, uint32_t t) {
    g = find_group(sg, S.ngroups, t);
    const GroupDev &G = sg[g];
    int tri = (int)(t - G.tri_base);
    int ix[3], iy[3];
    float z[3];
    project_ortho(G, tri, S.sh, S.bias, ix, iy, z);
    V2 uv[3] = {V2{0, 0}, V2{0, 0}, V2{0, 0}};
    if (ALPHA) {
#pragma unroll
      for (int k = 0; k < 3; k++) uv[k] = mul2(ld2(G.uv + ((size_t)tri * 3 + k) * 2), z[k]);
    }
    if (iy[0] > iy[1]) { swap_(iy[0], iy[1]); swap_(ix[0], ix[1]); swap_(z[0], z[1]); if (ALPHA) swap_(uv[0], uv[1]); }
    if (iy[1] > iy[2]) { swap_(iy[1], iy[2]); swap_(ix[1], ix[2]); swap_(z[1], z[2]); if (ALPHA) swap_(uv[1], uv[2]); }
    if (iy[0] > iy[1]) { swap_(iy[0], iy[1]); swap_(ix[0], ix[1]); swap_(z[0], z[1]); if (ALPHA) swap_(uv[0], uv[1]); }
    x1 = ix[0]; x2 = ix[1]; x3 = ix[2]; y1 = iy[0]; y2 = iy[1]; y3 = iy[2];
    z1 = z[0]; z2 = z[1]; z3 = z[2];
    if (!((y1 < S.sh.dim) && (y3 >= 0))) return false;
    finish(uv);
    return true;
  }

  // drawmin.c:49-51 (split vertex) and the first half's slopes, from the
  // sorted vertices
  __device__ __forceinline__ void finish(const V2 uv[3]) {
    float hgt = (float)(y3 - y1);   // (0: one row, the split vertex is not used)
    float q = quot_fast((float)(y2 - y1), hgt, recip_rn(hgt));
    safe = z_safe(z1, z2, z3, hgt);
    x4 = f2i((float)x1 + q * (float)(x3 - x1));
    z4 = z1 + q * (z3 - z1);
    if (ALPHA) {
      u1 = uv[0].x; u2 = uv[1].x; u3 = uv[2].x; v1 = uv[0].y; v2 = uv[1].y; v3 = uv[2].y;
      u4 = u1 + q * (u3 - u1);
      v4 = v1 + q * (v3 - v1);
    }
    slopes();
    start_half0();
    left = y3 - y1 + 1;
  }

  // The caster of record r (the setup projected and sorted it).  Only
  // casters with rows on the map have units.
  __device__ __forceinline__ void init_rec(const ShadowParams &S, const GroupDev *sg, uint32_t r) {
    uint4 a = S.rec[2 * (size_t)r], b = S.rec[2 * (size_t)r + 1];
    x1 = unpack_x(a.x); y1 = unpack_y(a.x);
    x2 = unpack_x(a.y); y2 = unpack_y(a.y);
    x3 = unpack_x(a.z); y3 = unpack_y(a.z);
    z1 = __uint_as_float(a.w); z2 = __uint_as_float(b.x); z3 = __uint_as_float(b.y);
    g = (int)(b.w >> 8);
    V2 uv[3] = {V2{0, 0}, V2{0, 0}, V2{0, 0}};
    if (ALPHA) {
      const GroupDev &G = sg[g];
      size_t v0 = ((size_t)b.z - (size_t)G.tri_base) * 3;
      uv[0] = mul2(ld2(G.uv + (v0 + (b.w & 3)) * 2), z1);
      uv[1] = mul2(ld2(G.uv + (v0 + ((b.w >> 2) & 3)) * 2), z2);
      uv[2] = mul2(ld2(G.uv + (v0 + ((b.w >> 4) & 3)) * 2), z3);
    }
    finish(uv);
  }

  // Restricts the walk to the rows ty0..ty1 of a tile: replays the rows
  // before the first of them and leaves in `left` the rows up to the last
  // (rows outside the tile in between are skipped as they come).  The walk
  // visits bottom-half rows y1..y2 (positions 0..n0-1), then top-half rows
  // y3 down to y2 + 1.
  __device__ __forceinline__ bool clip_rows(int ty0, int ty1) {
    int n0 = y2 - y1 + 1;
    int a0 = max(y1, ty0) - y1, a1 = min(y2, ty1) - y1;
    int blo = max(y2 + 1, ty0), bhi = min(y3, ty1);
    bool ha = a0 <= a1, hb = blo <= bhi;
    if (!ha && !hb) return false;
    int first = ha ? a0 : n0 + (y3 - bhi);
    int last = hb ? n0 + (y3 - blo) : a1;
    seek(first);
    left = last - first + 1;
    return true;
  }

  int left;      // rows left in this lane's chunk (a whole caster: y3 - y1 + 1)

  // advances one row of the current half
  __device__ __forceinline__ void step() {
    cx1 += s1; cx2 += s2; cz1 += sz1; cz2 += sz2;
    if (ALPHA) { cu1 += su1; cv1 += sv1; cu2 += su2; cv2 += sv2; }
  }
  __device__ __forceinline__ void next_row() {
    step();
    cy += half == 0 ? 1 : -1;
    if (half == 0 && cy > y2) start_half1();
  }
  // to row `first` of the walk (see SmallLane)
  __device__ __forceinline__ void seek(int first) {
    int n0 = y2 - y1 + 1;
    if (first >= n0) {
      start_half1();
      first -= n0;
    }
    for (int r = 0; r < first; r++) step();
    cy += half == 0 ? first : -first;
  }

  // chunk `chunk` of the caster's rows: replays the accumulation up to its
  // first row, so every interpolant equals the serial walk's
  __device__ __forceinline__ bool init_chunk(const ShadowParams &S, const GroupDev *sg, uint32_t t, int chunk) {
    if (!init(S, sg, t)) return false;
    int rows = left;
    int cl = chunk_len(rows, shadow_min_chunk(S, ALPHA));
    int first = chunk * cl;
    if (first >= rows) return false;
    left = min(cl, rows - first);
    seek(first);
    return true;
  }

  // writes the current row's span into `slot`, advances; returns its pixels
  __device__ __forceinline__ int emit(float *map, int dim, const GroupDev *sg, SpanQ<ALPHA> &q, int slot, int &addr,
                                      int &x, bool &live) {
    int cnt = 0;
    if (cy >= 0 && cy < dim) {
      int lo = max(f2i(half == 0 ? cx2 : cx1), 0), hi = min(f2i(half == 0 ? cx1 : cx2), dim - 1);
      cnt = hi >= lo ? hi - lo + 1 : 0;
      x = lo;
      addr = cy * dim + lo;
      if (cnt && !span_put<ALPHA>(q, slot, safe, lo, 0u, cx1, cx2, cz1, cz2, V2{cu1, cv1}, V2{cu2, cv2}, g)) {
        shadow_serial<ALPHA>(map, sg, q, slot, cnt, addr, x);
        cnt = 0;
      }
    }
    next_row();
    live = --left > 0;
    return cnt;
  }

  // emit() inside a tile: the current row lies in rows ty0..ty1; its span is
  // clipped to columns tx0..tx1 and written with its texel offset in the
  // tile (row stride TROW) and its depth floor.  Then advances to the next
  // row in the tile.  A span whose depth floor lies above every texel it
  // covers (by the tile's sub-block maxima `smax`) is not queued.
  __device__ __forceinline__ int emit_tile(int *tile, const GroupDev *sg, SpanQ<ALPHA> &q, int slot, int tx0, int tx1,
                                           int ty0, int ty1, const int *smax, int &addr, int &x, bool &live) {
    int lo = max(f2i(half == 0 ? cx2 : cx1), tx0), hi = min(f2i(half == 0 ? cx1 : cx2), tx1);
    int cnt = hi >= lo ? hi - lo + 1 : 0;
    int floor_bits = 0;
    if (cnt) {
      floor_bits = depth_floor_bits(cz1, cz2);
      const int *row = smax + ((cy - ty0) >> SUB_LOG) * SUBS;
      int m = INT_MIN;
      for (int bx = (lo - tx0) >> SUB_LOG; bx <= (hi - tx0) >> SUB_LOG; bx++) m = max(m, row[bx]);
      if (m < floor_bits) cnt = 0;
    }
    x = lo;
    addr = (cy - ty0) * TROW + (lo - tx0);
    if (cnt && !span_put<ALPHA>(q, slot, safe, lo, (uint32_t)floor_bits, cx1, cx2, cz1, cz2, V2{cu1, cv1},
                                V2{cu2, cv2}, g)) {
      shadow_serial<ALPHA>(reinterpret_cast<float *>(tile), sg, q, slot, cnt, addr, x);
      cnt = 0;
    }
    next_row();
    --left;
    while (left > 0 && (cy < ty0 || cy > ty1)) {
      next_row();
      --left;
    }
    live = left > 0;
    return cnt;
  }
};

template <bool ALPHA>
__device__ __forceinline__ void shadow_warp_loop(const ShadowParams &S, const GroupDev *sg, SpanQ<ALPHA> &q, int lane,
                                                 int ctr_list, int ctr_work) {
  // work items: row chunks of the casters when S.items is given, else casters
  const bool chunked = S.items != nullptr;
  uint32_t n = chunked ? S.ctr[ALPHA ? CTR_SH_ITEMS_A : CTR_SH_ITEMS] : S.ctr[ctr_list];
  uint32_t cap_items = S.cap_list * MAX_CHUNKS;
  int dim = S.sh.dim;
  // A caster's item may be as wide as the map, and a claim of several such items is
  // one warp's chain.  The more texels the map has an item, the wider they can be:
  // fewer than 8 a claim from 1,024 texels an item.  With 8 throughout, 376
  // triangles over 4096 and 2048 cascades (4K) took 1452 us a frame, now 496; 816
  // 640, now 486; 176 over 1024 and 512 (720p) 273, now 102; 41,800 there 156, now 157.
  const uint32_t least = min(max(n / max((uint32_t)(dim * dim) / 8192u, 1u), 1u), CLAIM_LEAST);
  const uint32_t per = claim_size(n, (uint32_t)S.claim_k, least);
  while (true) {
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(&S.ctr[ctr_work], per);
    base = __shfl_sync(FULL, base, 0);
    if (base >= n) break;
    ShadowLane<ALPHA> L;
    bool live = false;
    if ((uint32_t)lane < per && base + lane < n) {
      uint32_t idx = base + lane;
      if (chunked) {
        uint32_t item = S.items[ALPHA ? cap_items - 1 - idx : idx];
        uint32_t pos = item >> CHUNK_BITS;
        live = L.init_chunk(S, sg, S.list[ALPHA ? S.cap_list - 1 - pos : pos], (int)(item & (MAX_CHUNKS - 1)));
      } else {
        live = L.init(S, sg, S.list[ALPHA ? S.cap_list - 1 - idx : idx]);
      }
    }
    for (int round = 0; __any_sync(FULL, live); round++) {
      if (round == LOOP_LIMIT) {
        if (lane == 0) atomicOr(&S.ctr[CTR_LIMIT], 1u);
        break;
      }
      RowPair r = {};
      if (live) r.cnt[0] = L.emit(S.map, dim, sg, q, lane, r.addr[0], r.x[0], live);
      if (live) r.cnt[1] = L.emit(S.map, dim, sg, q, lane + SLOT2, r.addr[1], r.x[1], live);
      if constexpr (ALPHA)
        fill_rows<true>(q, lane, r, [&](int off, int p) { return caster_first(S.map, q, off, p); },
                        [&](const CasterFrag &f) { caster_second(S.map, sg, q, f); });
      else
        fill_rows<false>(q, lane, r, [&](int off, int p) { shadow_pixel(S.map, q, off, p); }, [](int) {});
    }
  }
}

// Blocks per SM: the opaque casters fit 9 in 56 registers without spills, the
// alpha-tested ones 7 in 72 with 20 bytes of them.  With an earlier build of both
// 204 -> 199 and 84 -> 80 us per cascade against 8 and 6 blocks.
template <bool ALPHA>
__global__ void __launch_bounds__(128, ALPHA ? 7 : 9) k_shadow_raster(ShadowParams S) {
  __shared__ GroupDev sg[64];
  __shared__ SpanQ<ALPHA> qs[4];
  for (int i = threadIdx.x; i < S.ngroups; i += blockDim.x) sg[i] = S.groups[i];
  __syncthreads();
  int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  shadow_warp_loop<ALPHA>(S, sg, qs[w], lane, ALPHA ? CTR_SH_LIST_A : CTR_SH_LIST, ALPHA ? CTR_SH_WORK_A : CTR_SH_WORK);
}

}  // namespace axr
