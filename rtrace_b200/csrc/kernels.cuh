// Wavefront kernels of one render.  Per reflection depth (queue level):
//   k_trace    closest hit per queued ray (World::hit, src/ray.rs:699);
//              misses get their background/grid colour here, hits are
//              compacted into the level's hit list (warp ballot + one atomic
//              per warp)
//   k_shaft    per hit: its record (point, normal, texture coordinates), and
//              per light whether all of its shadow rays are unblocked, all
//              blocked, or a few of the scene's primitives (or more) are in
//              the way; point lights are answered here
//   k_part     the disk lights in between: the light's sample points, their
//              rays and the sum of the unblocked ones' terms, one group of
//              lanes per (hit, light)
//   k_walk     k_part's walked pairs, where a level has many
//   k_light    per hit: ambient + the lights' contributions in the
//              reference's summation order (unblocked disk lights sampled
//              here), fog, and the reflection ray, appended to the next
//              level's queue (warp ballot + one atomic per warp)
// then, deepest level first, k_fold blends reflections into their parents
// (src/lighting.rs:469-493), and k_pixels/k_outline_* produce the image.
#pragma once

#include <cuda_fp16.h>

#include "denoise.hpp"
#include "dscene.cuh"

namespace rtb {

struct RayBuf {
  double *ox, *oy, *oz, *dx, *dy, *dz;
  uint64_t* seed;
};
struct LevelBuf {
  double *r, *g, *b, *refl;
  int* child;
};
// The shading records of a chunk's hits (k_shaft), relative to the chunk.
struct HitBuf {
  double *px, *py, *pz, *nx, *ny, *nz, *u, *v;
  int* mat;  // material, and bit 30: has texture coordinates
};
// What k_shaft found for (hit, light), by pair = light * chunk_hits + hit:
// st[pair] >= 0: a few primitives are in the way, the entry of `cand` that
// holds them; else one of the codes below.  The disk lights' lit, listed and
// walked pairs are queued for k_part as {hit, light}; two lit lights of one
// diameter, whose samples share their offsets, as one entry {hit, light |
// other light << 16}.
enum { PAIR_LIT = -1, PAIR_DARK = -2, PAIR_WALK = -3 };
enum { PART_LIT = 0, PART_LIST = 1, PART_WALK = 2, PART_LIT2 = 3 };  // k_part's classes
struct PairBuf {
  int* st;
  double* sum[3];  // the light's contribution
  int* vis;        // unblocked rays
  int2* queue[4];
  int2* cand;            // RTB_CAND candidates (Cone) per listed pair
  unsigned char* ncand;
  int* n;  // queue lengths: [0, 4) of the level, [4, 8) of the fallback
};

#define RTB_MAX_LEVELS 64

struct DFrame {
  DScene S;
  DCam C;
  int W, H, S_per_px, aa, max_depth, use_kd, outline, camera_mode;
  // The frame buffers hold image rows [y0, y0 + H) of an image of height
  // Himg (a row band; y0 = 0 and H = Himg for a whole image).  Camera
  // coordinates and seeds use absolute rows.
  int y0, Himg;
  // Shadow rays per disk light at the current level, set by the host (the
  // reference casts 16), and log2 of the lanes that share a light in k_part.
  int dsamp, lanes_log2;
  int walk;  // k_walk runs at this level, where walked pairs are many
  // Learned soft shadows (extension): at level 0 each disk light gets one
  // ray, and its visibility comes from the denoiser's vhat
  // ([plane][slot][H][W], plane = sample index within the pixel).
  int learned;
  int feat_on;          // write the feature image (and vis_aov) at level 0
  __half* feat;         // [plane][H][W][FEAT_CHANNELS]
  float* vhat;          // denoised visibility, read by k_light at level 0
  float* vis_aov;       // optional: per slot visible/dsamp of level-0 hits
  int n_slots;          // disk lights that are denoiser slots (<= DN_MAX_SLOTS)
  // Confidence-gated fallback (learned shadows): for a level-0 hit whose
  // estimated visibility error (vconf, layout of vhat) exceeds conf_thr on
  // some slot, those slots are shaded by the plain path.  k_fb_select keeps
  // each hit's slot bits in fb_flag (fbn[0] counts such hits, fbn[1] their
  // slots) and queues their pairs anew for k_part launches with fb_mode set.
  float* vconf;
  float conf_thr;
  int fb_mode, fb_dsamp;
  int* fbn;
  unsigned char* fb_flag;
  uint64_t seed;
  long long n_primary;
  long long n_corner;  // quincunx corner rays, (W+1)(H+1)
  RayBuf q[2];
  int* hobj;  // per queued ray: World index of the hit, -1 miss
  int* haux;
  int* hent;
  double* ht;
  int* hit_ray;  // per hit slot: queued ray index
  LevelBuf* levels;  // device array [max_depth]
  int* counts;       // device: [0, L] queue sizes, [L+1 ..] hit counts per level
  int* nhits;        // device [max_depth]
  HitBuf hr;
  PairBuf pair;
  long long chunk_hits;  // hits whose records and pairs are held at once
  // per primary ray outline data (pobj: World index of the hit object)
  double *pdepth, *pnx, *pny, *pnz;
  unsigned char* phit;
  int* pobj;
  // per pixel
  double *cr, *cg, *cb;
  double *dep, *nx, *ny, *nz;
  int* oid;  // per pixel: object of the nearest sample (outline object-ID term), or null
  unsigned char* valid;
  double* mask;
  unsigned char* rgb;
  double* linear;  // optional pixel colours (3 per pixel) before quantisation
  unsigned long long* stats;  // [2..5] trace work, [6..9] shadow work (nodes, tris, spheres, verify)
  int* err;
  double o_wd, o_wn, o_thr, o_color[3], o_thick, o_wid;
  int o_use8, o_radius;
};

__device__ __forceinline__ int warp_alloc(int* counter, bool want) {
  unsigned m = __ballot_sync(0xffffffffu, want);
  int lane = threadIdx.x & 31;
  int base = 0;
  if (m) {
    int leader = __ffs(m) - 1;
    if (lane == leader) base = atomicAdd(counter, __popc(m));
    base = __shfl_sync(0xffffffffu, base, leader);
  }
  return want ? base + __popc(m & ((1u << lane) - 1u)) : -1;
}

__device__ __forceinline__ void warp_sum_add(unsigned long long* ctr, unsigned long long v) {
  for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
  if ((threadIdx.x & 31) == 0 && v) atomicAdd(ctr, v);
}

// slot 0: trace counters (stats[2..5]), 1: shadow counters (stats[6..9])
__device__ __forceinline__ void flush_work(const DFrame& F, const Work& w, int slot) {
  unsigned long long* b = F.stats + 2 + 4 * slot;
  warp_sum_add(b + 0, w.nodes);
  warp_sum_add(b + 1, w.tris);
  warp_sum_add(b + 2, w.spheres);
  warp_sum_add(b + 3, w.verify);
}

// --------------------------------------------------------------------------
// Camera rays
// --------------------------------------------------------------------------
// Camera::get_ray (src/camera.rs:155-167) followed by Ray::new's normalise
__device__ __forceinline__ void camera_ray(const DCam& c, double u, double v, V3* o, V3* d) {
  V3 vp = ld3(c.llc) + u * ld3(c.hor) + v * ld3(c.ver);
  if (c.persp) {
    V3 dir = normalize(vp - ld3(c.origin));
    *o = ld3(c.origin);
    *d = normalize(dir);
  } else {
    *o = vp;
    *d = normalize(ld3(c.vdir));
  }
}

// Several frames in one launch (batched small jobs): T holds the frames,
// and job j owns blocks [b0[j], b0[j + 1]) of the grid (b0[nj] = the grid
// size).  The job of this block, by binary search.
__device__ __forceinline__ int job_of_block(const int* __restrict__ b0, int nj) {
  int lo = 0, hi = nj - 1;
  const int b = (int)blockIdx.x;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (b0[mid] <= b) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}
// queue levels of a frame: max_depth clamped to [1, RTB_MAX_LEVELS]
__device__ __forceinline__ int frame_levels(const DFrame& F) {
  return F.max_depth < 1 ? 1 : (F.max_depth > RTB_MAX_LEVELS ? RTB_MAX_LEVELS : F.max_depth);
}

// Start of a frame: queue sizes and hit counts to zero except the level-0
// queue, which holds the primary rays; work counters and the error word
// cleared.  One block of 128 threads (levels <= RTB_MAX_LEVELS).  A kernel
// rather than memsets and a host copy, so that the whole frame is device
// work a CUDA graph can hold.
__device__ __forceinline__ void frame_init_body(const DFrame& F, int levels) {
  for (int i = threadIdx.x; i < levels + 2; i += blockDim.x) F.counts[i] = i == 0 ? (int)F.n_primary : 0;
  for (int i = threadIdx.x; i < levels + 1; i += blockDim.x) F.nhits[i] = 0;
  if (threadIdx.x < 16) F.stats[threadIdx.x] = 0;
  if (threadIdx.x == 0) *F.err = 0;
  if (threadIdx.x < 4 && F.fbn) F.fbn[threadIdx.x] = 0;
}
__global__ void k_frame_init(const __grid_constant__ DFrame F, int levels) { frame_init_body(F, levels); }
// one block per frame
__global__ void k_frame_init_multi(const DFrame* __restrict__ T) {
  const DFrame& F = T[blockIdx.x];
  frame_init_body(F, frame_levels(F));
}

__device__ __forceinline__ void raygen_body(const DFrame& F, int bid, int nblk) {
  const uint64_t GOLD = 0x9E3779B97F4A7C15ULL;
  long long n = F.n_primary;
  for (long long i = bid * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)nblk * blockDim.x) {
    double u, v;
    uint64_t seed;
    if (F.aa == RT_AA_QUINCUNX) {
      // render_quincunx (src/renderer.rs:752-897)
      double pw = 1.0 / (double)F.W, ph = 1.0 / (double)F.Himg;
      if (i < F.n_corner) {
        unsigned cx = (unsigned)(i % (F.W + 1)), cy = (unsigned)(F.y0 + i / (F.W + 1));
        u = rclamp((double)cx * pw, 0.0, 1.0);
        v = rclamp(1.0 - (double)cy * ph, 0.0, 1.0);
        seed = F.seed * GOLD + (uint64_t)cx + (uint64_t)cy * 0x85EBCA6BULL;
      } else {
        long long j = i - F.n_corner;
        unsigned x = (unsigned)(j % F.W), y = (unsigned)(F.y0 + j / F.W);
        u = ((double)x + 0.5) * pw;
        v = 1.0 - ((double)y + 0.5) * ph;
        seed = F.seed * GOLD + (uint64_t)x * 0x85EBCA6BULL + (uint64_t)y * 0xC2B2AE35ULL + 0x12345678ULL;
      }
    } else {
      // render_standard (src/renderer.rs:445-584)
      long long pix = i / F.S_per_px;
      unsigned s = (unsigned)(i % F.S_per_px);
      unsigned x = (unsigned)(pix % F.W), y = (unsigned)(F.y0 + pix / F.W);
      double wm1 = (double)(unsigned)(F.W - 1), hm1 = (double)(unsigned)(F.Himg - 1);
      double pu = (double)x / wm1;
      double pv = (double)(unsigned)(F.Himg - 1 - y) / hm1;
      double pwid = 1.0 / wm1, phei = 1.0 / hm1;
      uint64_t pseed = F.seed * GOLD + (uint64_t)x * 0x85EBCA6BULL + (uint64_t)y * 0xC2B2AE35ULL;
      seed = pseed + (uint64_t)s * 0x1F845FEDULL;
      if (F.aa == RT_AA_NO_JITTER) {
        u = pu;
        v = pv;
      } else {
        // The pixel's StdRng stream: sample s draws u64 number 2s and 2s+1
        // (samples == 1: numbers 0 and 1), i.e. words 4s..4s+3, which sit in
        // ChaCha block s / 4.
        uint32_t key[8], blk[16];
        pcg32_key(pseed, key);
        chacha_block(key, (uint64_t)(s >> 2), 6, blk);
        int w0 = 4 * (s & 3);
        uint64_t r0 = ((uint64_t)blk[w0 + 1] << 32) | blk[w0];
        uint64_t r1 = ((uint64_t)blk[w0 + 3] << 32) | blk[w0 + 2];
        const double scale = 1.0 / 9007199254740992.0;
        double f0 = scale * (double)(r0 >> 11), f1 = scale * (double)(r1 >> 11);
        if (F.S_per_px == 1) {
          double ju = f0 - 0.5, jv = f1 - 0.5;
          u = pu + ju * pwid;
          v = pv + jv * phei;
        } else {
          const double PI = 3.141592653589793;
          double ang = 2.0 * PI * (double)s / (double)F.S_per_px;
          double phase = f0 * 2.0 * PI;
          double ra = ang + phase;
          double rad = 0.5 * f1;
          double ju = rad * cos(ra), jv = rad * sin(ra);
          u = pu + ju * pwid;
          v = pv + jv * phei;
        }
      }
    }
    V3 o, d;
    camera_ray(F.C, u, v, &o, &d);
    RayBuf q = F.q[0];
    q.ox[i] = o.x;
    q.oy[i] = o.y;
    q.oz[i] = o.z;
    q.dx[i] = d.x;
    q.dy[i] = d.y;
    q.dz[i] = d.z;
    q.seed[i] = seed;
  }
}
__global__ void k_raygen(const __grid_constant__ DFrame F) {
  raygen_body(F, blockIdx.x, gridDim.x);
}
__global__ void k_raygen_multi(const DFrame* __restrict__ T, const int* __restrict__ b0, int nj) {
  const int j = job_of_block(b0, nj);
  const DFrame& F = T[j];
  raygen_body(F, blockIdx.x - b0[j], b0[j + 1] - b0[j]);
}


// Rays (or cones) a warp takes at a time.  A warp's walk lasts as long as its
// longest lane's, and its gathered loads as long as their slowest, so where
// the n items do not fill 16 warps of an SM each warp takes fewer, down to 4.
// Thumbnail (128x128 icosphere) 0.387 -> 0.356 ms; the 48 mixed frames of a
// batch on one lane: trace 33.5 -> 28 ms, cones 67 -> 50 (39 with a thread per
// light, SPLIT_HITS).  With 4 warps of an SM as the limit 29 and 41, with
// 32 no better, and without one the deep levels of large frames lost a third.
// Spreading frames that do fill the chip costs: the 1080p icosphere 4.49 ms
// becomes 4.73 with 24 lanes a warp, 5.02 with 16, 5.91 with 8.
// Scenes without a tree have no walks to spread.  (16 warps on each of a
// B200's 148 SMs.)
#define WALK_WARPS (16 * 148)
__device__ __forceinline__ int walk_lanes(const DScene& S, long long n, int nblk) {
  const long long warps = min((long long)nblk * (blockDim.x >> 5), (long long)WALK_WARPS);
  int lanes = 32;
  while (S.has_bvh && lanes > 4 && n <= warps * (lanes >> 1)) lanes >>= 1;
  return lanes;
}

// A step of a stage is done: a warp's rays are traced, a light's cones walked
// or a round of its samples taken.  Counted for the waits of k_levels' grid
// barrier; the stages' own launches pass no counter.
__device__ __forceinline__ void step_done(unsigned* steps) {
  if (steps && (threadIdx.x & 31) == 0) atomicAdd(steps, 1u);
}

// Level 0 walks its rays in tiles of pixels (tile_place) from this many up:
// a warp's walks then share more of their nodes.  4K terrain 11.98 -> 11.18
// ms (trace 3.48 -> 3.05, cones 3.39 -> 3.08; with tiles 16 x 2 11.52), 2560x1440
// 6.15 -> 5.76; 1,000 spheres at 4 spp 17.06 -> 17.00.  An icosphere frame is
// the same at 2560x1440 (7.45) and 4K (15.7 -> 15.6), but at 1080p it takes
// 4.56 ms against 4.48 in rows (trace 0.65 against 0.59: its hard rays lie in
// fewer warps, and few warps are active at that size as it is).
#define TILED_RAYS (3 << 20)
__device__ __forceinline__ int primary_place(const DFrame& F, int i) {
  if (F.aa != RT_AA_QUINCUNX) return (int)tile_place(i, F.W, F.H, F.S_per_px);
  if (i < F.n_corner) return (int)tile_place(i, F.W + 1, F.H + 1, 1);
  return (int)(F.n_corner + tile_place((unsigned)(i - F.n_corner), F.W, F.H, 1));
}

// --------------------------------------------------------------------------
// Closest hit + hit compaction; misses resolve to their background here.
// Bound by the latency of its node loads (17 warps of an SM active at 6
// blocks, 35% of the issue slots): 8 blocks of 128 per SM (64 registers) took
// 3.45 ms on the 4K terrain, 6 blocks 3.75, 7 3.55, 10 3.65, 12 4.9 (in rows;
// 3.05 in tiles, TILED_RAYS).
// --------------------------------------------------------------------------
template <bool COUNT>
__device__ __forceinline__ void trace_body(const DFrame& F, int level, int bid, int nblk, unsigned* steps = nullptr) {
  int n = F.counts[level];
  RayBuf q = F.q[level & 1];
  LevelBuf L = F.levels[level];
  if (bid == 0 && threadIdx.x < 8) F.pair.n[threadIdx.x] = 0;  // for this level's k_shaft
  Work w{0, 0, 0, 0};
  const int lanes = walk_lanes(F.S, n, nblk), wpb = blockDim.x >> 5, lane = threadIdx.x & 31;
  const bool tiled = level == 0 && n >= TILED_RAYS && F.S.has_bvh;
  const long long stride = (long long)nblk * wpb * lanes;
  for (long long base = ((long long)bid * wpb + (threadIdx.x >> 5)) * lanes; base < n; base += stride) {
    int i = (int)base + lane;
    const bool active = lane < lanes && i < n;
    if (tiled && active) i = primary_place(F, i);
    bool hit = false;
    WHit h{-1, 0, 0.0, -1};
    if (active) {
      V3 o = mk(q.ox[i], q.oy[i], q.oz[i]);
      V3 d = mk(q.dx[i], q.dy[i], q.dz[i]);
      RayC r;  // the object tests need no more of it
      r.o = o;
      r.d = d;
      r.dd = dot(d, d);
      h = world_closest(F.S, r, 0.001, F.use_kd != 0, F.err, COUNT ? &w : nullptr);
      hit = h.obj >= 0;
      if (!hit) {
        // ray_color_with_camera / ray_color miss branch (src/lighting.rs:497-505)
        V3 g;
        V3 c = (F.camera_mode && grid_color(F.C, o, d, &g)) ? g : ld3(F.S.bg);
        L.r[i] = c.x;
        L.g[i] = c.y;
        L.b[i] = c.z;
        L.refl[i] = 0.0;
        L.child[i] = -1;
        if (level == 0 && F.outline) F.phit[i] = 0;
      }
    }
    int slot = warp_alloc(&F.nhits[level], hit);
    if (hit) {
      F.hobj[slot] = h.obj;
      F.haux[slot] = h.aux;
      F.hent[slot] = h.ent;
      F.ht[slot] = h.t;
      F.hit_ray[slot] = i;
    }
    step_done(steps);
  }
  if (COUNT) flush_work(F, w, 0);
}
template <bool COUNT>
__global__ void __launch_bounds__(128, 8) k_trace(const __grid_constant__ DFrame F, int level) {
  trace_body<COUNT>(F, level, blockIdx.x, gridDim.x);
}
template <bool COUNT>
__global__ void __launch_bounds__(128, 8) k_trace_multi(const DFrame* __restrict__ T, const int* __restrict__ b0, int nj, int level) {
  const int j = job_of_block(b0, nj);
  const DFrame& F = T[j];
  if (level >= frame_levels(F)) return;
  trace_body<COUNT>(F, level, blockIdx.x - b0[j], b0[j + 1] - b0[j]);
}


// --------------------------------------------------------------------------
// Shading
// --------------------------------------------------------------------------
struct SMat {
  V3 c;
  double ka, kd, ks, shin;
};

// apply_texture (src/lighting.rs:9-54) + the colour parse of phong_lighting
__device__ __forceinline__ SMat effective_material(const DMat& m, const HitRec& h) {
  SMat s;
  s.c = ld3(m.color);
  s.ka = m.ambient;
  s.kd = m.diffuse;
  s.ks = m.specular;
  s.shin = m.shininess;
  if (h.has_uv) {
    if (m.texture == 1) {
      double um = fabs(rfract(h.u / m.cell_size));
      double vm = fabs(rfract(h.v / m.cell_size));
      double hw = m.half_width;
      bool onu = um <= hw || um >= (1.0 - hw);
      bool onv = vm <= hw || vm >= (1.0 - hw);
      if (onu || onv) s.c = ld3(m.grid_color);
    } else if (m.texture == 2) {
      int32_t cu = sat_i32(floor(h.u)), cv = sat_i32(floor(h.v));
      int32_t sum = (int32_t)((uint32_t)cu + (uint32_t)cv);
      if (sum % 2 != 0) {
        s.c = ld3(m.cb_color);
        s.ka = m.cb_ambient;
        s.kd = m.cb_diffuse;
        s.ks = m.cb_specular;
        s.shin = m.cb_shininess;
      }
    }
  }
  return s;
}

// diffuse + specular of one light sample (src/lighting.rs:124-141, 191-208)
__device__ __forceinline__ V3 light_term(const SMat& m, const HitRec& h, V3 ldir, V3 lc, double li, V3 view) {
  double ds = rmax(dot(h.n, ldir), 0.0);
  V3 diffuse = m.kd * ds * li * cmul(lc, m.c);
  V3 spec = mk(0.0, 0.0, 0.0);
  if (ds > 0.0) {
    // reflect(-ldir, n) before its normalisation: where the view lies
    // behind it (by more than the rounding of either dot product), the
    // clamped cosine is 0 and its power is 0
    const V3 i = -ldir;
    const V3 v = i - 2.0 * dot(i, h.n) * h.n;
    double ss = 0.0;
    if (!(dot(view, v) < -1e-10 * sum_abs(v)) || !(m.shin > 0.0)) {
      const double c = rmax(dot(view, normalize(v)), 0.0);
      ss = c > 0.0 || !(m.shin > 0.0) ? spec_pow(c, m.shin) : 0.0;
    }
    spec = m.ks * ss * li * lc;
  }
  return diffuse + spec;
}

__device__ __forceinline__ HitRec load_hit(const DFrame& F, int level, int h, RayC* rc, uint64_t* seed) {
  RayBuf q = F.q[level & 1];
  int i = F.hit_ray[h];
  V3 o = mk(q.ox[i], q.oy[i], q.oz[i]);
  V3 d = mk(q.dx[i], q.dy[i], q.dz[i]);
  *seed = q.seed[i];
  *rc = make_rayc(o, d);
  WHit w{F.hobj[h], F.haux[h], F.ht[h], F.hent[h]};
  return finalize_hit(F.S, *rc, w);
}

__device__ __forceinline__ void store_hit(const HitBuf& B, long long hl, const HitRec& h) {
  B.px[hl] = h.p.x;
  B.py[hl] = h.p.y;
  B.pz[hl] = h.p.z;
  B.nx[hl] = h.n.x;
  B.ny[hl] = h.n.y;
  B.nz[hl] = h.n.z;
  B.u[hl] = h.u;
  B.v[hl] = h.v;
  B.mat[hl] = h.mat | (h.has_uv ? 1 << 30 : 0);
}
__device__ __forceinline__ HitRec read_hit(const HitBuf& B, long long hl) {
  HitRec h;
  h.p = mk(B.px[hl], B.py[hl], B.pz[hl]);
  h.n = mk(B.nx[hl], B.ny[hl], B.nz[hl]);
  h.u = B.u[hl];
  h.v = B.v[hl];
  const int m = B.mat[hl];
  h.mat = m & ((1 << 30) - 1);
  h.has_uv = (m >> 30) & 1;
  return h;
}

// Light sampling of calculate_diffuse_light_contribution (src/lighting.rs:
// 145-217), sample_disk_light_point (:69-97), sample_disk_point (:57-66):
// the stream's seed, the same for every light of a hit, and the disk's frame.
__device__ __forceinline__ uint64_t light_seed(uint64_t seed, V3 p) {
  return seed * 0x9E3779B97F4A7C15ULL + sat_u64(p.x * 1000.0) * 0x85EBCA6BULL + sat_u64(p.y * 1000.0) * 0xC2B2AE35ULL +
         sat_u64(p.z * 1000.0) * 0x6C8E9CF5ULL;
}
struct Disk {
  V3 lp, bu, bv;
  double radius;
};
__device__ __forceinline__ Disk make_disk(const DLight& L, V3 p) {
  Disk d;
  d.lp = ld3(L.pos);
  d.radius = L.diameter / 2.0;
  const V3 cdir = normalize(d.lp - p);
  const V3 up = fabs(cdir.x) < 0.9 ? mk(1.0, 0.0, 0.0) : mk(0.0, 1.0, 0.0);
  d.bu = normalize(cross(up, cdir));
  d.bv = normalize(cross(cdir, d.bu));
  return d;
}
// The direction to the disk's point (dx, dy) and its distance: normalize(v)
// divides by norm(v), one square root for both.
__device__ __forceinline__ V3 disk_dir(const Disk& d, V3 p, double dx, double dy, double* dist) {
  const V3 sp = d.lp + dx * d.bu + dy * d.bv;
  const V3 sv = sp - p;
  *dist = norm(sv);
  return sv / *dist;
}
// The next accepted disk offset of the stream; false (and the watchdog's
// error) if 4096 attempts did not give one.
__device__ __forceinline__ bool next_offset(StdRng& rng, double radius, double* dx, double* dy, int* err) {
  for (int it = 0; it < 4096; it++) {
    if (!rng.range(-radius, radius, dx) || !rng.range(-radius, radius, dy)) break;
    if (*dx * *dx + *dy * *dy <= radius * radius) return true;
  }
  atomicOr(err, ERR_WATCHDOG);
  return false;
}

// Hit records and light classes of hits [c0, c1) of the level's hit list.
// One thread per hit, one cone per disk light (shaft_collect): where nothing
// is in the cone, which holds for most hits, the light's rays are never
// traced.  Lit, listed and walked pairs (counted with up to eight candidates a
// list and no limit on nodes): 1080p icosphere frame 90, 0.2 and 7%,
// 1,000-sphere frame 69, 15 and 0%, 4K terrain 93, 7 and 0.5%.  Walking every ray took 3.3, 21.5 and 19.1
// ms; the cones take 0.62, 3.2 and 3.1.  Bound by the latency of its node
// loads (37% of the issue slots): 8 blocks per SM (64 registers) 3.4 ms on the
// 1,000-sphere frame where 6 blocks took 3.5 and unbounded (128 registers) 4.0.
// SPLIT: up to SPLIT_HITS hits, each pair of hit and light takes a thread of its
// own, as so few hits leave warps free and a thread's lights queue up: the deep
// levels of 1,000 spheres under 40 point lights (1280x720) 8.7 -> 5.8 ms, 16
// lights 3.9 -> 2.8, 12 disk lights 12.4 -> 10.8; with twice the hits 5.6, 2.7,
// 10.7.  Level 0 of frames whose rays are far more leaves it out, and so do
// their other levels where a hit has few lights: it costs the 1,000-sphere
// frame 0.3 ms, and the learned one 0.2 on its deep levels.
#define SPLIT_HITS (1 << 16)

template <bool COUNT, bool SPLIT>
__device__ __forceinline__ void shaft_body(const DFrame& F, int level, long long c0, int bid, int nblk,
                                           unsigned* steps = nullptr) {
  __shared__ int2 s_cand[RTB_CAND][128];
  const DScene& S = F.S;
  const long long nh = F.nhits[level];
  const long long c1 = c0 + F.chunk_hits < nh ? c0 + F.chunk_hits : nh;
  unsigned long long culled = 0;  // shadow rays not traced (lights facing away)
  Work w{0, 0, 0, 0};
  // one thread per hit, or, where hits are few, per hit and light
  const long long nhc = c1 > c0 ? c1 - c0 : 0;
  const bool split = SPLIT && S.n_lights > 1 && nhc <= SPLIT_HITS;
  const long long items = split ? nhc * S.n_lights : nhc;
  const int lanes = walk_lanes(S, items, nblk), wpb = blockDim.x >> 5, lane = threadIdx.x & 31;
  const long long stride = (long long)nblk * wpb * lanes;
  for (long long base = ((long long)bid * wpb + (threadIdx.x >> 5)) * lanes; base < items; base += stride) {
    const long long item = base + lane;
    const bool active = lane < lanes && item < items;
    const int l0 = split && active ? (int)(item / nhc) : 0;
    const long long hl = split ? item - l0 * nhc : item;
    RayC rc;
    uint64_t seed;
    HitRec hr;
    V3 so = mk(0.0, 0.0, 0.0);
    if (active) {
      hr = load_hit(F, level, (int)(c0 + hl), &rc, &seed);
      if (l0 == 0) store_hit(F.hr, hl, hr);
      so = hr.p + 0.001 * hr.n;
    }
    // Lights the surface faces away from: the reference's light term is
    // exactly zero there (diffuse max(n . l, 0) = 0, specular only when
    // n . l > 0), so their shadow rays cannot change the image and are not
    // traced.  A disk light qualifies when every point of the disk is
    // behind the surface: n . (centre - p) + radius < 0, with a margin far
    // above the rounding of the sample directions' dot products.  Not where
    // the rays' visibility is itself an output (the denoiser's features and
    // visibility images at level 0).
    const bool may_cull = !(level == 0 && F.feat_on);
    // the hit's lit disk lights, queued in pairs after the others (lit pairs of
    // a learned level 0 only where they fall back, by k_fb_select)
    const bool pairing = !split && S.n_lights <= 32, shaded = !(F.learned && level == 0);
    for (int k = 0; k < (split ? 1 : S.n_lights); k++) {
      const int li = split ? l0 : k;
      const DLight& L0 = S.lights[li];
      int st = PAIR_DARK, nc = 0, queue = -1;
      if (active) {
        const V3 lp = ld3(L0.pos);
        const V3 lv = lp - hr.p;
        const double dist = norm(lv);
        const V3 ldir = lv / dist;
        if (!L0.disk) {
          // calculate_point_light_contribution (src/lighting.rs:100-142)
          const double facing = dot(hr.n, lv);
          if (may_cull && facing < 0.0 && facing < -1e-9 * (norm(lp) + (norm(hr.p) + 1.0))) {
            culled++;
          } else {
            // Ray::new normalises the (already unit) light direction once more
            st = shadow_walk(S, so, normalize(ldir), 0.001, dist, F.use_kd != 0, F.err, COUNT ? &w : nullptr)
                     ? PAIR_DARK : PAIR_LIT;
          }
        } else {
          const double radius = L0.diameter / 2.0;
          // gen_range(-radius..radius) panics on an empty or infinite range
          bool ok = -radius < radius;
          if (!ok) atomicOr(F.err, ERR_EMPTY_RANGE);
          if (ok && !isfinite(radius - -radius)) {
            atomicOr(F.err, ERR_RANGE_OVERFLOW);
            ok = false;
          }
          const double facing = dot(hr.n, lv) + radius;
          if (ok && may_cull && facing < 0.0 &&
              facing < -1e-9 * (norm(lp) + (norm(hr.p) + 1.0) + radius)) {
            ok = false;  // facing away from the whole disk
            culled += (unsigned long long)F.dsamp;
          }
          if (ok) {
            Cone cone;
            nc = make_cone(so, hr.n, ldir, dist, radius, &cone)
                     ? shaft_collect(S, cone, &s_cand[0][threadIdx.x], 128, F.err, COUNT ? &w : nullptr)
                     : (int)CONE_MANY;
            if (nc == 0) st = PAIR_LIT, queue = PART_LIT;
            else if (nc > 0) queue = PART_LIST;
            else if (nc == CONE_MANY) st = PAIR_WALK, queue = PART_WALK;
          }
        }
      }
      if (queue == PART_LIT && (pairing || !shaded)) queue = -1;
#pragma unroll
      for (int c = 0; c < 3; c++) {
        if (c == PART_LIT && pairing) continue;
        const int at = warp_alloc(F.pair.n + c, queue == c);
        if (queue == c) {
          F.pair.queue[c][at] = make_int2((int)hl, li);
          if (c == PART_LIST) st = at;
        }
      }
      if (queue == PART_LIST) {
        F.pair.ncand[st] = (unsigned char)nc;
        for (int j = 0; j < nc; j++) F.pair.cand[(size_t)st * RTB_CAND + j] = s_cand[j][threadIdx.x];
      }
      if (active) F.pair.st[li * F.chunk_hits + hl] = st;
      step_done(steps);
    }
    unsigned lit = 0;
    if (shaded && pairing && active)
      for (int k = 0; k < S.n_lights; k++)
        if (S.lights[k].disk && F.pair.st[k * F.chunk_hits + hl] == PAIR_LIT) lit |= 1u << k;
    while (__any_sync(0xffffffffu, lit != 0)) {
      const bool some = lit != 0;
      const int a = some ? __ffs(lit) - 1 : 0;
      lit &= lit - 1;
      int b = -1;  // another of the same diameter
      for (unsigned m = lit; m && b < 0; m &= m - 1)
        if (S.lights[__ffs(m) - 1].diameter == S.lights[a].diameter) b = __ffs(m) - 1;
      if (b >= 0) lit &= ~(1u << b);
      const int at2 = warp_alloc(F.pair.n + PART_LIT2, some && b >= 0);
      const int at1 = warp_alloc(F.pair.n + PART_LIT, some && b < 0);
      if (some) F.pair.queue[b >= 0 ? PART_LIT2 : PART_LIT][b >= 0 ? at2 : at1] = make_int2((int)hl, b >= 0 ? a | b << 16 : a);
    }
  }
  warp_sum_add(F.stats + 10, culled);
  if (COUNT) flush_work(F, w, 1);
}
template <bool COUNT, bool SPLIT>
__global__ void __launch_bounds__(128, 8) k_shaft(const __grid_constant__ DFrame F, int level, long long c0) {
  shaft_body<COUNT, SPLIT>(F, level, c0, blockIdx.x, gridDim.x);
}
__global__ void __launch_bounds__(128, 8) k_shaft_multi(const DFrame* __restrict__ T, const int* __restrict__ b0, int nj, int level) {
  const int j = job_of_block(b0, nj);
  const DFrame& F = T[j];
  if (level >= frame_levels(F)) return;
  shaft_body<false, true>(F, level, 0, blockIdx.x - b0[j], b0[j + 1] - b0[j]);
}

// The disk lights that are not dark.  A group of g lanes shares a pair: each
// lane makes blocks of the pair's ChaCha stream (lane j the j-th of a round;
// a block is four rejection-sampling attempts), the accepted offsets are
// compacted in stream order into the group's ring in shared memory, and each
// lane takes one sample: its ray, the test against the pair's candidates
// (PART_WALK: against the scene; PART_LIT: none) and its light term.  The
// terms are then added in sample order, as the reference adds them.
//
// g: a lane per sample (at most 32) makes the most of few pairs; a pair per
// lane (g = 1) saves the work that a group's lanes repeat (the hit, the
// light's frame, the blocks beyond those the samples need), so g halves
// while the pairs still fill the chip.  Walked pairs keep more of them, as a
// pair's rays take similar walks: g halves from 2^22 lanes on (2^18 to 2^21,
// 1280x720: 8 to 37% more on a low light over terrain, up to 9% less under
// lights wider than their distance; never: 14% more there).
//
// Bound by instruction issue and by the code's own size: at 900 instructions
// per sample and warp the loop outgrows the instruction cache.  1,000-sphere
// frame (17.2 M pairs of 16 rays), k_part: 16 lanes for each listed pair and
// one thread per hit for the lit ones 27 ms; lanes per pair by their number
// 15.2; whole exponents of the specular term by squaring 14.3; two lit lights
// of a hit on one stream, each light through the same code, the ChaCha rounds
// and the power not unrolled 11.6 (that loop unrolled: 13.6, the light's: 13.9
// with it).  4 blocks per SM; 3 take 12.3, 5 13.9.
//
// Rand's gen_range(-r..r) retries when rounding reaches r; with the scale
// 2r and a significand of at most 1 - 2^-52 the result is at most r - 2 ulp,
// so for normal r it never does.  Radii below 1e-290, where these steps
// leave the normal range, draw serially (StdRng) on the group's first lane.
#define PART_RING 8         // ring entries per lane; a round adds at most 4
#define PART_FILL (1 << 17)  // lanes that fill the chip
#define WALK_FILL (1 << 22)  // and lanes that share out many walks
#define WALK_MANY (1 << 18)  // walked pairs that k_walk takes
struct PartShared {
  double2 off[4][32 * PART_RING];
  double term[4][3][32];
};
// log2 of the lanes that share a pair of this class, and its warps' tasks.
template <int KIND>
__device__ __forceinline__ int part_lanes(const DFrame& F, int n) {
  int lg = F.lanes_log2;
  while (lg > 0 && ((long long)n << (lg - 1)) >= (KIND == PART_WALK ? WALK_FILL : PART_FILL)) lg--;
  return lg;
}
template <int KIND>
__device__ __forceinline__ int part_tasks(const DFrame& F) {
  const int n = F.pair.n[(F.fb_mode ? 4 : 0) + KIND];
  const int per_warp = 32 >> part_lanes<KIND>(F, n);
  return (n + per_warp - 1) / per_warp;
}
// Warp w of nw takes the class's tasks w, w + nw, ...
template <int KIND, bool COUNT>
__device__ __forceinline__ void part_body(const DFrame& F, int level, long long c0, PartShared& sm, long long w0,
                                          long long nw, unsigned* steps) {
  constexpr int NL = KIND == PART_LIT2 ? 2 : 1;  // lights of an entry
  constexpr bool LIT = KIND == PART_LIT || KIND == PART_LIT2;
  const unsigned FULL = 0xffffffffu;
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const DScene& S = F.S;
  const int n = F.pair.n[(F.fb_mode ? 4 : 0) + KIND];
  const int lg = part_lanes<KIND>(F, n);
  const int g = 1 << lg, member = lane & (g - 1), gbase = lane & ~(g - 1);
  const unsigned gmask = g == 32 ? FULL : ((1u << g) - 1u) << gbase;
  const unsigned lower = gmask & ((1u << lane) - 1u);
  double2* ring = sm.off[wid] + gbase * PART_RING;
  const int rmask = g * PART_RING - 1;
  const int per_warp = 32 >> lg;
  const int dsamp = F.dsamp;
  // the learned pass only counts the unblocked rays
  const bool shade = !(F.learned && level == 0 && !F.fb_mode);
  const V3 campos = ld3(F.C.campos);
  Work w{0, 0, 0, 0};
  for (long long base = w0 * per_warp; base < n; base += nw * per_warp) {
    const long long at = base + (lane >> lg);
    const bool have = at < n;
    int2 hl = make_int2(0, 0);
    HitRec hr{mk(0, 0, 0), mk(0, 0, 1), 0, 0, 0.0, 0.0};
    Disk disk[NL];
#pragma unroll
    for (int u = 0; u < NL; u++) disk[u] = Disk{mk(0, 0, 1), mk(1, 0, 0), mk(0, 1, 0), 1.0};
    uint32_t key[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    SMat m{};
    V3 view = mk(0, 0, 1);
    int ent = 0, nc = 0;
    int li[NL] = {};
    if (have) {
      hl = F.pair.queue[KIND][at];
      hr = read_hit(F.hr, hl.x);
#pragma unroll
      for (int u = 0; u < NL; u++) {
        li[u] = NL == 1 ? hl.y : (hl.y >> (16 * u)) & 0xffff;
        disk[u] = make_disk(S.lights[li[u]], hr.p);
      }
      pcg32_key(light_seed(F.q[level & 1].seed[F.hit_ray[c0 + hl.x]], hr.p), key);
      if (KIND != PART_WALK) {
        m = effective_material(S.mat[hr.mat], hr);
        view = normalize(campos - hr.p);
      }
      if (KIND == PART_LIST) {
        ent = F.pair.st[li[0] * F.chunk_hits + hl.x];
        nc = F.pair.ncand[ent];
      }
    }
    const double radius = disk[0].radius, r2 = radius * radius;
    const bool serial = radius < 1e-290;
    V3 tot[NL];
#pragma unroll
    for (int u = 0; u < NL; u++) tot[u] = mk(0.0, 0.0, 0.0);
    int got = 0, visible = 0, rounds = 0;  // offsets drawn, unblocked samples, ChaCha rounds
    for (int s0 = 0; s0 < dsamp; s0 += g) {
      step_done(steps);
      const int need = min(dsamp, s0 + g);
      // Draw until every group holds its next samples.  A lane that draws
      // while others wait costs nothing, so groups draw ahead whenever the
      // round fits their ring, and mostly stay in step.
      while (__any_sync(FULL, have && got < need)) {
        const bool draw = have && !serial && got < dsamp && got - s0 <= (PART_RING - 4) * g;
        unsigned acc = 0;
        double2 off[4];
        if (draw) {
          uint32_t b[16];
          chacha_block(key, (uint64_t)((long long)rounds * g + member), 6, b);
          const double scale = radius - -radius;
#pragma unroll
          for (int a = 0; a < 4; a++) {
            const uint64_t u0 = ((uint64_t)b[4 * a + 1] << 32) | b[4 * a], u1 = ((uint64_t)b[4 * a + 3] << 32) | b[4 * a + 2];
            off[a].x = (bitsd((u0 >> 12) | (1023ULL << 52)) - 1.0) * scale + -radius;
            off[a].y = (bitsd((u1 >> 12) | (1023ULL << 52)) - 1.0) * scale + -radius;
            if (off[a].x * off[a].x + off[a].y * off[a].y <= r2) acc |= 1u << a;
          }
        }
        if (have && serial && got < need) {
          if (member == 0) {
            StdRng rng;
            rng.init(light_seed(F.q[level & 1].seed[F.hit_ray[c0 + hl.x]], hr.p));
            for (int k = 0; k < need; k++) {
              double dx = 0.0, dy = 0.0;
              if (!next_offset(rng, radius, &dx, &dy, F.err)) break;
              if (k >= s0) ring[k & rmask] = make_double2(dx, dy);
            }
          }
          got = need;
        }
        // the accepted offsets in stream order: attempt a of lane j follows
        // all attempts of the lanes before it
        int pos = got;
        if (g == 1) {
          got += __popc(acc);
        } else {
#pragma unroll
          for (int a = 0; a < 4; a++) {
            const unsigned v = __ballot_sync(FULL, (acc >> a) & 1u);
            pos += __popc(v & lower);
            got += __popc(v & gmask);
          }
        }
#pragma unroll
        for (int a = 0; a < 4; a++)
          if ((acc >> a) & 1u) ring[pos++ & rmask] = off[a];
        if (draw && ++rounds > 4096 * 8) {
          atomicOr(F.err, ERR_WATCHDOG);
          got = need;
        }
      }
      __syncwarp();
      const bool on = have && s0 + member < need;
      const double2 o = on ? ring[(s0 + member) & rmask] : make_double2(0.0, 0.0);
#pragma unroll 1
      for (int u = 0; u < NL; u++) {
        bool seen = false;
        V3 dir = mk(0.0, 0.0, 1.0);
        if (on) {
          double dist;
          dir = disk_dir(disk[u], hr.p, o.x, o.y, &dist);
          seen = true;
          if (!LIT) {
            const V3 so = hr.p + 0.001 * hr.n;
            const V3 rd = normalize(dir);  // Ray::new normalises once more
            if (KIND == PART_WALK) {
              seen = !shadow_walk(S, so, rd, 0.001, dist, F.use_kd != 0, F.err, COUNT ? &w : nullptr);
            } else {
              for (int j = 0; j < nc && seen; j++)
                seen = !ray_blocked_by(S, F.pair.cand[(size_t)ent * RTB_CAND + j], so, rd, 0.001, dist, F.use_kd != 0,
                                       COUNT ? &w : nullptr);
            }
          }
        }
        V3 term = mk(0.0, 0.0, 0.0);
        if (seen && shade) {
          const DLight& L0 = S.lights[li[u]];
          if (KIND == PART_WALK) {  // not kept across the walk
            m = effective_material(S.mat[hr.mat], hr);
            view = normalize(campos - hr.p);
          }
          term = light_term(m, hr, dir, ld3(L0.color), L0.intensity, view);
        }
        if (g == 1) {
          if (u == 0) visible += seen ? 1 : 0;
          if (seen) tot[u] = tot[u] + term;
          continue;
        }
        if (u == 0) visible += __popc(__ballot_sync(FULL, seen) & gmask);
        sm.term[wid][0][lane] = term.x;
        sm.term[wid][1][lane] = term.y;
        sm.term[wid][2][lane] = term.z;
        __syncwarp();
        // blocked samples add zero: the sum is never -0.  Three lanes add one
        // component each (in tot.x); groups of two lanes add all three.
        if (g >= 4) {
          if (member < 3)
            for (int k = 0; k < need - s0; k++) tot[u].x += sm.term[wid][member][gbase + k];
        } else if (member == 0) {
          for (int k = 0; k < need - s0; k++)
            tot[u] = tot[u] + mk(sm.term[wid][0][gbase + k], sm.term[wid][1][gbase + k], sm.term[wid][2][gbase + k]);
        }
        __syncwarp();
      }
    }
    if (have) {
      const double cnt = (double)dsamp;  // 16.0 in the reference
      const double part = (double)visible / cnt;
#pragma unroll
      for (int u = 0; u < NL; u++) {
        const long long pair = li[u] * F.chunk_hits + hl.x;
        if (shade) {
          if (g >= 4) {
            if (member < 3) F.pair.sum[member][pair] = tot[u].x / cnt * part;
          } else if (member == 0) {
            F.pair.sum[0][pair] = tot[u].x / cnt * part;
            F.pair.sum[1][pair] = tot[u].y / cnt * part;
            F.pair.sum[2][pair] = tot[u].z / cnt * part;
          }
        }
        if (member == 0) F.pair.vis[pair] = visible;
      }
    }
  }
  if (COUNT) flush_work(F, w, 1);
}
// One launch for the four queues, a quarter of the blocks each: the walks, whose
// slowest lanes take longest, start first and the other queues' blocks run
// beside them.  A grid whose blocks are all resident (k_levels) goes through
// the queues' tasks as one sequence.
template <bool COUNT>
__device__ __forceinline__ void part_all(const DFrame& F, int level, long long c0, int bid, int nblk, bool resident,
                                         unsigned* steps = nullptr) {
  __shared__ PartShared sm;
  const int wid = threadIdx.x >> 5;
  // a learned level 0 takes the lit pairs' shading from the network
  const bool lit = F.fb_mode || !(F.learned && level == 0);
  const int each = nblk / 4, part = each && !resident ? min(bid / each, 3) : -1;
  const long long none = 1LL << 40;  // no task of the class
  long long nw = 4LL * nblk, w0 = 4LL * bid + wid;
  if (part >= 0) {
    nw = 4LL * (part < 3 ? each : nblk - 3 * each);
    w0 = 4LL * (bid - part * each) + wid;
  }
  // the warp's first task of a class that follows `tasks` others
  auto next = [&](int tasks) { w0 = (w0 + nw - tasks % nw) % nw; };
  auto mine = [&](int k) { return part < 0 || part == k ? w0 : none; };
  part_body<PART_WALK, COUNT>(F, level, c0, sm, F.walk && F.pair.n[PART_WALK] >= WALK_MANY ? none : mine(0), nw, steps);
  if (part < 0) next(part_tasks<PART_WALK>(F));
  part_body<PART_LIST, COUNT>(F, level, c0, sm, mine(1), nw, steps);
  if (part < 0) next(part_tasks<PART_LIST>(F));
  part_body<PART_LIT2, COUNT>(F, level, c0, sm, lit ? mine(2) : none, nw, steps);
  if (part < 0) next(part_tasks<PART_LIT2>(F));
  part_body<PART_LIT, COUNT>(F, level, c0, sm, lit ? mine(3) : none, nw, steps);
}
// The walked pairs of a level where they are many, before k_part: walks wait
// for their node loads, and without the other classes' code 6 blocks of 128
// share an SM (80 registers; 8 blocks within 4%, 10 up to 60% slower).
// 1280x720: icosphere under a light as wide as its distance 7.2 -> 6.2 ms, low
// light over terrain 9.7 -> 8.5, 1,000 spheres under lights of diameter 16 11.0
// -> 10.2.  Fewer than 2^18 pairs (2^20: the first two as without) fill the
// chip beside the other queues' blocks, and frames with few walks pay 8 us for
// a launch that returns.
template <bool COUNT>
__global__ void __launch_bounds__(128, 6) k_walk(const __grid_constant__ DFrame F, int level, long long c0) {
  __shared__ PartShared sm;
  if (F.pair.n[PART_WALK] < WALK_MANY) return;
  part_body<PART_WALK, COUNT>(F, level, c0, sm, 4LL * blockIdx.x + (threadIdx.x >> 5), 4LL * gridDim.x, nullptr);
}
template <bool COUNT>
__global__ void __launch_bounds__(128, 4) k_part(const __grid_constant__ DFrame F, int level, long long c0) {
  part_all<COUNT>(F, level, c0, blockIdx.x, gridDim.x, false);
}
__global__ void __launch_bounds__(128, 4) k_part_multi(const DFrame* __restrict__ T, const int* __restrict__ b0, int nj, int level) {
  const int j = job_of_block(b0, nj);
  const DFrame& F = T[j];
  if (level >= frame_levels(F)) return;
  part_all<false>(F, level, 0, blockIdx.x - b0[j], b0[j + 1] - b0[j], false);
}

// phong_lighting's sum, fog and the reflection ray (src/lighting.rs:220-288,
// 297-319, 437-496) for hits [c0, c1), one thread per hit.
__device__ __forceinline__ void light_body(const DFrame& F, int level, long long c0, int bid, int nblk) {
  const DScene& S = F.S;
  const long long nh = F.nhits[level];
  const long long c1 = c0 + F.chunk_hits < nh ? c0 + F.chunk_hits : nh;
  const RayBuf q = F.q[level & 1];
  RayBuf qn = F.q[(level + 1) & 1];
  LevelBuf L = F.levels[level];
  const bool can_reflect = (F.max_depth - level) > 1;
  const bool learned = level == 0 && F.learned;
  const V3 campos = ld3(F.C.campos);
  const long long stride = (long long)nblk * blockDim.x;
  for (long long base = c0 + bid * (long long)blockDim.x; base < c1; base += stride) {
    const long long h = base + threadIdx.x;
    const bool active = h < c1;
    bool emit = false;
    V3 ro = mk(0, 0, 0), rd = mk(0, 0, 0);
    int i = -1;
    V3 color = mk(0.0, 0.0, 0.0);
    double refl = 0.0;
    if (active) {
      const long long hl = h - c0;
      const HitRec hr = read_hit(F.hr, hl);
      i = F.hit_ray[h];
      const DMat& mat = S.mat[hr.mat];
      const SMat m = effective_material(mat, hr);
      color = m.ka * S.amb_int * cmul(ld3(S.amb_color), m.c);
      const V3 view = normalize(campos - hr.p);
      long long vix = 0;  // slot 0 of this sample in the visibility planes
      unsigned falls = 0u;
      if (learned) {
        const long long pix = i / F.S_per_px;
        vix = ((long long)(i % F.S_per_px) * DN_MAX_SLOTS * F.H) * F.W + pix;
        falls = F.fb_flag ? F.fb_flag[h] : 0u;
      }
      int slot = 0;
      for (int li = 0; li < S.n_lights; li++) {
        const DLight& L0 = S.lights[li];
        const long long pair = li * F.chunk_hits + hl;
        const int st = F.pair.st[pair];
        const bool estimate = learned && L0.disk && !((falls >> slot) & 1u);
        V3 contrib = mk(0.0, 0.0, 0.0);
        if (estimate || (!L0.disk && st == PAIR_LIT)) {
          const V3 lv = ld3(L0.pos) - hr.p;
          contrib = light_term(m, hr, lv / norm(lv), ld3(L0.color), L0.intensity, view);
          if (estimate) {
            // extension: the light-centre term times the squared visibility
            // estimate, the expectation of the reference's
            // (sum of visible terms / n) * (visible / n)
            double vh = (double)F.vhat[vix + (long long)slot * F.H * F.W];
            vh = rclamp(vh, 0.0, 1.0);
            contrib = contrib * (vh * vh);
          }
        } else if (L0.disk) {
          if (st != PAIR_DARK) contrib = mk(F.pair.sum[0][pair], F.pair.sum[1][pair], F.pair.sum[2][pair]);
          // fallback of a learned render: the plain visibility replaces the
          // estimate in the visibility output
          if (learned)
            F.vhat[vix + (long long)slot * F.H * F.W] =
                (float)(st != PAIR_DARK ? F.pair.vis[pair] : 0) / (float)F.fb_dsamp;
        }
        if (L0.disk) slot++;
        color = color + contrib;
      }
      if (S.has_fog) {
        double dist = norm(hr.p - campos);
        double f;
        if (dist <= S.fog_start) f = 0.0;
        else if (dist >= S.fog_end) f = 1.0;
        else f = (dist - S.fog_start) / (S.fog_end - S.fog_start);
        f = 1.0 - exp(-S.fog_density * f);
        f = rclamp(f, 0.0, 1.0);
        color = color * (1.0 - f) + ld3(S.fog_color) * f;
      }
      if (mat.has_refl && mat.refl > 0.0 && can_reflect) {
        emit = true;
        refl = mat.refl;
        V3 vd = normalize(campos - hr.p);
        ro = hr.p + 0.001 * hr.n;
        rd = normalize(reflect(-vd, hr.n));
      }
      if (level == 0 && F.outline) {
        F.phit[i] = 1;
        F.pobj[i] = F.hobj[h];
        F.pdepth[i] = norm(hr.p - campos);
        F.pnx[i] = hr.n.x;
        F.pny[i] = hr.n.y;
        F.pnz[i] = hr.n.z;
      }
    }
    int slot = warp_alloc(&F.counts[level + 1], emit);
    if (active) {
      L.r[i] = color.x;
      L.g[i] = color.y;
      L.b[i] = color.z;
      L.refl[i] = refl;
      L.child[i] = slot;
      if (emit) {
        qn.ox[slot] = ro.x;
        qn.oy[slot] = ro.y;
        qn.oz[slot] = ro.z;
        qn.dx[slot] = rd.x;
        qn.dy[slot] = rd.y;
        qn.dz[slot] = rd.z;
        qn.seed[slot] = q.seed[i];
      }
    }
  }
}
__global__ void __launch_bounds__(128, 6) k_light(const __grid_constant__ DFrame F, int level, long long c0) {
  light_body(F, level, c0, blockIdx.x, gridDim.x);
}
__global__ void __launch_bounds__(128, 6) k_light_multi(const DFrame* __restrict__ T, const int* __restrict__ b0, int nj, int level) {
  const int j = job_of_block(b0, nj);
  const DFrame& F = T[j];
  if (level >= frame_levels(F)) return;
  light_body(F, level, 0, blockIdx.x - b0[j], b0[j + 1] - b0[j]);
}


// Confidence gate of learned shadows: the slots of a level-0 hit whose
// estimated visibility error is above conf_thr go to fb_flag, to be shaded
// by the plain path, and their pairs to k_part's queues (whose entries the
// learned pass is done with), unless they are dark.
__global__ void __launch_bounds__(128) k_fb_select(DFrame F) {
  const long long nh = F.nhits[0];
  const long long plane_px = (long long)F.H * F.W;
  for (long long base = blockIdx.x * (long long)blockDim.x; base < nh; base += (long long)gridDim.x * blockDim.x) {
    const long long h = base + threadIdx.x;
    unsigned mask = 0;
    if (h < nh) {
      const int i = F.hit_ray[h];
      const long long pix = i / F.S_per_px, plane = i % F.S_per_px;
      for (int j = 0; j < F.n_slots; j++)
        if (F.vconf[(plane * DN_MAX_SLOTS + j) * plane_px + pix] > F.conf_thr) mask |= 1u << j;
      F.fb_flag[h] = (unsigned char)mask;
    }
    // every lane of the warp takes part in each allocation
    warp_alloc(F.fbn, mask != 0);
    int slot = 0;
    for (int li = 0; li < F.S.n_lights; li++) {
      if (!F.S.lights[li].disk) continue;
      const int st = (mask >> slot) & 1u ? F.pair.st[li * F.chunk_hits + h] : (int)PAIR_DARK;
      const int queue = st >= 0 ? PART_LIST : st == PAIR_LIT ? PART_LIT : st == PAIR_WALK ? PART_WALK : -1;
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const int at = warp_alloc(F.pair.n + 4 + c, queue == c);
        if (queue == c) F.pair.queue[c][at] = make_int2((int)h, li);
      }
      slot++;
    }
    const unsigned slots = __reduce_add_sync(0xffffffffu, (unsigned)__popc(mask));
    if ((threadIdx.x & 31) == 0 && slots) atomicAdd(F.fbn + 1, (int)slots);
  }
}

// Denoiser input of the level-0 hits [c0, c1): one FEAT_CHANNELS FP16
// pixel per (sample plane, pixel); misses stay zero (FEAT_VALID = 0).  Also
// the plain visibility (visible / dsamp) of each slot into vis_aov.
__global__ void __launch_bounds__(128) k_features(DFrame F, long long c0) {
  const DScene& S = F.S;
  long long nh = F.nhits[0];
  long long c1 = c0 + F.chunk_hits < nh ? c0 + F.chunk_hits : nh;
  V3 campos = ld3(F.C.campos);
  const long long plane_px = (long long)F.H * F.W;
  for (long long h = c0 + blockIdx.x * (long long)blockDim.x + threadIdx.x; h < c1;
       h += (long long)gridDim.x * blockDim.x) {
    const HitRec hr = read_hit(F.hr, h - c0);
    int i = F.hit_ray[h];
    long long pix = i / F.S_per_px;
    long long plane = i % F.S_per_px;
    float f[FEAT_CHANNELS];
#pragma unroll
    for (int c = 0; c < FEAT_CHANNELS; c++) f[c] = 0.f;
    f[FEAT_VALID] = 1.f;
    double d = norm(hr.p - campos);
    f[FEAT_DEPTH] = (float)(d / (d + 4.0));
    f[FEAT_NX] = (float)hr.n.x;
    f[FEAT_NX + 1] = (float)hr.n.y;
    f[FEAT_NX + 2] = (float)hr.n.z;
    int slot = 0;
    for (int li = 0; li < S.n_lights; li++) {
      const DLight& L0 = S.lights[li];
      if (!L0.disk) continue;
      if (slot < DN_MAX_SLOTS) {
        const long long pair = li * F.chunk_hits + h - c0;
        const int st = F.pair.st[pair];
        const int visible = st == PAIR_LIT ? F.dsamp : st == PAIR_DARK ? 0 : F.pair.vis[pair];
        float v = (float)visible / (float)F.dsamp;
        V3 lp = ld3(L0.pos);
        double dist = norm(lp - hr.p);
        V3 cdir = normalize(lp - hr.p);
        double cosc = rmax(dot(hr.n, cdir), 0.0);
        double ang = rclamp(0.5 * L0.diameter / dist, 0.0, 1.0);
        const float fv[4] = {v, (float)cosc, (float)ang, 1.f};
#pragma unroll
        for (int s = 0; s < DN_MAX_SLOTS; s++)
          if (s == slot)
            for (int c = 0; c < 4; c++) f[FEAT_SLOT0 + FEAT_SLOT_STRIDE * s + c] = fv[c];
        if (F.vis_aov) F.vis_aov[(plane * DN_MAX_SLOTS + slot) * plane_px + pix] = v;
      }
      slot++;
    }
    __align__(16) __half hv[FEAT_CHANNELS];
#pragma unroll
    for (int c = 0; c < FEAT_CHANNELS; c++) hv[c] = __float2half_rn(f[c]);
    uint4* dst = reinterpret_cast<uint4*>(F.feat + (plane * plane_px + pix) * FEAT_CHANNELS);
    const uint4* src = reinterpret_cast<const uint4*>(hv);
    dst[0] = src[0];
    dst[1] = src[1];
  }
}

// Pixel-level feature: for each slot, the mean cast-ray visibility over the
// samples of the pixel whose primary ray hit, written into every hit
// sample's FEAT_PIXEL_VIS + slot channel, so that the network of each
// sample plane sees the pixel's other samples too.  One thread per pixel.
__global__ void __launch_bounds__(128) k_feat_pixel_mean(DFrame F) {
  const long long plane_px = (long long)F.H * F.W;
  for (long long pix = blockIdx.x * (long long)blockDim.x + threadIdx.x; pix < plane_px;
       pix += (long long)gridDim.x * blockDim.x) {
    float sum[DN_MAX_SLOTS] = {0.f, 0.f};
    int n = 0;
    for (int s = 0; s < F.S_per_px; s++) {
      const __half* f = F.feat + ((long long)s * plane_px + pix) * FEAT_CHANNELS;
      if (__half2float(f[FEAT_VALID]) > 0.f) {
        n++;
#pragma unroll
        for (int j = 0; j < DN_MAX_SLOTS; j++) sum[j] += __half2float(f[FEAT_SLOT0 + FEAT_SLOT_STRIDE * j]);
      }
    }
    if (n == 0) continue;
    for (int s = 0; s < F.S_per_px; s++) {
      __half* f = F.feat + ((long long)s * plane_px + pix) * FEAT_CHANNELS;
      if (__half2float(f[FEAT_VALID]) > 0.f) {
#pragma unroll
        for (int j = 0; j < DN_MAX_SLOTS; j++) f[FEAT_PIXEL_VIS + j] = __float2half_rn(sum[j] / (float)n);
      }
    }
  }
}

// color * (1 - r) + reflected * r, deepest level first: each primary ray's
// chain of reflections is followed down and blended back up.  One launch
// for all levels; only the level-0 colours are written.
__device__ __forceinline__ void fold_body(const DFrame& F, int bid, int nblk) {
  const long long n = F.n_primary;
  const LevelBuf L0 = F.levels[0];
  for (long long i = bid * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)nblk * blockDim.x) {
    int at[RTB_MAX_LEVELS];
    int d = 0, c = L0.child[i];
    if (c < 0) continue;
    at[0] = (int)i;
    while (c >= 0) {
      at[++d] = c;
      c = F.levels[d].child[c];
    }
    LevelBuf B = F.levels[d];
    V3 col = mk(B.r[at[d]], B.g[at[d]], B.b[at[d]]);
    for (d--; d >= 0; d--) {
      B = F.levels[d];
      const int k = at[d];
      const double r = B.refl[k], q = 1.0 - r;
      col = mk(B.r[k] * q + col.x * r, B.g[k] * q + col.y * r, B.b[k] * q + col.z * r);
    }
    L0.r[i] = col.x;
    L0.g[i] = col.y;
    L0.b[i] = col.z;
  }
}
__global__ void k_fold(const __grid_constant__ DFrame F) { fold_body(F, blockIdx.x, gridDim.x); }
__global__ void k_fold_multi(const DFrame* __restrict__ T, const int* __restrict__ b0, int nj) {
  const int j = job_of_block(b0, nj);
  fold_body(T[j], blockIdx.x - b0[j], b0[j + 1] - b0[j]);
}


// --------------------------------------------------------------------------
// Per-pixel resolve, outline, quantise
// --------------------------------------------------------------------------
__device__ __forceinline__ void store_rgb(const DFrame& F, long long p, V3 c) {
  F.rgb[3 * p + 0] = sat_u8(rclamp(c.x, 0.0, 1.0) * 255.0);
  F.rgb[3 * p + 1] = sat_u8(rclamp(c.y, 0.0, 1.0) * 255.0);
  F.rgb[3 * p + 2] = sat_u8(rclamp(c.z, 0.0, 1.0) * 255.0);
  if (F.linear) {
    F.linear[3 * p + 0] = c.x;
    F.linear[3 * p + 1] = c.y;
    F.linear[3 * p + 2] = c.z;
  }
}

__device__ __forceinline__ void pixels_body(const DFrame& F, int bid, int nblk) {
  long long np = (long long)F.W * F.H;
  LevelBuf L = F.levels[0];
  for (long long p = bid * (long long)blockDim.x + threadIdx.x; p < np; p += (long long)nblk * blockDim.x) {
    V3 c;
    if (F.max_depth <= 0) {
      // ray_color returns black before any World::hit (src/lighting.rs:450-452)
      c = mk(0.0, 0.0, 0.0);
      if (F.aa == RT_AA_QUINCUNX) {
        c = (c + c + c + c + c) / 5.0;
      } else {
        V3 t = mk(0.0, 0.0, 0.0);
        for (int s = 0; s < F.S_per_px; s++) t = t + c;
        c = t / (double)F.S_per_px;
      }
      if (F.outline) F.valid[p] = 0;
    } else if (F.aa == RT_AA_QUINCUNX) {
      // (center + tl + tr + bl + br) / 5 (src/renderer.rs:873-886)
      long long x = p % F.W, y = p / F.W;
      long long W1 = F.W + 1;
      long long ci = F.n_corner + p;
      long long k0 = y * W1 + x, k1 = y * W1 + x + 1, k2 = (y + 1) * W1 + x, k3 = (y + 1) * W1 + x + 1;
      V3 cc = mk(L.r[ci], L.g[ci], L.b[ci]);
      V3 c0 = mk(L.r[k0], L.g[k0], L.b[k0]);
      V3 c1 = mk(L.r[k1], L.g[k1], L.b[k1]);
      V3 c2 = mk(L.r[k2], L.g[k2], L.b[k2]);
      V3 c3 = mk(L.r[k3], L.g[k3], L.b[k3]);
      c = (cc + c0 + c1 + c2 + c3) / 5.0;
    } else {
      // sum / samples; outline keeps the nearest sample's depth and normal
      // (src/renderer.rs:548-552, 690-702)
      V3 t = mk(0.0, 0.0, 0.0);
      bool have = false;
      double pd = 0.0;
      V3 pn = mk(0.0, 0.0, 0.0);
      int po = -1;
      for (int s = 0; s < F.S_per_px; s++) {
        long long i = p * F.S_per_px + s;
        t = t + mk(L.r[i], L.g[i], L.b[i]);
        if (F.outline && F.phit[i]) {
          double d = F.pdepth[i];
          if (!have || d < pd) {
            have = true;
            pd = d;
            pn = mk(F.pnx[i], F.pny[i], F.pnz[i]);
            po = F.pobj[i];
          }
        }
      }
      c = t / (double)F.S_per_px;
      if (F.outline) {
        F.valid[p] = have ? 1 : 0;
        if (F.oid) F.oid[p] = po;
        F.dep[p] = pd;
        F.nx[p] = pn.x;
        F.ny[p] = pn.y;
        F.nz[p] = pn.z;
      }
    }
    if (F.outline) {
      F.cr[p] = c.x;
      F.cg[p] = c.y;
      F.cb[p] = c.z;
    } else {
      store_rgb(F, p, c);
    }
  }
}
__global__ void k_pixels(const __grid_constant__ DFrame F) {
  pixels_body(F, blockIdx.x, gridDim.x);
}
__global__ void k_pixels_multi(const DFrame* __restrict__ T, const int* __restrict__ b0, int nj) {
  const int j = job_of_block(b0, nj);
  const DFrame& F = T[j];
  pixels_body(F, blockIdx.x - b0[j], b0[j + 1] - b0[j]);
}


// Queue levels [first, levels) in one cooperative launch, a grid barrier
// between the stages, until a level's queue is empty; then the reflections
// of all levels are folded.  Most levels that a frame may have are empty, and
// launching their stages took 2 us each on a small frame (the 400x300 sphere
// frame: 0.235 ms in 42 launches, 0.106 in 11) and 8 us with a large frame's
// grids (the 1080p icosphere frame 4.89 -> 4.58 ms).
//
// The barrier: the blocks are co-resident (cooperative launch), bar[0]
// counts their arrivals and each stage waits for the next multiple of the
// grid.  A stage may last as long as its work takes: a block waits on while
// others arrive or do steps (bar[2], step_done).  One that sees neither for
// `limit` nanoseconds sets the watchdog's error and leaves, and so, at their
// next barrier, do the others.  A step is one walk of the scene at most, and
// the host admits scenes only where that is far shorter (kCoopWalk).
__device__ __forceinline__ bool grid_barrier(unsigned* bar, unsigned* target, unsigned long long limit, int* err) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    volatile unsigned* vb = bar;
    *target += gridDim.x;
    __threadfence();
    atomicAdd(bar, 1u);
    unsigned long long t0, t;
    unsigned seen = vb[0] + vb[2];
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
    bool ok = true;
    while ((int)(vb[0] - *target) < 0) {
      asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
      if (t - t0 > limit) {
        const unsigned now = vb[0] + vb[2];
        if (now == seen) {
          atomicOr(err, ERR_BARRIER);
          ok = false;
          break;
        }
        seen = now;
        t0 = t;
      }
    }
    __threadfence();
    s_ok = ok ? 1 : 0;
  }
  __syncthreads();
  return s_ok != 0;
}
__global__ void __launch_bounds__(128, 4) k_levels(const __grid_constant__ DFrame F, int first, int levels, unsigned* bar,
                                                     unsigned long long limit) {
  const int bid = blockIdx.x, nblk = gridDim.x;
  unsigned target = 0;
  unsigned* steps = bar + 2;
  bool ok = true;
  for (int l = first; ok && l < levels; l++) {
    if (*(volatile int*)&F.counts[l] == 0) break;
    trace_body<false>(F, l, bid, nblk, steps);
    if (!(ok = grid_barrier(bar, &target, limit, F.err))) break;
    if (*(volatile int*)&F.nhits[l] == 0) break;
    shaft_body<false, true>(F, l, 0, bid, nblk, steps);
    if (!(ok = grid_barrier(bar, &target, limit, F.err))) break;
    if (*(volatile int*)&F.pair.n[0] + *(volatile int*)&F.pair.n[1] + *(volatile int*)&F.pair.n[2] + *(volatile int*)&F.pair.n[3] > 0) {
      part_all<false>(F, l, 0, bid, nblk, true, steps);
      if (!(ok = grid_barrier(bar, &target, limit, F.err))) break;
    }
    light_body(F, l, 0, bid, nblk);
    if (!(ok = grid_barrier(bar, &target, limit, F.err))) break;
  }
  if (ok) fold_body(F, bid, nblk);
  // the last block to leave clears the barrier for the next launch
  if (threadIdx.x == 0 && atomicAdd(bar + 1, 1u) == gridDim.x - 1) {
    bar[0] = 0;
    bar[1] = 0;
  }
}

// detect_edges / compute_edge_strength (src/outline.rs:113-182): one tile of
// OT_X x OT_Y pixels with a one-pixel halo staged in shared memory.
#define OT_X 32
#define OT_Y 8
__global__ void __launch_bounds__(OT_X* OT_Y) k_outline_mask(DFrame F) {
  __shared__ double sd[OT_Y + 2][OT_X + 2];
  __shared__ double snx[OT_Y + 2][OT_X + 2], sny[OT_Y + 2][OT_X + 2], snz[OT_Y + 2][OT_X + 2];
  __shared__ unsigned char sv[OT_Y + 2][OT_X + 2];
  __shared__ int so[OT_Y + 2][OT_X + 2];
  const bool ids = F.oid && F.o_wid != 0.0;
  int x0 = blockIdx.x * OT_X - 1, y0 = blockIdx.y * OT_Y - 1;
  for (int k = threadIdx.y * OT_X + threadIdx.x; k < (OT_X + 2) * (OT_Y + 2); k += OT_X * OT_Y) {
    int lx = k % (OT_X + 2), ly = k / (OT_X + 2);
    int gx = x0 + lx, gy = y0 + ly;
    unsigned char v = 0;
    double d = 0, a = 0, b = 0, c = 0;
    int o = -1;
    if (gx >= 0 && gy >= 0 && gx < F.W && gy < F.H) {
      long long p = (long long)gy * F.W + gx;
      v = F.valid[p];
      d = F.dep[p];
      a = F.nx[p];
      b = F.ny[p];
      c = F.nz[p];
      if (ids) o = F.oid[p];
    }
    so[ly][lx] = o;
    sv[ly][lx] = v;
    sd[ly][lx] = d;
    snx[ly][lx] = a;
    sny[ly][lx] = b;
    snz[ly][lx] = c;
  }
  __syncthreads();
  int gx = blockIdx.x * OT_X + threadIdx.x, gy = blockIdx.y * OT_Y + threadIdx.y;
  if (gx >= F.W || gy >= F.H) return;
  int lx = threadIdx.x + 1, ly = threadIdx.y + 1;
  bool cf = sv[ly][lx] != 0;
  double cd = sd[ly][lx];
  V3 cn = mk(snx[ly][lx], sny[ly][lx], snz[ly][lx]);
  // neighbour lists of get_4_neighbors / get_8_neighbors (src/outline.rs:185-224)
  int ndx[8], ndy[8], nn = 0;
  if (F.o_use8) {
    for (int dy = -1; dy <= 1; dy++)
      for (int dx = -1; dx <= 1; dx++) {
        if (dx == 0 && dy == 0) continue;
        if (gx + dx >= 0 && gy + dy >= 0) {
          ndx[nn] = dx;
          ndy[nn] = dy;
          nn++;
        }
      }
  } else {
    if (gx > 0) { ndx[nn] = -1; ndy[nn] = 0; nn++; }
    ndx[nn] = 1; ndy[nn] = 0; nn++;
    if (gy > 0) { ndx[nn] = 0; ndy[nn] = -1; nn++; }
    ndx[nn] = 0; ndy[nn] = 1; nn++;
  }
  double maxe = 0.0;
  for (int k = 0; k < nn; k++) {
    int qx = gx + ndx[k], qy = gy + ndy[k];
    bool nf = false;
    double nd = 0.0;
    V3 nnv = mk(0, 0, 0);
    if (qx < F.W && qy < F.H) {  // get_depth / get_normal bounds (src/outline.rs:68-82)
      nf = sv[ly + ndy[k]][lx + ndx[k]] != 0;
      nd = sd[ly + ndy[k]][lx + ndx[k]];
      nnv = mk(snx[ly + ndy[k]][lx + ndx[k]], sny[ly + ndy[k]][lx + ndx[k]], snz[ly + ndy[k]][lx + ndx[k]]);
    }
    double e;
    if (cf && nf) {
      double dd = fabs(cd - nd);
      double ndd = dd / rmax(cd * 0.1, 0.1);
      double dp = rclamp(dot(cn, nnv), -1.0, 1.0);
      e = F.o_wd * ndd + F.o_wn * (1.0 - dp);
      // extension: different objects on either side of the edge
      if (ids && so[ly][lx] != so[ly + ndy[k]][lx + ndx[k]]) e = e + F.o_wid;
    } else if (cf != nf) {
      e = F.o_wd * 2.0 + F.o_wn * 2.0;
    } else {
      e = 0.0;
    }
    maxe = rmax(maxe, e);
  }
  double m = 0.0;
  if (maxe > F.o_thr) m = (maxe - F.o_thr) / rmax(1.0 - F.o_thr, 0.001);
  F.mask[(long long)gy * F.W + gx] = m;
}

// dilate_edges + blend_colors + quantise (src/outline.rs:227-278,
// src/renderer.rs:899-912); the mask tile with a halo of `radius` pixels is
// staged in dynamic shared memory.
__global__ void __launch_bounds__(OT_X* OT_Y) k_outline_apply(DFrame F) {
  extern __shared__ double sm[];
  int R = F.o_radius;
  int TW = OT_X + 2 * R, TH = OT_Y + 2 * R;
  int x0 = blockIdx.x * OT_X - R, y0 = blockIdx.y * OT_Y - R;
  for (int k = threadIdx.y * OT_X + threadIdx.x; k < TW * TH; k += OT_X * OT_Y) {
    int lx = k % TW, ly = k / TW;
    int gx = x0 + lx, gy = y0 + ly;
    double v = 0.0;
    if (gx >= 0 && gy >= 0 && gx < F.W && gy < F.H) v = F.mask[(long long)gy * F.W + gx];
    sm[k] = v;
  }
  __syncthreads();
  int gx = blockIdx.x * OT_X + threadIdx.x, gy = blockIdx.y * OT_Y + threadIdx.y;
  if (gx >= F.W || gy >= F.H) return;
  int lx = threadIdx.x + R, ly = threadIdx.y + R;
  double ms = sm[ly * TW + lx];
  if (R > 0) {
    double th = F.o_thick;
    for (int dy = -R; dy <= R; dy++)
      for (int dx = -R; dx <= R; dx++) {
        int nx = gx + dx, ny = gy + dy;
        if (nx >= 0 && ny >= 0 && nx < F.W && ny < F.H) {
          double dist = sqrt((double)(dx * dx + dy * dy));
          if (dist <= th) {
            double fo = 1.0 - (dist / th);
            ms = rmax(ms, sm[(ly + dy) * TW + (lx + dx)] * fo);
          }
        }
      }
  }
  long long p = (long long)gy * F.W + gx;
  V3 c = mk(F.cr[p], F.cg[p], F.cb[p]);
  if (ms > 0.0) {
    double w = rclamp(rmin(ms, 1.0), 0.0, 1.0);
    c = mk(c.x * (1.0 - w) + F.o_color[0] * w, c.y * (1.0 - w) + F.o_color[1] * w,
           c.z * (1.0 - w) + F.o_color[2] * w);
  }
  store_rgb(F, p, c);
}

// k_outline_apply for radii whose mask tile does not fit in shared memory
// (outline thickness above 65): the same dilation, reading the mask from
// global memory (its neighbourhood stays in L1/L2).  One thread per pixel.
__global__ void __launch_bounds__(256) k_outline_apply_wide(DFrame F) {
  const int R = F.o_radius;
  const double th = F.o_thick;
  const long long n = (long long)F.W * F.H;
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x) {
    const int gx = (int)(p % F.W), gy = (int)(p / F.W);
    double ms = F.mask[p];
    for (int dy = -R; dy <= R; dy++) {
      const int ny = gy + dy;
      if (ny < 0 || ny >= F.H) continue;
      for (int dx = -R; dx <= R; dx++) {
        const int nx = gx + dx;
        if (nx < 0 || nx >= F.W) continue;
        double dist = sqrt((double)(dx * dx + dy * dy));
        if (dist <= th) {
          double fo = 1.0 - (dist / th);
          ms = rmax(ms, __ldg(F.mask + (long long)ny * F.W + nx) * fo);
        }
      }
    }
    V3 c = mk(F.cr[p], F.cg[p], F.cb[p]);
    if (ms > 0.0) {
      double w = rclamp(rmin(ms, 1.0), 0.0, 1.0);
      c = mk(c.x * (1.0 - w) + F.o_color[0] * w, c.y * (1.0 - w) + F.o_color[1] * w,
             c.z * (1.0 - w) + F.o_color[2] * w);
    }
    store_rgb(F, p, c);
  }
}

// --------------------------------------------------------------------------
// Unit kernels for the parity tests and the FP64 rate probe
// --------------------------------------------------------------------------
// Eight independent add/multiply chains per thread; each iteration issues
// 16 FP64 add and 16 FP64 multiply instructions.
__global__ void k_fp64_rate(double* out, int iters, double a, double b) {
  double x[8], y[8];
  for (int k = 0; k < 8; k++) {
    x[k] = threadIdx.x * 1e-3 + k;
    y[k] = blockIdx.x * 1e-3 + k;
  }
  for (int i = 0; i < iters; i++) {
#pragma unroll
    for (int k = 0; k < 8; k++) {
      x[k] = x[k] * a + b;
      y[k] = y[k] * b + a;
    }
  }
  double s = 0;
  for (int k = 0; k < 8; k++) s += x[k] + y[k];
  if (s == 12345.678) out[0] = s;  // keeps the chains live
}
// Read bandwidth of a buffer small enough to stay in L2: 16-byte loads
// with ld.global.cg (cached in L2, not L1, so no pass is served by L1),
// four independent loads per thread in flight, `reps` passes over the
// buffer.  n16 is the buffer's size in 16-byte vectors, a multiple of
// 4 * gridDim.x * blockDim.x.
__global__ void k_l2_read(const uint4* __restrict__ buf, long long n16, int reps, unsigned* out) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  unsigned acc = 0;
  for (int r = 0; r < reps; r++) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n16; i += 4 * stride) {
      uint4 a = __ldcg(buf + i), b = __ldcg(buf + i + stride), c = __ldcg(buf + i + 2 * stride),
            d = __ldcg(buf + i + 3 * stride);
      acc ^= a.x ^ a.y ^ a.z ^ a.w ^ b.x ^ b.y ^ b.z ^ b.w ^ c.x ^ c.y ^ c.z ^ c.w ^ d.x ^ d.y ^ d.z ^ d.w;
    }
  }
  if (acc == 0x9E3779B9u) out[0] = acc;  // keeps the loads live
}
__global__ void k_debug_rng(const uint64_t* seeds, long long n, int nw, uint32_t* out) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    StdRng r;
    r.init(seeds[i]);
    for (int k = 0; k < nw; k++) out[i * nw + k] = r.u32();
  }
}
__global__ void k_debug_disk(const uint64_t* seeds, long long n, double radius, double* out, int* err) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    StdRng r;
    r.init(seeds[i]);
    for (int s = 0; s < 16; s++) {
      double dx = 0, dy = 0;
      for (int it = 0;; it++) {
        if (it >= 4096 || !r.range(-radius, radius, &dx) || !r.range(-radius, radius, &dy)) {
          atomicOr(err, ERR_WATCHDOG);
          break;
        }
        if (dx * dx + dy * dy <= radius * radius) break;
      }
      out[i * 32 + 2 * s] = dx;
      out[i * 32 + 2 * s + 1] = dy;
    }
  }
}
// Mesh queries for the parity tests: closest hit as the renderer runs it
// (mode 0: BVH search + reference-leaf verification), the plain reference
// k-d walk (mode 1), any-hit as shadow rays run it (mode 2),
// and for every k-d leaf the cell-based visit test against the root walk
// (mode 3: out = {leaves where they differ, where they agree, leaves the
// walk visits}).  128 threads per block.
__global__ void __launch_bounds__(128) k_debug_mesh(DMesh M, int use_kd, int mode, const double* rays, long long n,
                                                    double tmin, double tmax, double* out, int* err) {
  for (long long base = blockIdx.x * (long long)blockDim.x + (threadIdx.x & ~31); base < n;
       base += (long long)gridDim.x * blockDim.x) {
    const long long i = base + (threadIdx.x & 31);
    const bool valid = i < n;
    V3 o = mk(0.0, 0.0, 0.0), d = mk(0.0, 0.0, 1.0);
    if (valid) {
      const double* rr = rays + 6 * i;
      o = mk(rr[0], rr[1], rr[2]);
      d = normalize(mk(rr[3], rr[4], rr[5]));
    }
    RayC r = make_rayc(o, d);
    double closest = tmax;
    int best = -1;
    double* oo = out + 8 * (valid ? i : 0);
    if (mode == 3) {
      // every k-d leaf: the cell-based visit test against the root walk
      if (valid) {
        double agree = 0.0, visited = 0.0, differ = 0.0;
        for (int k = 0; k < M.n_nodes; k++) {
          if (hi32(__ldg(M.nodes + 4 * (size_t)k + 3).y) >= 0) continue;
          unsigned key;
          const bool a = kd_leaf_visited_cell(M, r, k, nullptr), b = kd_leaf_visited(M, r, k, &key);
          if (a == b) agree += 1.0;
          else differ += 1.0;
          if (b) visited += 1.0;
        }
        for (int k = 0; k < 8; k++) oo[k] = 0.0;
        oo[0] = differ;
        oo[1] = agree;
        oo[2] = visited;
      }
      continue;
    }
    if (mode == 2) {
      if (valid) {
        for (int k = 0; k < 8; k++) oo[k] = 0.0;
        oo[0] = shadow_mesh(M, o, d, tmin, tmax, use_kd != 0, err, nullptr) ? 1.0 : 0.0;
      }
      continue;
    }
    bool hit = valid && (mode == 0 ? mesh_closest(M, o, d, tmin, closest, best, use_kd != 0, err, nullptr)
                                   : (mesh_bounds(M, r, tmin, closest) &&
                                      mesh_kd_walk(M, r, tmin, closest, best, err, nullptr)));
    if (!valid) continue;
    for (int k = 0; k < 8; k++) oo[k] = 0.0;
    if (hit) {
      const double2* E = M.brute + 5 * (size_t)best;
      double2 q1 = E[1], q2 = E[2], q3 = E[3], q4 = E[4];
      V3 e1 = mk(q1.y, q2.x, q2.y), e2 = mk(q3.x, q3.y, q4.x);
      double a = dot(e1, cross(r.d, e2));
      double4 nn = M.normals[best];
      V3 nv = mk(nn.x, nn.y, nn.z);
      if (a < 0.0) nv = -nv;
      V3 p = r.o + closest * r.d;
      V3 fn = face_normal(r.d, nv);
      oo[0] = 1.0;
      oo[1] = closest;
      oo[2] = p.x;
      oo[3] = p.y;
      oo[4] = p.z;
      oo[5] = fn.x;
      oo[6] = fn.y;
      oo[7] = fn.z;
    }
  }
}

}  // namespace rtb
