// kf_raycast.cu — surface prediction by ray marching the TSDF.
//
// Reference: gFusion::raycast (src/gFusion.cpp:1289-1366) and shaders/raycast.cs:133-321:
// view = m_pose * invK; ray origin = pose translation, direction = R * K^-1 (u, v, 1)
// (unnormalised: t is camera z); slab test against [0, volDim]^3 clipped to
// [nearPlane, farPlane]; no hit if the first sample is negative; march with largeStep
// until a sample drops below 0.8, then with step = voxel size (stepSize(), Q9), stop at
// the first negative sample; refine t + step * f_tt / (f_t - f_tt); trilinear samples
// (interpVol :69-82, no weight test, border-clamped taps); normal = normalised
// central-difference trilinear gradient (getGradient :229-276), zero when its length is
// zero.  Misses write zero vertex and normal.
//
// B200 design: one thread per pixel, 32-wide tiles so a warp's rays stay coherent and its
// trilinear taps share L1 lines; the value plane alone is read (2 B per tap for the
// 16-bit storages).  The march position is t0 + k * step (one rounding) rather than the
// reference's repeated float addition.  Once the march is in its fine-step phase it
// skips every brick that holds no negative value (no sample there can be the first
// negative one), keeping the sample positions tb + k * step and re-evaluating the sample
// before a hit for the refinement, so the result is the unskipped march's.  The flags are
// read as bits, 4^3 bricks to a word: 32 KB for 512^3, which stays in L1, and a zero word
// skips 32 voxels at once.
// What bounds it: the chain of a ray's samples (13 coarse, 16 skips and 22 fine ones on average
// at 512^3) and its tail, a few rays of 200 steps that graze surfaces.  Device us per view,
// one sample at a time with word flags and exactly verified skips -> now: 512^3 102 -> 60,
// 768^3 293 -> 168, 128^3 46 -> 32, 16 batched sessions 672 -> 567.
#include "kf_internal.cuh"

namespace {

struct RayArgs {
  const void* vol;
  int nx, ny, nz;
  float sx, sy, sz;         // volSize / volDim
  float gx, gy, gz;         // volDim / volSize * 0.5 (getGradient scale, :273)
  float dimx, dimy, dimz;
  float step, large_step, nearp, farp;
  int max_steps;
  int W, H;
  float ikx, iky, ikcx, ikcy;  // getInverseCameraMatrix: 1/fx, 1/fy, -cx/fx, -cy/fy (float)
  float4* out_v;
  float4* out_n;
  const KfDevState* st;
  KfDevState* st_out;
  float inv_step;
  const unsigned long long* neg;  // NEG bits
  int wx, wy;
};

// 32 x ROWS pixel tiles (ROWS one of KF_RAY_ROWS, chosen per session: default 4, or the
// autotuner's pick): ray lengths vary a lot, and small blocks keep the SMs evenly loaded to
// the end of the launch (512 x 424 in 32 x 4 tiles gives 1,696 blocks).  Every choice
// computes the same maps.

template <int S>
struct Sampler {
  typedef typename Vox<S>::V V;
  const V* f;
  int nx, ny, nz;
  uint32_t sxy;
  __device__ __forceinline__ float tap(int x, int y, int z) const {
    return Vox<S>::raw(f, (uint32_t)x + (uint32_t)nx * (uint32_t)y + sxy * (uint32_t)z);
  }
  // The base voxel of a sample and the weights of its far taps.  floor by an add rounded down
  // (exact below 2^22): the rounding and conversion instructions run at a quarter rate.
  struct Cell {
    int x, y, z;
    float fx, fy, fz;
  };
  static __device__ __forceinline__ int floor_of(float q, float* frac) {
    constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23
    const float t = __fadd_rd(q, kMagic);
    *frac = q - (t - kMagic);
    return __float_as_int(t) - 0x4B400000;
  }
  static __device__ __forceinline__ Cell cell(float qx, float qy, float qz) {
    Cell c;
    c.x = floor_of(qx, &c.fx);
    c.y = floor_of(qy, &c.fy);
    c.z = floor_of(qz, &c.fz);
    return c;
  }
  // interpVol (raycast.cs:69-82) before the final * (1/32766), taps clamped to the volume.
  // The 8 taps share one base offset.
  __device__ __forceinline__ float interp(const Cell& p) const {
    const int lx = min(max(p.x, 0), nx - 1), ly = min(max(p.y, 0), ny - 1), lz = min(max(p.z, 0), nz - 1);
    const int ux = max(min(p.x + 1, nx - 1), 0), uy = max(min(p.y + 1, ny - 1), 0), uz = max(min(p.z + 1, nz - 1), 0);
    const uint32_t b = (uint32_t)lx + (uint32_t)nx * (uint32_t)ly + sxy * (uint32_t)lz;
    const uint32_t ox = (uint32_t)(ux - lx), oy = (uint32_t)(uy - ly) * (uint32_t)nx,
                   oz = (uint32_t)(uz - lz) * sxy;
    const float fx = p.fx, fy = p.fy, fz = p.fz;
    const float c000 = Vox<S>::raw(f, b), c100 = Vox<S>::raw(f, b + ox);
    const float c010 = Vox<S>::raw(f, b + oy), c110 = Vox<S>::raw(f, b + ox + oy);
    const float c001 = Vox<S>::raw(f, b + oz), c101 = Vox<S>::raw(f, b + ox + oz);
    const float c011 = Vox<S>::raw(f, b + oy + oz), c111 = Vox<S>::raw(f, b + ox + oy + oz);
    return ((c000 * (1 - fx) + c100 * fx) * (1 - fy) + (c010 * (1 - fx) + c110 * fx) * fy) * (1 - fz) +
           ((c001 * (1 - fx) + c101 * fx) * (1 - fy) + (c011 * (1 - fx) + c111 * fx) * fy) * fz;
  }
  // q in voxel coordinates (world * volSize / volDim - 0.5)
  __device__ __forceinline__ float interp_raw(float qx, float qy, float qz) const { return interp(cell(qx, qy, qz)); }
};

// An integer 0 <= i < 2^23 as float without a conversion instruction.
__device__ __forceinline__ float float_of(int i) { return __int_as_float(0x4B000000 | i) - 8388608.0f; }

// A pixel's ray (raycast.cs:133-152) for view rows s_view (m_pose * invK): direction, slab
// clipped to the near and far planes, and the ray in voxel coordinates:
// q(t) = (o + d t) * volSize / volDim - 0.5 = q0 + t dq.
struct Ray {
  float dx, dy, dz;
  float tnear, tfar;
  float q0x, q0y, q0z, dqx, dqy, dqz;
};

__device__ __forceinline__ Ray make_ray(const RayArgs& a, const float* s_view, int x, int y) {
  Ray r;
  const float ox = s_view[3], oy = s_view[7], oz = s_view[11];
  const float fxp = (float)x, fyp = (float)y;
  r.dx = fmaf(s_view[0], fxp, fmaf(s_view[1], fyp, s_view[2]));
  r.dy = fmaf(s_view[4], fxp, fmaf(s_view[5], fyp, s_view[6]));
  r.dz = fmaf(s_view[8], fxp, fmaf(s_view[9], fyp, s_view[10]));
  // slab test (raycast.cs:141-152)
  const float ix = 1.0f / r.dx, iy = 1.0f / r.dy, iz = 1.0f / r.dz;
  const float tbx = -1.0f * ix * ox, tby = -1.0f * iy * oy, tbz = -1.0f * iz * oz;
  const float ttx = ix * (a.dimx - ox), tty = iy * (a.dimy - oy), ttz = iz * (a.dimz - oz);
  const float tminx = fminf(ttx, tbx), tminy = fminf(tty, tby), tminz = fminf(ttz, tbz);
  const float tmaxx = fmaxf(ttx, tbx), tmaxy = fmaxf(tty, tby), tmaxz = fmaxf(ttz, tbz);
  const float largest_tmin = fmaxf(fmaxf(tminx, tminy), fmaxf(tminx, tminz));
  const float smallest_tmax = fminf(fminf(tmaxx, tmaxy), fminf(tmaxx, tmaxz));
  r.tnear = fmaxf(largest_tmin, a.nearp);
  r.tfar = fminf(smallest_tmax, a.farp);
  r.q0x = fmaf(ox, a.sx, -0.5f);
  r.q0y = fmaf(oy, a.sy, -0.5f);
  r.q0z = fmaf(oz, a.sz, -0.5f);
  r.dqx = r.dx * a.sx;
  r.dqy = r.dy * a.sy;
  r.dqz = r.dz * a.sz;
  return r;
}

// Empty-space skipping in the fine phase.  A sample's eight taps lie in the brick of its base
// voxel; a brick without a negative value (or 4^3 of them, a zero word) cannot hold the first
// negative sample.  Such samples change nothing but f_t, so the march jumps to the first
// sample past the region's exit plane; the positions stay tb + k * step, as in the unskipped
// march.  Exit along an axis: t = edge * r + e with r the reciprocal slope; e moves the plane
// inwards by more than the positions' rounding, so that every skipped sample lies in the
// region.
struct Exits {
  float rx, ry, rz, ex, ey, ez;
};

__device__ __forceinline__ Exits make_exits(const RayArgs& a, const Ray& ray) {
  Exits v;
  auto axis = [](float dq, float q0, int n, float* r, float* e) {
    *r = dq != 0.0f ? 1.0f / dq : 0.0f;
    *e = dq != 0.0f ? -q0 * *r - (0.01f + 1e-6f * (fabsf(q0) + (float)n)) * fabsf(*r) : 1e30f;
  };
  axis(ray.dqx, ray.q0x, a.nx, &v.rx, &v.ex);
  axis(ray.dqy, ray.q0y, a.ny, &v.ry, &v.ey);
  axis(ray.dqz, ray.q0z, a.nz, &v.rz, &v.ez);
  return v;
}

// The NEG words a ray passes, the last one kept.
struct NegWord {
  uint32_t at = 0xffffffffu;
  unsigned long long word = 0;
};

// Whether the sample in cell p of a fine march (from tb) may be negative; else *next is the
// number of the first sample past the region without a negative value that p lies in.
template <class Cell>
__device__ __forceinline__ bool may_be_negative(const RayArgs& a, const Ray& ray, const Exits& v, const Cell& p,
                                                float tb, NegWord* nw, float* next) {
  const int vx = min(max(p.x, 0), a.nx - 1), vy = min(max(p.y, 0), a.ny - 1), vz = min(max(p.z, 0), a.nz - 1);
  const uint32_t w = kf_neg_word(vx >> 3, vy >> 3, vz >> 3, a.wx, a.wy);
  if (w != nw->at) {
    nw->at = w;
    nw->word = __ldg(a.neg + w);
  }
  if (nw->word >> ((vx >> 3 & 3) | (vy >> 3 & 3) << 2 | (vz >> 3 & 3) << 4) & 1u) return true;
  const int sh = nw->word ? 3 : 5;
  const float te = fminf(fminf(fmaf(float_of(((vx >> sh) + (ray.dqx > 0.0f)) << sh), v.rx, v.ex),
                               fmaf(float_of(((vy >> sh) + (ray.dqy > 0.0f)) << sh), v.ry, v.ey)),
                         fmaf(float_of(((vz >> sh) + (ray.dqz > 0.0f)) << sh), v.rz, v.ez));
  *next = floorf((fminf(te, ray.tfar) - tb) * a.inv_step) + 1.0f;
  return false;
}

// The sample number after k; from 2^24 on the next one that exists (a march of that many steps
// visits every representable position, as with integer numbers rounded to float).
__device__ __forceinline__ float after(float k) {
  const float r = k + 1.0f;
  return r > k ? r : __int_as_float(__float_as_int(k) + 1);
}

// Samples a thread takes together.  One 512 x 424 view is 46 warps per SM, too few to hide the
// taps' latency one sample at a time; a batch fills the GPU and is bound by issue, where
// discarded samples cost (device us at 1 / 2 / 3 / 4 samples: 512^3 79 / 65 / 60 / 58, 768^3
// 259 / 190 / 168 / 163, 128^3 37 / 33 / 32 / 33; 16 batched sessions 578 / 567 / 604 / 655).
constexpr int kAheadOne = 3, kAheadBatch = 2;

// raycast.cs:153-199 for one ray by one thread: the hit's t, 0 for a miss.  AHEAD consecutive
// samples are taken together and examined in order (the positions do not depend on the
// samples); those past the first that matters are discarded.
template <int S, int AHEAD>
__device__ __forceinline__ float march_ray(const RayArgs& a, const Sampler<S>& smp, const Ray& ray) {
  if (!(ray.tnear < ray.tfar)) return 0.0f;
  const float scale = Vox<S>::kRawToF;
  float t = ray.tnear, stepsize = a.large_step;
  auto cell = [&](float tt) {
    return Sampler<S>::cell(fmaf(tt, ray.dqx, ray.q0x), fmaf(tt, ray.dqy, ray.q0y), fmaf(tt, ray.dqz, ray.q0z));
  };
  float f_t = smp.interp(cell(t)) * scale;
  if (!(f_t >= 0.0f)) return 0.0f;
  const Exits v = make_exits(a, ray);
  float tb = t;
  float k = 0.0f;          // sample number since tb
  bool fine = false;       // stepsize == step (the reference never switches back)
  bool prev_known = true;  // f_t holds the sample just before t
  NegWord nw;
  // bounded march: a NaN sample keeps largeStep, so cap the step count
  for (int n = 0; t < ray.tfar && n < a.max_steps; ++n) {
    const auto p = cell(t);
    float next;
    if (fine && !may_be_negative(a, ray, v, p, tb, &nw, &next)) {
      k = fmaxf(after(k), next);
      t = fmaf(k, stepsize, tb);
      prev_known = false;
      continue;
    }
    float ts[AHEAD], fs[AHEAD];
    ts[0] = t;
    fs[0] = smp.interp(p) * scale;
#pragma unroll
    for (int i = 1; i < AHEAD; ++i) {
      ts[i] = fmaf(k + (float)i, stepsize, tb);
      fs[i] = smp.interp(cell(ts[i])) * scale;
    }
    float f_tt = fs[0];
    bool on = true;  // the samples so far change nothing but f_t
#pragma unroll
    for (int i = 1; i < AHEAD; ++i) {
      on = on && !(f_tt < (fine ? 0.0f : 0.8f)) && ts[i] < ray.tfar;
      if (on) {
        f_t = f_tt;
        prev_known = true;
        f_tt = fs[i];
        k += 1.0f;
        t = ts[i];
      }
    }
    if (f_tt < 0.0f) {
      if (!prev_known) f_t = smp.interp(cell(fmaf(k - 1.0f, stepsize, tb))) * scale;
      return t + stepsize * f_tt / (f_t - f_tt);
    }
    if (f_tt < 0.8f && !fine) {
      fine = true;
      stepsize = a.step;
      tb = t;
      k = 0.0f;
    }
    f_t = f_tt;
    prev_known = true;
    k = after(k);
    t = fmaf(k, stepsize, tb);
  }
  return 0.0f;
}

// The pixel's vertex and normal for a hit at ht (0: none).
template <int S>
__device__ __forceinline__ void write_pixel(const RayArgs& a, const Sampler<S>& smp, const float* s_view, const Ray& ray,
                                            int x, int y, float ht) {
  const float scale = Vox<S>::kRawToF;
  const size_t o = (size_t)y * a.W + x;
  if (ht > 0.0f) {
    const float hx = fmaf(ray.dx, ht, s_view[3]), hy = fmaf(ray.dy, ht, s_view[7]), hz = fmaf(ray.dz, ht, s_view[11]);
    a.out_v[o] = make_float4(hx, hy, hz, 1.0f);
    // getGradient (raycast.cs:229-276)
    const float qx = hx * a.sx - 0.5f, qy = hy * a.sy - 0.5f, qz = hz * a.sz - 0.5f;
    const float bx = floorf(qx), by = floorf(qy), bz = floorf(qz);
    const float f3[3] = {qx - bx, qy - by, qz - bz};
    const int bi[3] = {(int)bx, (int)by, (int)bz};
    const int n3[3] = {a.nx, a.ny, a.nz};
    int ll[3], lu[3], ul[3], uu[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      ll[k] = min(max(bi[k] - 1, 0), n3[k] - 1);
      lu[k] = min(max(bi[k], 0), n3[k] - 1);
      ul[k] = max(min(bi[k] + 1, n3[k] - 1), 0);
      uu[k] = max(min(bi[k] + 2, n3[k] - 1), 0);
    }
    float g[3];
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
      float acc = 0.0f;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const int cc[3] = {c & 1, (c >> 1) & 1, (c >> 2) & 1};
        int pa[3], pb[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          if (k == ax) {
            pa[k] = cc[k] ? uu[k] : ul[k];
            pb[k] = cc[k] ? lu[k] : ll[k];
          } else {
            pa[k] = cc[k] ? ul[k] : lu[k];
            pb[k] = pa[k];
          }
        }
        const float w = (cc[0] ? f3[0] : 1.0f - f3[0]) * (cc[1] ? f3[1] : 1.0f - f3[1]) *
                        (cc[2] ? f3[2] : 1.0f - f3[2]);
        acc = fmaf(w, smp.tap(pa[0], pa[1], pa[2]) - smp.tap(pb[0], pb[1], pb[2]), acc);
      }
      g[ax] = acc;
    }
    const float gx = g[0] * a.gx * scale, gy = g[1] * a.gy * scale, gz = g[2] * a.gz * scale;
    const float len = sqrtf(gx * gx + gy * gy + gz * gz);
    if (len == 0.0f)
      a.out_n[o] = make_float4(0.f, 0.f, 0.f, 0.f);
    else
      a.out_n[o] = make_float4(gx / len, gy / len, gz / len, 1.0f);
  } else {
    a.out_v[o] = make_float4(0.f, 0.f, 0.f, 0.f);
    a.out_n[o] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

template <int S>
__device__ __forceinline__ Sampler<S> make_sampler(const RayArgs& a) {
  Sampler<S> smp;
  smp.f = reinterpret_cast<const typename Vox<S>::V*>(a.vol);
  smp.nx = a.nx; smp.ny = a.ny; smp.nz = a.nz;
  smp.sxy = (uint32_t)a.nx * (uint32_t)a.ny;
  return smp;
}

// view = m_pose * invK (gFusion.cpp:1296) from the FP32 pose rows and float invK; thread
// t < 12 writes element t of the 3x4 rows.
__device__ __forceinline__ void raycast_view(const RayArgs& a, float* s_view, int t) {
  const int r = t >> 2, c = t & 3;
  const float* P = a.st->pose_rows;
  float v;
  if (c == 0) v = P[r * 4 + 0] * a.ikx;
  else if (c == 1) v = P[r * 4 + 1] * a.iky;
  else if (c == 2) v = fmaf(P[r * 4 + 0], a.ikcx, fmaf(P[r * 4 + 1], a.ikcy, P[r * 4 + 2]));
  else v = P[r * 4 + 3];
  s_view[r * 4 + c] = v;
}

// Lane l of warp w in a 32 x ROWS tile.
template <int ROWS>
__device__ __forceinline__ int tile_x(int w, int l) {
  return ROWS == 2 ? w * 16 + (l & 15) : (w & 3) * 8 + (l & 7);
}
template <int ROWS>
__device__ __forceinline__ int tile_y(int w, int l) {
  return ROWS == 2 ? l >> 4 : (w >> 2) * 4 + (l >> 3);
}

// BATCH: blockIdx.z selects the session's arguments in `many`.
template <int S, bool BATCH, int ROWS>
__global__ void __launch_bounds__(32 * ROWS, BATCH ? 28 / ROWS : 1) raycast_kernel(RayArgs one, const RayArgs* many) {
  static_assert(ROWS == 2 || ROWS == 4 || ROWS == 8, "raycast tile rows: 2, 4 or 8");
  __shared__ RayArgs s_args;
  __shared__ float s_view[12];  // rows of m_pose * invK: (R K^-1 | t)
  if constexpr (BATCH) {
    const int tid = threadIdx.y * 32 + threadIdx.x;
    const int* src = reinterpret_cast<const int*>(many + blockIdx.z);
    for (int k = tid; k < (int)(sizeof(RayArgs) / 4); k += 32 * ROWS) reinterpret_cast<int*>(&s_args)[k] = __ldg(src + k);
    __syncthreads();
  }
  const RayArgs& a = BATCH ? s_args : one;
  if (threadIdx.y == 0 && threadIdx.x < 12) raycast_view(a, s_view, threadIdx.x);
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.y == 1 && threadIdx.x < 16)
    a.st_out->raycast_pose[threadIdx.x] = a.st->pose[threadIdx.x];
  __syncthreads();
  // each warp takes a compact patch of the 32 x ROWS tile (16 x 2 pixels in 2-row tiles,
  // 8 x 4 otherwise): neighbouring rays march through the same bricks and end at similar
  // depths, so a warp's taps share cache lines and its lanes finish together (measured
  // ~1 % faster than a 32 x 1 row per warp)
  const int t = threadIdx.y * 32 + threadIdx.x, w = t >> 5, l = t & 31;
  const int x = blockIdx.x * 32 + tile_x<ROWS>(w, l), y = blockIdx.y * ROWS + tile_y<ROWS>(w, l);
  if (x >= a.W || y >= a.H) return;
  const Sampler<S> smp = make_sampler<S>(a);
  const Ray ray = make_ray(a, s_view, x, y);
  write_pixel<S>(a, smp, s_view, ray, x, y, march_ray<S, BATCH ? kAheadBatch : kAheadOne>(a, smp, ray));
}

// The same rays as a persistent sweep: one block per resident slot, and every warp takes
// the next row segment of 32 pixels from a device counter until the image is done, so no
// warp waits for another and long rays do not leave SMs idle at the end of the launch.
// The last warp to find the queue empty resets the counter (and its own completion count)
// for the next launch.  Every pixel runs the same march: the maps are the tiled kernel's.
template <int S>
__global__ void __launch_bounds__(256) raycast_sweep_kernel(RayArgs a, unsigned* queue) {
  __shared__ float s_view[12];
  const int lane = threadIdx.x & 31;
  if (threadIdx.x < 12) raycast_view(a, s_view, threadIdx.x);
  if (blockIdx.x == 0 && threadIdx.x >= 32 && threadIdx.x < 48)
    a.st_out->raycast_pose[threadIdx.x - 32] = a.st->pose[threadIdx.x - 32];
  __syncthreads();
  const int segs_x = (a.W + 31) / 32;
  const unsigned nseg = (unsigned)segs_x * (unsigned)a.H;
  for (;;) {
    unsigned seg = 0;
    if (lane == 0) seg = atomicAdd(queue, 1u);
    seg = __shfl_sync(0xffffffffu, seg, 0);
    if (seg >= nseg) break;
    const int y = (int)(seg / (unsigned)segs_x);
    const int x = (int)(seg % (unsigned)segs_x) * 32 + lane;
    if (x < a.W) {
      const Sampler<S> smp = make_sampler<S>(a);
      const Ray ray = make_ray(a, s_view, x, y);
      write_pixel<S>(a, smp, s_view, ray, x, y, march_ray<S, kAheadOne>(a, smp, ray));
    }
  }
  // every warp drew one ticket past the end; the last of them resets the queue
  if (lane == 0) {
    const unsigned warps = gridDim.x * (blockDim.x / 32);
    if (atomicAdd(queue + 1, 1u) == warps - 1) {
      queue[0] = 0u;
      queue[1] = 0u;
    }
  }
}

// Volume ray-sum image (gFusion::intensityProjection, src/gFusion.cpp:1368-1409, and
// shaders/mip.cs:52-104): the raycast's view, slab test and near/far clipping, then samples
// every largeStep from tnear while t < tfar, summing the positive interpolated values into
// x; the pixel is (sum, 0, 0, 1), misses included (mip.cs's other two branches add zero or
// are unreachable).  Sample positions are tnear + k * largeStep (one rounding, as in the
// raycast).  The reference dispatches it on demand, never from the frame loop; so does this.
template <int S>
__global__ void __launch_bounds__(128) mip_kernel(RayArgs a, float4* out) {
  __shared__ float s_view[12];
  if (threadIdx.y == 0 && threadIdx.x < 12) {
    const int r = threadIdx.x >> 2, c = threadIdx.x & 3;
    const float* P = a.st->pose_rows;
    float v;
    if (c == 0) v = P[r * 4 + 0] * a.ikx;
    else if (c == 1) v = P[r * 4 + 1] * a.iky;
    else if (c == 2) v = fmaf(P[r * 4 + 0], a.ikcx, fmaf(P[r * 4 + 1], a.ikcy, P[r * 4 + 2]));
    else v = P[r * 4 + 3];
    s_view[r * 4 + c] = v;
  }
  __syncthreads();
  const int x = blockIdx.x * 32 + threadIdx.x;
  const int y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= a.W || y >= a.H) return;
  Sampler<S> smp;
  smp.f = reinterpret_cast<const typename Vox<S>::V*>(a.vol);
  smp.nx = a.nx; smp.ny = a.ny; smp.nz = a.nz;
  smp.sxy = (uint32_t)a.nx * (uint32_t)a.ny;

  const float ox = s_view[3], oy = s_view[7], oz = s_view[11];
  const float fxp = (float)x, fyp = (float)y;
  const float dx = fmaf(s_view[0], fxp, fmaf(s_view[1], fyp, s_view[2]));
  const float dy = fmaf(s_view[4], fxp, fmaf(s_view[5], fyp, s_view[6]));
  const float dzv = fmaf(s_view[8], fxp, fmaf(s_view[9], fyp, s_view[10]));
  // slab test (mip.cs:61-77, as raycast.cs:141-152)
  const float ix = 1.0f / dx, iy = 1.0f / dy, iz = 1.0f / dzv;
  const float tbx = -1.0f * ix * ox, tby = -1.0f * iy * oy, tbz = -1.0f * iz * oz;
  const float ttx = ix * (a.dimx - ox), tty = iy * (a.dimy - oy), ttz = iz * (a.dimz - oz);
  const float tminx = fminf(ttx, tbx), tminy = fminf(tty, tby), tminz = fminf(ttz, tbz);
  const float tmaxx = fmaxf(ttx, tbx), tmaxy = fmaxf(tty, tby), tmaxz = fmaxf(ttz, tbz);
  const float largest_tmin = fmaxf(fmaxf(tminx, tminy), fmaxf(tminx, tminz));
  const float smallest_tmax = fminf(fminf(tmaxx, tmaxy), fminf(tmaxx, tmaxz));
  const float tnear = fmaxf(largest_tmin, a.nearp);
  const float tfar = fminf(smallest_tmax, a.farp);

  float sum = 0.0f;
  if (tnear < tfar) {
    const float scale = Vox<S>::kRawToF;
    const float q0x = fmaf(ox, a.sx, -0.5f), q0y = fmaf(oy, a.sy, -0.5f), q0z = fmaf(oz, a.sz, -0.5f);
    const float dqx = dx * a.sx, dqy = dy * a.sy, dqz = dzv * a.sz;
    // bounded: max_steps covers (far - near) / min(step, largeStep) samples
    for (int k = 0; k < a.max_steps; ++k) {
      const float t = fmaf((float)k, a.large_step, tnear);
      if (!(t < tfar)) break;
      const float f = smp.interp_raw(fmaf(t, dqx, q0x), fmaf(t, dqy, q0y), fmaf(t, dqz, q0z)) * scale;
      if (f > 0.0f) sum += f;
    }
  }
  out[(size_t)y * a.W + x] = make_float4(sum, 0.0f, 0.0f, 1.0f);
}

// Exact brick flags from the volume itself: only a brick whose flag is set can lose it, so a
// block reads 32 flag words, and its 8 warps check the set ones against the volume, three
// planes at a time until each set bit is confirmed: NEG by a negative value over the voxels
// [8B, 8B+8], SET by a nonzero bit in a value or weight of [8B, 8B+8).  The NEG bits are
// cleared first and set here.  The set bricks come in runs along x, hence few words per block
// (at most four bricks in a row for a warp, whose latency the launch waits for).
template <int S>
__global__ void __launch_bounds__(256) refresh_bricks_kernel(const void* vol, size_t count, int nx, int ny, int nz,
                                                             int bx, int by, int bz, uint32_t* bricks,
                                                             unsigned long long* negs, int wx, int wy) {
  typedef typename Vox<S>::V V;
  typedef typename Vox<S>::Wt Wt;
  const V* f = reinterpret_cast<const V*>(vol);
  const Wt* wt = reinterpret_cast<const Wt*>(reinterpret_cast<const char*>(vol) + count * sizeof(V));
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t n = (uint32_t)bx * by * bz, base = blockIdx.x * 32u;
  const uint32_t word = base + lane < n ? bricks[base + lane] & (KF_BRICK_NEG | KF_BRICK_SET) : 0u;
  auto bits = [](const auto& v) {
    uint32_t b = 0;
    memcpy(&b, &v, sizeof(v));
    return b;
  };
  __syncthreads();  // every warp has read the words that the warps rewrite below
  int turn = 0;
  for (unsigned todo = __ballot_sync(0xffffffffu, word != 0); todo; todo &= todo - 1, ++turn) {
    if ((turn & 7) != warp) continue;
    const int k = __ffs(todo) - 1;
    const uint32_t had = __shfl_sync(0xffffffffu, word, k), b = base + k;
    const int cx = (int)(b % bx), cy = (int)(b / bx % by), cz = (int)(b / ((uint32_t)bx * by));
    // the lane's columns of a plane: two of the brick's own 64, one of the +1 layer's 17
    const int x = 8 * cx + (lane & 7), y = 8 * cy + (lane >> 3);
    const int ex = lane < 9 ? 8 * cx + 8 : 8 * cx + lane - 9, ey = lane < 9 ? 8 * cy + lane : 8 * cy + 8;
    const bool in0 = x < nx && y < ny, in1 = x < nx && y + 4 < ny, in2 = lane < 17 && ex < nx && ey < ny;
    const V zero = Vox<S>::encode_value(0.0f);
    uint32_t found = 0;
    for (int d0 = 0; d0 <= 8 && (had & ~found); d0 += 3) {
      V v[3][3];
      uint32_t i0[3];
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const bool in = 8 * cz + d0 + j < nz;
        const uint32_t row = (uint32_t)nx * (uint32_t)ny * (uint32_t)(8 * cz + d0 + j);
        i0[j] = row + (uint32_t)nx * (uint32_t)y + (uint32_t)x;
        v[j][0] = in && in0 ? f[i0[j]] : zero;
        v[j][1] = in && in1 ? f[i0[j] + 4u * (uint32_t)nx] : zero;
        v[j][2] = in && in2 ? f[row + (uint32_t)nx * (uint32_t)ey + (uint32_t)ex] : zero;
      }
      bool neg = false, set = false;
#pragma unroll
      for (int j = 0; j < 3; ++j) {
#pragma unroll
        for (int c = 0; c < 3; ++c) neg |= Vox<S>::raw_nc(&v[j][c], 0) < 0.0f;
        set |= d0 + j < 8 && (bits(v[j][0]) | bits(v[j][1])) != 0;
      }
      if ((had & ~found & KF_BRICK_SET) && !__any_sync(0xffffffffu, set)) {
#pragma unroll
        for (int j = 0; j < 3; ++j)
          if (d0 + j < 8 && 8 * cz + d0 + j < nz)
            set |= (in0 && bits(wt[i0[j]]) != 0) || (in1 && bits(wt[i0[j] + 4u * (uint32_t)nx]) != 0);
      }
      if (__any_sync(0xffffffffu, neg)) found |= KF_BRICK_NEG;
      if (__any_sync(0xffffffffu, set)) found |= KF_BRICK_SET;
    }
    found &= had;
    if (lane == 0) {
      bricks[b] = found;
      if (found & KF_BRICK_NEG) atomicOr(negs + kf_neg_word(cx, cy, cz, wx, wy), kf_neg_bit(cx, cy, cz));
    }
  }
}

}  // namespace

int kf_refresh_bricks(kf_session* s, cudaStream_t stream) {
  KF_CUDA_TRY(s, cudaMemsetAsync(s->d_neg, 0, (size_t)s->wx * s->wy * s->wz * 8, stream));
  const uint32_t nb = (uint32_t)s->bx * s->by * s->bz;
  const int grid = (int)((nb + 31) / 32);
#define KF_REFRESH(S)                                                                                               \
  refresh_bricks_kernel<S><<<grid, 256, 0, stream>>>(s->d_vol, s->vol_count, s->cfg.nx, s->cfg.ny, s->cfg.nz, s->bx, \
                                                     s->by, s->bz, s->d_bricks, s->d_neg, s->wx, s->wy)
  switch (s->cfg.storage) {
    case KF_STORAGE_F32F32: KF_REFRESH(KF_STORAGE_F32F32); break;
    case KF_STORAGE_F16U16: KF_REFRESH(KF_STORAGE_F16U16); break;
    default: KF_REFRESH(KF_STORAGE_RG16I); break;
  }
#undef KF_REFRESH
  KF_CUDA_TRY(s, cudaGetLastError());
  kf_note_launch(s, 1);
  s->frames_since_rebuild = 0;
  return KF_OK;
}

int kf_rebuild_bricks(kf_session* s, cudaStream_t stream) {
  // a volume from elsewhere: every flag is set, then checked
  const size_t nb = (size_t)s->bx * s->by * s->bz;
  KF_CUDA_TRY(s, cudaMemsetAsync(s->d_bricks, KF_BRICK_NEG | KF_BRICK_SET, nb * 4, stream));
  return kf_refresh_bricks(s, stream);
}

int kf_note_integrate(kf_session* s, cudaStream_t stream) {
  if (++s->frames_since_rebuild < KF_BRICK_REBUILD_EVERY) return KF_OK;
  return kf_refresh_bricks(s, stream);
}

int kf_reset_bricks(kf_session* s) {
  // an all-zero volume has no negative value
  const size_t words = kf_flag_words(s->bx, s->by, s->bz);
  KF_CUDA_TRY(s, cudaMemsetAsync(s->d_bricks, 0, words * 4, s->stream));
  s->frames_since_rebuild = 0;
  return KF_OK;
}

namespace {

RayArgs make_ray_args(kf_session* s) {
  RayArgs a;
  a.vol = s->d_vol;
  a.nx = s->cfg.nx; a.ny = s->cfg.ny; a.nz = s->cfg.nz;
  a.dimx = s->cfg.dim_x; a.dimy = s->cfg.dim_y; a.dimz = s->cfg.dim_z;
  a.sx = (float)a.nx / a.dimx; a.sy = (float)a.ny / a.dimy; a.sz = (float)a.nz / a.dimz;
  a.gx = a.dimx / (float)a.nx * 0.5f; a.gy = a.dimy / (float)a.ny * 0.5f; a.gz = a.dimz / (float)a.nz * 0.5f;
  // stepSize() (gFusion.h:72-81) and largeStep = 0.75 mu (gFusion.cpp:1302)
  const float mind = fminf(fminf(a.dimx, a.dimy), a.dimz);
  const float maxn = (float)max(max(a.nx, a.ny), a.nz);
  a.step = mind / maxn;
  a.large_step = 0.75f * s->cfg.mu;
  a.nearp = s->cfg.near_plane;
  a.farp = s->cfg.far_plane;
  {
    const float smin = fminf(a.step, a.large_step > 0.0f ? a.large_step : a.step);
    const double n = (double)(a.farp - a.nearp) / (double)smin + 16.0;
    a.max_steps = (int)fmin(n, 1.0e8);
  }
  a.W = s->W[0]; a.H = s->H[0];
  a.ikx = 1.0f / s->intr.fx;
  a.iky = 1.0f / s->intr.fy;
  a.ikcx = -s->intr.cx / s->intr.fx;
  a.ikcy = -s->intr.cy / s->intr.fy;
  a.out_v = s->d_ref_vertex;
  a.out_n = s->d_ref_normal;
  a.st = s->d_state;
  a.st_out = s->d_state;
  a.inv_step = 1.0f / a.step;
  a.neg = s->d_neg;
  a.wx = s->wx; a.wy = s->wy;
  return a;
}

template <bool BATCH, int ROWS>
void launch_ray_rows(int storage, dim3 grid, cudaStream_t st, const RayArgs& a, const RayArgs* many) {
  dim3 block(32, ROWS);
  switch (storage) {
    case KF_STORAGE_F32F32: raycast_kernel<KF_STORAGE_F32F32, BATCH, ROWS><<<grid, block, 0, st>>>(a, many); break;
    case KF_STORAGE_F16U16: raycast_kernel<KF_STORAGE_F16U16, BATCH, ROWS><<<grid, block, 0, st>>>(a, many); break;
    default: raycast_kernel<KF_STORAGE_RG16I, BATCH, ROWS><<<grid, block, 0, st>>>(a, many); break;
  }
}

template <bool BATCH>
void launch_ray(int storage, int rows, dim3 grid, cudaStream_t st, const RayArgs& a, const RayArgs* many) {
  if (rows == 2) launch_ray_rows<BATCH, 2>(storage, grid, st, a, many);
  else if (rows == 8) launch_ray_rows<BATCH, 8>(storage, grid, st, a, many);
  else launch_ray_rows<BATCH, 4>(storage, grid, st, a, many);
}

RayArgs retarget(RayArgs a, const kf_scratch_target* t) {
  if (t) {
    a.out_v = t->out_v;
    a.out_n = t->out_n;
    a.st_out = t->st_out;
  }
  return a;
}

}  // namespace

int kf_launch_raycast_shape(kf_session* s, int rows, const kf_scratch_target* t) {
  const RayArgs a = retarget(make_ray_args(s), t);
  if (rows == 1) {
    // persistent sweep: every resident slot of 256 threads, the queue in the session state
    const void* fn = s->cfg.storage == KF_STORAGE_F32F32   ? (const void*)raycast_sweep_kernel<KF_STORAGE_F32F32>
                     : s->cfg.storage == KF_STORAGE_F16U16 ? (const void*)raycast_sweep_kernel<KF_STORAGE_F16U16>
                                                           : (const void*)raycast_sweep_kernel<KF_STORAGE_RG16I>;
    const int blocks = kf_occupancy_blocks(s, fn, 256, 0, 64);
    if (blocks <= 0) return KF_ERR_CUDA;
    unsigned* q = s->d_state->ray_queue;
    switch (s->cfg.storage) {
      case KF_STORAGE_F32F32: raycast_sweep_kernel<KF_STORAGE_F32F32><<<blocks, 256, 0, s->stream>>>(a, q); break;
      case KF_STORAGE_F16U16: raycast_sweep_kernel<KF_STORAGE_F16U16><<<blocks, 256, 0, s->stream>>>(a, q); break;
      default: raycast_sweep_kernel<KF_STORAGE_RG16I><<<blocks, 256, 0, s->stream>>>(a, q); break;
    }
    KF_CUDA_TRY(s, cudaGetLastError());
    kf_note_launch(s);
    return KF_OK;
  }
  dim3 grid((a.W + 31) / 32, (a.H + rows - 1) / rows);
  launch_ray<false>(s->cfg.storage, rows, grid, s->stream, a, nullptr);
  KF_CUDA_TRY(s, cudaGetLastError());
  kf_note_launch(s);
  return KF_OK;
}

int kf_launch_raycast(kf_session* s) { return kf_launch_raycast_shape(s, s->ray_rows, nullptr); }

int kf_launch_intensity_projection(kf_session* s, float4* out) {
  const RayArgs a = make_ray_args(s);
  dim3 grid((a.W + 31) / 32, (a.H + 3) / 4);
  dim3 block(32, 4);
  switch (s->cfg.storage) {
    case KF_STORAGE_F32F32: mip_kernel<KF_STORAGE_F32F32><<<grid, block, 0, s->stream>>>(a, out); break;
    case KF_STORAGE_F16U16: mip_kernel<KF_STORAGE_F16U16><<<grid, block, 0, s->stream>>>(a, out); break;
    default: mip_kernel<KF_STORAGE_RG16I><<<grid, block, 0, s->stream>>>(a, out); break;
  }
  KF_CUDA_TRY(s, cudaGetLastError());
  kf_note_launch(s);
  return KF_OK;
}

// ---- batched: every member's raycast in one launch (blockIdx.z = member) ----
int kf_batch_prepare_raycast(kf_batch* b, const kf_scratch_target* over) {
  const int n = (int)b->members.size();
  RayArgs* h = nullptr;
  b->ray_args = kf_batch_table(b, sizeof(RayArgs) * n, reinterpret_cast<void**>(&h));
  if (!b->ray_args) return KF_ERR_CAPACITY;
  for (int e = 0; e < n; ++e) h[e] = retarget(make_ray_args(b->members[e]), over ? over + e : nullptr);
  return KF_OK;
}

int kf_batch_launch_raycast(kf_batch* b, int n) {
  kf_session* s0 = b->members[0];
  const int rows = b->ray_rows;
  dim3 grid((s0->W[0] + 31) / 32, (s0->H[0] + rows - 1) / rows, n);
  launch_ray<true>(s0->cfg.storage, rows, grid, b->stream, RayArgs{}, static_cast<const RayArgs*>(b->ray_args));
  KF_CUDA_TRY(b, cudaGetLastError());
  b->launches += 1;
  return KF_OK;
}
