// kf_integrate.cu — TSDF fusion of one depth frame.
//
// Reference: gFusion::integrate (src/gFusion.cpp:1234-1287) and shaders/integrate.cs:52-169:
// one thread per (x, y) voxel column marching z; voxel centre ((i + 0.5) * volDim /
// volSize) to camera by inverse(m_pose); skip z < 1e-4, pixels outside the 512x424
// image (:54, Q11) and zero depth; eta = (d - z) * sqrt(1 + (x/z)^2 + (y/z)^2); if
// eta > -mu the running average (w*F + min(1, eta/mu)) / (w + 1) is kept only when it is
// below 0.2, clamped to [-0.1, 0.2] with w = min(w + 1, maxWeight); otherwise (and for
// eta <= -mu) value and weight are zeroed (Q8).
//
// B200 design: two launches.  The plan kernel tests every 8^3 brick, one thread each, and
// lists the bricks the frame can change; the integrate kernel runs the reference's tests on
// the voxels of the listed bricks only.  Of the voxels that project into the image about six
// in ten lie more than mu behind the surface (rewritten with zero, which changes nothing in
// a brick that holds only zeros) and three in ten see a zero depth pixel (skipped), so most
// bricks drop out on the farthest depth of the tiles their projection covers.
// What bounds it: instruction issue and the L1 request rate, not DRAM (194 MB read and 64 MB
// written for 63 M listed voxels of a 768^3 room frame).  Integrate at 512^3 F16U16 (both
// launches): 181 -> 50 us, at 768^3 427 -> 206 us, 16 batched sessions 917 -> 412 us.
#include "kf_internal.cuh"

namespace {

struct IntArgs {
  void* vol;
  size_t count_voxels;
  int nx, ny, nz;
  float dimx, dimy, dimz;
  const float* depth;
  int W, H;
  float fx, fy, cx, cy;
  float mu, inv_mu, maxw;
  int band;  // Q8
  const int* gate;
  const KfDevState* st;
  uint32_t* bricks;
  int bx, by, bz;
  unsigned long long* neg;
  int wx, wy;
  // the farthest depths of 8x8 and 16x16 pixel tiles (kf_pyramid.cu)
  const float* tiles8;
  const float* tiles16;
  int tw8, tw16;
  uint32_t* list;   // planned bricks
  unsigned* count;  // their number (zero between launches)
};

template <class T>
__device__ __forceinline__ uint32_t bits_of(const T& v) {
  uint32_t b = 0;
  memcpy(&b, &v, sizeof(T));
  return b;
}

// True when the box of voxel centres [b0, b1] (index space, inclusive) lies entirely on the
// outside of one of the five half-spaces whose intersection is the set of voxels
// integrate.cs can touch: z >= 1e-4, 0 <= u <= W-1, 0 <= v <= H-1 (u, v the +0.5-rounded
// projection).  Conservative: a box that is not culled is tested voxel by voxel.  Called by
// a whole warp: lane & 7 evaluates one corner, the ballots combine them.
__device__ __forceinline__ bool box_outside_frustum(const IntArgs& a, const float* inv, const int* b0, const int* b1) {
  const float vx = a.dimx / a.nx, vy = a.dimy / a.ny, vz = a.dimz / a.nz;
  const float kx0 = a.cx + 0.5f, kx1 = a.cx + 0.5f - (float)(a.W - 1);
  const float ky0 = a.cy + 0.5f, ky1 = a.cy + 0.5f - (float)(a.H - 1);
  const int c = threadIdx.x & 7;
  const float wx = ((c & 1 ? b1[0] : b0[0]) + 0.5f) * vx;
  const float wy = ((c & 2 ? b1[1] : b0[1]) + 0.5f) * vy;
  const float wz = ((c & 4 ? b1[2] : b0[2]) + 0.5f) * vz;
  const float X = inv[0] * wx + inv[1] * wy + inv[2] * wz + inv[3];
  const float Y = inv[4] * wx + inv[5] * wy + inv[6] * wz + inv[7];
  const float Z = inv[8] * wx + inv[9] * wy + inv[10] * wz + inv[11];
  const unsigned o0 = __ballot_sync(0xffffffffu, Z - 1e-4f < 0.0f);
  const unsigned o1 = __ballot_sync(0xffffffffu, a.fx * X + kx0 * Z < 0.0f);
  const unsigned o2 = __ballot_sync(0xffffffffu, -(a.fx * X + kx1 * Z) < 0.0f);
  const unsigned o3 = __ballot_sync(0xffffffffu, a.fy * Y + ky0 * Z < 0.0f);
  const unsigned o4 = __ballot_sync(0xffffffffu, -(a.fy * Y + ky1 * Z) < 0.0f);
  return (o0 & 0xffu) == 0xffu || (o1 & 0xffu) == 0xffu || (o2 & 0xffu) == 0xffu ||
         (o3 & 0xffu) == 0xffu || (o4 & 0xffu) == 0xffu;
}

// A batched launch: plan block b belongs to the entry e with prefix[e] <= b < prefix[e + 1];
// the integrate kernel walks all entries' lists (counts[e] bricks each) as one.
struct IntBatch {
  const IntArgs* args;
  const uint32_t* prefix;  // n + 1 entries
  unsigned* counts;        // n counts
  unsigned* done;          // blocks of the integrate launch that are through (zero between launches)
  int n;
};

// A plan block covers 8 x 8 x 4 bricks; list entries hold the brick's coordinates (at most
// 512 per axis) and whether it held anything but zeros.
constexpr int kPlanX = 8, kPlanY = 8, kPlanZ = 4;
constexpr uint32_t kEntrySet = 1u << 27;
__device__ __forceinline__ uint32_t entry_of(int bx, int by, int bz) {
  return (uint32_t)bx | (uint32_t)by << 9 | (uint32_t)bz << 18;
}

// Whether integrate.cs may change a voxel of brick (bx, by, bz), whose flag word is `word`.
// False only when no voxel of it can: the brick (grown by half a voxel on every side, which
// also covers the rounding of the per-voxel positions) lies outside the view frustum, or on
// every depth pixel that its projection may touch the voxels are skipped (depth 0) or, in a
// brick that holds only zeros, zeroed (d - z <= -mu).  The ray-length factor is >= 1, so
// d - z <= -mu, with a margin for rounding, implies eta <= -mu.
__device__ __forceinline__ bool brick_changes(const IntArgs& a, const float* inv, int bx, int by, int bz,
                                              uint32_t word) {
  const float vx = a.dimx / a.nx, vy = a.dimy / a.ny, vz = a.dimz / a.nz;
  const float wx = (float)(bx * KF_BRICK) * vx, wy = (float)(by * KF_BRICK) * vy, wz = (float)(bz * KF_BRICK) * vz;
  const float ex = (float)min(KF_BRICK, a.nx - bx * KF_BRICK) * vx, ey = (float)min(KF_BRICK, a.ny - by * KF_BRICK) * vy,
              ez = (float)min(KF_BRICK, a.nz - bz * KF_BRICK) * vz;
  float o[3], ax[3], ay[3], az[3], mag = 0.0f;  // the low corner and the three edges in camera space
  bool bounded = true;
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    o[r] = inv[r * 4] * wx + inv[r * 4 + 1] * wy + inv[r * 4 + 2] * wz + inv[r * 4 + 3];
    ax[r] = inv[r * 4] * ex;
    ay[r] = inv[r * 4 + 1] * ey;
    az[r] = inv[r * 4 + 2] * ez;
    const float m = fabsf(inv[r * 4]) * a.dimx + fabsf(inv[r * 4 + 1]) * a.dimy + fabsf(inv[r * 4 + 2]) * a.dimz +
                    fabsf(inv[r * 4 + 3]);
    bounded = bounded && m < 1e30f;  // row by row: a maximum would drop a NaN
    mag = fmaxf(mag, m);
  }
  if (!bounded) return true;
  // outside one of the five half-spaces: the largest value over the corners is negative
  auto top = [&](float kx, float ky, float kz) {
    return kx * o[0] + ky * o[1] + kz * o[2] + fmaxf(0.0f, kx * ax[0] + ky * ax[1] + kz * ax[2]) +
           fmaxf(0.0f, kx * ay[0] + ky * ay[1] + kz * ay[2]) + fmaxf(0.0f, kx * az[0] + ky * az[1] + kz * az[2]);
  };
  const float ku = a.cx + 0.5f, kv = a.cy + 0.5f;
  const float W1 = (float)(a.W - 1), H1 = (float)(a.H - 1);
  if (top(0.0f, 0.0f, 1.0f) < 1e-4f || top(a.fx, 0.0f, ku) < 0.0f || top(-a.fx, 0.0f, W1 - ku) < 0.0f ||
      top(0.0f, a.fy, kv) < 0.0f || top(0.0f, -a.fy, H1 - kv) < 0.0f)
    return false;
  const float zmin = o[2] + fminf(0.0f, ax[2]) + fminf(0.0f, ay[2]) + fminf(0.0f, az[2]);
  if (!(zmin > 0.01f)) return true;  // reaches the camera plane: no bounded projection
  // the pixels it may touch: the bounding box of the corners' projections (every corner is in
  // front of the camera), a pixel and the positions' rounding wider
  float u0 = 1e30f, u1 = -1e30f, v0 = 1e30f, v1 = -1e30f;
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const float X = o[0] + (c & 1 ? ax[0] : 0.0f) + (c & 2 ? ay[0] : 0.0f) + (c & 4 ? az[0] : 0.0f);
    const float Y = o[1] + (c & 1 ? ax[1] : 0.0f) + (c & 2 ? ay[1] : 0.0f) + (c & 4 ? az[1] : 0.0f);
    const float Z = o[2] + (c & 1 ? ax[2] : 0.0f) + (c & 2 ? ay[2] : 0.0f) + (c & 4 ? az[2] : 0.0f);
    const float iz = __fdividef(1.0f, Z);
    const float u = fmaf(a.fx, X * iz, ku), v = fmaf(a.fy, Y * iz, kv);
    u0 = fminf(u0, u);
    u1 = fmaxf(u1, u);
    v0 = fminf(v0, v);
    v1 = fmaxf(v1, v);
  }
  const float slack = 4e-6f * mag;
  const float m = 1.0f + slack * fmaxf(a.fx, a.fy) * __fdividef(1.0f, zmin);
  u0 = fmaxf(u0 - m, 0.0f);
  v0 = fmaxf(v0 - m, 0.0f);
  u1 = fminf(u1 + m, W1);
  v1 = fminf(v1 + m, H1);
  if (u0 > u1 || v0 > v1) return false;
  const float reach = word & KF_BRICK_SET ? -INFINITY : zmin - a.mu - 1e-4f * (zmin + a.mu) - slack;
  const int x0 = (int)u0, x1 = (int)u1, y0 = (int)v0, y1 = (int)v1;
  // tiles of the finest level that covers the box in few reads; a box too wide for that is
  // a brick close to the camera
  int sh = 3, tw = a.tw8;
  const float* t = a.tiles8;
  if (((x1 >> 3) - (x0 >> 3) + 1) * ((y1 >> 3) - (y0 >> 3) + 1) > 16) {
    sh = 4;
    tw = a.tw16;
    t = a.tiles16;
    if (((x1 >> 4) - (x0 >> 4) + 1) * ((y1 >> 4) - (y0 >> 4) + 1) > 100) return true;
  }
  // no early exit: the loads do not wait for one another
  float far = -INFINITY;
  for (int ty = y0 >> sh; ty <= y1 >> sh; ++ty)
#pragma unroll 4
    for (int tx = x0 >> sh; tx <= x1 >> sh; ++tx) far = fmaxf(far, __ldg(t + ty * tw + tx));
  return far * 0.001f > reach;
}

template <bool BATCH>
__global__ void __launch_bounds__(256) plan_kernel(IntArgs one, IntBatch batch) {
  __shared__ unsigned s_n[9];
  int local = blockIdx.x, e = 0;
  if constexpr (BATCH) {
    // binary search of the entry (uniform over the block)
    int lo = 0, hi = batch.n - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (__ldg(batch.prefix + mid) <= blockIdx.x) lo = mid; else hi = mid - 1;
    }
    e = lo;
    local = (int)(blockIdx.x - __ldg(batch.prefix + e));
  }
  const IntArgs& a = BATCH ? batch.args[e] : one;
  if (a.gate && *(volatile const int*)a.gate == 0) return;
  float inv[12];  // inverse(m_pose), rows of [R^T | -R^T t] (integrate uses glm::inverse, :1242)
#pragma unroll
  for (int k = 0; k < 12; ++k) inv[k] = a.st->inv_rows[k];
  const int gx = (a.bx + kPlanX - 1) / kPlanX, gy = (a.by + kPlanY - 1) / kPlanY;
  const int x0 = local % gx * kPlanX, y0 = local / gx % gy * kPlanY, z0 = local / (gx * gy) * kPlanZ;
  // the whole block's box first (every warp finds the same answer); one voxel of margin
  {
    const int b0[3] = {x0 * KF_BRICK - 1, y0 * KF_BRICK - 1, z0 * KF_BRICK - 1};
    const int b1[3] = {(x0 + kPlanX) * KF_BRICK, (y0 + kPlanY) * KF_BRICK, (z0 + kPlanZ) * KF_BRICK};
    if (box_outside_frustum(a, inv, b0, b1)) return;
  }
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int bx = x0 + (tid & 7), by = y0 + ((tid >> 3) & 7), bz = z0 + (tid >> 6);
  bool work = false;
  uint32_t word = 0;
  if (bx < a.bx && by < a.by && bz < a.bz) {
    word = a.bricks[(uint32_t)bx + (uint32_t)a.bx * ((uint32_t)by + (uint32_t)a.by * (uint32_t)bz)];
    work = brick_changes(a, inv, bx, by, bz, word);
  }
  const unsigned mine = __ballot_sync(0xffffffffu, work);
  if (lane == 0) s_n[warp] = __popc(mine);
  __syncthreads();
  if (tid == 0) {
    unsigned n = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      const unsigned c = s_n[w];
      s_n[w] = n;
      n += c;
    }
    s_n[8] = n ? atomicAdd(a.count, n) : 0u;
  }
  __syncthreads();
  if (work)
    a.list[s_n[8] + s_n[warp] + __popc(mine & ((1u << lane) - 1u))] =
        entry_of(bx, by, bz) | (word & KF_BRICK_SET ? kEntrySet : 0u);
}

// Hardware reciprocal and reciprocal square root of normal numbers: the values of __fdividef
// and rsqrtf without their scaling of denormals, which no operand here is.
__device__ __forceinline__ float mufu_rcp(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float mufu_rsqrt(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Half of a listed brick by one warp: lane = (x, y) column (8 x 4 of them), its 8 voxels
// along z in registers.  The loads of a step (depth pixels, then values and weights) are
// issued for all 8 voxels together: a column waits for two memory latencies, not sixteen.
// 64 registers, no spills: a variant with fewer instructions (border tests left out for inner
// bricks, the ray length only near the surface) spilled and was slower.
template <int S>
__device__ __forceinline__ void integrate_half_brick(const IntArgs& a, uint32_t entry, int half, int lane) {
  typedef typename Vox<S>::V V;
  typedef typename Vox<S>::Wt Wt;
  const int bx = entry & 511, by = (entry >> 9) & 511, bz = (entry >> 18) & 511;
  const int x = bx * KF_BRICK + (lane & 7), y = by * KF_BRICK + 4 * half + (lane >> 3), z0 = bz * KF_BRICK;
  const bool was_set = (entry & kEntrySet) != 0;
  const int zend = (x < a.nx && y < a.ny) ? min(KF_BRICK, a.nz - z0) : 0;

  // getVolumePosition (integrate.cs:16-19; along z as (i + 0.5) * voxel size) and
  // delta = rotate(invTrack, (0,0,vz)): the camera-space position is computed directly at
  // the brick's first voxel and steps by delta inside it (:57-62)
  const float cxw = (x + 0.5f) * a.dimx / a.nx;
  const float cyw = (y + 0.5f) * a.dimy / a.ny;
  const float vz = a.dimz / a.nz;
  const float czw = (z0 + 0.5f) * vz;
  const float* inv = a.st->inv_rows;  // inverse(m_pose), rows of [R^T | -R^T t] (glm::inverse, :1242)
  float pos[3], dz[3];
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    pos[r] = fmaf(inv[r * 4 + 2], czw, fmaf(inv[r * 4 + 0], cxw, fmaf(inv[r * 4 + 1], cyw, inv[r * 4 + 3])));
    dz[r] = __fmul_rn(inv[r * 4 + 2], vz);  // kept rounded: the steps below are plain adds
  }
  const float fW1 = (float)(a.W - 1), fH1 = (float)(a.H - 1);
  const float ku = a.cx + 0.5f, kv = a.cy + 0.5f;
  float pz[8], len[8], d[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    d[j] = 0.0f;
    const float px = pos[0], py = pos[1];
    pz[j] = pos[2];
    const float iz = mufu_rcp(pz[j]);  // 2 ulp
    const float rx = px * iz;  // pos.x / pos.z
    const float ry = py * iz;
    // cameraX.x / cameraX.z + 0.5 = fx * x/z + cx + 0.5 (K has no skew, :67)
    const float u = fmaf(a.fx, rx, ku);
    const float v = fmaf(a.fy, ry, kv);
    const float r2 = fmaf(rx, rx, fmaf(ry, ry, 1.0f));
    len[j] = __fmul_rn(r2, mufu_rsqrt(r2));  // sqrt(r2), r2 >= 1
    const bool out = pz[j] < 0.0001f || u < 0.0f || u > fW1 || v < 0.0f || v > fH1;
    // a position beyond FP32 makes u or v a NaN, which passes the border test: column or row 0,
    // as a NaN converts to (fmaxf returns its other operand)
    if (j < zend && !out) d[j] = __ldg(a.depth + kf_trunc_index(fmaxf(v, 0.0f), fmaxf(u, 0.0f), (uint32_t)a.W));
#pragma unroll
    for (int r = 0; r < 3; ++r) pos[r] += dz[r];
  }
  V* vf = reinterpret_cast<V*>(a.vol);
  Wt* vw = reinterpret_cast<Wt*>(reinterpret_cast<char*>(a.vol) + a.count_voxels * sizeof(V));
  const uint32_t slice = (uint32_t)a.nx * (uint32_t)a.ny;
  const uint32_t idx0 = (uint32_t)x + (uint32_t)a.nx * (uint32_t)y + (uint32_t)z0 * slice;
  V oldv[8];
  Wt oldw[8];
  uint32_t fuse = 0, hit = 0;  // bit j: voxel j is averaged; sees a depth
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float dm = __fmul_rn(d[j], 0.001f);
    if (dm != 0.0f) hit |= 1u << j;
    // explicitly rounded: no launch fuses the scaling into the subtraction
    d[j] = __fmul_rn(__fsub_rn(dm, pz[j]), len[j]);
    if (dm != 0.0f && d[j] > -a.mu) {
      fuse |= 1u << j;
      oldv[j] = vf[idx0 + j * slice];
      oldw[j] = vw[idx0 + j * slice];
    }
  }
  bool set = false, neg = false, neg0 = false;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    if (fuse >> j & 1u) {
      const float sdf = fminf(1.0f, __fmul_rn(d[j], a.inv_mu));
      const float F = __fmul_rn(Vox<S>::raw_nc(&oldv[j], 0), Vox<S>::kRawToF);
      const float w = Vox<S>::weight(&oldw[j], 0);
      const float wd = fmaf(w, F, sdf) * mufu_rcp(w + 1.0f);
      float nF, nw;
      if (!a.band) {
        // the reference's earlier update (integrate.cs:115-150)
        nF = fminf(fmaxf(wd, -1.0f), 1.0f);
        nw = fminf(w + 1.0f, a.maxw);
      } else if (wd < 0.2f) {
        nF = fminf(fmaxf(wd, -0.1f), 0.2f);
        nw = fminf(w + 1.0f, a.maxw);
      } else {
        nF = 0.0f;
        nw = 0.0f;
      }
      const V ev = Vox<S>::encode_value(nF);
      const Wt ew = Vox<S>::encode_weight(nw);
      if (bits_of(ev) != bits_of(oldv[j])) vf[idx0 + j * slice] = ev;
      if (bits_of(ew) != bits_of(oldw[j])) vw[idx0 + j * slice] = ew;
      set |= (bits_of(ev) | bits_of(ew)) != 0;
      // a non-negative nF never stores a negative value
      neg |= nF < 0.0f;
      if (j == 0) neg0 = nF < 0.0f;
    }
  }
  if (was_set && __any_sync(0xffffffffu, (hit & ~fuse) != 0)) {
    // eta <= -mu: zeroed (already zero in a brick that held only zeros)
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if ((hit & ~fuse) >> j & 1u) {
        vf[idx0 + j * slice] = Vox<S>::encode_value(0.0f);
        vw[idx0 + j * slice] = Vox<S>::encode_weight(0.0f);
      }
  }
  // Brick flags: lane c merges corner c of the dilation (a brick's low x, y or z layer is
  // also the +1 layer of the brick below it) and sets the brick's flags where they are still
  // clear (and with a new NEG its bit).
  const unsigned b_set = __ballot_sync(0xffffffffu, set), b_neg = __ballot_sync(0xffffffffu, neg),
                 b_neg0 = __ballot_sync(0xffffffffu, neg0);
  if (lane < 8 && (b_set | b_neg)) {
    const int gx = bx - (lane & 1), gy = by - ((lane >> 1) & 1), gz = bz - (lane >> 2);
    unsigned m = lane & 4 ? b_neg0 : b_neg;
    if (lane & 1) m &= 0x01010101u;
    if (lane & 2) m &= half ? 0u : 0xffu;
    uint32_t want = m ? KF_BRICK_NEG : 0u;
    if (lane == 0 && b_set) want |= KF_BRICK_SET;
    if (want && gx >= 0 && gy >= 0 && gz >= 0) {
      uint32_t* w = &a.bricks[(uint32_t)gx + (uint32_t)a.bx * ((uint32_t)gy + (uint32_t)a.by * (uint32_t)gz)];
      const uint32_t had = *(volatile uint32_t*)w;
      if (want & ~had) atomicOr(w, want);
      if (want & ~had & KF_BRICK_NEG) atomicOr(a.neg + kf_neg_word(gx, gy, gz, a.wx, a.wy), kf_neg_bit(gx, gy, gz));
    }
  }
}

// Small volumes: every warp tests one brick and runs it, or (split 1) half of it, at once, which saves the list and a
// launch.  A warp's test costs about as many instructions as half a brick's voxels, all lanes
// doing the same, so it pays only while the launches' latency dominates (see kSmallBricks).
template <int S>
__global__ void __launch_bounds__(256, 4) integrate_small_kernel(IntArgs a, int split) {
  if (a.gate && *(volatile const int*)a.gate == 0) return;
  const int lane = threadIdx.x & 31, w = blockIdx.x * 8 + (threadIdx.x >> 5), b = w >> split;
  if (b >= a.bx * a.by * a.bz) return;
  const int bx = b % a.bx, by = b / a.bx % a.by, bz = b / (a.bx * a.by);
  const uint32_t word = a.bricks[b];
  if (!brick_changes(a, a.st->inv_rows, bx, by, bz, word)) return;
  const uint32_t entry = entry_of(bx, by, bz) | (word & KF_BRICK_SET ? kEntrySet : 0u);
#pragma unroll 1
  for (int half = w & split; half < 2; half += 1 + split) integrate_half_brick<S>(a, entry, half, lane);
}

// Persistent: every warp takes `chunk` half-bricks of the list(s) per step until they are
// through; the last block zeroes the counts for the next plan.
template <int S, bool BATCH>
__global__ void __launch_bounds__(256, 4) integrate_kernel(IntArgs one, IntBatch batch, int chunk) {
  __shared__ uint32_t s_first[BATCH ? 257 : 1];  // first half-brick of each entry
  __shared__ uint32_t s_warp[BATCH ? 8 : 1];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t total;
  if constexpr (BATCH) {
    const uint32_t c = tid < batch.n ? 2u * *(volatile const unsigned*)(batch.counts + tid) : 0u;
    uint32_t inc = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += u;
    }
    if (lane == 31) s_warp[warp] = inc;
    __syncthreads();
    for (int w = 0; w < warp; ++w) inc += s_warp[w];
    s_first[tid] = inc - c;
    if (tid == 255) s_first[256] = inc;
    __syncthreads();
    total = s_first[256];
  } else {
    total = 2u * *(volatile const unsigned*)one.count;
  }
  const uint32_t step = gridDim.x * 8u * (uint32_t)chunk;
  for (uint32_t t0 = (blockIdx.x * 8u + warp) * (uint32_t)chunk; t0 < total; t0 += step)
    for (uint32_t t = t0; t < min(t0 + (uint32_t)chunk, total); ++t) {
      if constexpr (BATCH) {
        int lo = 0, hi = batch.n - 1;
        while (lo < hi) {
          const int mid = (lo + hi + 1) >> 1;
          if (s_first[mid] <= t) lo = mid; else hi = mid - 1;
        }
        const uint32_t k = t - s_first[lo];
        integrate_half_brick<S>(batch.args[lo], batch.args[lo].list[k >> 1], (int)(k & 1u), lane);
      } else {
        integrate_half_brick<S>(one, one.list[t >> 1], (int)(t & 1u), lane);
      }
    }
  __syncthreads();  // every warp of the block has read the counts
  if (tid == 0) {
    unsigned* done = BATCH ? batch.done : one.count + 1;
    if (atomicAdd(done, 1u) == gridDim.x - 1) {
      if constexpr (BATCH) {
        for (int e = 0; e < batch.n; ++e) batch.counts[e] = 0u;
      } else {
        *one.count = 0u;
      }
      *done = 0u;
    }
  }
}

}  // namespace

namespace {

IntArgs make_int_args(kf_session* s, int gated) {
  IntArgs a;
  a.vol = s->d_vol;
  a.count_voxels = s->vol_count;
  a.nx = s->cfg.nx; a.ny = s->cfg.ny; a.nz = s->cfg.nz;
  a.dimx = s->cfg.dim_x; a.dimy = s->cfg.dim_y; a.dimz = s->cfg.dim_z;
  a.depth = s->d_depth[0];
  a.W = s->W[0]; a.H = s->H[0];
  a.fx = s->intr.fx; a.fy = s->intr.fy; a.cx = s->intr.cx; a.cy = s->intr.cy;
  a.mu = s->cfg.mu;
  a.inv_mu = 1.0f / s->cfg.mu;
  a.maxw = s->cfg.max_weight;
  a.band = (s->cfg.quirks & KF_Q8_NARROW_BAND) ? 1 : 0;
  a.gate = gated ? &s->d_state->do_integrate : nullptr;
  a.st = s->d_state;
  a.bricks = s->d_bricks;
  a.bx = s->bx; a.by = s->by; a.bz = s->bz;
  a.neg = s->d_neg;
  a.wx = s->wx; a.wy = s->wy;
  a.tiles8 = s->d_tiles;
  a.tw8 = (a.W + 7) / 8;
  a.tiles16 = s->d_tiles + (size_t)a.tw8 * ((a.H + 7) / 8);
  a.tw16 = (a.W + 15) / 16;
  a.count = s->d_plan;
  a.list = s->d_plan + KF_PLAN_HEAD;
  return a;
}

uint32_t plan_blocks(const IntArgs& a) {
  return (uint32_t)((a.bx + kPlanX - 1) / kPlanX) * ((a.by + kPlanY - 1) / kPlanY) * ((a.bz + kPlanZ - 1) / kPlanZ);
}

// Volumes of at most this many bricks take the one-launch form.  Per call, one launch against
// two (B200, a warp per brick, back to back, events included): 64^3 18.5 / 27.2 us, 128^3 21.5 / 26.8, 160^3
// 26.4 / 29.4, 192^3 33.0 / 31.3, 256^3 53 / 41.  The line lies between 160^3 and 192^3.
constexpr int kSmallBricks = 8192;
// Up to this many bricks a warp takes half a brick: the launch is one wave either way and bound by
// a warp's chain, so testing every brick twice costs less than the second half.  Device us with
// a warp per brick / per half: 80 x 52 x 80 11.0 / 8.8, 81^3 11.2 / 9.7, 108^3 11.0 / 10.3, 91 x 124
// x 124 (3,072 bricks) 10.7 / 9.9, 129 x 132 x 205 (7,514) 15.7 / 18.7.
constexpr int kSplitBricks = 3072;

int brick_count(const IntArgs& a) { return a.bx * a.by * a.bz; }

cudaError_t launch_int_small(int storage, cudaStream_t st, const IntArgs& a) {
  const int split = brick_count(a) <= kSplitBricks ? 1 : 0;
  const int grid = ((brick_count(a) << split) + 7) / 8;
  switch (storage) {
    case KF_STORAGE_F32F32: integrate_small_kernel<KF_STORAGE_F32F32><<<grid, 256, 0, st>>>(a, split); break;
    case KF_STORAGE_F16U16: integrate_small_kernel<KF_STORAGE_F16U16><<<grid, 256, 0, st>>>(a, split); break;
    default: integrate_small_kernel<KF_STORAGE_RG16I><<<grid, 256, 0, st>>>(a, split); break;
  }
  return cudaGetLastError();
}

// Four blocks of 256 threads per SM (the register budget), one wave.
template <bool BATCH>
cudaError_t launch_int(int storage, int num_sms, uint32_t plan, int zc, cudaStream_t st, const IntArgs& a,
                       const IntBatch& b) {
  plan_kernel<BATCH><<<plan, 256, 0, st>>>(a, b);
  if (cudaError_t e = cudaGetLastError()) return e;
  const int grid = 4 * num_sms, chunk = zc / KF_BRICK;
  switch (storage) {
    case KF_STORAGE_F32F32: integrate_kernel<KF_STORAGE_F32F32, BATCH><<<grid, 256, 0, st>>>(a, b, chunk); break;
    case KF_STORAGE_F16U16: integrate_kernel<KF_STORAGE_F16U16, BATCH><<<grid, 256, 0, st>>>(a, b, chunk); break;
    default: integrate_kernel<KF_STORAGE_RG16I, BATCH><<<grid, 256, 0, st>>>(a, b, chunk); break;
  }
  return cudaGetLastError();
}

IntArgs retarget(IntArgs a, const kf_scratch_target* t) {
  if (t) {
    a.vol = t->vol;
    a.bricks = t->bricks;
    a.neg = t->neg;
  }
  return a;
}

}  // namespace

// Whether the session's integrate takes the listed form, the only one that has a chunk.
bool kf_integrate_has_chunk(const kf_session* s) { return s->bx * s->by * s->bz > kSmallBricks; }

int kf_launch_integrate_shape(kf_session* s, int gated, int zc, const kf_scratch_target* t) {
  const IntArgs a = retarget(make_int_args(s, gated), t);
  if (!kf_integrate_has_chunk(s)) {
    KF_CUDA_TRY(s, launch_int_small(s->cfg.storage, s->stream, a));
    kf_note_launch(s);
    return KF_OK;
  }
  KF_CUDA_TRY(s, launch_int<false>(s->cfg.storage, s->num_sms, plan_blocks(a), zc, s->stream, a, IntBatch{}));
  kf_note_launch(s, 2);
  return KF_OK;
}

int kf_launch_integrate(kf_session* s, int gated) { return kf_launch_integrate_shape(s, gated, s->int_zc, nullptr); }

// ---- batched: every member's gated frame-step integrate in one launch ----
int kf_batch_prepare_integrate(kf_batch* b, const kf_scratch_target* over) {
  const int n = (int)b->members.size();
  IntArgs* h = nullptr;
  uint32_t* hp = nullptr;
  b->int_args = kf_batch_table(b, sizeof(IntArgs) * n, reinterpret_cast<void**>(&h));
  b->int_prefix = static_cast<const uint32_t*>(kf_batch_table(b, 4 * (size_t)(n + 1), reinterpret_cast<void**>(&hp)));
  if (!b->int_args || !b->int_prefix) return KF_ERR_CAPACITY;
  uint64_t total = 0;
  for (int e = 0; e < n; ++e) {
    // the autotuner's timing runs ungated into scratch copies
    h[e] = over ? retarget(make_int_args(b->members[e], 0), over + e) : make_int_args(b->members[e], 1);
    h[e].count = b->d_plan + e;
    hp[e] = (uint32_t)total;
    total += plan_blocks(h[e]);
  }
  if (total >= (1ull << 31)) return KF_ERR_CAPACITY;
  hp[n] = (uint32_t)total;
  b->int_blocks = (uint32_t)total;
  return KF_OK;
}

int kf_batch_launch_integrate(kf_batch* b) {
  const IntBatch batch = {static_cast<const IntArgs*>(b->int_args), b->int_prefix, b->d_plan, b->d_plan + b->cap,
                          (int)b->members.size()};
  KF_CUDA_TRY(b, launch_int<true>(b->members[0]->cfg.storage, b->num_sms, b->int_blocks, b->int_zc, b->stream, IntArgs{},
                                  batch));
  b->launches += 2;
  return KF_OK;
}
