// kf_mcubes.cu — marching-cubes extraction: histoPyramid path and classic scan path.
//
// Reference: MCubes::histoPyramids (src/mcubes.cpp:206-389) with
// shaders/histoPyramids.cs:42-174 (classifyCubes, constructHPLevel) and
// shaders/traverseHistoPyramids.cs:54-260 (traverseHPLevel); the classic path of
// shaders/marchingCubes.cs:102-305 (classify / compact / generate, dead code in the
// reference) on top of the prefix sum (prefixSum.cs); export mcubes.cpp:391-509.
//
// histoPyramid semantics kept: cube corners in the reference's y/z-swapped order
// {000,100,001,101,010,110,011,111}; "positive found" over the first 7 corners (Q13);
// cubes within 10 voxels of the border left empty (Q15); cubeIndex bits f0,f1,f3,f2,
// f4,f5,f7,f6 -> 1..128; base texel = nrOfTriangles | cubeIndex << 16; level k+1 = 2x2x2
// sum; traversal descends the levels with the reference's running-sum comparison;
// vertices at mix(p0, p1, a) in voxel-index units with a = 0.5 outside [0, 1], w = 0.
// The pyramid is padded to a power of two P >= N with zero counts (the reference only
// supports power-of-two N, Q16).
//
// B200 design: a surface crosses few bricks, so the extraction works on tiles of 32 x 8 x 8
// cubes (a warp each) whose brick flags say that they may hold a negative value; with an iso
// level at or below zero no other cube can have a triangle (above zero every tile is looked
// at).  A tile's corner signs are loaded row by row, each value once per tile, and kept as
// bits; the case indices (a byte per cube) and the triangle counts come from the bits.
//  - histoPyramid order: the traversal numbers the triangles in the Morton order of their
//    cubes (children x fastest, then z, then y), so the pyramid's levels are not needed: the
//    counts per 8^3 brick in Morton order are prefix-summed, and a warp per brick lists its
//    triangles in shared memory in the same order and writes them.
//  - classic order and the welded mesh: voxel order, so counts per 32-voxel row segment are
//    prefix-summed.
// The vertex buffer holds more than the last extraction needed, so the generating kernel is
// launched without waiting for the count; without a buffer (the first extraction), or when it
// turns out too small, it is allocated for the count and the kernel launched (again).
// Device us per extraction at 512^3 F16U16, 1.28 M triangles: 925 -> 112 (123 MB of vertices
// and normals alone take 19); classic 205 x 160 x 131 F32, 158 k triangles: 90 -> 58; welded
// 384^3, 553 k triangles: 1,040 -> 150.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <new>
#include <vector>

#include "kf_internal.cuh"

#define KF_MC_TABLE_QUAL static __device__ const
#include "generated/kf_mc_tables.inc"

namespace kf_mc_host {
#undef KF_MC_TABLE_QUAL
#define KF_MC_TABLE_QUAL [[maybe_unused]] static const
#include "generated/kf_mc_tables.inc"
}  // namespace kf_mc_host

namespace {

__constant__ int c_bourke[8][3] = {{0, 0, 0}, {1, 0, 0}, {1, 1, 0}, {0, 1, 0},
                                   {0, 0, 1}, {1, 0, 1}, {1, 1, 1}, {0, 1, 1}};
__constant__ int c_bourke_edge[12][2] = {{0, 1}, {1, 2}, {2, 3}, {3, 0}, {4, 5}, {5, 6},
                                         {6, 7}, {7, 4}, {0, 4}, {1, 5}, {2, 6}, {3, 7}};

constexpr int kTileCubes = 32 * 8 * 8;

// The three extractions: histoPyramid (y/z-swapped corner order), classic, welded mesh.
constexpr int kHisto = 0, kClassic = 1, kMesh = 2;

struct McArgs {
  const void* vol;
  int nx, ny, nz;
  float iso;
  int q13, q15;
  const unsigned long long* neg;  // NEG bits; null: every tile is looked at
  int wx, wy;
  int tx, ty, tz;        // tiles of 32 x 8 x 8 cubes
  uint32_t* list;        // the listed tiles
  uint32_t* listed;      // their number
  uint8_t* cases;        // case index per cube, kTileCubes bytes per listed tile (z, y, x)
  uint32_t* counts;      // histoPyramid: triangles per brick in Morton order; else vertices
                         // (classic) or triangles (mesh) per row segment
  const uint32_t* offsets;  // their exclusive prefix sum
  uint32_t cap;          // triangles (classic: vertices) the output buffers hold
  float4* out;
  float4* nout;          // the triangle's face normal cross(v1 - v0, v2 - v0) per vertex, w = 0
  int shader_units;      // Q24: marchingCubes.cs's output convention (see classic_vertex)
  float vsx, vsy, vsz;   // its voxelSize (mCubeConfig, mcubes.h:30-39): 1000 * dim / size
  // welded mesh
  uint32_t* mask;        // edge bits: per row segment one word for each axis, bit = voxel
  uint32_t* vcounts;     // vertices per segment
  const uint32_t* voffsets;
  float* pos;
  float* nrm;
  uint32_t* idx;
  uint32_t vcap;
  float dimx, dimy, dimz;
};

// getVolumeData (histoPyramids.cs:95-107): the raw int16 for RG16I, the value otherwise
template <int S>
__device__ __forceinline__ float mc_raw(const void* vol, size_t i) {
  return Vox<S>::raw(reinterpret_cast<const typename Vox<S>::V*>(vol), i);
}

__device__ __forceinline__ size_t mc_index(const McArgs& a, int x, int y, int z) {
  return (size_t)x + (size_t)a.nx * ((size_t)y + (size_t)a.ny * z);
}
// Row segment of tile column tx in row (y, z): 32 voxels, in voxel order.
__device__ __forceinline__ uint32_t mc_segment(const McArgs& a, int tx, int y, int z) {
  return (uint32_t)tx + (uint32_t)a.tx * ((uint32_t)y + (uint32_t)a.ny * (uint32_t)z);
}

// Lists the tiles of which some cube may have a triangle (a tile is four bricks along x).
__global__ void __launch_bounds__(256) tile_list_kernel(McArgs a) {
  const uint32_t t = blockIdx.x * 256u + threadIdx.x, n = (uint32_t)a.tx * a.ty * a.tz;
  const int lane = threadIdx.x & 31;
  bool on = t < n;
  if (on && a.neg) {
    const int x = (int)(t % a.tx), y = (int)(t / a.tx % a.ty), z = (int)(t / ((uint32_t)a.tx * a.ty));
    const unsigned long long w = __ldg(a.neg + kf_neg_word(4 * x, y, z, a.wx, a.wy));
    on = (w >> ((y & 3) << 2 | (z & 3) << 4) & 15ull) != 0;
  }
  const unsigned m = __ballot_sync(0xffffffffu, on);
  uint32_t at = 0;
  if (lane == 0 && m) at = atomicAdd(a.listed, (uint32_t)__popc(m));
  at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << lane) - 1u));
  if (on) a.list[at] = t;
}

// A warp's share of the listed tiles' work, `parts` parts each, in turn over the grid.
template <class F>
__device__ __forceinline__ void for_each_part(const McArgs& a, uint32_t parts, F&& f) {
  const uint32_t total = __ldg(a.listed) * parts;
  for (uint32_t k = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); k < total; k += gridDim.x * (blockDim.x >> 5)) {
    const uint32_t slot = k / parts, t = __ldg(a.list + slot);
    f((int)(t % a.tx), (int)(t / a.tx % a.ty), (int)(t / ((uint32_t)a.tx * a.ty)), a.cases + (size_t)slot * kTileCubes,
      (int)(k % parts));
  }
}

// Half of a tile (four z) by a warp, lane = cube along x: visit(y, z, ci) for every row, with
// the cube's case index (0 where it is skipped or no corner is positive).  Corners beyond the
// volume repeat the last voxel (sampleVolume clamps, marchingCubes.cs:70-78; the other two
// extractions skip such cubes).
template <int S, int KIND, class F>
__device__ __forceinline__ void walk_half_tile(const McArgs& a, int tx, int ty, int tz, int half, F&& visit) {
  const int lane = threadIdx.x & 31;
  const int x = 32 * tx + lane, X = min(x, a.nx - 1), X1 = min(32 * tx + 32, a.nx - 1);
  const int y0 = 8 * ty, z0 = 8 * tz + 4 * half;
  // bit r: row y0 + r; s below iso, p above zero; 0 at x, 1 at x + 1
  uint32_t s0 = 0, s1 = 0, p0 = 0, p1 = 0;
  for (int dz = 0; dz <= 4; ++dz) {
    const int z = z0 + dz;
    const int Z = min(z, a.nz - 1);  // planes past the volume: their cubes are skipped below
    float v[9];
#pragma unroll
    for (int r = 0; r < 9; ++r) v[r] = mc_raw<S>(a.vol, mc_index(a, X, min(y0 + r, a.ny - 1), Z));
    // the column past the tile: row r by lane r
    const float e = mc_raw<S>(a.vol, mc_index(a, X1, min(y0 + min(lane, 8), a.ny - 1), Z));
    uint32_t t0 = 0, q0 = 0;
#pragma unroll
    for (int r = 0; r < 9; ++r) {
      t0 |= (uint32_t)(v[r] < a.iso) << r;
      q0 |= (uint32_t)(v[r] > 0.0f) << r;
    }
    const uint32_t te = __ballot_sync(0xffffffffu, e < a.iso) & 0x1ffu, qe = __ballot_sync(0xffffffffu, e > 0.0f) & 0x1ffu;
    uint32_t t1 = __shfl_down_sync(0xffffffffu, t0, 1), q1 = __shfl_down_sync(0xffffffffu, q0, 1);
    if (lane == 31) {
      t1 = te;
      q1 = qe;
    }
    if (dz > 0) {
      const int zc = z - 1;  // the cubes between the last plane and this one
      const uint32_t any = s0 | s1 | t0 | t1;  // rows with a corner below iso
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const int y = y0 + r;
        if (y >= a.ny) {
          visit(y, zc, 0u);
          continue;
        }
        uint32_t ci = 0;
        if (any >> r & 3u) {
          bool skip = x >= a.nx || zc >= a.nz;
          if (KIND == kHisto && a.q15)  // histoPyramids.cs:117
            skip |= x <= 10 || x >= a.nx - 10 || y <= 10 || y >= a.ny - 10 || zc <= 10 || zc >= a.nz - 10;
          else if (KIND != kClassic)
            skip |= x >= a.nx - 1 || y >= a.ny - 1 || zc >= a.nz - 1;
          // "positive found" over the first 7 corners (Q13): without (1,1,1) in the y/z-swapped
          // order, without (0,1,1) in the classic one
          uint32_t pos = (p0 | p1 | (KIND == kHisto ? q0 : q1)) >> r & 3u;
          pos |= (KIND == kHisto ? q1 : q0) >> r & (a.q13 ? 1u : 3u);
          if (pos && !skip) {
            const uint32_t b000 = s0 >> r & 1u, b100 = s1 >> r & 1u, b010 = s0 >> (r + 1) & 1u, b110 = s1 >> (r + 1) & 1u;
            const uint32_t b001 = t0 >> r & 1u, b101 = t1 >> r & 1u, b011 = t0 >> (r + 1) & 1u, b111 = t1 >> (r + 1) & 1u;
            if (KIND == kHisto)  // histoPyramids.cs:158-166
              ci = b000 | b100 << 1 | b101 << 2 | b001 << 3 | b010 << 4 | b110 << 5 | b111 << 6 | b011 << 7;
            else
              ci = b000 | b100 << 1 | b110 << 2 | b010 << 3 | b001 << 4 | b101 << 5 | b111 << 6 | b011 << 7;
          }
        }
        visit(y, zc, ci);
      }
    }
    s0 = t0; s1 = t1; p0 = q0; p1 = q1;
  }
}

// Triangles per case, in shared memory (lanes look up different cases).
__device__ __forceinline__ void load_counts(uint8_t* s_nt) {
  for (int k = threadIdx.x; k < 256; k += blockDim.x) s_nt[k] = kf_mc_nr_triangles[k];
  __syncthreads();
}

// Morton code of a brick in the traversal's child order (x lowest, then z, then y; c_hp order
// {000,100,001,101,010,110,011,111}).
__host__ __device__ inline uint32_t spread3(uint32_t v) {
  v = (v | v << 16) & 0x030000ffu;
  v = (v | v << 8) & 0x0300f00fu;
  v = (v | v << 4) & 0x030c30c3u;
  return (v | v << 2) & 0x09249249u;
}
__host__ __device__ inline uint32_t gather3(uint32_t v) {
  v &= 0x09249249u;
  v = (v | v >> 2) & 0x030c30c3u;
  v = (v | v >> 4) & 0x0300f00fu;
  v = (v | v >> 8) & 0x030000ffu;
  return (v | v >> 16) & 0x3ffu;
}
__host__ __device__ inline uint32_t morton_xzy(uint32_t x, uint32_t y, uint32_t z) {
  return spread3(x) | spread3(z) << 1 | spread3(y) << 2;
}

// classifyCubes (histoPyramids.cs:108-174): case bytes and triangles per brick.
template <int S>
__global__ void __launch_bounds__(256) histo_classify_kernel(McArgs a) {
  __shared__ uint8_t s_nt[256];
  load_counts(s_nt);
  const int lane = threadIdx.x & 31;
  for_each_part(a, 2, [&](int tx, int ty, int tz, uint8_t* cases, int half) {
    uint32_t n = 0;
    walk_half_tile<S, kHisto>(a, tx, ty, tz, half, [&](int y, int z, uint32_t ci) {
      cases[(z & 7) << 8 | (y & 7) << 5 | lane] = (uint8_t)ci;
      n += s_nt[ci];
    });
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
    if ((lane & 7) == 0 && n) atomicAdd(a.counts + morton_xzy(4 * tx + (lane >> 3), ty, tz), n);
  });
}

__device__ __forceinline__ float4 face_normal(float4 a, float4 b, float4 c) {
  const float ux = b.x - a.x, uy = b.y - a.y, uz = b.z - a.z;
  const float vx = c.x - a.x, vy = c.y - a.y, vz = c.z - a.z;
  return make_float4(uy * vz - uz * vy, uz * vx - ux * vz, ux * vy - uy * vx, 0.0f);
}

// The 32 triangles (or fewer) of a warp to out[3 * first ..] and their normals, staged so that
// the stores are whole lines; lane = triangle.
__device__ __forceinline__ void store_triangles(const McArgs& a, float4* stage, size_t first, uint32_t n,
                                                const float4* vo, const float4& fn) {
  const uint32_t lane = threadIdx.x & 31;
  __syncwarp();
#pragma unroll
  for (int v = 0; v < 3; ++v) stage[3 * lane + v] = vo[v];
  stage[96 + lane] = fn;
  __syncwarp();
#pragma unroll
  for (int v = 0; v < 3; ++v) {
    const uint32_t j = lane + 32 * v;
    if (j < 3 * n) {
      a.out[3 * first + j] = stage[j];
      a.nout[3 * first + j] = stage[96 + j / 3];
    }
  }
}

constexpr int kGenWarps = 4;  // warps per block of the generating kernels

// traverseHistoPyramids.cs:54-260 for the triangles of one brick by a warp: their cubes in
// Morton order, listed first, so that the lanes then take triangles and not cubes.
template <int S>
__global__ void __launch_bounds__(32 * kGenWarps) histo_generate_kernel(McArgs a) {
  __shared__ uint8_t s_nt[256];
  __shared__ uint16_t s_list[kGenWarps][512 * 5];  // cube (9 bits of Morton code), triangle (3 bits)
  __shared__ float4 s_stage[kGenWarps][128];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  load_counts(s_nt);
  uint16_t* list = s_list[warp];
  for_each_part(a, 4, [&](int tx, int ty, int tz, const uint8_t* tile, int part) {
    // a tile's bricks past the volume may have no place in the counts: at most 8 voxels a side
    // make one count, at most 16 eight, and the first codes of the four parts are 0, 1, 8 and 9
    if (32 * tx + 8 * part >= a.nx) return;
    const uint32_t code = morton_xzy(4 * tx + part, ty, tz), total = __ldg(a.counts + code), off = __ldg(a.offsets + code);
    if (!total || off + total > a.cap || off + total < off) return;  // none, or it does not fit
    const int bx = 32 * tx + 8 * part, by = 8 * ty, bz = 8 * tz;
    const uint8_t* cases = tile + 8 * part;  // + x + 32 y + 256 z
    // lane: cubes 16 * lane .. + 15, i.e. four x of each of 2 x 2 rows
    const uint32_t m = 16u * lane;
    const int lx = (int)gather3(m), lz = (int)gather3(m >> 1), ly = (int)gather3(m >> 2);
    uint32_t rows[4];  // by (y0, z0): four case bytes
    uint32_t n = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      rows[q] = __ldg(reinterpret_cast<const uint32_t*>(cases + lx + 32 * (ly + (q >> 1)) + 256 * (lz + (q & 1))));
#pragma unroll
      for (int j = 0; j < 4; ++j) n += s_nt[rows[q] >> (8 * j) & 255u];
    }
    uint32_t at = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t u = __shfl_up_sync(0xffffffffu, at, o);
      if (lane >= o) at += u;
    }
    at -= n;
    __syncwarp();
    // Morton order inside the lane's 16 cubes: x0, z0, y0, x1
#pragma unroll
    for (int c = 0; c < 16; ++c) {
      const int q = (c >> 2 & 1) << 1 | (c >> 1 & 1), xi = (c & 1) | (c >> 3) << 1;
      const uint32_t nt = s_nt[rows[q] >> (8 * xi) & 255u];
      for (uint32_t j = 0; j < nt; ++j) list[at++] = (uint16_t)((m + c) << 3 | j);
    }
    __syncwarp();
    for (uint32_t i0 = 0; i0 < total; i0 += 32) {
      float4 vo[3] = {}, fn = {};
      if (i0 + lane < total) {
        const uint32_t ent = list[i0 + lane], cube = ent >> 3, j = ent & 7u;
        const int x = (int)gather3(cube), z = (int)gather3(cube >> 1), y = (int)gather3(cube >> 2);
        const int cx = bx + x, cy = by + y, cz = bz + z;
        const uint32_t ci = __ldg(cases + x + 32 * y + 256 * z);
#pragma unroll
        for (int v = 0; v < 3; ++v) {
          const int edge = kf_mc_tri_table[ci * 16 + 3 * j + v];
          const uint8_t* o = &kf_mc_offsets3[edge * 6];
          const int p0x = cx + o[0], p0y = cy + o[1], p0z = cz + o[2];
          const int p1x = cx + o[3], p1y = cy + o[4], p1z = cz + o[5];
          const float v0 = mc_raw<S>(a.vol, mc_index(a, p0x, p0y, p0z));
          const float v1 = mc_raw<S>(a.vol, mc_index(a, p1x, p1y, p1z));
          float al = (a.iso - v0) / (v1 - v0);
          if (al > 1.0f || al < 0.0f) al = 0.5f;  // traverseHistoPyramids.cs:213-216
          vo[v] = make_float4(p0x * (1.0f - al) + p1x * al, p0y * (1.0f - al) + p1y * al,
                              p0z * (1.0f - al) + p1z * al, 0.0f);
        }
        fn = face_normal(vo[0], vo[1], vo[2]);
      }
      store_triangles(a, s_stage[warp], (size_t)off + i0, min(total - i0, 32u), vo, fn);
    }
    __syncwarp();
  });
}

// ---- classic path (marchingCubes.cs) ---------------------------------------------------
// launchClassifyVoxel: case bytes and vertices per row segment.
template <int S>
__global__ void __launch_bounds__(256) classic_classify_kernel(McArgs a) {
  __shared__ uint8_t s_nt[256];
  load_counts(s_nt);
  const int lane = threadIdx.x & 31;
  for_each_part(a, 2, [&](int tx, int ty, int tz, uint8_t* cases, int half) {
    walk_half_tile<S, kClassic>(a, tx, ty, tz, half, [&](int y, int z, uint32_t ci) {
      cases[(z & 7) << 8 | (y & 7) << 5 | lane] = (uint8_t)ci;
      if (!__any_sync(0xffffffffu, ci != 0)) return;
      const uint32_t n = __reduce_add_sync(0xffffffffu, 3u * s_nt[ci]);
      if (lane == 0) a.counts[mc_segment(a, tx, y, z)] = n;
    });
  });
}

// One row's triangles listed in cube order (cube << 3 | triangle) by its warp; returns their number.
__device__ __forceinline__ uint32_t list_row(uint16_t* list, uint32_t nt) {
  const int lane = threadIdx.x & 31;
  uint32_t at = nt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t u = __shfl_up_sync(0xffffffffu, at, o);
    if (lane >= o) at += u;
  }
  const uint32_t total = __shfl_sync(0xffffffffu, at, 31);
  at -= nt;
  __syncwarp();
  for (uint32_t j = 0; j < nt; ++j) list[at++] = (uint16_t)(lane << 3 | j);
  __syncwarp();
  return total;
}

// launchGenerateTriangles: the cubes' triangles at their offsets, in voxel order; a warp per
// (tile, z), row by row.
template <int S>
__global__ void __launch_bounds__(32 * kGenWarps) classic_generate_kernel(McArgs a) {
  __shared__ uint8_t s_nt[256];
  __shared__ uint16_t s_list[kGenWarps][32 * 5];
  __shared__ float4 s_stage[kGenWarps][128];
  load_counts(s_nt);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for_each_part(a, 8, [&](int tx, int ty, int tz, const uint8_t* cases, int dz) {
    const int z = 8 * tz + dz;
    if (z >= a.nz) return;
    for (int r = 0; r < 8; ++r) {
      const int y = 8 * ty + r;
      if (y >= a.ny) break;
      const uint32_t seg = mc_segment(a, tx, y, z), count = __ldg(a.counts + seg), first = __ldg(a.offsets + seg);
      if (!count || first + count > a.cap || first + count < first) continue;  // none, or it does not fit
      const uint8_t* row = cases + (dz << 8 | r << 5);
      const uint32_t total = list_row(s_list[warp], s_nt[__ldg(row + lane)]);
      for (uint32_t i0 = 0; i0 < total; i0 += 32) {
        float4 vo[3] = {}, fn = {};
        if (i0 + lane < total) {
          const uint32_t ent = s_list[warp][i0 + lane], j = ent & 7u, ci = __ldg(row + (ent >> 3));
          const int x = 32 * tx + (int)(ent >> 3);
          // corner positions: voxel-index units, or with Q24 the shader's p = -1 + gridPos *
          // voxelSize plus the corner's voxelSize offset (launchGenerateTriangles, :205-220)
          float px = (float)x, py = (float)y, pz = (float)z, sx = 1.0f, sy = 1.0f, sz = 1.0f;
          if (a.shader_units) {
            px = -1.0f + (float)x * a.vsx;
            py = -1.0f + (float)y * a.vsy;
            pz = -1.0f + (float)z * a.vsz;
            sx = a.vsx; sy = a.vsy; sz = a.vsz;
          }
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            const int e = kf_mc_tri_table[ci * 16 + 3 * j + k];
            const int p = c_bourke_edge[e][0], q = c_bourke_edge[e][1];
            // sampleVolume clamps to gridSize - 1 (marchingCubes.cs:70-78)
            const float fp = mc_raw<S>(a.vol, mc_index(a, min(x + c_bourke[p][0], a.nx - 1),
                                                       min(y + c_bourke[p][1], a.ny - 1), min(z + c_bourke[p][2], a.nz - 1)));
            const float fq = mc_raw<S>(a.vol, mc_index(a, min(x + c_bourke[q][0], a.nx - 1),
                                                       min(y + c_bourke[q][1], a.ny - 1), min(z + c_bourke[q][2], a.nz - 1)));
            const float t = (a.iso - fp) / (fq - fp);  // vertexInterp (:81-85)
            const float ax = c_bourke[p][0] ? px + sx : px, ay = c_bourke[p][1] ? py + sy : py,
                        az = c_bourke[p][2] ? pz + sz : pz;
            const float bx = c_bourke[q][0] ? px + sx : px, by = c_bourke[q][1] ? py + sy : py,
                        bz = c_bourke[q][2] ? pz + sz : pz;
            vo[k] = make_float4(ax * (1.0f - t) + bx * t, ay * (1.0f - t) + by * t, az * (1.0f - t) + bz * t, 1.0f);
          }
          // calcNormal (:87-93) on the unscaled positions, one per triangle
          fn = face_normal(vo[0], vo[1], vo[2]);
          if (a.shader_units) {  // pos[index] of :290-299: / 128 * voxelSize.x, z negated
#pragma unroll
            for (int k = 0; k < 3; ++k)
              vo[k] = make_float4((vo[k].x / 128.0f) * a.vsx, (vo[k].y / 128.0f) * a.vsx, -(vo[k].z / 128.0f) * a.vsx, 1.0f);
          }
        }
        store_triangles(a, s_stage[warp], (size_t)(first / 3) + i0, min(total - i0, 32u), vo, fn);
      }
    }
  });
}

// ---- welded mesh: one vertex per cut voxel edge, indexed triangles ----------------------
// Export form (no counterpart in the reference, whose exportMesh writes the triangle soup
// with normal (1,1,1), mcubes.cpp:451-500).  Cubes are the interior cubes [0, n-2]^3 in the
// classic path's Bourke corner order and case table; a triangle vertex lies on a cube edge,
// which belongs to the voxel at its lower end and its axis.  Every edge a triangle uses is
// marked (a cube with triangles uses exactly its cut edges), the marks are counted per row
// segment and prefix-summed: an edge's vertex index is its rank among the marked edges in
// voxel order, then axis order, the same whatever the launch.  Positions are world metres
// ((voxel index + 0.5) * dim / size, the voxel centres of integrate.cs:16-19); normals the
// normalised TSDF gradient (central differences at the edge's two voxels, interpolated).
// per Bourke edge (corners c_bourke_edge): the voxel at its lower end (offset from the
// cube's corner 0) and its axis
__constant__ int c_edge_owner[12][4] = {{0, 0, 0, 0}, {1, 0, 0, 1}, {0, 1, 0, 0}, {0, 0, 0, 1},
                                        {0, 0, 1, 0}, {1, 0, 1, 1}, {0, 1, 1, 0}, {0, 0, 1, 1},
                                        {0, 0, 0, 2}, {1, 0, 0, 2}, {1, 1, 0, 2}, {0, 1, 0, 2}};

// Marks the edges and counts the triangles per segment.  Lane e collects the warp's marks of
// edge e (a ballot each); an owner one voxel further along x moves the bits by one, the last
// of them into the next segment.
template <int S>
__global__ void __launch_bounds__(256) mesh_mark_kernel(McArgs a) {
  __shared__ uint8_t s_nt[256];
  load_counts(s_nt);
  const int lane = threadIdx.x & 31;
  for_each_part(a, 2, [&](int tx, int ty, int tz, uint8_t* cases, int half) {
    walk_half_tile<S, kMesh>(a, tx, ty, tz, half, [&](int y, int z, uint32_t ci) {
      cases[(z & 7) << 8 | (y & 7) << 5 | lane] = (uint8_t)ci;
      if (!__any_sync(0xffffffffu, ci != 0)) return;
      const uint32_t nt = s_nt[ci], n = __reduce_add_sync(0xffffffffu, nt);
      if (!n) return;
      if (lane == 0) a.counts[mc_segment(a, tx, y, z)] = n;
      const uint32_t edges = nt ? kf_mc_edge_table[ci] : 0u;
      uint32_t bits = 0;
#pragma unroll
      for (int e = 0; e < 12; ++e) {
        const uint32_t b = __ballot_sync(0xffffffffu, edges >> e & 1u);
        if (lane == e) bits = b;
      }
      if (lane < 12 && bits) {
        const int ox = c_edge_owner[lane][0], axis = c_edge_owner[lane][3];
        const uint32_t seg = mc_segment(a, tx, y + c_edge_owner[lane][1], z + c_edge_owner[lane][2]);
        const uint32_t here = bits << ox;
        if (here) atomicOr(a.mask + 3 * (size_t)seg + axis, here);
        if (ox && bits >> 31) atomicOr(a.mask + 3 * (size_t)(seg + 1) + axis, 1u);
      }
    });
  });
}

// Vertices per segment, of the listed tiles.
__global__ void __launch_bounds__(256) mesh_count_kernel(McArgs a) {
  for_each_part(a, 2, [&](int tx, int ty, int tz, const uint8_t*, int half) {
    const int r = (threadIdx.x & 31) + 32 * half;
    const int y = 8 * ty + (r & 7), z = 8 * tz + (r >> 3);
    if (y >= a.ny || z >= a.nz) return;
    const uint32_t seg = mc_segment(a, tx, y, z);
    const uint32_t* m = a.mask + 3 * (size_t)seg;
    const uint32_t n = (uint32_t)(__popc(m[0]) + __popc(m[1]) + __popc(m[2]));
    if (n) a.vcounts[seg] = n;
  });
}

template <int S>
__device__ __forceinline__ float mesh_val(const McArgs& a, int x, int y, int z) {
  x = min(max(x, 0), a.nx - 1);
  y = min(max(y, 0), a.ny - 1);
  z = min(max(z, 0), a.nz - 1);
  return mc_raw<S>(a.vol, mc_index(a, x, y, z));
}

// A marked edge's rank in its segment: the marked edges of earlier voxels, then of earlier axes.
__device__ __forceinline__ uint32_t mesh_rank(const uint32_t* m, int bit, int axis) {
  const uint32_t m0 = m[0], m1 = m[1], m2 = m[2], below = (1u << bit) - 1u;
  return (uint32_t)(__popc(m0 & below) + __popc(m1 & below) + __popc(m2 & below)) +
         (axis > 0 ? m0 >> bit & 1u : 0u) + (axis > 1 ? m1 >> bit & 1u : 0u);
}

// A warp per (tile, z), row by row: the row's marked edges listed in rank order, then a lane each.
template <int S>
__global__ void __launch_bounds__(32 * kGenWarps) mesh_vertex_kernel(McArgs a) {
  __shared__ uint8_t s_list[kGenWarps][96];  // voxel, axis << 5
  const int lane = threadIdx.x & 31;
  uint8_t* list = s_list[threadIdx.x >> 5];
  const float hx = 0.5f * a.nx / a.dimx, hy = 0.5f * a.ny / a.dimy, hz = 0.5f * a.nz / a.dimz;
  for_each_part(a, 8, [&](int tx, int ty, int tz, const uint8_t*, int dz) {
    const int z = 8 * tz + dz;
    if (z >= a.nz) return;
    for (int r = 0; r < 8; ++r) {
      const int y = 8 * ty + r;
      if (y >= a.ny) break;
      const uint32_t seg = mc_segment(a, tx, y, z), count = __ldg(a.vcounts + seg), first = __ldg(a.voffsets + seg);
      if (!count || first + count > a.vcap || first + count < first) continue;  // none, or it does not fit
      const uint32_t* m = a.mask + 3 * (size_t)seg;
      __syncwarp();
#pragma unroll
      for (int k = 0; k < 3; ++k)
        if (m[k] >> lane & 1u) list[mesh_rank(m, lane, k)] = (uint8_t)(lane | k << 5);
      __syncwarp();
      for (uint32_t i = lane; i < count; i += 32) {
        const int axis = list[i] >> 5, x = 32 * tx + (list[i] & 31);
        const size_t out = (size_t)first + i;
        const int x1 = x + (axis == 0), y1 = y + (axis == 1), z1 = z + (axis == 2);
        const float f0 = mesh_val<S>(a, x, y, z), f1 = mesh_val<S>(a, x1, y1, z1);
        const float t = (a.iso - f0) / (f1 - f0);  // vertexInterp (marchingCubes.cs:81-85)
        const float px = x + t * (x1 - x), py = y + t * (y1 - y), pz = z + t * (z1 - z);
        a.pos[3 * out + 0] = (px + 0.5f) * a.dimx / a.nx;
        a.pos[3 * out + 1] = (py + 0.5f) * a.dimy / a.ny;
        a.pos[3 * out + 2] = (pz + 0.5f) * a.dimz / a.nz;
        // central-difference gradients at both voxels (world units), interpolated
        float g[3];
        {
          const float g0x = (mesh_val<S>(a, x + 1, y, z) - mesh_val<S>(a, x - 1, y, z)) * hx;
          const float g0y = (mesh_val<S>(a, x, y + 1, z) - mesh_val<S>(a, x, y - 1, z)) * hy;
          const float g0z = (mesh_val<S>(a, x, y, z + 1) - mesh_val<S>(a, x, y, z - 1)) * hz;
          const float g1x = (mesh_val<S>(a, x1 + 1, y1, z1) - mesh_val<S>(a, x1 - 1, y1, z1)) * hx;
          const float g1y = (mesh_val<S>(a, x1, y1 + 1, z1) - mesh_val<S>(a, x1, y1 - 1, z1)) * hy;
          const float g1z = (mesh_val<S>(a, x1, y1, z1 + 1) - mesh_val<S>(a, x1, y1, z1 - 1)) * hz;
          g[0] = g0x + t * (g1x - g0x);
          g[1] = g0y + t * (g1y - g0y);
          g[2] = g0z + t * (g1z - g0z);
        }
        const float len = sqrtf(g[0] * g[0] + g[1] * g[1] + g[2] * g[2]);
        const float il = len > 0.0f ? 1.0f / len : 0.0f;
        a.nrm[3 * out + 0] = g[0] * il;
        a.nrm[3 * out + 1] = g[1] * il;
        a.nrm[3 * out + 2] = g[2] * il;
      }
    }
  });
}

__global__ void __launch_bounds__(32 * kGenWarps) mesh_index_kernel(McArgs a) {
  __shared__ uint8_t s_nt[256];
  __shared__ uint16_t s_list[kGenWarps][32 * 5];
  load_counts(s_nt);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for_each_part(a, 8, [&](int tx, int ty, int tz, const uint8_t* cases, int dz) {
    const int z = 8 * tz + dz;
    if (z >= a.nz) return;
    for (int r = 0; r < 8; ++r) {
      const int y = 8 * ty + r;
      if (y >= a.ny) break;
      const uint32_t seg = mc_segment(a, tx, y, z), count = __ldg(a.counts + seg), first = __ldg(a.offsets + seg);
      if (!count || first + count > a.cap || first + count < first) continue;  // none, or it does not fit
      const uint8_t* row = cases + (dz << 8 | r << 5);
      list_row(s_list[warp], s_nt[__ldg(row + lane)]);
      // lane = index: table vertices (0, 1, 2) stored as (0, 2, 1), counter-clockwise seen from
      // the positive (free-space) side, so facet normals point along the TSDF gradient
      for (uint32_t i = lane; i < 3 * count; i += 32) {
        const uint32_t ent = s_list[warp][i / 3], k = i % 3, ci = __ldg(row + (ent >> 3));
        const int e = kf_mc_tri_table[ci * 16 + 3 * (ent & 7u) + (k == 0 ? 0u : 3u - k)];
        const int bit = (int)(ent >> 3) + c_edge_owner[e][0];
        const uint32_t own = mc_segment(a, tx, y + c_edge_owner[e][1], z + c_edge_owner[e][2]) + (uint32_t)(bit >> 5);
        a.idx[3 * (size_t)first + i] =
            __ldg(a.voffsets + own) + mesh_rank(a.mask + 3 * (size_t)own, bit & 31, c_edge_owner[e][3]);
      }
    }
  });
}

// Grows a device buffer to at least `bytes`, by 1.5x steps so that a mesh that grows
// from one extraction to the next does not reallocate (and synchronise) every time.
int ensure(kf_session* s, void** p, size_t* cap, size_t bytes) {
  if (*cap >= bytes && *p) return KF_OK;
  bytes = std::max(bytes, *cap + *cap / 2);
  cudaFree(*p);
  *p = nullptr;
  *cap = 0;
  if (cudaMalloc(p, bytes) != cudaSuccess) {
    cudaGetLastError();
    s->last_error = "marching cubes: out of device memory";
    return KF_ERR_OUT_OF_MEMORY;
  }
  *cap = bytes;
  return KF_OK;
}

// Bytes for the vertex buffer: the vertices needed now, but at least room for one triangle
// per 64 cubes (fused scenes reach one triangle per 200-600 cubes), so a mesh that grows as
// frames are fused does not reallocate: a reallocation frees and allocates device memory,
// which synchronises the device and takes the driver's locks, whose wait is unbounded on a
// shared machine.
size_t vertex_bytes(size_t ncube, size_t nverts) {
  return std::max<size_t>(16, std::max(nverts, ncube / 64 * 3) * 16);
}

McArgs make_mc_args(kf_session* s, float iso) {
  McArgs a{};
  a.vol = s->d_vol;
  a.nx = s->cfg.nx; a.ny = s->cfg.ny; a.nz = s->cfg.nz;
  a.iso = iso;
  a.q13 = (s->cfg.quirks & KF_Q13_MC_FIRST_SEVEN) ? 1 : 0;
  a.q15 = (s->cfg.quirks & KF_Q15_MC_BORDER_SKIP) ? 1 : 0;
  a.neg = iso <= 0.0f ? s->d_neg : nullptr;  // a corner below iso is then negative
  a.wx = s->wx; a.wy = s->wy;
  a.tx = (a.nx + 31) / 32; a.ty = (a.ny + 7) / 8; a.tz = (a.nz + 7) / 8;
  a.dimx = s->cfg.dim_x; a.dimy = s->cfg.dim_y; a.dimz = s->cfg.dim_z;
  return a;
}

size_t tile_count(const McArgs& a) { return (size_t)a.tx * a.ty * a.tz; }

// rounded up, so that the arrays of that many words behind one another are 16-byte aligned
size_t segment_count(const McArgs& a) { return ((size_t)a.tx * a.ny * a.nz + 3) & ~(size_t)3; }

#define KF_MC_LAUNCH(kernel, grid, threads, ...)                                                             \
  do {                                                                                                       \
    switch (s->cfg.storage) {                                                                                \
      case KF_STORAGE_F32F32: kernel<KF_STORAGE_F32F32><<<grid, threads, 0, s->stream>>>(__VA_ARGS__); break; \
      case KF_STORAGE_F16U16: kernel<KF_STORAGE_F16U16><<<grid, threads, 0, s->stream>>>(__VA_ARGS__); break; \
      default: kernel<KF_STORAGE_RG16I><<<grid, threads, 0, s->stream>>>(__VA_ARGS__); break;                 \
    }                                                                                                        \
    KF_CUDA_TRY(s, cudaGetLastError());                                                                     \
    kf_note_launch(s);                                                                                      \
  } while (0)

// The vertex and normal buffers' capacity in vertices, with room for at least `nverts`.
int ensure_soup(kf_session* s, size_t nverts) {
  const size_t bytes = vertex_bytes((size_t)s->cfg.nx * s->cfg.ny * s->cfg.nz, nverts);
  int rc = ensure(s, (void**)&s->d_mc_vertices, &s->mc_vertex_cap, bytes);
  if (!rc) rc = ensure(s, (void**)&s->d_mc_normals, &s->mc_normal_cap, bytes);
  return rc;
}
// What the two buffers hold, in units of `vertices` vertices (1, or 3: triangles).  The kernels
// count units in 32 bits, not bytes or vertices: a soup of more than 2^32 / 3 triangles fits too.
constexpr uint32_t soup_room(size_t vertex_cap, size_t normal_cap, size_t vertices) {
  const size_t units = (vertex_cap < normal_cap ? vertex_cap : normal_cap) / (16 * vertices);
  return units < 0xffffffffu ? (uint32_t)units : 0xffffffffu;
}
static_assert(soup_room((size_t)1500000000 * 48, (size_t)1500000000 * 48, 3) == 1500000000u &&
                  soup_room((size_t)1 << 36, (size_t)1 << 37, 1) == 0xffffffffu && soup_room(95, 960, 3) == 1,
              "an extraction repeats until its count fits");

// Words of an extraction's tile list: the list, its length.
size_t list_words(const McArgs& a) { return tile_count(a) + 1; }

// The list that belongs to the case bytes of histopyramid() and classic().
uint32_t* case_tiles(const kf_session* s, const McArgs& a) {
  return reinterpret_cast<uint32_t*>(s->d_mc_cases + tile_count(a) * kTileCubes);
}

// Lays the list out at w, zeroes its length and fills it.
int list_tiles(kf_session* s, McArgs* a, uint32_t* w) {
  const size_t n = tile_count(*a);
  a->list = w;
  a->listed = w + n;
  KF_CUDA_TRY(s, cudaMemsetAsync(a->listed, 0, 4, s->stream));
  tile_list_kernel<<<(int)((n + 255) / 256), 256, 0, s->stream>>>(*a);
  KF_CUDA_TRY(s, cudaGetLastError());
  kf_note_launch(s);
  return KF_OK;
}

// Grids of the kernels that walk the list: their warps take the parts in turn.
int walk_blocks(const kf_session* s) { return 6 * s->num_sms; }
int gen_blocks(const kf_session* s) { return 16 * s->num_sms; }  // 512^3: 104, 74, 73, 64 us at 4, 8, 12, 16
constexpr int kGenThreads = 32 * kGenWarps;

// Prefix sum of the counts; its result is on the way to two pinned words.
int scan_counts(kf_session* s, const uint32_t* counts, uint32_t* offsets, uint64_t n, uint32_t* scratch, size_t words,
                uint32_t* host) {
  const uint32_t* result = nullptr;
  if (int rc = kf_scan_u32(counts, offsets, n, s->stream, scratch, words, &result)) return rc;
  KF_CUDA_TRY(s, cudaMemcpyAsync(host, result, 8, cudaMemcpyDeviceToHost, s->stream));
  return KF_OK;
}
int scan_check(kf_session* s, const uint32_t* host) {
  if (!host[1]) return KF_OK;
  s->last_error = "prefix sum: a wait for another block gave up";
  return KF_ERR_CUDA;
}

int histopyramid(kf_session* s, float iso, uint32_t* n_tri) {
  McArgs a = make_mc_args(s, iso);
  uint32_t side = 1;  // bricks per side of the pyramid's power-of-two cube
  while (side < (uint32_t)std::max(s->bx, std::max(s->by, s->bz))) side <<= 1;
  const uint32_t codes = side * side * side;
  const size_t sw = kf_scan_scratch_words(codes);
  int rc;
  // case bytes, then the list of their tiles
  if ((rc = ensure(s, (void**)&s->d_mc_cases, &s->mc_case_cap, tile_count(a) * kTileCubes + list_words(a) * 4))) return rc;
  // counts[codes], offsets[codes], scan scratch
  if ((rc = ensure(s, (void**)&s->d_mc_scratch, &s->mc_scratch_words, (2 * (size_t)codes + sw) * 4))) return rc;
  uint32_t* offs = s->d_mc_scratch + codes;
  a.cases = s->d_mc_cases;
  a.counts = s->d_mc_scratch;
  a.offsets = offs;
  KF_CUDA_TRY(s, cudaMemsetAsync(a.counts, 0, (size_t)codes * 4, s->stream));
  if ((rc = list_tiles(s, &a, case_tiles(s, a)))) return rc;
  KF_MC_LAUNCH(histo_classify_kernel, walk_blocks(s), 256, a);
  // and the triangle count (glGetTexImage of the top texel at mcubes.cpp:290-300)
  if ((rc = scan_counts(s, a.counts, offs, codes, offs + codes, sw, s->h_u32_scalar))) return rc;
  for (;;) {
    a.cap = soup_room(s->mc_vertex_cap, s->mc_normal_cap, 3);
    a.out = s->d_mc_vertices;
    a.nout = s->d_mc_normals;
    if (a.out && a.nout) KF_MC_LAUNCH(histo_generate_kernel, gen_blocks(s), kGenThreads, a);
    KF_CUDA_TRY(s, cudaStreamSynchronize(s->stream));
    if ((rc = scan_check(s, s->h_u32_scalar))) return rc;
    const uint32_t T = s->h_u32_scalar[0];
    if (a.out && a.nout && T <= a.cap) {
      *n_tri = T;
      return KF_OK;
    }
    if ((rc = ensure_soup(s, (size_t)T * 3))) return rc;
  }
}

int classic(kf_session* s, float iso, uint32_t* n_tri) {
  if ((size_t)s->cfg.nx * s->cfg.ny * s->cfg.nz >= (1ull << 32)) return KF_ERR_INVALID_ARGUMENT;
  McArgs a = make_mc_args(s, iso);
  const size_t n = segment_count(a), sw = kf_scan_scratch_words(n);
  int rc;
  // case bytes, then the list of their tiles
  if ((rc = ensure(s, (void**)&s->d_mc_cases, &s->mc_case_cap, tile_count(a) * kTileCubes + list_words(a) * 4))) return rc;
  // counts[n], offsets[n], scan scratch
  if ((rc = ensure(s, (void**)&s->d_mc_scratch, &s->mc_scratch_words, (2 * n + sw) * 4))) return rc;
  uint32_t* offs = s->d_mc_scratch + n;
  a.cases = s->d_mc_cases;
  a.counts = s->d_mc_scratch;
  a.offsets = offs;
  a.shader_units = (s->cfg.quirks & KF_Q24_MC_SHADER_UNITS) ? 1 : 0;
  a.vsx = 1000.0f * s->cfg.dim_x / (float)a.nx;
  a.vsy = 1000.0f * s->cfg.dim_y / (float)a.ny;
  a.vsz = 1000.0f * s->cfg.dim_z / (float)a.nz;
  KF_CUDA_TRY(s, cudaMemsetAsync(a.counts, 0, n * 4, s->stream));
  if ((rc = list_tiles(s, &a, case_tiles(s, a)))) return rc;
  KF_MC_LAUNCH(classic_classify_kernel, walk_blocks(s), 256, a);
  if ((rc = scan_counts(s, a.counts, offs, n, offs + n, sw, s->h_u32_scalar))) return rc;
  for (;;) {
    a.cap = soup_room(s->mc_vertex_cap, s->mc_normal_cap, 1);
    a.out = s->d_mc_vertices;
    a.nout = s->d_mc_normals;
    if (a.out && a.nout) KF_MC_LAUNCH(classic_generate_kernel, gen_blocks(s), kGenThreads, a);
    KF_CUDA_TRY(s, cudaStreamSynchronize(s->stream));
    if ((rc = scan_check(s, s->h_u32_scalar))) return rc;
    const uint32_t nverts = s->h_u32_scalar[0];
    if (a.out && a.nout && nverts <= a.cap) {
      *n_tri = nverts / 3;
      return KF_OK;
    }
    if ((rc = ensure_soup(s, nverts))) return rc;
  }
}

int copy_vertices_host(kf_session* s, std::vector<float>& v) {
  v.resize((size_t)s->mc_triangles * 3 * 4);
  if (v.empty()) return KF_OK;
  KF_CUDA_TRY(s, cudaMemcpyAsync(v.data(), s->d_mc_vertices, v.size() * 4, cudaMemcpyDeviceToHost, s->stream));
  KF_CUDA_TRY(s, cudaStreamSynchronize(s->stream));
  return KF_OK;
}

// The welded mesh of the current volume.
int extract_mesh(kf_session* s, float iso, uint32_t* nv_out, uint32_t* nt_out) {
  if ((size_t)s->cfg.nx * s->cfg.ny * s->cfg.nz >= (1ull << 32)) return KF_ERR_INVALID_ARGUMENT;
  McArgs a = make_mc_args(s, iso);
  const size_t n = segment_count(a), sw = kf_scan_scratch_words(n);
  s->mesh_valid = 0;
  int rc;
  if ((rc = ensure(s, (void**)&s->d_mesh_cases, &s->mesh_case_cap, tile_count(a) * kTileCubes))) return rc;
  // triangles[n], vertices[n], edge marks[3 n], triangle offsets[n], vertex offsets[n], scan
  // scratch twice, tile list
  if ((rc = ensure(s, (void**)&s->d_mesh_scratch, &s->mesh_scratch_cap, (7 * n + 2 * sw + list_words(a)) * 4))) return rc;
  uint32_t* w = s->d_mesh_scratch;
  uint32_t *toff = w + 5 * n, *voff = w + 6 * n, *scr = w + 7 * n;
  a.cases = s->d_mesh_cases;
  a.counts = w;
  a.vcounts = w + n;
  a.mask = w + 2 * n;
  a.offsets = toff;
  a.voffsets = voff;
  KF_CUDA_TRY(s, cudaMemsetAsync(w, 0, 5 * n * 4, s->stream));
  if ((rc = list_tiles(s, &a, scr + 2 * sw))) return rc;
  KF_MC_LAUNCH(mesh_mark_kernel, walk_blocks(s), 256, a);
  mesh_count_kernel<<<walk_blocks(s), 256, 0, s->stream>>>(a);
  KF_CUDA_TRY(s, cudaGetLastError());
  kf_note_launch(s);
  if ((rc = scan_counts(s, a.counts, toff, n, scr, sw, s->h_u32_scalar))) return rc;
  if ((rc = scan_counts(s, a.vcounts, voff, n, scr + sw, sw, s->h_u32_scalar + 2))) return rc;
  for (;;) {
    // launched for what the buffers hold, and again if that was too little
    a.vcap = (uint32_t)std::min<size_t>(std::min(s->mesh_pos_cap, s->mesh_nrm_cap) / 12, 0xffffffffu);
    a.cap = (uint32_t)std::min<size_t>(s->mesh_idx_cap / 12, 0xffffffffu);
    a.pos = s->d_mesh_pos;
    a.nrm = s->d_mesh_nrm;
    a.idx = s->d_mesh_idx;
    if (a.vcap) KF_MC_LAUNCH(mesh_vertex_kernel, gen_blocks(s), kGenThreads, a);
    if (a.cap) {
      mesh_index_kernel<<<gen_blocks(s), kGenThreads, 0, s->stream>>>(a);
      KF_CUDA_TRY(s, cudaGetLastError());
      kf_note_launch(s);
    }
    KF_CUDA_TRY(s, cudaStreamSynchronize(s->stream));
    if ((rc = scan_check(s, s->h_u32_scalar)) || (rc = scan_check(s, s->h_u32_scalar + 2))) return rc;
    const uint32_t T = s->h_u32_scalar[0], NV = s->h_u32_scalar[2];
    if ((uint64_t)T * 3 >= (1ull << 32)) return KF_ERR_CAPACITY;
    if (NV <= a.vcap && T <= a.cap) {
      s->mesh_vertices = NV;
      s->mesh_triangles = T;
      s->mesh_valid = 1;
      *nv_out = NV;
      *nt_out = T;
      return KF_OK;
    }
    if ((rc = ensure(s, (void**)&s->d_mesh_pos, &s->mesh_pos_cap, std::max<size_t>(12, (size_t)NV * 12)))) return rc;
    if ((rc = ensure(s, (void**)&s->d_mesh_nrm, &s->mesh_nrm_cap, std::max<size_t>(12, (size_t)NV * 12)))) return rc;
    if ((rc = ensure(s, (void**)&s->d_mesh_idx, &s->mesh_idx_cap, std::max<size_t>(12, (size_t)T * 12)))) return rc;
  }
}

int copy_mesh_host(kf_session* s, std::vector<float>& pos, std::vector<float>& nrm, std::vector<uint32_t>& idx) {
  pos.resize((size_t)s->mesh_vertices * 3);
  nrm.resize((size_t)s->mesh_vertices * 3);
  idx.resize((size_t)s->mesh_triangles * 3);
  if (!pos.empty()) {
    KF_CUDA_TRY(s, cudaMemcpyAsync(pos.data(), s->d_mesh_pos, pos.size() * 4, cudaMemcpyDeviceToHost, s->stream));
    KF_CUDA_TRY(s, cudaMemcpyAsync(nrm.data(), s->d_mesh_nrm, nrm.size() * 4, cudaMemcpyDeviceToHost, s->stream));
  }
  if (!idx.empty())
    KF_CUDA_TRY(s, cudaMemcpyAsync(idx.data(), s->d_mesh_idx, idx.size() * 4, cudaMemcpyDeviceToHost, s->stream));
  KF_CUDA_TRY(s, cudaStreamSynchronize(s->stream));
  return KF_OK;
}

}  // namespace

int kf_mc_run(kf_session* s, float iso, int method, uint32_t* n_tri) {
  cudaEvent_t e0 = s->ev[0], e1 = s->ev[1];
  cudaEventRecord(e0, s->stream);
  s->mc_valid = 0;
  int rc = (method == KF_MC_SCAN) ? classic(s, iso, n_tri) : histopyramid(s, iso, n_tri);
  if (rc) return rc;
  cudaEventRecord(e1, s->stream);
  cudaEventSynchronize(e1);
  cudaEventElapsedTime(&s->stage_ms[5], e0, e1);
  s->mc_triangles = *n_tri;
  s->mc_valid = 1;
  return KF_OK;
}

extern "C" {

int kf_mc_extract(kf_session* s, float iso, int method, uint32_t* n) {
  if (!s || !n || (method != KF_MC_HISTOPYRAMID && method != KF_MC_SCAN)) return KF_ERR_INVALID_ARGUMENT;
  return kf_mc_run(s, iso, method, n);
}

int kf_mc_copy_vertices(kf_session* s, float* v, uint64_t max_vertices) {
  if (!s || (!v && s->mc_triangles)) return KF_ERR_INVALID_ARGUMENT;
  if (!s->mc_valid) return KF_ERR_STATE;
  const uint64_t n = (uint64_t)s->mc_triangles * 3;
  if (max_vertices < n) return KF_ERR_CAPACITY;
  if (!n) return KF_OK;
  return kf_copy_to_host(s, v, s->d_mc_vertices, n * 16);
}

int kf_mc_copy_normals(kf_session* s, float* n4, uint64_t max_vertices) {
  if (!s || (!n4 && s->mc_triangles)) return KF_ERR_INVALID_ARGUMENT;
  if (!s->mc_valid) return KF_ERR_STATE;
  const uint64_t n = (uint64_t)s->mc_triangles * 3;
  if (max_vertices < n) return KF_ERR_CAPACITY;
  if (!n) return KF_OK;
  return kf_copy_to_host(s, n4, s->d_mc_normals, n * 16);
}

int kf_mc_copy_base_level(kf_session* s, uint32_t* base, uint64_t count) {
  if (!s || !base) return KF_ERR_INVALID_ARGUMENT;
  if (!s->mc_valid) return KF_ERR_STATE;
  if (count != (uint64_t)s->cfg.nx * s->cfg.ny * s->cfg.nz) return KF_ERR_INVALID_ARGUMENT;
  // the listed tiles' case bytes, expanded to texels; cubes of the other tiles are empty
  const McArgs a = make_mc_args(s, 0.0f);
  const size_t tiles = tile_count(a);
  std::vector<uint32_t> list;
  std::vector<uint8_t> cases;
  try {
    list.resize(tiles + 1);
  } catch (const std::bad_alloc&) {
    return KF_ERR_OUT_OF_MEMORY;
  }
  KF_CUDA_TRY(s, cudaMemcpyAsync(list.data(), case_tiles(s, a), (tiles + 1) * 4, cudaMemcpyDeviceToHost, s->stream));
  KF_CUDA_TRY(s, cudaStreamSynchronize(s->stream));
  const size_t listed = list[tiles];
  try {
    cases.resize(listed * kTileCubes);
  } catch (const std::bad_alloc&) {
    return KF_ERR_OUT_OF_MEMORY;
  }
  if (listed)
    KF_CUDA_TRY(s, cudaMemcpyAsync(cases.data(), s->d_mc_cases, cases.size(), cudaMemcpyDeviceToHost, s->stream));
  std::memset(base, 0, count * 4);
  KF_CUDA_TRY(s, cudaStreamSynchronize(s->stream));
  for (size_t k = 0; k < listed; ++k) {
    const int x0 = 32 * (int)(list[k] % a.tx), y0 = 8 * (int)(list[k] / a.tx % a.ty), z0 = 8 * (int)(list[k] / ((uint32_t)a.tx * a.ty));
    for (int z = z0; z < std::min(z0 + 8, a.nz); ++z)
      for (int y = y0; y < std::min(y0 + 8, a.ny); ++y) {
        const uint8_t* c = &cases[k * kTileCubes + (size_t)((z - z0) << 8 | (y - y0) << 5)];
        uint32_t* b = base + (size_t)a.nx * ((size_t)y + (size_t)a.ny * z);
        for (int x = x0; x < std::min(x0 + 32, a.nx); ++x)
          b[x] = kf_mc_host::kf_mc_nr_triangles[c[x - x0]] | (uint32_t)c[x - x0] << 16;
      }
  }
  return KF_OK;
}

int kf_mc_export_stl(kf_session* s, const char* path) {
  // exportMesh (mcubes.cpp:429-509): 80-byte header (zeroed here), uint32 triangle count
  // (4x with Q18), then per triangle normal (1,1,1), three vertices, uint16 0
  if (!s || !path) return KF_ERR_INVALID_ARGUMENT;
  if (!s->mc_valid) return KF_ERR_STATE;
  std::vector<float> v;
  int rc = copy_vertices_host(s, v);
  if (rc) return rc;
  FILE* f = std::fopen(path, "wb");
  if (!f) return KF_ERR_IO;
  char hdr[80];
  std::memset(hdr, 0, sizeof(hdr));
  const uint32_t T = s->mc_triangles;
  const uint32_t count = (s->cfg.quirks & KF_Q18_STL_COUNT_X4) ? 4 * T : T;
  bool ok = std::fwrite(hdr, 1, 80, f) == 80 && std::fwrite(&count, 4, 1, f) == 1;
  std::vector<unsigned char> rec((size_t)T * 50);
  const float nrm[3] = {1.0f, 1.0f, 1.0f};
  const uint16_t attr = 0;
  for (uint32_t t = 0; t < T; ++t) {
    unsigned char* r = &rec[(size_t)t * 50];
    std::memcpy(r, nrm, 12);
    for (int k = 0; k < 3; ++k) std::memcpy(r + 12 + 12 * k, &v[((size_t)t * 3 + k) * 4], 12);
    std::memcpy(r + 48, &attr, 2);
  }
  ok = ok && (T == 0 || std::fwrite(rec.data(), 1, rec.size(), f) == rec.size());
  ok = (std::fclose(f) == 0) && ok;
  return ok ? KF_OK : KF_ERR_IO;
}

int kf_mc_extract_mesh(kf_session* s, float iso, uint32_t* n_vertices, uint32_t* n_triangles) {
  if (!s || !n_vertices || !n_triangles) return KF_ERR_INVALID_ARGUMENT;
  return extract_mesh(s, iso, n_vertices, n_triangles);
}

int kf_mc_copy_mesh(kf_session* s, float* positions3, float* normals3, uint32_t* indices3, uint64_t max_vertices,
                    uint64_t max_triangles) {
  if (!s) return KF_ERR_INVALID_ARGUMENT;
  if (!s->mesh_valid) return KF_ERR_STATE;
  const uint64_t nv = s->mesh_vertices, nt = s->mesh_triangles;
  if (max_vertices < nv || max_triangles < nt) return KF_ERR_CAPACITY;
  if ((nv && (!positions3 && !normals3)) || (nt && !indices3 && !positions3 && !normals3)) return KF_ERR_INVALID_ARGUMENT;
  int rc = KF_OK;
  if (nv && positions3) rc = kf_copy_to_host(s, positions3, s->d_mesh_pos, nv * 12);
  if (!rc && nv && normals3) rc = kf_copy_to_host(s, normals3, s->d_mesh_nrm, nv * 12);
  if (!rc && nt && indices3) rc = kf_copy_to_host(s, indices3, s->d_mesh_idx, nt * 12);
  return rc;
}

int kf_mc_export_mesh_ply(kf_session* s, const char* path) {
  // binary little-endian PLY: vertex x y z nx ny nz (float), face list (uchar, uint32)
  if (!s || !path) return KF_ERR_INVALID_ARGUMENT;
  if (!s->mesh_valid) return KF_ERR_STATE;
  std::vector<float> pos, nrm;
  std::vector<uint32_t> idx;
  int rc = copy_mesh_host(s, pos, nrm, idx);
  if (rc) return rc;
  FILE* f = std::fopen(path, "wb");
  if (!f) return KF_ERR_IO;
  const unsigned long long NV = s->mesh_vertices, NT = s->mesh_triangles;
  std::fprintf(f, "ply\nformat binary_little_endian 1.0\nelement vertex %llu\nproperty float x\nproperty float y\n"
               "property float z\nproperty float nx\nproperty float ny\nproperty float nz\nelement face %llu\n"
               "property list uchar uint vertex_indices\nend_header\n", NV, NT);
  std::vector<float> vrec((size_t)NV * 6);
  for (size_t i = 0; i < NV; ++i)
    for (int k = 0; k < 3; ++k) {
      vrec[i * 6 + k] = pos[i * 3 + k];
      vrec[i * 6 + 3 + k] = nrm[i * 3 + k];
    }
  bool ok = NV == 0 || std::fwrite(vrec.data(), 4, vrec.size(), f) == vrec.size();
  std::vector<unsigned char> frec((size_t)NT * 13);
  for (size_t t = 0; t < NT; ++t) {
    frec[t * 13] = 3;
    std::memcpy(&frec[t * 13 + 1], &idx[t * 3], 12);
  }
  ok = ok && (NT == 0 || std::fwrite(frec.data(), 1, frec.size(), f) == frec.size());
  ok = (std::fclose(f) == 0) && ok;
  return ok ? KF_OK : KF_ERR_IO;
}

int kf_mc_export_mesh_stl(kf_session* s, const char* path) {
  // binary STL of the welded mesh: zeroed 80-byte header, the triangle count, per triangle
  // its unit facet normal (from the vertex positions, counter-clockwise), three vertices
  if (!s || !path) return KF_ERR_INVALID_ARGUMENT;
  if (!s->mesh_valid) return KF_ERR_STATE;
  std::vector<float> pos, nrm;
  std::vector<uint32_t> idx;
  int rc = copy_mesh_host(s, pos, nrm, idx);
  if (rc) return rc;
  FILE* f = std::fopen(path, "wb");
  if (!f) return KF_ERR_IO;
  char hdr[80];
  std::memset(hdr, 0, sizeof(hdr));
  const uint32_t T = s->mesh_triangles;
  bool ok = std::fwrite(hdr, 1, 80, f) == 80 && std::fwrite(&T, 4, 1, f) == 1;
  std::vector<unsigned char> rec((size_t)T * 50);
  const uint16_t attr = 0;
  for (uint32_t t = 0; t < T; ++t) {
    const float* p0 = &pos[(size_t)idx[3 * t] * 3];
    const float* p1 = &pos[(size_t)idx[3 * t + 1] * 3];
    const float* p2 = &pos[(size_t)idx[3 * t + 2] * 3];
    const float ux = p1[0] - p0[0], uy = p1[1] - p0[1], uz = p1[2] - p0[2];
    const float vx = p2[0] - p0[0], vy = p2[1] - p0[1], vz = p2[2] - p0[2];
    float nv[3] = {uy * vz - uz * vy, uz * vx - ux * vz, ux * vy - uy * vx};
    const float len = std::sqrt(nv[0] * nv[0] + nv[1] * nv[1] + nv[2] * nv[2]);
    for (float& c : nv) c = len > 0.0f ? c / len : 0.0f;
    unsigned char* r = &rec[(size_t)t * 50];
    std::memcpy(r, nv, 12);
    std::memcpy(r + 12, p0, 12);
    std::memcpy(r + 24, p1, 12);
    std::memcpy(r + 36, p2, 12);
    std::memcpy(r + 48, &attr, 2);
  }
  ok = ok && (T == 0 || std::fwrite(rec.data(), 1, rec.size(), f) == rec.size());
  ok = (std::fclose(f) == 0) && ok;
  return ok ? KF_OK : KF_ERR_IO;
}

int kf_mc_export_ply(kf_session* s, const char* path) {
  // exportPointCloud (mcubes.cpp:391-427): ASCII PLY of the vertex buffer
  if (!s || !path) return KF_ERR_INVALID_ARGUMENT;
  if (!s->mc_valid) return KF_ERR_STATE;
  std::vector<float> v;
  int rc = copy_vertices_host(s, v);
  if (rc) return rc;
  FILE* f = std::fopen(path, "w");
  if (!f) return KF_ERR_IO;
  const unsigned long long n = (unsigned long long)s->mc_triangles * 3;
  std::fprintf(f, "ply\nformat ascii 1.0\nelement vertex %llu\nproperty float x\nproperty float y\n"
               "property float z\nend_header\n", n);
  for (unsigned long long i = 0; i < n; ++i) std::fprintf(f, "%g %g %g\n", v[i * 4], v[i * 4 + 1], v[i * 4 + 2]);
  const bool bad = std::ferror(f);
  return (std::fclose(f) == 0 && !bad) ? KF_OK : KF_ERR_IO;
}

}  // extern "C"
