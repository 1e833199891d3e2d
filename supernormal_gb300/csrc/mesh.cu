// Mesh extraction on the device: SDF lattice query points and marching cubes.
//
// The reference extracts a mesh from the SDF on a res^3 lattice over the
// bounding box (models/renderer.py:9-34, extract_fields + extract_geometry,
// called from exp_runner.py for validation meshes and the Chamfer / F-score
// evaluation) with PyMCubes on the host.  Here the lattice points are formed
// per slab on the device, the field kernels evaluate them, and marching
// cubes runs over the lattice:
//   1. one bit per point (inside: value > threshold), 32 points per word;
//   2. per tile of words: edges that carry a vertex (their ends lie on
//      different sides), per axis, and triangles of the cut cubes; exclusive
//      scans of the tile sums -> totals and first numbers;
//   3. vertices at the linear-interpolation crossing of each such edge,
//      numbered axis by axis in lattice order (shared by the cubes that meet
//      at the edge, so the mesh is indexed and watertight);
//   4. each cube's triangles as vertex numbers.
//
// The triangle table is generated at compile time (make_mc_table) rather than
// transcribed: on every cube face the sign changes are paired so that each
// inside corner is cut off on its own (the same pairing from both cubes that
// share the face, so no cracks), the face segments are oriented from the
// crossing where the face boundary (counter-clockwise around the outward
// normal) enters the inside to the next crossing where it leaves, the
// segments chain into closed loops, and each loop is fanned into triangles
// from a vertex none of whose diagonals lies on a cube face; the right-hand
// normals then point from the inside to the outside.
#include "common.cuh"
#include "scan.cuh"

namespace sn {
namespace {

// Corner c of a cube is (dx, dy, dz) = (c & 1, c >> 1 & 1, c >> 2 & 1).
// Edge e = axis * 4 + the two other corner bits of its lower corner.
constexpr int kMcMaxTri = 5;

struct McTable {
  uint8_t ntri[256];
  int8_t edge[256][3 * kMcMaxTri];
  uint8_t max_tri;
};

constexpr int mc_edge_of(int c0, int axis) {
  return axis == 0 ? ((c0 >> 1) & 3) : axis == 1 ? (4 + ((c0 & 1) | (((c0 >> 2) & 1) << 1))) : (8 + (c0 & 3));
}

// Faces of the cube edge e as a 6-bit mask (bit 2 * axis + side).
constexpr int mc_edge_faces(int e) {
  const int axis = e >> 2, o = e & 3;
  const int x0 = axis == 0 ? 1 : 0, x1 = axis == 2 ? 1 : 2;  // the other two axes, low first
  return (1 << (2 * x0 + (o & 1))) | (1 << (2 * x1 + ((o >> 1) & 1)));
}

constexpr McTable make_mc_table() {
  McTable t{};
  t.max_tri = 0;
  for (int cs = 0; cs < 256; ++cs) {
    int next[12] = {-1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1};
    for (int a = 0; a < 3; ++a) {
      const int b = (a + 1) % 3, c = (a + 2) % 3;  // e_b x e_c = e_a
      for (int s = 0; s < 2; ++s) {
        // corners counter-clockwise around the outward normal (+e_a if s, else -e_a)
        int q[4] = {0, 0, 0, 0};
        const int bc[4][2] = {{0, 0}, {1, 0}, {1, 1}, {0, 1}};
        for (int i = 0; i < 4; ++i) {
          const int k = s ? i : (4 - i) % 4;
          q[i] = (s << a) | (bc[k][0] << b) | (bc[k][1] << c);
        }
        int cross_edge[4] = {0, 0, 0, 0};
        bool cross_entry[4] = {false, false, false, false};
        int nc = 0;
        for (int i = 0; i < 4; ++i) {
          const int p = q[i], r = q[(i + 1) % 4];
          const bool ip = (cs >> p) & 1, ir = (cs >> r) & 1;
          if (ip != ir) {
            const int lo = p < r ? p : r;
            const int axis = (p ^ r) == 1 ? 0 : (p ^ r) == 2 ? 1 : 2;
            cross_edge[nc] = mc_edge_of(lo, axis);
            cross_entry[nc] = ir;   // the boundary walk enters the inside here
            ++nc;
          }
        }
        for (int i = 0; i < nc; ++i) {
          if (!cross_entry[i]) continue;
          for (int j = 1; j < nc; ++j) {
            const int k = (i + j) % nc;
            if (!cross_entry[k]) {
              next[cross_edge[i]] = cross_edge[k];
              break;
            }
          }
        }
      }
    }
    bool seen[12] = {false, false, false, false, false, false, false, false, false, false, false, false};
    int nt = 0;
    for (int e0 = 0; e0 < 12; ++e0) {
      if (next[e0] < 0 || seen[e0]) continue;
      int loop[12] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
      int n = 0;
      for (int e = e0; !seen[e]; e = next[e]) {
        seen[e] = true;
        loop[n++] = e;
      }
      // fan apex: a vertex none of whose diagonals lies on a cube face, so no
      // diagonal can coincide with one of the neighbouring cube's (such a pair
      // would make the edge shared by four triangles); every loop has one
      int ap = 0;
      for (int c = 0; c < n; ++c) {
        bool good = true;
        for (int j = 0; j < n; ++j)
          if (j != c && j != (c + 1) % n && j != (c + n - 1) % n &&
              (mc_edge_faces(loop[c]) & mc_edge_faces(loop[j])) != 0)
            good = false;
        if (good) {
          ap = c;
          break;
        }
      }
      for (int i = 1; i + 1 < n; ++i) {
        t.edge[cs][3 * nt + 0] = (int8_t)loop[ap];
        t.edge[cs][3 * nt + 1] = (int8_t)loop[(ap + i) % n];
        t.edge[cs][3 * nt + 2] = (int8_t)loop[(ap + i + 1) % n];
        ++nt;
      }
    }
    t.ntri[cs] = (uint8_t)nt;
    if (nt > t.max_tri) t.max_tri = (uint8_t)nt;
  }
  return t;
}

constexpr McTable kMcHost = make_mc_table();
static_assert(kMcHost.max_tri <= kMcMaxTri, "marching-cubes table: too many triangles in a case");
static_assert(kMcHost.ntri[0] == 0 && kMcHost.ntri[255] == 0, "marching-cubes table: empty and full cubes");
static_assert(kMcHost.ntri[1] == 1 && kMcHost.ntri[3] == 2 && kMcHost.ntri[15] == 2,
              "marching-cubes table: corner, edge and face cases");
// In global memory: blocks stage it, lanes reading different entries, which a
// constant bank would serve one after the other.
__device__ __align__(16) const McTable kMc = make_mc_table();

struct Lattice {
  int nx, ny, nz;
  int W;            // 32-bit words per row of nz lattice points
  int words;        // nx * ny * W
  float thr;
};

// The passes work on one bit per lattice point (inside: value > threshold),
// 32 consecutive k of a row per word, so the values are read once and every
// later pass reads 1/32 of their bytes: on a 256^3 lattice 2 MB instead of
// twelve gathered reads of 64 MB, with one division pair per word instead of
// per edge.  Words are numbered row-major, so words x bits in order is the
// lattice order and the vertex and triangle numbers come out of popcounts.
// Measured on a 256^3 lattice, counts and outputs with the host's wait between:
// 2.01 ms with one scan entry per edge, 0.105 ms so; the bit pass (64 MB, read
// once) is the largest kernel and the host's round trip the largest part.
struct MeshWork {
  uint32_t* bits;   // words
  int2* edges;      // 3 * words: {id of the word's first vertex, its edge mask}, axis-major
  int32_t* tiles;   // 4 * n_tiles: vertices of axis 0, 1, 2, then triangles
  int n_tiles;
};

constexpr int kMeshThreads = 512;   // words per tile, one per thread
constexpr int kBitWords = 8;        // words per warp and step of the bit pass (loads in flight)

__global__ void __launch_bounds__(256)
mesh_bits_kernel(Lattice L, const float* __restrict__ u, uint32_t* __restrict__ bits) {
  const int lane = threadIdx.x & 31;
  const int warps = (int)((gridDim.x * blockDim.x) >> 5);
  for (int w0 = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * kBitWords; w0 < L.words;
       w0 += warps * kBitWords) {
    int row = w0 / L.W, wi = w0 - row * L.W;
    float v[kBitWords];
#pragma unroll
    for (int i = 0; i < kBitWords; ++i) {
      const int k = 32 * wi + lane;
      // a NaN or a point past the row's end compares false: outside
      v[i] = (w0 + i < L.words && k < L.nz) ? __ldg(u + (int64_t)row * L.nz + k) : __int_as_float(0x7fc00000);
      if (++wi == L.W) {
        wi = 0;
        ++row;
      }
    }
    uint32_t mine = 0;
#pragma unroll
    for (int i = 0; i < kBitWords; ++i) {
      const uint32_t b = __ballot_sync(0xffffffffu, v[i] > L.thr);
      if (lane == i) mine = b;
    }
    if (lane < kBitWords && w0 + lane < L.words) bits[w0 + lane] = mine;
  }
}

// Position of word w and the bits around it.
struct WordView {
  int i, j, k0;          // lattice coordinates of the word's first point
  uint32_t b[4], n[4];   // bits of the rows (dx, dy) = (0,0) (1,0) (0,1) (1,1) at k and at k + 1
  uint32_t valid_z;      // k + 1 < nz
  bool x, y;             // i + 1 < nx, j + 1 < ny
};

__device__ __forceinline__ WordView word_view(const Lattice& L, const uint32_t* __restrict__ bits, int w) {
  WordView v;
  const int row = w / L.W, wi = w - row * L.W;
  v.i = row / L.ny;
  v.j = row - v.i * L.ny;
  v.k0 = 32 * wi;
  v.x = v.i + 1 < L.nx;
  v.y = v.j + 1 < L.ny;
  const int left = L.nz - 1 - v.k0;  // cubes along z from this word's first point on
  v.valid_z = left >= 32 ? 0xffffffffu : (1u << left) - 1u;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const bool in = (!(c & 1) || v.x) && (!(c & 2) || v.y);
    const int q = w + ((c & 1) ? L.ny * L.W : 0) + ((c & 2) ? L.W : 0);
    v.b[c] = in ? bits[q] : 0u;
    v.n[c] = (v.b[c] >> 1) | ((in && wi + 1 < L.W) ? bits[q + 1] << 31 : 0u);
  }
  return v;
}

// Flagged edges of the word's points along each axis.
__device__ __forceinline__ void edge_masks(const WordView& v, uint32_t m[3]) {
  m[0] = v.x ? v.b[0] ^ v.b[1] : 0u;
  m[1] = v.y ? v.b[0] ^ v.b[2] : 0u;
  m[2] = (v.b[0] ^ v.n[0]) & v.valid_z;
}

// Cubes of the word that the surface cuts.
__device__ __forceinline__ uint32_t cut_cubes(const WordView& v) {
  if (!v.x || !v.y) return 0u;
  const uint32_t any = v.b[0] | v.b[1] | v.b[2] | v.b[3] | v.n[0] | v.n[1] | v.n[2] | v.n[3];
  const uint32_t all = v.b[0] & v.b[1] & v.b[2] & v.b[3] & v.n[0] & v.n[1] & v.n[2] & v.n[3];
  return any & ~all & v.valid_z;
}

__device__ __forceinline__ int cube_case(const WordView& v, int k) {
  int cs = 0;
#pragma unroll
  for (int c = 0; c < 4; ++c) cs |= (int)((v.b[c] >> k) & 1u) << c | (int)((v.n[c] >> k) & 1u) << (4 + c);
  return cs;
}

__device__ __forceinline__ void stage_ntri(uint8_t* s_ntri) {
  if (threadIdx.x < 64)
    reinterpret_cast<uint32_t*>(s_ntri)[threadIdx.x] = reinterpret_cast<const uint32_t*>(kMc.ntri)[threadIdx.x];
}

__device__ __forceinline__ int word_triangles(const WordView& v, const uint8_t* s_ntri) {
  int n = 0;
  for (uint32_t m = cut_cubes(v); m; m &= m - 1) n += s_ntri[cube_case(v, __ffs(m) - 1)];
  return n;
}

// Sums over the block's words of the three edge counts (21 bits each: at most
// 512 * 32 per axis) and of the triangles.
__global__ void __launch_bounds__(kMeshThreads)
mesh_count_kernel(Lattice L, const uint32_t* __restrict__ bits, int n_tiles, int32_t* __restrict__ tiles) {
  __shared__ __align__(4) uint8_t s_ntri[256];
  __shared__ int red[kMeshThreads / 32][4];
  stage_ntri(s_ntri);
  __syncthreads();
  int s[4] = {0, 0, 0, 0};
  const int w = blockIdx.x * kMeshThreads + threadIdx.x;
  if (w < L.words) {
    const WordView v = word_view(L, bits, w);
    uint32_t m[3];
    edge_masks(v, m);
#pragma unroll
    for (int a = 0; a < 3; ++a) s[a] = __popc(m[a]);
    s[3] = word_triangles(v, s_ntri);
  }
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    s[a] = __reduce_add_sync(0xffffffffu, s[a]);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][a] = s[a];
  }
  __syncthreads();
  if (threadIdx.x < 4) {
    int t = 0;
    for (int q = 0; q < kMeshThreads / 32; ++q) t += red[q][threadIdx.x];
    tiles[threadIdx.x * n_tiles + blockIdx.x] = t;
  }
}

// Exclusive prefix of one value per thread over the block.
template <typename T>
__device__ __forceinline__ T block_prefix(T v, T* s_warp) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  T incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  T off = 0;
  for (int q = 0; q < warp; ++q) off += s_warp[q];
  return off + incl - v;
}

// Vertex numbers and masks of every word, and the vertices themselves.
__global__ void __launch_bounds__(kMeshThreads)
mesh_vertices_kernel(Lattice L, const float* __restrict__ u, const uint32_t* __restrict__ bits, int n_tiles,
                     const int32_t* __restrict__ tiles, int2* __restrict__ edges, float3 origin, float3 spacing,
                     float* __restrict__ verts, int64_t cap) {
  __shared__ unsigned long long s_warp[kMeshThreads / 32];
  const int w = blockIdx.x * kMeshThreads + threadIdx.x;
  WordView v;
  uint32_t m[3] = {0u, 0u, 0u};
  if (w < L.words) {
    v = word_view(L, bits, w);
    edge_masks(v, m);
  }
  const unsigned long long pre =
      block_prefix((unsigned long long)__popc(m[0]) | (unsigned long long)__popc(m[1]) << 21 |
                       (unsigned long long)__popc(m[2]) << 42,
                   s_warp);
  if (w >= L.words) return;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    int id = tiles[a * n_tiles + blockIdx.x] + (int)((pre >> (21 * a)) & 0x1fffffu);
    edges[(int64_t)a * L.words + w] = make_int2(id, (int)m[a]);
    if (!verts) continue;
    for (uint32_t r = m[a]; r; r &= r - 1, ++id) {
      if (id >= cap) break;
      const int k = v.k0 + __ffs(r) - 1;
      const int64_t p = ((int64_t)v.i * L.ny + v.j) * L.nz + k;
      const int64_t q = p + (a == 0 ? (int64_t)L.ny * L.nz : a == 1 ? (int64_t)L.nz : 1);
      const float u0 = u[p], u1 = u[q];
      const float t = (L.thr - u0) / (u1 - u0);
      float pos[3] = {(float)v.i, (float)v.j, (float)k};
      pos[a] += t;
      verts[3 * (int64_t)id + 0] = fmaf(pos[0], spacing.x, origin.x);
      verts[3 * (int64_t)id + 1] = fmaf(pos[1], spacing.y, origin.y);
      verts[3 * (int64_t)id + 2] = fmaf(pos[2], spacing.z, origin.z);
    }
  }
}

// Each cube's triangles as vertex numbers: the number of an edge's vertex is
// its word's first number plus the edges flagged below it in the word.  A surface
// along z cuts all 32 cubes of a word and most words have none, so the block lists
// its cut cubes first and then takes them a thread each: with a thread walking its
// own word's cubes (three dependent reads a vertex) the longest word was the time,
// 50 us for a 256^3 lattice's 140 k triangles with the tables staged from constant
// memory, 34 us from global memory and only where a tile has cubes, 13 us so.
constexpr int kMeshList = 2048;   // cubes listed at a time
__global__ void __launch_bounds__(kMeshThreads)
mesh_triangles_kernel(Lattice L, const uint32_t* __restrict__ bits, const int32_t* __restrict__ tiles_tri,
                      const int2* __restrict__ edges, int32_t* __restrict__ tris, int64_t cap) {
  __shared__ __align__(4) uint8_t s_ntri[256];
  __shared__ __align__(4) int8_t s_edge[256 * 3 * kMcMaxTri];
  __shared__ unsigned long long s_warp[kMeshThreads / 32];
  __shared__ uint2 s_cube[kMeshList];   // {word | cube << 9 | case << 14, first triangle}
  __shared__ int s_total;
  static_assert(kMeshThreads <= 512, "nine bits for the word");
  stage_ntri(s_ntri);
  __syncthreads();
  const int w0 = blockIdx.x * kMeshThreads;
  WordView v;
  uint32_t cut = 0u;
  int n = 0;
  if (w0 + (int)threadIdx.x < L.words) {
    v = word_view(L, bits, w0 + threadIdx.x);
    cut = cut_cubes(v);
    n = word_triangles(v, s_ntri);
  }
  if (!__syncthreads_or(n)) return;   // most tiles: nothing to stage the edges for
  for (int e = threadIdx.x; e < 256 * 3 * kMcMaxTri / 4; e += blockDim.x)
    reinterpret_cast<uint32_t*>(s_edge)[e] = reinterpret_cast<const uint32_t*>(&kMc.edge[0][0])[e];
  const unsigned long long pre =
      block_prefix((unsigned long long)__popc(cut) | (unsigned long long)n << 32, s_warp);
  const int first = (int)(pre & 0xffffffffu);   // of this word's cubes among the block's
  if (threadIdx.x == kMeshThreads - 1) s_total = first + __popc(cut);
  const int64_t id0 = tiles_tri[blockIdx.x];
  for (int base = 0;; base += kMeshList) {
    int at = first - base, tri = (int)(pre >> 32);
    if (at < kMeshList && at + __popc(cut) > 0) {
      for (uint32_t r = cut; r; r &= r - 1, ++at) {
        const int b = __ffs(r) - 1, cs = cube_case(v, b);
        if (at >= 0 && at < kMeshList) s_cube[at] = make_uint2(threadIdx.x | b << 9 | cs << 14, tri);
        tri += s_ntri[cs];
      }
    }
    __syncthreads();   // (the first time: the edges and the total too)
    const int listed = min(kMeshList, s_total - base);
    for (int q = threadIdx.x; q < listed; q += kMeshThreads) {
      const uint2 cube = s_cube[q];
      const int w = w0 + (int)(cube.x & 511u), b = (int)(cube.x >> 9) & 31, cs = (int)(cube.x >> 14);
      int64_t id = id0 + cube.y;
      for (int t = 0; t < s_ntri[cs] && id < cap; ++t, ++id) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const int e = s_edge[cs * 3 * kMcMaxTri + 3 * t + c];
          const int axis = e >> 2, b0 = e & 1, b1 = (e >> 1) & 1;  // the two other corner bits, low axis first
          const int di = axis == 0 ? 0 : b0, dj = axis == 1 ? 0 : (axis == 0 ? b0 : b1), dk = axis == 2 ? 0 : b1;
          const int kb = b + dk;  // 32: the first point of the row's next word
          const int at_w = w + (di ? L.ny * L.W : 0) + (dj ? L.W : 0) + (kb >> 5);
          const int2 ev = edges[(int64_t)axis * L.words + at_w];
          tris[3 * id + c] = ev.x + __popc((uint32_t)ev.y & ((1u << (kb & 31)) - 1u));
        }
      }
    }
    if (base + kMeshList >= s_total) break;
    __syncthreads();   // the list is read
  }
}

// Points of a slab of lattice rows: row r is the points along the inner axis at
// (a0 + r / nb, r % nb) of the two outer ones, XFAST: inner x, outer (y, z); else
// inner z, outer (x, y).  The coordinates are formed in double and rounded once, per
// axis instead of per point, and FP64 is slow here: the inner axis is staged in
// shared memory, and a warp takes four rows at a time, whose eight outer coordinates
// are one double expression of eight lanes (with every thread forming its row's two,
// a slab of 2 M points took 27 us; now 12 us, 2 TB/s).
// x fastest: neighbouring x hit neighbouring table entries at every level (the hash
// keeps the low bits of x), so a warp that walks along x touches half the lines of
// one that walks along z.  Few long rows are cut along the inner axis over grid.y
// until the chip is full (2 x 2 rows of 100,000 points, field and all: 3,417 -> 151 us).
constexpr int kLatticeInner = 1024;  // inner coordinates staged at a time
constexpr int kLatticeRows = 4;      // rows a warp takes at a time
// Rows of at most kLatticeShort points: a lane forms the outer coordinates of one, and the
// warp writes its 32 rows as one run (extract_fields of 3000 x 3000 x 2 with a cheap
// query, four rows a warp 772 us, now 290).
constexpr int kLatticeShort = 32;
template <bool XFAST, bool SHORT>
__global__ void __launch_bounds__(256)
lattice_points_kernel(int64_t a0, int64_t n_rows, int n_inner, int nb, double3 lo, double3 step, float* __restrict__ x) {
  __shared__ float s_in[kLatticeInner];
  const double lo_in = XFAST ? lo.x : lo.z, step_in = XFAST ? step.x : step.z;
  const double lo_a = XFAST ? lo.y : lo.x, step_a = XFAST ? step.y : step.x;
  const double lo_b = XFAST ? lo.z : lo.y, step_b = XFAST ? step.z : step.y;
  const int lane = threadIdx.x & 31;
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5, warps = gridDim.x * (int64_t)blockDim.x >> 5;
  for (int64_t i0 = blockIdx.y * (int64_t)kLatticeInner; i0 < n_inner; i0 += (int64_t)gridDim.y * kLatticeInner) {
    const int ni = (int)min((int64_t)kLatticeInner, n_inner - i0);
    __syncthreads();
    for (int i = threadIdx.x; i < ni; i += blockDim.x) s_in[i] = (float)(lo_in + step_in * (double)(i0 + i));
    __syncthreads();
    if constexpr (SHORT) {   // (one piece: ni is n_inner)
      const int w = 3 * ni;
      const uint32_t inv_w = (1u << 20) / w + 1;   // e / w = e * inv_w >> 20 for e < 32 w: e w < 2^20
      for (int64_t r0 = warp * 32; r0 < n_rows; r0 += warps * 32) {
        const int64_t mine = min(r0 + lane, n_rows - 1), ia = mine / nb, ib = mine - ia * nb;
        const float oa = (float)(lo_a + step_a * (double)(a0 + ia)), ob = (float)(lo_b + step_b * (double)ib);
        const int total = (int)min((int64_t)32, n_rows - r0) * w;
        float* run = x + r0 * w;
        for (int e0 = 0; e0 < total; e0 += 32) {
          const int e = e0 + lane, q = min((int)((uint32_t)e * inv_w >> 20), 31), f = e - q * w, i = f / 3, d = f - 3 * i;
          const float pa = __shfl_sync(0xffffffffu, oa, q), pb = __shfl_sync(0xffffffffu, ob, q);
          if (e < total) run[e] = d == (XFAST ? 0 : 2) ? s_in[i] : d == (XFAST ? 1 : 0) ? pa : pb;
        }
      }
      continue;
    }
    for (int64_t r0 = warp * kLatticeRows; r0 < n_rows; r0 += warps * kLatticeRows) {
      // lanes 0..3: the first outer coordinate of their row, lanes 4..7 the second
      const int64_t mine = r0 + (lane & (kLatticeRows - 1));
      const bool second = lane & kLatticeRows;
      const double at = second ? (double)(mine % nb) : (double)(a0 + mine / nb);
      const float outer = (float)((second ? lo_b : lo_a) + (second ? step_b : step_a) * at);
#pragma unroll
      for (int q = 0; q < kLatticeRows; ++q) {
        const float pa = __shfl_sync(0xffffffffu, outer, q), pb = __shfl_sync(0xffffffffu, outer, kLatticeRows + q);
        if (r0 + q >= n_rows) break;
        float* row = x + 3 * ((r0 + q) * n_inner + i0);
        for (int f = lane; f < 3 * ni; f += 32) {
          const int i = f / 3, d = f - 3 * i;
          row[f] = d == (XFAST ? 0 : 2) ? s_in[i] : d == (XFAST ? 1 : 0) ? pa : pb;
        }
      }
    }
  }
}

template <bool XFAST>
void launch_lattice_points(int64_t a0, int64_t n_rows, int n_inner, int nb, double3 lo, double3 step, float* x,
                           cudaStream_t st) {
  if (n_inner <= kLatticeShort) {
    lattice_points_kernel<XFAST, true><<<stride_grid(n_rows, 256, 8), 256, 0, st>>>(a0, n_rows, n_inner, nb, lo, step, x);
    return;
  }
  const unsigned most = 8u * (unsigned)num_sms(), blocks = stride_grid(n_rows, 8 * kLatticeRows, 8);
  const unsigned chunks = (unsigned)((n_inner + (int64_t)kLatticeInner - 1) / kLatticeInner), y = most / blocks;
  lattice_points_kernel<XFAST, false><<<dim3(blocks, y < 1 ? 1 : y < chunks ? y : chunks), 256, 0, st>>>(
      a0, n_rows, n_inner, nb, lo, step, x);
}

// u[i, j, k] = sign * in[j - j0, k, i]: 32 x 32 tiles through shared memory (all of a
// row's in grid.x: the other two axes of a grid end at 65,535).
__global__ void __launch_bounds__(256)
lattice_store_kernel(int64_t j0, int nx, int ny, int nz, float sign, const float* __restrict__ in,
                     float* __restrict__ u) {
  __shared__ float tile[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int tiles_x = (nx + 31) / 32;
  const int ib = (int)(blockIdx.x % tiles_x) * 32, kb = (int)(blockIdx.x / tiles_x) * 32;
  const int64_t j = blockIdx.y;
#pragma unroll
  for (int r = ty; r < 32; r += 8)
    if (kb + r < nz && ib + tx < nx) tile[r][tx] = in[(j * nz + kb + r) * nx + ib + tx];
  __syncthreads();
#pragma unroll
  for (int r = ty; r < 32; r += 8)
    if (ib + r < nx && kb + tx < nz) u[((int64_t)(ib + r) * ny + j0 + j) * nz + kb + tx] = sign * tile[tx][r];
}

__global__ void negate_kernel(int64_t n, const float* __restrict__ in, float* __restrict__ out) {
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x)
    out[p] = -in[p];
}

// Layout of the workspace of a lattice.
MeshWork mesh_work(const Lattice& L, void* ws) {
  MeshWork m;
  m.n_tiles = (L.words + kMeshThreads - 1) / kMeshThreads;
  m.edges = reinterpret_cast<int2*>((reinterpret_cast<uintptr_t>(ws) + 7) & ~(uintptr_t)7);
  m.bits = reinterpret_cast<uint32_t*>(m.edges + 3 * (int64_t)L.words);
  m.tiles = reinterpret_cast<int32_t*>(m.bits + L.words);
  return m;
}

int mesh_lattice(Lattice& L, const float* values, int nx, int ny, int nz, float threshold, const void* ws) {
  SN_REQUIRE(nx >= 2 && ny >= 2 && nz >= 2, "marching_cubes: resolution must be >= 2 per axis");
  const int64_t n = (int64_t)nx * ny * nz;
  SN_REQUIRE(3 * n < ((int64_t)1 << 31), "marching_cubes: %lld lattice edges exceed int32 ids", (long long)(3 * n));
  SN_REQUIRE(values && ws, "marching_cubes: null buffer");
  L.nx = nx;
  L.ny = ny;
  L.nz = nz;
  L.W = (nz + 31) / 32;
  L.words = nx * ny * L.W;   // at most n / 2 < 2^30
  L.thr = threshold;
  return SN_OK;
}

int mesh_count(const Lattice& L, const float* values, int32_t* counts, void* ws, cudaStream_t st) {
  const MeshWork m = mesh_work(L, ws);
  const int64_t steps = ((int64_t)L.words + kBitWords - 1) / kBitWords;
  mesh_bits_kernel<<<stride_grid(steps * 32, 256, 8), 256, 0, st>>>(L, values, m.bits);
  mesh_count_kernel<<<m.n_tiles, kMeshThreads, 0, st>>>(L, m.bits, m.n_tiles, m.tiles);
  scan_tile_offsets<<<1, kScanThreads, 0, st>>>(m.tiles, 3 * (int64_t)m.n_tiles, counts);
  scan_tile_offsets<<<1, kScanThreads, 0, st>>>(m.tiles + 3 * (int64_t)m.n_tiles, m.n_tiles, counts + 1);
  return check_launch("marching_cubes", 4);
}

int mesh_emit(const Lattice& L, const float* values, const double* lo, const double* hi, int64_t vert_cap,
              int64_t tri_cap, float* vertices, int32_t* triangles, void* ws, cudaStream_t st) {
  const MeshWork m = mesh_work(L, ws);
  const float3 origin = make_float3((float)lo[0], (float)lo[1], (float)lo[2]);
  const float3 spacing = make_float3((float)((hi[0] - lo[0]) / (L.nx - 1)), (float)((hi[1] - lo[1]) / (L.ny - 1)),
                                     (float)((hi[2] - lo[2]) / (L.nz - 1)));
  mesh_vertices_kernel<<<m.n_tiles, kMeshThreads, 0, st>>>(L, values, m.bits, m.n_tiles, m.tiles, m.edges, origin,
                                                           spacing, vert_cap > 0 ? vertices : nullptr, vert_cap);
  if (tri_cap == 0) return check_launch("marching_cubes");
  mesh_triangles_kernel<<<m.n_tiles, kMeshThreads, 0, st>>>(L, m.bits, m.tiles + 3 * (int64_t)m.n_tiles, m.edges,
                                                            triangles, tri_cap);
  return check_launch("marching_cubes", 2);
}

}  // namespace
}  // namespace sn

using namespace sn;

extern "C" {

int sn_lattice_points(int64_t i0, int64_t n_i, int nx, int ny, int nz, const double* bound_min,
                      const double* bound_max, float* x_out, void* stream) {
  SN_REQUIRE(nx >= 2 && ny >= 2 && nz >= 2, "lattice_points: resolution must be >= 2 per axis");
  SN_REQUIRE(i0 >= 0 && n_i >= 0 && i0 + n_i <= nx, "lattice_points: slab [%lld, %lld) outside [0, %d)",
             (long long)i0, (long long)(i0 + n_i), nx);
  SN_REQUIRE(bound_min && bound_max && (n_i == 0 || x_out), "lattice_points: null buffer");
  if (n_i == 0) return SN_OK;
  const double3 lo = make_double3(bound_min[0], bound_min[1], bound_min[2]);
  const double3 st = make_double3((bound_max[0] - bound_min[0]) / (nx - 1), (bound_max[1] - bound_min[1]) / (ny - 1),
                                  (bound_max[2] - bound_min[2]) / (nz - 1));
  launch_lattice_points<false>(i0, n_i * ny, nz, ny, lo, st, x_out, as_stream(stream));
  return check_launch("lattice_points");
}

static int lattice_slab(int64_t first, int64_t count, int nx, int ny, int nz, int along) {
  SN_REQUIRE(nx >= 2 && ny >= 2 && nz >= 2, "lattice: resolution must be >= 2 per axis");
  SN_REQUIRE(first >= 0 && count >= 0 && first + count <= along, "lattice: slab [%lld, %lld) outside [0, %d)",
             (long long)first, (long long)(first + count), along);
  return SN_OK;
}

int sn_lattice_points_x(int64_t j0, int64_t n_j, int nx, int ny, int nz, const double* bound_min,
                        const double* bound_max, float* x_out, void* stream) {
  SN_TRY(lattice_slab(j0, n_j, nx, ny, nz, ny));
  SN_REQUIRE(bound_min && bound_max && (n_j == 0 || x_out), "lattice_points_x: null buffer");
  if (n_j == 0) return SN_OK;
  const double3 lo = make_double3(bound_min[0], bound_min[1], bound_min[2]);
  const double3 st = make_double3((bound_max[0] - bound_min[0]) / (nx - 1), (bound_max[1] - bound_min[1]) / (ny - 1),
                                  (bound_max[2] - bound_min[2]) / (nz - 1));
  launch_lattice_points<true>(j0, n_j * nz, nx, nz, lo, st, x_out, as_stream(stream));
  return check_launch("lattice_points_x");
}

int sn_lattice_store(int64_t j0, int64_t n_j, int nx, int ny, int nz, int negate, const float* values, float* u,
                     void* stream) {
  SN_TRY(lattice_slab(j0, n_j, nx, ny, nz, ny));
  SN_REQUIRE(n_j == 0 || (values && u), "lattice_store: null buffer");
  const int64_t tiles = (int64_t)((nx + 31) / 32) * ((nz + 31) / 32);
  SN_REQUIRE(tiles < (int64_t)1 << 31, "lattice_store: rows of %d x %d points", nx, nz);
  for (int64_t a = 0; a < n_j; a += 65535) {  // grid.y limit
    const int64_t m = n_j - a < 65535 ? n_j - a : 65535;
    lattice_store_kernel<<<dim3((unsigned)tiles, (unsigned)m), 256, 0, as_stream(stream)>>>(
        j0 + a, nx, ny, nz, negate ? -1.0f : 1.0f, values + a * nz * nx, u);
    SN_TRY(check_launch("lattice_store"));
  }
  return SN_OK;
}

int sn_negate(int64_t n, const float* in, float* out, void* stream) {
  SN_REQUIRE(n >= 0 && (n == 0 || (in && out)), "negate: bad arguments");
  if (n == 0) return SN_OK;
  negate_kernel<<<stride_grid(n, 256, 8), 256, 0, as_stream(stream)>>>(n, in, out);
  return check_launch("negate");
}

size_t sn_marching_cubes_workspace_bytes(int nx, int ny, int nz) {
  if (nx < 2 || ny < 2 || nz < 2) return 0;
  const int64_t words = (int64_t)nx * ny * ((nz + 31) / 32);
  const int64_t tiles = (words + kMeshThreads - 1) / kMeshThreads;
  const size_t b = (size_t)words * (3 * sizeof(int2) + sizeof(uint32_t)) + (size_t)(4 * tiles) * sizeof(int32_t) + 8;
  return (b + 255) & ~(size_t)255;
}

int sn_marching_cubes_count(const float* values, int nx, int ny, int nz, float threshold, int32_t* counts,
                            void* workspace, void* stream) {
  Lattice L;
  SN_TRY(mesh_lattice(L, values, nx, ny, nz, threshold, workspace));
  SN_REQUIRE(counts != nullptr, "marching_cubes_count: counts is null");
  return mesh_count(L, values, counts, workspace, as_stream(stream));
}

int sn_marching_cubes_emit(const float* values, int nx, int ny, int nz, float threshold, const double* bound_min,
                           const double* bound_max, int64_t vert_cap, int64_t tri_cap, float* vertices,
                           int32_t* triangles, void* workspace, void* stream) {
  Lattice L;
  SN_TRY(mesh_lattice(L, values, nx, ny, nz, threshold, workspace));
  SN_REQUIRE(bound_min && bound_max, "marching_cubes_emit: null bounds");
  SN_REQUIRE(vert_cap >= 0 && tri_cap >= 0 && (vert_cap == 0 || vertices) && (tri_cap == 0 || triangles),
             "marching_cubes: output capacity without a buffer");
  return mesh_emit(L, values, bound_min, bound_max, vert_cap, tri_cap, vertices, triangles, workspace,
                   as_stream(stream));
}

int sn_marching_cubes(const float* values, int nx, int ny, int nz, float threshold, const double* bound_min,
                      const double* bound_max, int64_t vert_cap, int64_t tri_cap, float* vertices,
                      int32_t* triangles, int32_t* counts, void* workspace, void* stream) {
  Lattice L;
  SN_TRY(mesh_lattice(L, values, nx, ny, nz, threshold, workspace));
  SN_REQUIRE(counts && bound_min && bound_max, "marching_cubes: null buffer");
  SN_REQUIRE(vert_cap >= 0 && tri_cap >= 0 && (vert_cap == 0 || vertices) && (tri_cap == 0 || triangles),
             "marching_cubes: output capacity without a buffer");
  SN_TRY(mesh_count(L, values, counts, workspace, as_stream(stream)));
  if (vert_cap == 0 && tri_cap == 0) return SN_OK;
  return mesh_emit(L, values, bound_min, bound_max, vert_cap, tri_cap, vertices, triangles, workspace,
                   as_stream(stream));
}

}  // extern "C"
