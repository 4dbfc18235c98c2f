// Integer half of the path: voxel hash table, 27-tap neighbour maps, the reference's row order and
// per-block tap lists, 2x subdivision maps, row gather and the up-block skip add.
//
// Results are defined by the reference (src/spconv.cu:13-75, src/sdec.cu:21-57 of trellis2-cuda) and are
// bit-exact with it; the layout of the work is not.  The pool-backed builders hash 2x2x2 BRICKS of voxels
// (8 probes per row instead of 27, k_brick_*); the allocation-free builder keeps the per-voxel table with one
// 16-byte {key, row} slot per probe and one thread per (row, tap) entry (k_hash_insert / k_neighbors).
// Nothing is built on the host.
#include "common.cuh"
#include <cub/cub.cuh>

namespace {

struct __align__(16) Slot { unsigned long long key; uint32_t val; uint32_t pad; };
static constexpr unsigned long long KEY_EMPTY = ~0ull;

__device__ __forceinline__ uint32_t mix32(unsigned long long k) {   // src/spconv.cu:13
  k ^= k >> 33; k *= 0xff51afd7ed558ccdull; k ^= k >> 33; return (uint32_t)k;
}
__device__ __forceinline__ unsigned long long pack_key(int b, int x, int y, int z, int W, int H, int D) {  // src/spconv.cu:16
  return (((unsigned long long)b * W + x) * H + y) * D + z;
}

__global__ void k_hash_insert(const int4* __restrict__ coords, int n, int W, int H, int D, Slot* table, uint32_t mask) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int4 q = coords[i];
  unsigned long long k = pack_key(q.x, q.y, q.z, q.w, W, H, D);
  // at most `mask + 1` probes: the table holds >= 2n slots, so this bound is never reached on valid input
  for (uint32_t s = mix32(k) & mask, it = 0; it <= mask; s = (s + 1) & mask, ++it) {
    unsigned long long prev = atomicCAS(&table[s].key, KEY_EMPTY, k);
    if (prev == KEY_EMPTY || prev == k) { atomicMin(&table[s].val, (uint32_t)i); return; }  // duplicates: lowest row wins
  }
}

constexpr int NB_ROWS = 32;                 // rows per CTA of the neighbour kernel
constexpr int NB_THREADS = 288;             // 32 rows * 27 taps = 864 entries = 3 per thread
__global__ void __launch_bounds__(NB_THREADS) k_neighbors(const int4* __restrict__ coords, int n, int W, int H, int D,
                                                          const Slot* __restrict__ table, uint32_t mask,
                                                          uint32_t* __restrict__ nbr, int* __restrict__ gray, int* __restrict__ bin) {
  __shared__ uint32_t s_mask[NB_ROWS];
  i64 row0 = (i64)blockIdx.x * NB_ROWS;
  if (threadIdx.x < NB_ROWS) s_mask[threadIdx.x] = 0;
  __syncthreads();
  int rows = (int)min((i64)NB_ROWS, (i64)n - row0);
#pragma unroll
  for (int e = threadIdx.x; e < NB_ROWS * 27; e += NB_THREADS) {
    int lr = e / 27, v = e - lr * 27;
    if (lr >= rows) break;
    int4 q = coords[row0 + lr];
    int x = q.y + v / 9 - 1, y = q.z + (v / 3) % 3 - 1, z = q.w + v % 3 - 1;   // src/spconv.cu:27
    uint32_t r = NBR_EMPTY;
    if (x >= 0 && x < W && y >= 0 && y < H && z >= 0 && z < D) {
      unsigned long long k = pack_key(q.x, x, y, z, W, H, D);
      for (uint32_t s = mix32(k) & mask, it = 0; it <= mask; s = (s + 1) & mask, ++it) {
        uint4 raw = __ldg(reinterpret_cast<const uint4*>(table + s));
        unsigned long long sk = ((unsigned long long)raw.y << 32) | raw.x;
        if (sk == KEY_EMPTY) break;
        if (sk == k) { r = raw.z; break; }
      }
    }
    nbr[(row0 + lr) * 27 + v] = r;
    if (r != NBR_EMPTY) atomicOr(&s_mask[lr], 1u << v);
  }
  __syncthreads();
  if (threadIdx.x < rows) {
    uint32_t g = s_mask[threadIdx.x], b = g;
#pragma unroll
    for (int v = 1; v < 27; v++) b ^= g >> v;       // gray -> binary, src/spconv.cu:34
    gray[row0 + threadIdx.x] = (int)g;
    if (bin) bin[row0 + threadIdx.x] = (int)b;
  }
}

// ---- brick table: one slot per occupied 2x2x2 block of voxels, holding the 8 row indices of its cells.
// The 27 neighbours of a voxel always lie in exactly 8 bricks (2 per axis), so a row costs 8 key probes and 8
// 32-byte value reads instead of 27 probes; the value reads of one row are shared by up to 8 taps each.
struct __align__(16) BrickVals { uint32_t v[8]; };

__device__ __forceinline__ unsigned long long brick_key(int b, int bx, int by, int bz, int Wb, int Hb, int Db) {
  return (((unsigned long long)b * Wb + bx) * Hb + by) * Db + bz;
}

__global__ void k_brick_insert(const int4* __restrict__ coords, int n, int Wb, int Hb, int Db, unsigned long long* keys,
                               BrickVals* vals, uint32_t mask) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int4 q = coords[i];
  unsigned long long k = brick_key(q.x, q.y >> 1, q.z >> 1, q.w >> 1, Wb, Hb, Db);
  int sub = (q.y & 1) | ((q.z & 1) << 1) | ((q.w & 1) << 2);
  for (uint32_t s = mix32(k) & mask, it = 0; it <= mask; s = (s + 1) & mask, ++it) {
    unsigned long long prev = atomicCAS(&keys[s], KEY_EMPTY, k);
    if (prev == KEY_EMPTY || prev == k) { atomicMin(&vals[s].v[sub], (uint32_t)i); return; }   // duplicates: lowest row wins
  }
}

// Where a voxel's 8 bricks come from: the hash table.
struct HashBricks {
  const int4* coords; int W, H, D, Wb, Hb, Db; const unsigned long long* keys; const BrickVals* vals; uint32_t mask;
  // parity of the voxel in its brick, and the 8 rows of brick t = (sx, sy, sz) of its 2x2x2 neighbourhood of bricks: along one
  // axis the offsets -1, 0, +1 fall into brick lo = (c-1)>>1 or hi = lo + 1: odd c -> {lo, lo, hi}, even c -> {lo, hi, hi}
  __device__ __forceinline__ int load(i64 row, int t, uint32_t* v) const {
    const int4 q = __ldg(coords + row);
    const int bx = ((q.y - 1) >> 1) + (t & 1), by = ((q.z - 1) >> 1) + ((t >> 1) & 1), bz = ((q.w - 1) >> 1) + (t >> 2);
    if (bx >= 0 && by >= 0 && bz >= 0 && bx < Wb && by < Hb && bz < Db) {
      const unsigned long long k = brick_key(q.x, bx, by, bz, Wb, Hb, Db);
      for (uint32_t s = mix32(k) & mask, it = 0; it <= mask; s = (s + 1) & mask, ++it) {
        const unsigned long long sk = __ldg(keys + s);
        if (sk == KEY_EMPTY) break;
        if (sk == k) {
          const uint4 a = __ldg(reinterpret_cast<const uint4*>(vals + s)), b = __ldg(reinterpret_cast<const uint4*>(vals + s) + 1);
          v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
          break;
        }
      }
      // a neighbour outside the grid is absent (src/spconv.cu:28): with an odd extent the last brick reaches one cell past it
      if (2 * bx + 1 >= W) v[1] = v[3] = v[5] = v[7] = NBR_EMPTY;
      if (2 * by + 1 >= H) v[2] = v[3] = v[6] = v[7] = NBR_EMPTY;
      if (2 * bz + 1 >= D) v[4] = v[5] = v[6] = v[7] = NBR_EMPTY;
    }
    return (q.y & 1) | ((q.z & 1) << 1) | ((q.w & 1) << 2);
  }
};

// The map of a subdivided level: one warp per four parents, lane = tap.  A lane holds info[q] = {row of the first child, 8-bit set of
// children} of a parent's neighbour in its tap's direction, loaded once for all of the parent's children (which lie in slot order one
// behind the other); the neighbour of child s in direction v is child (s + v) & 1 of the parent's neighbour (s + v) >> 1 along
// each axis, so its row is a shuffle and a popcount away.  Three loads depend on one another here, which with one parent per
// warp was the whole time (269 us for 3,288,465 children, as much as 8 threads per child that each look a brick up); four
// parents' loads are in flight together (218 us).
constexpr int CHILD_PARENTS = 4;
__global__ void __launch_bounds__(256) k_child_neighbors(const uint32_t* __restrict__ pnbr, const uint2* __restrict__ info, int n,
                                                         uint32_t* __restrict__ nbr, int* __restrict__ gray) {
  const int p0 = (int)((blockIdx.x * 256ll + threadIdx.x) >> 5) * CHILD_PARENTS, lane = threadIdx.x & 31;
  uint32_t q[CHILD_PARENTS];
  uint2 own[CHILD_PARENTS], f[CHILD_PARENTS];
#pragma unroll
  for (int k = 0; k < CHILD_PARENTS; k++) {
    own[k] = p0 + k < n ? __ldg(info + p0 + k) : make_uint2(0u, 0u);
    q[k] = p0 + k < n && lane < 27 ? __ldg(pnbr + (i64)(p0 + k) * 27 + lane) : NBR_EMPTY;
  }
#pragma unroll
  for (int k = 0; k < CHILD_PARENTS; k++) f[k] = q[k] != NBR_EMPTY ? __ldg(info + q[k]) : make_uint2(0u, 0u);
  // per axis and slot bit b: with d = tap offset + 1 (0..2), b + d + 1 is twice the neighbour's offset + 1, plus its slot bit; parent tap in
  // the low byte, slot above
  const int v = lane < 27 ? lane : 26, d[3] = {v / 9, (v / 3) % 3, v % 3}, mul[3] = {9, 3, 1};
  int to[3][2];
#pragma unroll
  for (int a = 0; a < 3; a++)
#pragma unroll
    for (int b = 0; b < 2; b++) to[a][b] = ((b + d[a] + 1) >> 1) * mul[a] | ((b + d[a] + 1) & 1) << (8 + a);
#pragma unroll
  for (int k = 0; k < CHILD_PARENTS; k++) {
    uint32_t row = own[k].x;
    for (uint32_t kids = own[k].y; kids; kids &= kids - 1, row++) {
      const int s = __ffs(kids) - 1;
      const int at = (s & 1 ? to[0][1] : to[0][0]) + (s & 2 ? to[1][1] : to[1][0]) + (s & 4 ? to[2][1] : to[2][0]);
      const uint32_t first = __shfl_sync(0xffffffffu, f[k].x, at & 31), set = __shfl_sync(0xffffffffu, f[k].y, at & 31);
      const int slot = at >> 8;
      const uint32_t r = set >> slot & 1 ? first + __popc(set & ((1u << slot) - 1)) : NBR_EMPTY;
      if (lane < 27) nbr[(i64)row * 27 + lane] = r;
      const uint32_t m = __ballot_sync(0xffffffffu, lane < 27 && r != NBR_EMPTY);
      if (lane == 0) gray[row] = (int)m;
    }
  }
}

// 8 threads per row fetch the rows of its 8 bricks (64 cells) into shared memory; then a warp writes four rows of the map, lane = tap:
// 27 consecutive words per store, and the presence mask is the ballot.  Bound by instruction issue, so the work per entry is
// what was cut: the fetching threads used to pick their taps out of the 8 cells and store them one by one (1,000,003 rows:
// 130 -> 107 us; with the CTA's rows gathered in shared memory and stored in 16-byte pieces: 125).
__global__ void __launch_bounds__(256) k_brick_neighbors(const HashBricks bricks, int n, uint32_t* __restrict__ nbr, int* __restrict__ gray,
                                                         int* __restrict__ bin, int* __restrict__ iota) {
  __shared__ __align__(16) uint32_t s_cell[32][64];
  __shared__ int s_par[32];
  const i64 row0 = (i64)blockIdx.x * 32;
  {
    const int lr = threadIdx.x >> 3, t = threadIdx.x & 7;
    const i64 row = row0 + lr;
    if (row < n) {
      uint32_t v[8];
#pragma unroll
      for (int e = 0; e < 8; e++) v[e] = NBR_EMPTY;
      const int par = bricks.load(row, t, v);
      *(uint4*)&s_cell[lr][t * 8] = make_uint4(v[0], v[1], v[2], v[3]);
      *(uint4*)&s_cell[lr][t * 8 + 4] = make_uint4(v[4], v[5], v[6], v[7]);
      if (t == 0) s_par[lr] = par;
    }
  }
  __syncwarp();               // a warp finishes the four rows that it has fetched
  const int lane = threadIdx.x & 31, lr0 = (threadIdx.x >> 5) * 4;
  // Tap v = (dx + 1) * 9 + (dy + 1) * 3 + (dz + 1) (src/spconv.cu:27).  Along an axis the 4 cells of the two bricks are numbered
  // 0..3; offset d of an even coordinate is cell d + 2, of an odd one d + 1.  A cell's place: brick bits in 3..5, cell bits in 0..2.
  const int v = lane < 27 ? lane : 26, dx = v / 9, dy = (v / 3) % 3, dz = v % 3;
  auto place = [](int c) { return (c >> 1) * 8 + (c & 1); };
  const int x0 = place(dx + 1), x1 = place(dx), y0 = place(dy + 1) * 2, y1 = place(dy) * 2, z0 = place(dz + 1) * 4, z1 = place(dz) * 4;
  uint32_t g = 0;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const i64 row = row0 + lr0 + i;
    if (row >= n) break;
    const int par = s_par[lr0 + i];
    const uint32_t r = s_cell[lr0 + i][(par & 1 ? x1 : x0) + (par & 2 ? y1 : y0) + (par & 4 ? z1 : z0)];
    if (lane < 27) nbr[row * 27 + lane] = r;
    const uint32_t m = __ballot_sync(0xffffffffu, lane < 27 && r != NBR_EMPTY);
    if (lane == i) g = m;
  }
  const i64 row = row0 + lr0 + lane;
  if (lane < 4 && row < n) {
    uint32_t b = g;                                 // gray -> binary (src/spconv.cu:34): XOR of all right shifts, as a prefix scan
    b ^= b >> 16; b ^= b >> 8; b ^= b >> 4; b ^= b >> 2; b ^= b >> 1;
    gray[row] = (int)g;
    if (bin) { bin[row] = (int)b; iota[row] = (int)row; }
  }
}

// one thread per query coordinate: the row of the voxel that sits there, or NBR_EMPTY
__global__ void k_brick_lookup(const int4* __restrict__ queries, i64 m, int W, int H, int D, int Wb, int Hb, int Db,
                               const unsigned long long* __restrict__ keys, const BrickVals* __restrict__ vals, uint32_t mask,
                               uint32_t* __restrict__ rows) {
  const i64 i = blockIdx.x * (i64)blockDim.x + threadIdx.x;
  if (i >= m) return;
  const int4 q = queries[i];
  uint32_t r = NBR_EMPTY;
  if (q.x >= 0 && q.y >= 0 && q.y < W && q.z >= 0 && q.z < H && q.w >= 0 && q.w < D) {
    const unsigned long long k = brick_key(q.x, q.y >> 1, q.z >> 1, q.w >> 1, Wb, Hb, Db);
    for (uint32_t s = mix32(k) & mask, it = 0; it <= mask; s = (s + 1) & mask, ++it) {
      const unsigned long long sk = __ldg(keys + s);
      if (sk == KEY_EMPTY) break;
      if (sk == k) { r = __ldg(&vals[s].v[(q.y & 1) | ((q.z & 1) << 1) | ((q.w & 1) << 2)]); break; }
    }
  }
  rows[i] = r;
}

// ---- valid(B1): one warp per block of B1 sorted rows
__global__ void k_block_or(const int* __restrict__ gray, const int* __restrict__ sorted, int n, int B1, int nb,
                           int* __restrict__ code, int* __restrict__ cnt) {
  int b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (b >= nb) return;
  int o = 0;
  i64 lo = (i64)b * B1, hi = min((i64)n, lo + B1);
  for (i64 i = lo + lane; i < hi; i += 32) o |= gray[sorted[i]];
  o = __reduce_or_sync(0xffffffffu, (unsigned)o);
  if (lane == 0) { code[b] = o; cnt[b] = __popc(o); }
}
__global__ void k_block_list(const int* __restrict__ code, const int* __restrict__ seg, int nb, int* __restrict__ list) {
  int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= nb) return;
  int c = code[b], s = seg[b];
  while (c) { list[s++] = __ffs(c) - 1; c &= c - 1; }
}

// ---- 2x subdivision
template <class T> __device__ __forceinline__ bool sub_keep(const T* sub, i64 e);
template <> __device__ __forceinline__ bool sub_keep<__half>(const __half* s, i64 e) { return __half2float(s[e]) > 0.f; }
template <> __device__ __forceinline__ bool sub_keep<__nv_bfloat16>(const __nv_bfloat16* s, i64 e) { return __bfloat162float(s[e]) > 0.f; }
template <> __device__ __forceinline__ bool sub_keep<uint8_t>(const uint8_t* s, i64 e) { return s[e] != 0; }

// With info: the parent's set of children as bits (k_c2s_emit adds the first child's row), and *partial is set when the
// children's map cannot be read off the parents' (t2sc_subdivide_neighbors): a parent outside the grid the parents' map was
// built in, one whose children would leave the children's grid, or one of several parents at one place, of which the
// parents' map names the first only.
template <class T> __global__ void k_c2s_count(const T* __restrict__ sub, int n, int* __restrict__ cnt, const int4* __restrict__ co,
                                               const uint32_t* __restrict__ nbr, int W, int H, int D, uint2* __restrict__ info, int* __restrict__ partial) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t bits = 0;
#pragma unroll
  for (int s = 0; s < 8; s++) bits |= (sub_keep<T>(sub, (i64)i * 8 + s) ? 1u : 0u) << s;
  cnt[i] = __popc(bits);
  if (info) {
    info[i].y = bits;
    const int4 q = co[i];
    if (q.x < 0 || (unsigned)q.y >= (unsigned)W || (unsigned)q.z >= (unsigned)H || (unsigned)q.w >= (unsigned)D || nbr[(i64)i * 27 + 13] != (uint32_t)i) atomicOr(partial, 1);
  }
}
template <class T> __global__ void k_c2s_emit(const T* __restrict__ sub, const int4* __restrict__ co, const int* __restrict__ off,
                                              int n, int4* __restrict__ nco, int* __restrict__ src, uint2* __restrict__ info) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int r = off[i]; int4 q = co[i];
  if (info) info[i].x = (uint32_t)r;
#pragma unroll
  for (int s = 0; s < 8; s++)
    if (sub_keep<T>(sub, (i64)i * 8 + s)) {
      nco[r] = make_int4(q.x, q.y * 2 + (s & 1), q.z * 2 + (s >> 1 & 1), q.w * 2 + (s >> 2 & 1));
      src[r++] = i * 8 + s;
    }
}

// ---- row gather / skip add, 16 bytes per thread
__global__ void k_gather_rows16(const uint4* __restrict__ x, const int* __restrict__ src, i64 m, int vec_per_row, uint4* __restrict__ y) {
  i64 i = blockIdx.x * (i64)blockDim.x + threadIdx.x;
  if (i >= m * vec_per_row) return;
  i64 r = i / vec_per_row; int c = (int)(i - r * vec_per_row);
  y[i] = __ldg(x + (i64)src[r] * vec_per_row + c);
}
template <class T> __global__ void k_add_skip(T* __restrict__ h, const T* __restrict__ x, const int* __restrict__ src, i64 m,
                                              int Co, int Cin, int rep) {
  i64 i = blockIdx.x * (i64)blockDim.x + threadIdx.x;
  if (i >= m * Co) return;
  i64 r = i / Co; int c = (int)(i - r * Co), p = src[r] >> 3, s = src[r] & 7, Cs = Cin / 8;
  h[i] = from_f<T>(to_f<T>(h[i]) + to_f<T>(x[(i64)p * Cin + s * Cs + c / rep]));
}

// 8 output channels per thread (16-byte accesses of h for the 16-bit types); Co % 8 == 0
template <class T> __global__ void k_add_skip8(T* __restrict__ h, const T* __restrict__ x, const int* __restrict__ src, i64 nvec,
                                               int vpr, int Cin, int rep) {
  const i64 i = blockIdx.x * (i64)blockDim.x + threadIdx.x;
  if (i >= nvec) return;
  const i64 r = nvec < (1ll << 31) ? (i64)((unsigned)i / (unsigned)vpr) : i / vpr;
  const int c0 = (int)(i - r * vpr) * 8, sv = src[r], Cs = Cin / 8;
  const T* xs = x + (i64)(sv >> 3) * Cin + (sv & 7) * Cs;
  T* hp = h + i * 8;
  T v[8];
  if constexpr (sizeof(T) == 2) *(uint4*)v = *(const uint4*)hp;
  else { *(float4*)v = *(const float4*)hp; *((float4*)v + 1) = *((const float4*)hp + 1); }
#pragma unroll
  for (int e = 0; e < 8; e++) v[e] = from_f<T>(to_f<T>(v[e]) + to_f<T>(xs[(c0 + e) / rep]));
  if constexpr (sizeof(T) == 2) *(uint4*)hp = *(const uint4*)v;
  else { *(float4*)hp = *(const float4*)v; *((float4*)hp + 1) = *((const float4*)v + 1); }
}

template <class T> void add_skip_pick(cudaStream_t st, void* h, const void* x, const int32_t* src, i64 m, int Co, int Cin, int rep) {
  if (Co % 8 == 0 && (uintptr_t)h % 16 == 0) {
    const i64 nvec = m * (Co / 8);
    k_add_skip8<T><<<cdiv_i(nvec, 256), 256, 0, st>>>((T*)h, (const T*)x, src, nvec, Co / 8, Cin, rep);
  } else {
    k_add_skip<T><<<cdiv_i(m * Co, 256), 256, 0, st>>>((T*)h, (const T*)x, src, m, Co, Cin, rep);
  }
}

}  // namespace

// ------------------------------------------------------------------------------------------ entry points
extern "C" int t2sc_build_neighbors(t2sc_ctx* ctx, const int32_t* coords, int64_t n, int W, int H, int D,
                                    uint32_t* nbr, int32_t* gray, int32_t* sorted) {
  T2_REQ(ctx, ctx != nullptr, "null context");
  T2_REQ(ctx, n >= 0 && n < (1ll << 30), "n=%lld", (long long)n);
  if (n == 0) return T2SC_OK;
  T2_REQ(ctx, coords && nbr && gray, "null tensor");
  T2_REQ(ctx, (uintptr_t)coords % 16 == 0, "coords must be 16-byte aligned");
  T2_REQ(ctx, W > 0 && H > 0 && D > 0, "grid extent %d %d %d", W, H, D);
  T2_CUDA(ctx, cudaSetDevice(ctx->device));
  uint32_t cap = 1; while (cap < 2u * (uint32_t)n) cap <<= 1;            // src/spconv.cu:40
  Scratch scratch(ctx);            // returned to the pool on every path out of this function
  int* bin = nullptr;
  char* table = nullptr;           // keys [cap] then brick rows [cap]: one allocation, one memset
  const int Wb = (W + 1) / 2, Hb = (H + 1) / 2, Db = (D + 1) / 2;
  const size_t table_bytes = (size_t)cap * (sizeof(unsigned long long) + sizeof(BrickVals));
  T2_CUDA(ctx, scratch.get(&table, table_bytes));
  unsigned long long* bkeys = (unsigned long long*)table; BrickVals* bvals = (BrickVals*)(table + (size_t)cap * sizeof(unsigned long long));
  T2_CUDA(ctx, cudaMemsetAsync(table, 0xff, table_bytes, ctx->stream));
  k_brick_insert<<<cdiv_i(n, 256), 256, 0, ctx->stream>>>((const int4*)coords, (int)n, Wb, Hb, Db, bkeys, bvals, cap - 1);
  T2_LAUNCHED(ctx);
  int* iota = nullptr;
  if (sorted) { T2_CUDA(ctx, scratch.get(&bin, (size_t)n)); T2_CUDA(ctx, scratch.get(&iota, (size_t)n)); }
  k_brick_neighbors<<<cdiv_i(n, 32), 256, 0, ctx->stream>>>(HashBricks{(const int4*)coords, W, H, D, Wb, Hb, Db, bkeys, bvals, cap - 1}, (int)n, nbr, gray, bin, iota);
  T2_LAUNCHED(ctx);
  if (sorted) {
    int* bs = nullptr; char* tmp = nullptr; size_t tb = 0;
    T2_CUDA(ctx, scratch.get(&bs, (size_t)n));
    // the key has 27 significant bits; radix sort is stable, so ties keep ascending row order
    T2_CUDA(ctx, cub::DeviceRadixSort::SortPairs(nullptr, tb, bin, bs, iota, sorted, (int)n, 0, 27, ctx->stream));
    T2_CUDA(ctx, scratch.get(&tmp, tb));
    T2_CUDA(ctx, cub::DeviceRadixSort::SortPairs(tmp, tb, bin, bs, iota, sorted, (int)n, 0, 27, ctx->stream));
  }
  return T2SC_OK;
}

extern "C" int t2sc_valid_taps(t2sc_ctx* ctx, const int32_t* gray, const int32_t* sorted, int64_t n, int B1,
                               int32_t* seg, int32_t* list, int64_t* total_host) {
  T2_REQ(ctx, ctx != nullptr, "null context");
  T2_REQ(ctx, n >= 0 && B1 > 0, "n=%lld B1=%d", (long long)n, B1);
  if (total_host) *total_host = 0;
  if (n == 0) return T2SC_OK;
  T2_REQ(ctx, gray && sorted && seg && list, "null tensor");
  T2_CUDA(ctx, cudaSetDevice(ctx->device));
  int nb = cdiv_i(n, B1);
  Scratch scratch(ctx);
  int* code = nullptr; char* tmp = nullptr; size_t tb = 0;
  T2_CUDA(ctx, scratch.get(&code, (size_t)nb));
  T2_CUDA(ctx, cudaMemsetAsync(seg, 0, sizeof(int), ctx->stream));
  k_block_or<<<cdiv_i((i64)nb * 32, 256), 256, 0, ctx->stream>>>(gray, sorted, (int)n, B1, nb, code, seg + 1);
  T2_LAUNCHED(ctx);
  T2_CUDA(ctx, cub::DeviceScan::InclusiveSum(nullptr, tb, seg + 1, seg + 1, nb, ctx->stream));
  T2_CUDA(ctx, scratch.get(&tmp, tb));
  T2_CUDA(ctx, cub::DeviceScan::InclusiveSum(tmp, tb, seg + 1, seg + 1, nb, ctx->stream));
  k_block_list<<<cdiv_i(nb, 256), 256, 0, ctx->stream>>>(code, seg, nb, list);
  T2_LAUNCHED(ctx);
  if (total_host) {
    int tot = 0;
    T2_CUDA(ctx, cudaMemcpyAsync(&tot, seg + nb, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    T2_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    *total_host = tot;
  }
  return T2SC_OK;
}

static int subdivide_count(t2sc_ctx* ctx, const void* sub, int sub_dtype, int64_t n, int32_t* off, int64_t* m_host,
                           const int32_t* coords, const uint32_t* nbr, int W, int H, int D, uint32_t* info, int* whole_host) {
  T2_REQ(ctx, ctx != nullptr, "null context");
  T2_REQ(ctx, n >= 0 && n < (1ll << 28), "n=%lld", (long long)n);
  T2_REQ(ctx, sub_dtype == T2SC_F16 || sub_dtype == T2SC_BF16 || sub_dtype == T2SC_U8, "sub dtype %d", sub_dtype);
  if (m_host) *m_host = 0;
  T2_REQ(ctx, off != nullptr, "null off");
  T2_CUDA(ctx, cudaSetDevice(ctx->device));
  T2_CUDA(ctx, cudaMemsetAsync(off, 0, sizeof(int), ctx->stream));
  if (n == 0) return T2SC_OK;
  T2_REQ(ctx, sub != nullptr, "null sub");
  Scratch scratch(ctx);
  int *cnt = nullptr, *partial = nullptr; char* tmp = nullptr; size_t tb = 0;
  T2_CUDA(ctx, scratch.get(&cnt, (size_t)n));
  if (info) {
    T2_CUDA(ctx, scratch.get(&partial, 1));
    T2_CUDA(ctx, cudaMemsetAsync(partial, 0, sizeof(int), ctx->stream));
  }
  int g = cdiv_i(n, 256);
  const int4* co = (const int4*)coords; uint2* inf = (uint2*)info;
  if (sub_dtype == T2SC_F16) k_c2s_count<__half><<<g, 256, 0, ctx->stream>>>((const __half*)sub, (int)n, cnt, co, nbr, W, H, D, inf, partial);
  else if (sub_dtype == T2SC_BF16) k_c2s_count<__nv_bfloat16><<<g, 256, 0, ctx->stream>>>((const __nv_bfloat16*)sub, (int)n, cnt, co, nbr, W, H, D, inf, partial);
  else k_c2s_count<uint8_t><<<g, 256, 0, ctx->stream>>>((const uint8_t*)sub, (int)n, cnt, co, nbr, W, H, D, inf, partial);
  T2_LAUNCHED(ctx);
  T2_CUDA(ctx, cub::DeviceScan::InclusiveSum(nullptr, tb, cnt, off + 1, (int)n, ctx->stream));
  T2_CUDA(ctx, scratch.get(&tmp, tb));
  T2_CUDA(ctx, cub::DeviceScan::InclusiveSum(tmp, tb, cnt, off + 1, (int)n, ctx->stream));
  if (m_host) {
    // both words land in the context's pinned block, so one wait covers them
    T2_CUDA(ctx, cudaMemcpyAsync(ctx->pinned, off + n, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    if (partial) T2_CUDA(ctx, cudaMemcpyAsync(ctx->pinned + 1, partial, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    T2_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    *m_host = ctx->pinned[0];
    if (whole_host) *whole_host = ctx->pinned[1] == 0;
  }
  return T2SC_OK;
}

extern "C" int t2sc_subdivide_count(t2sc_ctx* ctx, const void* sub, int sub_dtype, int64_t n, int32_t* off, int64_t* m_host) {
  return subdivide_count(ctx, sub, sub_dtype, n, off, m_host, nullptr, nullptr, 0, 0, 0, nullptr, nullptr);
}

extern "C" int t2sc_subdivide_count_info(t2sc_ctx* ctx, const void* sub, int sub_dtype, const int32_t* coords, const uint32_t* nbr, int W, int H, int D,
                                         int64_t n, int32_t* off, uint32_t* info, int64_t* m_host, int* whole_host) {
  T2_REQ(ctx, ctx != nullptr, "null context");
  T2_REQ(ctx, m_host && whole_host && W > 0 && H > 0 && D > 0, "null result or grid extent %d %d %d", W, H, D);
  *whole_host = 1;
  T2_REQ(ctx, n <= 0 || (coords && nbr && info), "null tensor");
  T2_REQ(ctx, (uintptr_t)coords % 16 == 0 && (uintptr_t)info % 8 == 0, "coords must be 16-byte aligned, info 8-byte");
  return subdivide_count(ctx, sub, sub_dtype, n, off, m_host, coords, nbr, W, H, D, info, whole_host);
}

extern "C" int t2sc_subdivide_emit(t2sc_ctx* ctx, const void* sub, int sub_dtype, const int32_t* coords, const int32_t* off,
                                   int64_t n, int32_t* child_coords, int32_t* src) {
  return t2sc_subdivide_emit_info(ctx, sub, sub_dtype, coords, off, n, child_coords, src, nullptr);
}

extern "C" int t2sc_subdivide_emit_info(t2sc_ctx* ctx, const void* sub, int sub_dtype, const int32_t* coords, const int32_t* off,
                                        int64_t n, int32_t* child_coords, int32_t* src, uint32_t* info) {
  T2_REQ(ctx, ctx != nullptr, "null context");
  T2_REQ(ctx, n >= 0 && n < (1ll << 28), "n=%lld", (long long)n);
  T2_REQ(ctx, sub_dtype == T2SC_F16 || sub_dtype == T2SC_BF16 || sub_dtype == T2SC_U8, "sub dtype %d", sub_dtype);
  if (n == 0) return T2SC_OK;
  T2_REQ(ctx, sub && coords && off && child_coords && src, "null tensor");
  T2_REQ(ctx, (uintptr_t)coords % 16 == 0 && (uintptr_t)child_coords % 16 == 0 && (uintptr_t)info % 8 == 0, "coords must be 16-byte aligned, info 8-byte");
  T2_CUDA(ctx, cudaSetDevice(ctx->device));
  int g = cdiv_i(n, 256);
  const int4* co = (const int4*)coords; int4* nco = (int4*)child_coords; uint2* inf = (uint2*)info;
  if (sub_dtype == T2SC_F16) k_c2s_emit<__half><<<g, 256, 0, ctx->stream>>>((const __half*)sub, co, off, (int)n, nco, src, inf);
  else if (sub_dtype == T2SC_BF16) k_c2s_emit<__nv_bfloat16><<<g, 256, 0, ctx->stream>>>((const __nv_bfloat16*)sub, co, off, (int)n, nco, src, inf);
  else k_c2s_emit<uint8_t><<<g, 256, 0, ctx->stream>>>((const uint8_t*)sub, co, off, (int)n, nco, src, inf);
  T2_LAUNCHED(ctx);
  return T2SC_OK;
}

// The children's neighbour map without a hash table: every neighbour of a child is a child of its parent or of one of the
// parent's 26 neighbours.  (On 3,288,465 children the table took a memset of 335 MB, an atomic insertion per row and eight
// probes per row.)
extern "C" int t2sc_subdivide_neighbors(t2sc_ctx* ctx, const uint32_t* parent_nbr, const uint32_t* info, int64_t n,
                                        uint32_t* nbr, int32_t* gray) {
  T2_REQ(ctx, ctx != nullptr, "null context");
  T2_REQ(ctx, n >= 0 && n < (1ll << 28), "n=%lld", (long long)n);
  if (n == 0) return T2SC_OK;
  T2_REQ(ctx, parent_nbr && info && nbr && gray && (uintptr_t)info % 8 == 0, "null or unaligned tensor");
  T2_CUDA(ctx, cudaSetDevice(ctx->device));
  k_child_neighbors<<<cdiv_i(n, 8 * CHILD_PARENTS), 256, 0, ctx->stream>>>(parent_nbr, (const uint2*)info, (int)n, nbr, gray);
  T2_LAUNCHED(ctx);
  return T2SC_OK;
}

extern "C" int t2sc_gather_rows(t2sc_ctx* ctx, const void* x, const int32_t* src, int64_t m, int C, int dtype, void* y) {
  T2_REQ(ctx, ctx != nullptr, "null context");
  size_t row_bytes = (size_t)C * dtype_size(dtype);
  T2_REQ(ctx, m >= 0 && C > 0 && row_bytes % 16 == 0, "m=%lld C=%d: rows must be a multiple of 16 bytes", (long long)m, C);
  if (m == 0) return T2SC_OK;
  T2_REQ(ctx, x && src && y && (uintptr_t)x % 16 == 0 && (uintptr_t)y % 16 == 0, "null or unaligned tensor");
  T2_CUDA(ctx, cudaSetDevice(ctx->device));
  int vpr = (int)(row_bytes / 16);
  k_gather_rows16<<<cdiv_i(m * vpr, 256), 256, 0, ctx->stream>>>((const uint4*)x, src, m, vpr, (uint4*)y);
  T2_LAUNCHED(ctx);
  return T2SC_OK;
}

extern "C" int t2sc_add_skip(t2sc_ctx* ctx, void* h, const void* x, const int32_t* src, int64_t m, int Co, int Cin, int rep, int dtype) {
  T2_REQ(ctx, ctx != nullptr, "null context");
  T2_REQ(ctx, m >= 0 && Co > 0 && Cin % 8 == 0 && rep > 0 && Co == (Cin / 8) * rep, "m=%lld Co=%d Cin=%d rep=%d", (long long)m, Co, Cin, rep);
  if (m == 0) return T2SC_OK;
  T2_REQ(ctx, h && x && src, "null tensor");
  T2_CUDA(ctx, cudaSetDevice(ctx->device));
  if (dtype == T2SC_F16) add_skip_pick<__half>(ctx->stream, h, x, src, m, Co, Cin, rep);
  else if (dtype == T2SC_BF16) add_skip_pick<__nv_bfloat16>(ctx->stream, h, x, src, m, Co, Cin, rep);
  else if (dtype == T2SC_F32) add_skip_pick<float>(ctx->stream, h, x, src, m, Co, Cin, rep);
  else return t2sc_fail(ctx, T2SC_ERR_ARG, "dtype %d", dtype);
  T2_LAUNCHED(ctx);
  return T2SC_OK;
}


// Neighbour rows of the contiguous row range [row_lo, row_hi) only, against the hash of ALL n rows: what one rank
// of a Morton-range partition needs (its owned rows, with global row indices in the map).  nbr [row_hi-row_lo, 27],
// gray [row_hi-row_lo].  No counterpart in the reference, which is single-GPU.
extern "C" int t2sc_build_neighbors_range(t2sc_ctx* ctx, const int32_t* coords, int64_t n, int W, int H, int D,
                                          int64_t row_lo, int64_t row_hi, uint32_t* nbr, int32_t* gray) {
  T2_REQ(ctx, ctx != nullptr, "null context");
  T2_REQ(ctx, n >= 0 && n < (1ll << 30) && row_lo >= 0 && row_lo <= row_hi && row_hi <= n, "n=%lld range [%lld,%lld)", (long long)n, (long long)row_lo, (long long)row_hi);
  if (row_hi == row_lo) return T2SC_OK;
  T2_REQ(ctx, coords && nbr && gray, "null tensor");
  T2_REQ(ctx, (uintptr_t)coords % 16 == 0, "coords must be 16-byte aligned");
  T2_REQ(ctx, W > 0 && H > 0 && D > 0, "grid extent %d %d %d", W, H, D);
  T2_CUDA(ctx, cudaSetDevice(ctx->device));
  uint32_t cap = 1; while (cap < 2u * (uint32_t)n) cap <<= 1;
  Scratch scratch(ctx);
  char* table = nullptr;
  const int Wb = (W + 1) / 2, Hb = (H + 1) / 2, Db = (D + 1) / 2;
  const size_t table_bytes = (size_t)cap * (sizeof(unsigned long long) + sizeof(BrickVals));
  T2_CUDA(ctx, scratch.get(&table, table_bytes));
  unsigned long long* bkeys = (unsigned long long*)table; BrickVals* bvals = (BrickVals*)(table + (size_t)cap * sizeof(unsigned long long));
  T2_CUDA(ctx, cudaMemsetAsync(table, 0xff, table_bytes, ctx->stream));
  k_brick_insert<<<cdiv_i(n, 256), 256, 0, ctx->stream>>>((const int4*)coords, (int)n, Wb, Hb, Db, bkeys, bvals, cap - 1);
  T2_LAUNCHED(ctx);
  const i64 m = row_hi - row_lo;
  k_brick_neighbors<<<cdiv_i(m, 32), 256, 0, ctx->stream>>>(HashBricks{(const int4*)coords + row_lo, W, H, D, Wb, Hb, Db, bkeys, bvals, cap - 1}, (int)m, nbr, gray, nullptr, nullptr);
  T2_LAUNCHED(ctx);
  return T2SC_OK;
}

// Rows of arbitrary query coordinates in the same voxel hash: what the reference's other hash users need of it
// (vhash_find of src/mesh.cu:7-19, used by the dual-grid quad search :54-72, and the hash half of the grid-sample
// neighbour build, src/glb.cu:545-552).
extern "C" int t2sc_voxel_lookup(t2sc_ctx* ctx, const int32_t* coords, int64_t n, int W, int H, int D,
                                 const int32_t* queries, int64_t m, uint32_t* rows) {
  T2_REQ(ctx, ctx != nullptr, "null context");
  T2_REQ(ctx, n >= 0 && n < (1ll << 30) && m >= 0, "n=%lld m=%lld", (long long)n, (long long)m);
  if (m == 0) return T2SC_OK;
  T2_REQ(ctx, queries && rows && (n == 0 || coords), "null tensor");
  T2_REQ(ctx, (uintptr_t)coords % 16 == 0 && (uintptr_t)queries % 16 == 0, "coords and queries must be 16-byte aligned");
  T2_REQ(ctx, W > 0 && H > 0 && D > 0, "grid extent %d %d %d", W, H, D);
  T2_CUDA(ctx, cudaSetDevice(ctx->device));
  uint32_t cap = 2; while (cap < 2u * (uint32_t)n) cap <<= 1;
  Scratch scratch(ctx);
  char* table = nullptr;
  const int Wb = (W + 1) / 2, Hb = (H + 1) / 2, Db = (D + 1) / 2;
  const size_t table_bytes = (size_t)cap * (sizeof(unsigned long long) + sizeof(BrickVals));
  T2_CUDA(ctx, scratch.get(&table, table_bytes));
  unsigned long long* bkeys = (unsigned long long*)table; BrickVals* bvals = (BrickVals*)(table + (size_t)cap * sizeof(unsigned long long));
  T2_CUDA(ctx, cudaMemsetAsync(table, 0xff, table_bytes, ctx->stream));
  if (n > 0) {
    k_brick_insert<<<cdiv_i(n, 256), 256, 0, ctx->stream>>>((const int4*)coords, (int)n, Wb, Hb, Db, bkeys, bvals, cap - 1);
    T2_LAUNCHED(ctx);
  }
  k_brick_lookup<<<cdiv_i(m, 256), 256, 0, ctx->stream>>>((const int4*)queries, m, W, H, D, Wb, Hb, Db, bkeys, bvals, cap - 1, rows);
  T2_LAUNCHED(ctx);
  return T2SC_OK;
}

// ------------------------------------------------------------------------------------------ allocation-free variant
// The hash table of this variant is a fixed array inside the library image instead of pool memory.
static __device__ __align__(256) unsigned char g_static_table[(size_t)2 * T2SC_STATIC_MAX_ROWS * sizeof(Slot)];
static Slot* g_static_table_ptr[64] = {nullptr};      // device address of the array, per device, resolved on first use

extern "C" int t2sc_build_neighbors_static(t2sc_ctx* ctx, const int32_t* coords, int64_t n, int W, int H, int D,
                                           uint32_t* nbr, int32_t* gray) {
  T2_REQ(ctx, ctx != nullptr, "null context");
  T2_REQ(ctx, n >= 0, "n=%lld", (long long)n);
  if (n > T2SC_STATIC_MAX_ROWS)
    return t2sc_fail(ctx, T2SC_ERR_UNSUPPORTED, "t2sc_build_neighbors_static: %lld rows exceed the built-in table (at most %d rows); "
                     "use t2sc_build_neighbors, which takes its table from the memory pool", (long long)n, T2SC_STATIC_MAX_ROWS);
  if (n == 0) return T2SC_OK;
  T2_REQ(ctx, coords && nbr && gray, "null tensor");
  T2_REQ(ctx, (uintptr_t)coords % 16 == 0, "coords must be 16-byte aligned");
  T2_REQ(ctx, W > 0 && H > 0 && D > 0, "grid extent %d %d %d", W, H, D);
  T2_REQ(ctx, ctx->device >= 0 && ctx->device < 64, "device %d", ctx->device);
  T2_CUDA(ctx, cudaSetDevice(ctx->device));
  if (!g_static_table_ptr[ctx->device]) {
    // In host code the array's name is only a handle; the kernels need its address on THIS device.
    void* p = nullptr;
    T2_CUDA(ctx, cudaGetSymbolAddress(&p, g_static_table));
    g_static_table_ptr[ctx->device] = (Slot*)p;
  }
  Slot* table = g_static_table_ptr[ctx->device];
  uint32_t cap = 1; while (cap < 2u * (uint32_t)n) cap <<= 1;
  // the array keeps the previous call's keys: every slot this call can probe is reset to "empty" first
  T2_CUDA(ctx, cudaMemsetAsync(table, 0xff, (size_t)cap * sizeof(Slot), ctx->stream));
  k_hash_insert<<<cdiv_i(n, 256), 256, 0, ctx->stream>>>((const int4*)coords, (int)n, W, H, D, table, cap - 1);
  T2_LAUNCHED(ctx);
  k_neighbors<<<cdiv_i(n, NB_ROWS), NB_THREADS, 0, ctx->stream>>>((const int4*)coords, (int)n, W, H, D, table, cap - 1, nbr, gray, nullptr);
  T2_LAUNCHED(ctx);
  return T2SC_OK;
}
