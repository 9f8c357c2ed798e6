// ffb_trace.cuh -- the hot kernels: fused emission + nearest-hit trace +
// per-(source, hit) histogram (form-factor counts), ray-batch casts (grid and
// brute force) and ray materialisation.
#pragma once

#include "ffb_grid.cuh"

namespace ffb {

// A unit of work of the fused kernel: `count` consecutive rays [j0, j0+count)
// of face `face` (index within its scene).  Rays j < front leave the front
// side, the others the rear.
struct Chunk {
  int32_t face;
  int32_t j0;
  int32_t count;
  int32_t front;
};

// Writes the work chunks of the emitting faces: src[i] = {face, front rays,
// front + rear rays, first chunk}; the face's rays [0, nf) become chunks of
// `rays` consecutive rays (the last one shorter), one warp per face.
__global__ void k_chunk_fill(const int4* __restrict__ src, int n, int rays, Chunk* __restrict__ chunks)
{
  const int lane = threadIdx.x & 31;
  const int warps = (int)((gridDim.x * blockDim.x) >> 5);
  for (int i = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); i < n; i += warps) {
    const int4 f = src[i];
    const int nc = (f.z + rays - 1) / rays;
    for (int j = lane; j < nc; j += 32)
      chunks[(uint32_t)f.w + (uint32_t)j] = Chunk{f.x, j * rays, min(rays, f.z - j * rays), f.y};
  }
}

// Statistics slots (uint64 each), accumulated once per warp.
enum { kStatTests = 0, kStatCells = 1, kStatRays = 2, kStatHits = 3, kStatJumps = 4, kStatSlots = 5 };

// The scene of a fused launch: its grid, its count matrix and where its
// faces start in the launch's frame table.
struct SceneSlot {
  GridView g;
  uint32_t* __restrict__ counts;              // n_cols * n_cols
  const int32_t* __restrict__ face_to_row;   // face -> matrix row/column (mesh), or null for identity
  int face_base;                              // first frame of the scene
  int n_cols;                                 // matrix side
};

// Scenes of one batch (ffb_batch_set); each is traced by its own launch.
constexpr int kMaxBatchScenes = 4096;

struct TraceParams {
  const float* __restrict__ frames;          // 20 floats per face, scenes concatenated
  const Chunk* __restrict__ chunks;
  int n_chunks;
  uint32_t key0, key1, epoch;
  const uint32_t* __restrict__ epoch_ptr;    // when set, the epoch is read from device memory
  const uint2* __restrict__ scene_keys;      // device Philox key of the scene, or null for (key0, key1)
  uint32_t* __restrict__ chunk_cursor;        // work counter, zero before the launch
  unsigned long long* __restrict__ stats;     // kStatSlots, or null
  // radiance sink (kPower): per-ray power of each (face, side) as 64-bit
  // fixed point, and the per-mesh absorbed power it adds to (mesh = the
  // scene's face_to_row of the hit face), in absorb_mask + 1 copies
  // absorb_stride apart (k_tally_sum)
  const unsigned long long* __restrict__ power;
  unsigned long long* __restrict__ absorb;
  uint32_t absorb_mask = 0, absorb_stride = 0;
  // when set: [0] gets the earliest block start and [1] the latest warp end
  // of the launch, in %globaltimer nanoseconds (atomicMin / atomicMax, so
  // several launches may share one pair)
  unsigned long long* __restrict__ span;
  int default_shape = 0;        // the launch's shape where none was chosen (host only)
  bool stream_records = false;  // test records bypass the L1 cache, see ldg8 (host only)
  SceneSlot scene;
};

__device__ __forceinline__ unsigned long long global_ns()
{
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

constexpr int kTraceThreads = 128;
constexpr int kWarpsPerBlock = kTraceThreads / 32;
// Blocks per SM the trace kernels are compiled for: 8 blocks of 128 threads
// cap registers at 64 per thread (32 warps per SM to hide L1/L2 latency).
#ifndef FFB_MIN_BLOCKS
#define FFB_MIN_BLOCKS 8
#endif
constexpr int kWarpHashLog2 = 9;
constexpr int kWarpHash = 1 << kWarpHashLog2;  // histogram slots per warp
constexpr uint32_t kEmptyKey = 0xFFFFFFFFu;
constexpr size_t kHashSmem = sizeof(uint32_t) * 2 * kWarpHash * kWarpsPerBlock;  // dynamic shared bytes with kHash
constexpr unsigned kFull = 0xFFFFFFFFu;

__device__ __forceinline__ void warp_stats(unsigned long long* stats, uint32_t tests, uint32_t cells, uint32_t rays,
                                           uint32_t hits, uint32_t jumps)
{
  if (!stats)
    return;
  unsigned long long v[kStatSlots] = {tests, cells, rays, hits, jumps};
#pragma unroll
  for (int k = 0; k < kStatSlots; ++k) {
    unsigned long long x = v[k];
    for (int o = 16; o > 0; o >>= 1)
      x += __shfl_xor_sync(kFull, x, o);
    if ((threadIdx.x & 31) == 0 && x)
      atomicAdd(stats + k, x);
  }
}

// Adds 1 to the bin of `key` in a warp's open-addressing table.  Returns true
// when the key took a new slot.  Keys are matrix indices row * n_cols + col.
__device__ __forceinline__ bool warp_hash_add(uint32_t* keys, uint32_t* vals, uint32_t key, uint32_t* counts)
{
  uint32_t s = (key * 2654435761u) >> (32 - kWarpHashLog2);
  volatile uint32_t* vk = keys;
  for (int probe = 0; probe < kWarpHash; ++probe) {
    uint32_t cur = vk[s];
    if (cur == kEmptyKey) {
      cur = atomicCAS(keys + s, kEmptyKey, key);
      if (cur == kEmptyKey) {
        atomicAdd(vals + s, 1u);
        return true;
      }
    }
    if (cur == key) {
      atomicAdd(vals + s, 1u);
      return false;
    }
    s = (s + 1) & (kWarpHash - 1);
  }
  atomicAdd(counts + key, 1u);  // full table; unreachable: flushed at half load
  return false;
}

// Adds every occupied bin of a warp's table to the global matrix and clears it.
__device__ __forceinline__ void warp_hash_flush(uint32_t* keys, uint32_t* vals, uint32_t* counts, int lane)
{
  __syncwarp();
  for (int i = lane; i < kWarpHash; i += 32) {
    const uint32_t k = keys[i];
    if (k != kEmptyKey) {
      atomicAdd(counts + k, vals[i]);
      keys[i] = kEmptyKey;
      vals[i] = 0;
    }
  }
  __syncwarp();
}

// ---------------------------------------------------------------------------
// Fused form-factor kernel.  Persistent warps, no block barriers.  Each warp
// keeps a current chunk (consecutive rays of one face; one global atomic per
// chunk) and emits its next 32 rays, one per lane, into a queue in shared
// memory whenever the queue is empty.  Idle lanes are refilled from the queue
// together once at least the shape's `refill` of them wait (or the whole warp
// is idle), so a warp may hold rays of several faces at once.  Emission by
// the idle lanes themselves, 6 to 8 of 32, took 15 of 167 warp instructions
// per ray.  Each iteration a lane tests up to the shape's `test` references
// of its cell and, when it has none left, moves on (stop, DDA step or
// empty-space jump; up to `adv` moves while it lands in empty cells): this
// order took 5 % less than moving before testing.  Letting a vote of the warp
// pick one kind of work per iteration filled more lanes and was 6 to 11 %
// slower: it waits for memory more often.  A finished hit adds one to the
// warp's shared-memory hash histogram keyed by the matrix index
// row(f) * n_cols + row(h); the warp flushes the table to the global uint32
// matrix with atomic adds when it is half full and at the end.
//
// kPower (the radiance equation, thermal_equation/radiance_cpu.cpp:142-180)
// replaces the matrix: a hit adds the per-ray power of the ray's (source
// face, side) to the absorbed power of the hit face's mesh, in 64-bit fixed
// point (integer sums: the same result whatever the order of the hits).
// kStats adds the test / cell / ray / hit counters (Tally); without it
// p.stats is ignored.  kStream: see ldg8.  kHash selects the warp histogram;
// without it each hit is one global reduction (red.global.add) into the
// matrix, which suits large, sparse matrices (distinct keys per warp, so the
// histogram merges little) and leaves the shared memory to the L1 cache.
//
// What bounds it: waiting for the loads of cell and test records from L1 and
// L2, each of which depends on the one before, with the 32 warps per SM that
// 64 registers leave; then issue (58 % of the slots, 146 warp instructions per
// ray, 14.7 of 32 lanes).  22.08 M rays in the closed room of 22 080 faces at
// 162^3 cells: 4.61 ms; 4.80 with the records cached in L1 (ldg8), 5.48 with
// emission by idle lanes and spills in the loop, 9.65 with the exact test for
// every reference.
// ---------------------------------------------------------------------------
#ifndef FFB_REFILL_MIN
#define FFB_REFILL_MIN 8
#endif
constexpr int kRefillMin = FFB_REFILL_MIN;
// cell advances and triangle tests a lane may do per iteration
#ifndef FFB_ADV_PER_ITER
#define FFB_ADV_PER_ITER 2
#endif
#ifndef FFB_TEST_PER_ITER
#define FFB_TEST_PER_ITER 2
#endif

// Launch shapes of the fused kernel, the choices of the autotuner
// (ffb_autotune): cell advances and triangle tests a lane may do per
// iteration, the idle lanes a warp waits for before it refills them, and the
// resident blocks of 128 threads per SM the kernel is compiled for (which
// caps its registers at 65536 / (128 * blocks)).  Shape 0 is the default; where
// a scene's grid lists few references per face, shape 12 (default_shape).
// The shape changes only the order in which lanes do their work, never a
// ray's result or the counts.
// With `coherent` set, a warp hands out the rays of each chunk it takes in
// the order of their directions (bins of an 8 x 8 Morton order on the Malley
// disk) instead of in index order, so that lanes refilled together trace
// rays of similar direction from the same face.
struct TraceShape {
  int adv, test, refill, blocks, coherent;
};
constexpr int kNumShapes = 14;
__host__ __device__ constexpr TraceShape trace_shape(int v)
{
  return v == 1 ? TraceShape{1, 1, 4, 8, 0}
       : v == 2 ? TraceShape{2, 1, 6, 8, 0}
       : v == 3 ? TraceShape{1, 2, 6, 8, 0}
       : v == 4 ? TraceShape{3, 3, 6, 8, 0}
       : v == 5 ? TraceShape{2, 2, 10, 8, 0}
       : v == 6 ? TraceShape{2, 2, 6, 6, 0}
       : v == 7 ? TraceShape{2, 2, 6, 8, 1}
       : v == 8 ? TraceShape{2, 2, 10, 8, 1}
       : v == 9 ? TraceShape{2, 2, 8, 7, 0}
       : v == 10 ? TraceShape{2, 4, 8, 8, 0}
       : v == 11 ? TraceShape{4, 2, 8, 8, 0}
       : v == 12 ? TraceShape{2, 3, 8, 8, 0}
       : v == 13 ? TraceShape{3, 2, 8, 8, 1}
                 : TraceShape{FFB_ADV_PER_ITER, FFB_TEST_PER_ITER, FFB_REFILL_MIN, FFB_MIN_BLOCKS, 0};
}

constexpr int kChunkRaysMax = 256;  // rays per chunk (the host's chunk size)
constexpr int kDirBins = 64;        // direction bins of the coherent hand-out

// Direction bin of ray j of a face (the draws of emit_ray): the Malley disk
// point (sqrt(r) cos phi, sqrt(r) sin phi) on an 8 x 8 grid, in Morton order.
__device__ __forceinline__ int direction_bin(uint32_t face, uint32_t j, uint32_t key0, uint32_t key1, uint32_t epoch)
{
  const uint4 x = philox4x32_10(make_uint4(j, face, epoch, 0x46464231u), key0, key1);
  const float rad = sqrtf(u01(x.z));
  float sphi, cphi;
  sincos_turn24(x.w >> 8, sphi, cphi);
  const int qx = min(7, max(0, (int)((rad * cphi + 1.f) * 4.f)));
  const int qy = min(7, max(0, (int)((rad * sphi + 1.f) * 4.f)));
  int code = 0;
#pragma unroll
  for (int b = 0; b < 3; ++b)
    code |= (((qx >> b) & 1) << (2 * b)) | (((qy >> b) & 1) << (2 * b + 1));
  return code;
}

// Order of the chunk's rays [0, count) by direction bin (a counting sort in
// the warp's shared memory: `cnt` kDirBins counters, `perm` the order).
__device__ __forceinline__ void direction_order(uint32_t face, uint32_t j0, int count, uint32_t key0, uint32_t key1,
                                                uint32_t epoch, uint32_t* cnt, uint8_t* perm, int lane)
{
  cnt[lane] = 0;
  cnt[lane + 32] = 0;
  __syncwarp();
  uint32_t code[kChunkRaysMax / 32];
#pragma unroll
  for (int m = 0; m < kChunkRaysMax / 32; ++m) {
    const int idx = m * 32 + lane;
    code[m] = 0;
    if (idx < count) {
      const int bin = direction_bin(face, j0 + (uint32_t)idx, key0, key1, epoch);
      code[m] = (uint32_t)bin | (atomicAdd(cnt + bin, 1u) << 8);
    }
  }
  __syncwarp();
  // exclusive scan of the counters, two per lane
  const uint32_t a = cnt[2 * lane], b = cnt[2 * lane + 1];
  uint32_t incl = a + b;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(kFull, incl, o);
    if (lane >= o)
      incl += y;
  }
  __syncwarp();
  cnt[2 * lane] = incl - a - b;
  cnt[2 * lane + 1] = incl - b;
  __syncwarp();
#pragma unroll
  for (int m = 0; m < kChunkRaysMax / 32; ++m) {
    const int idx = m * 32 + lane;
    if (idx < count)
      perm[cnt[code[m] & 0xFFu] + (code[m] >> 8)] = (uint8_t)idx;
  }
  __syncwarp();
}

// The lanes' test / cell / ray / hit / jump counters, in shared memory: five
// more registers a lane spill.  For 22 M rays in a closed room of 22 080
// faces they cost 0.7 ms of 6.2; these cost 0.4 of 5.2.
enum { kCountTests, kCountCells, kCountRays, kCountHits, kCountJumps };
template <bool kOn>
struct Tally {
  uint32_t (*n)[kTraceThreads];
  __device__ __forceinline__ void clear()
  {
    if constexpr (kOn) {
      __shared__ uint32_t s_count[kCountJumps + 1][kTraceThreads];
      n = s_count;
#pragma unroll
      for (int k = 0; k <= kCountJumps; ++k)
        n[k][threadIdx.x] = 0;
    }
  }
  __device__ __forceinline__ void add(int k, uint32_t x)
  {
    if constexpr (kOn)
      n[k][threadIdx.x] += x;
  }
  __device__ __forceinline__ void flush(unsigned long long* stats)
  {
    if constexpr (kOn)
      warp_stats(stats, n[kCountTests][threadIdx.x], n[kCountCells][threadIdx.x], n[kCountRays][threadIdx.x],
                 n[kCountHits][threadIdx.x], n[kCountJumps][threadIdx.x]);
  }
};

// Part of a lane's state (the first kVectors vectors of Tracer), set aside in
// local memory around a rare stretch of code that needs many registers: the
// exact test (one ray in twenty) and the emission of 32 rays.  Left to itself
// the compiler fits the loop into 64 registers by spilling 84 bytes a thread
// of what every iteration uses; 80 registers spill nothing but leave six
// blocks per SM.  22 M rays in a closed room, ms: 5.4 spilling, 5.9 with six
// blocks, 4.8 with this.  How much to set aside is measured for each variant:
// more than it takes to end the spills only adds stores.
template <int kVectors>
struct TracerHold {
  volatile float v[3 * kVectors + (kVectors == 0)];
  __device__ __forceinline__ explicit TracerHold(const Tracer& T)
  {
    const float3* a[6] = {&T.og, &T.dg, &T.po, &T.pd, &T.iv, &T.io};
#pragma unroll
    for (int k = 0; k < kVectors; ++k) {
      v[3 * k] = a[k]->x;
      v[3 * k + 1] = a[k]->y;
      v[3 * k + 2] = a[k]->z;
    }
  }
  __device__ __forceinline__ void release(Tracer& T) const
  {
    float3* a[6] = {&T.og, &T.dg, &T.po, &T.pd, &T.iv, &T.io};
#pragma unroll
    for (int k = 0; k < kVectors; ++k)
      *a[k] = f3(v[3 * k], v[3 * k + 1], v[3 * k + 2]);
  }
};

// Tests up to kTest pending references of the cell of each active lane; the
// ray for the exact test comes from shared memory (`ray`).
template <int kTest, int kHold, bool kFar, bool kStream>
__device__ __forceinline__ void warp_tests(Tracer& T, const GridView& g, bool active,
                                           const float4 (&ray)[2][kTraceThreads], uint32_t& n_tests)
{
  if (active && T.i < T.en) {
    int open = -1;
#pragma unroll
    for (int k = 0; k < kTest; ++k)
      if (T.i < T.en && open < 0)
        open = tracer_test<kFar, kStream>(T, g, n_tests);
    if (open >= 0) {
      const TracerHold<kHold> hold(T);
      const float4 q = ray[0][threadIdx.x], r = ray[1][threadIdx.x];
      tracer_exact(T, g, open, f3(q.x, q.y, q.z), f3(q.w, r.x, r.y), r.z);
      hold.release(T);
    }
  }
}

template <bool kStats, bool kHash, bool kPower, int kShape, bool kStream>
__global__ void __launch_bounds__(kTraceThreads, trace_shape(kShape).blocks)
    k_form_factors(const __grid_constant__ TraceParams p)
{
  constexpr TraceShape kS = trace_shape(kShape);
  // vectors set aside around the emission and the exact test (TracerHold)
  constexpr int kHoldFill = kS.coherent ? 4 : kStats ? 1 : 0, kHoldExact = kStats || kHash ? 6 : 3;
  extern __shared__ uint32_t s_hash[];  // kWarpsPerBlock x (keys, values) when kHash
  // coherent hand-out: per warp, direction-bin counters and the chunk's ray order
  __shared__ uint32_t s_bins[kS.coherent ? kWarpsPerBlock * kDirBins : 1];
  __shared__ uint8_t s_perm[kS.coherent ? kWarpsPerBlock * kChunkRaysMax : 1];
  // each lane's ray for the exact test: (origin, direction x), (direction y, z, start distance, row)
  __shared__ float4 s_ray[2][kTraceThreads];
  // rays of each warp that are emitted but not handed out: (origin, direction x), (direction y, z, -, row)
  __shared__ float4 s_queue[2][kTraceThreads];
  __shared__ int4 s_chunk[kWarpsPerBlock];  // (face, j, front, row)
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  Tally<kStats> count;
  count.clear();
  if (p.span && threadIdx.x == 0)
    atomicMin(p.span, global_ns());
  uint32_t* keys = s_hash + warp * 2 * kWarpHash;
  uint32_t* vals = keys + kWarpHash;
  if (kHash) {
    for (int i = lane; i < kWarpHash; i += 32) {
      keys[i] = kEmptyKey;
      vals[i] = 0;
    }
    __syncwarp();
  }
  const uint32_t epoch = p.epoch_ptr ? *p.epoch_ptr : p.epoch;
  const unsigned lane_below = (1u << lane) - 1u;
  int fill = 0;  // occupied slots (warp-uniform)
  // current chunk (warp-uniform); c_pos: its rays handed out so far
  int c_left = 0;
  const SceneSlot& S = p.scene;
  uint32_t key0 = p.key0, key1 = p.key1;
  if (p.scene_keys) {
    const uint2 k = p.scene_keys[0];
    key0 = k.x;
    key1 = k.y;
  }
  int q_pos = 0, q_end = 0;  // queued rays [q_pos, q_end) (warp-uniform)
  bool exhausted = false;
  // lane state
  Tracer T;
  bool active = false;
  for (;;) {
    unsigned need = __ballot_sync(kFull, !active);
    if ((__popc(need) < kS.refill && need != kFull) || (exhausted && q_pos == q_end))
      need = 0;
    while (need) {
      if (q_pos == q_end) {
        // the next 32 rays of the warp's chunks, one per lane (after every
        // lane has read the last ones)
        __syncwarp();
        const TracerHold<kHoldFill> hold(T);
        q_pos = q_end = 0;
        while (q_end < 32 && !exhausted) {
          if (c_left == 0) {
            int k = 0;
            if (lane == 0)
              k = (int)atomicAdd(p.chunk_cursor, 1u);
            k = __shfl_sync(kFull, k, 0);
            if (k >= p.n_chunks) {
              exhausted = true;
              break;
            }
            const Chunk ch = p.chunks[k];
            c_left = ch.count;
            __syncwarp();  // every lane has read the chunk before (a shuffle orders no memory)
            if (lane == 0)
              s_chunk[warp] = make_int4(ch.face, kS.coherent ? ch.j0 : ch.j0 + ch.count, ch.front,
                                        S.face_to_row ? __ldg(S.face_to_row + ch.face) : ch.face);
            __syncwarp();
            if (kS.coherent)
              direction_order((uint32_t)ch.face, (uint32_t)ch.j0, c_left, key0, key1, epoch, s_bins + warp * kDirBins,
                              s_perm + warp * kChunkRaysMax, lane);
          }
          const int take = min(32 - q_end, c_left), rank = lane - q_end;
          if (rank >= 0 && rank < take) {
            const int4 ch = s_chunk[warp];
            const int c_face = ch.x, c_front = ch.z, c_row = ch.w;
            const int j =
                ch.y + (kS.coherent ? (int)s_perm[warp * kChunkRaysMax + c_left - 1 - rank] : rank - c_left);
            float3 o, e;
            emit_ray(p.frames + 20 * ((size_t)S.face_base + c_face), (uint32_t)c_face, (uint32_t)j, c_front, key0, key1,
                     epoch, o, e);
            count.add(kCountRays, 1u);
            const float3 dir = sub3(e, o);
            s_queue[0][threadIdx.x] = make_float4(o.x, o.y, o.z, dir.x);
            s_queue[1][threadIdx.x] =
                make_float4(dir.y, dir.z, 0.f, __int_as_float(kPower ? 2 * c_face + (j >= c_front ? 1 : 0) : c_row));
          }
          c_left -= take;
          q_end += take;
        }
        __syncwarp();
        hold.release(T);
        if (q_end == 0)
          break;
      }
      const int take = min(__popc(need), q_end - q_pos);
      const int rank = __popc(need & lane_below);
      const bool mine = ((need >> lane) & 1u) && rank < take;
      if (mine) {
        const float4 q = s_queue[0][(threadIdx.x & ~31) + q_pos + rank];
        float4 r = s_queue[1][(threadIdx.x & ~31) + q_pos + rank];
        uint32_t n_cells = 0;
        active = tracer_begin<false>(T, S.g, f3(q.x, q.y, q.z), f3(q.w, r.x, r.y), &r.z, n_cells);
        count.add(kCountCells, n_cells);
        s_ray[0][threadIdx.x] = q;
        s_ray[1][threadIdx.x] = r;
      }
      need &= ~__ballot_sync(kFull, mine);
      q_pos += take;
    }
    if (exhausted && q_pos == q_end && !__any_sync(kFull, active))
      break;
    uint32_t n_tests = 0;
    warp_tests<kS.test, kHoldExact, false, kStream>(T, S.g, active, s_ray, n_tests);
    count.add(kCountTests, n_tests);
    int hit = -1;
    if (active && T.i >= T.en) {
      bool live = true;
      uint32_t n_cells = 0, n_jumps = 0;
#pragma unroll
      for (int k = 0; k < kS.adv; ++k)
        if (live && T.i >= T.en)
          live = tracer_advance(T, S.g, n_cells, n_jumps);
      count.add(kCountCells, n_cells);
      count.add(kCountJumps, n_jumps);
      if (!live) {
        active = false;
        hit = T.face;
      }
    }
    bool fresh = false;
    if (hit >= 0) {
      count.add(kCountHits, 1u);
      const int col = S.face_to_row ? __ldg(S.face_to_row + hit) : hit;
      const int my_row = __float_as_int(s_ray[1][threadIdx.x].w);
      if (kPower) {
        atomicAdd(p.absorb + (size_t)(blockIdx.x & p.absorb_mask) * p.absorb_stride + col, __ldg(p.power + my_row));
      } else {
        const uint32_t key = (uint32_t)my_row * (uint32_t)S.n_cols + (uint32_t)col;
        if (kHash)
          fresh = warp_hash_add(keys, vals, key, S.counts);
        else
          atomicAdd(S.counts + key, 1u);
      }
    }
    if (kHash) {
      fill += __popc(__ballot_sync(kFull, fresh));
      if (fill > kWarpHash / 2) {
        warp_hash_flush(keys, vals, S.counts, lane);
        fill = 0;
      }
    }
  }
  if (kHash)
    warp_hash_flush(keys, vals, S.counts, lane);
  count.flush(p.stats);
  if (p.span && lane == 0)
    atomicMax(p.span + 1, global_ns());
}

// ---------------------------------------------------------------------------
// Parallel rays from a disc (a distant source): the thermal_equation
// parallel_rays_cpu path (thermal_equation/parallel_rays_cpu.cpp:92-131)
// with emission, trace and the per-face tally fused.  Persistent warps take
// 32 ray indices at a time from a global cursor and emit them together into a
// queue, as k_form_factors does (10 M rays at 20 000 faces: 2.09
// ms; 2.23 with the idle lanes emitting and an atomic for each refill).  A hit
// on face h adds one to side_counts[2h] when the ray meets its front (dot(triangle_normal(h), direction) < 0, as the
// reference chooses the front absorbance) and to side_counts[2h + 1]
// otherwise.
// ---------------------------------------------------------------------------
template <bool kStats, bool kStream>
__global__ void __launch_bounds__(kTraceThreads, FFB_MIN_BLOCKS)
    k_parallel_rays(GridView g, const __grid_constant__ DiscSource src, const float* __restrict__ faces9,
                    unsigned long long n_rays, uint32_t key0, uint32_t key1, uint32_t epoch,
                    uint32_t* __restrict__ side_counts, uint32_t copy_mask, uint32_t copy_stride,
                    unsigned long long* __restrict__ cursor, unsigned long long* __restrict__ stats)
{
  __shared__ float4 s_ray[2][kTraceThreads], s_queue[2][kTraceThreads];  // as in k_form_factors
  const int lane = threadIdx.x & 31;
  const unsigned lane_below = (1u << lane) - 1u;
  Tally<kStats> count;
  count.clear();
  Tracer T;
  bool active = false;
  int q_pos = 0, q_end = 0;  // queued rays [q_pos, q_end)
  bool exhausted = false;
  for (;;) {
    unsigned need = __ballot_sync(kFull, !active);
    while ((__popc(need) >= kRefillMin || need == kFull) && !(exhausted && q_pos == q_end)) {
      if (q_pos == q_end) {
        // the next 32 rays, one per lane (after every lane has read the last ones)
        __syncwarp();
        const TracerHold<1> hold(T);
        q_pos = q_end = 0;
        unsigned long long next = 0;
        if (lane == 0)
          next = atomicAdd(cursor, 32ull);
        next = __shfl_sync(kFull, next, 0);
        if (next >= n_rays)
          exhausted = true;
        else
          q_end = (int)min(32ull, n_rays - next);
        if (lane < q_end) {
          float3 o, e;
          emit_disc_ray(src, next + lane, key0, key1, epoch, o, e);
          count.add(kCountRays, 1u);
          const float3 dir = sub3(e, o);
          s_queue[0][threadIdx.x] = make_float4(o.x, o.y, o.z, dir.x);
          s_queue[1][threadIdx.x] = make_float4(dir.y, dir.z, 0.f, 0.f);
        }
        __syncwarp();
        hold.release(T);
      }
      const int take = min(__popc(need), q_end - q_pos);
      const int rank = __popc(need & lane_below);
      if (((need >> lane) & 1u) && rank < take) {
        const float4 q = s_queue[0][(threadIdx.x & ~31) + q_pos + rank];
        float4 r = s_queue[1][(threadIdx.x & ~31) + q_pos + rank];
        uint32_t n_cells = 0;
        active = tracer_begin<true>(T, g, f3(q.x, q.y, q.z), f3(q.w, r.x, r.y), &r.z, n_cells);
        count.add(kCountCells, n_cells);
        s_ray[0][threadIdx.x] = q;
        s_ray[1][threadIdx.x] = r;
      }
      q_pos += take;
      // lanes whose ray passes the grid box are idle again
      need = __ballot_sync(kFull, !active);
    }
    if (exhausted && q_pos == q_end && !__any_sync(kFull, active))
      break;
    uint32_t n_tests = 0;
    warp_tests<FFB_TEST_PER_ITER, 4, true, kStream>(T, g, active, s_ray, n_tests);
    count.add(kCountTests, n_tests);
    if (active && T.i >= T.en) {
      bool live = true;
      uint32_t n_cells = 0, n_jumps = 0;
#pragma unroll
      for (int k = 0; k < FFB_ADV_PER_ITER; ++k)
        if (live && T.i >= T.en)
          live = tracer_advance(T, g, n_cells, n_jumps);
      count.add(kCountCells, n_cells);
      count.add(kCountJumps, n_jumps);
      if (!live) {
        active = false;
        const int h = T.face;
        if (h >= 0) {
          count.add(kCountHits, 1u);
          // triangle_normal (math/triangle.cpp:114-119), dot with the direction
          const float* q = faces9 + 9 * (size_t)h;
          const float3 p0 = f3(__ldg(q + 0), __ldg(q + 1), __ldg(q + 2));
          const float3 nrm = cross3(sub3(f3(__ldg(q + 3), __ldg(q + 4), __ldg(q + 5)), p0),
                                    sub3(f3(__ldg(q + 6), __ldg(q + 7), __ldg(q + 8)), p0));
          const float side = dot3(nrm, src.direction);
          atomicAdd(side_counts + (size_t)(blockIdx.x & copy_mask) * copy_stride + 2 * (size_t)h + (side < 0.f ? 0 : 1),
                    1u);
        }
      }
    }
  }
  if (kStats)
    count.flush(stats);
}

// out[i] = the sum of in[k * stride + i] over `copies` copies, i below n.
//
// The sinks with few counters (a distant source's tallies, the radiance
// equation's meshes) are bound by atomics that meet in the same cache lines:
// 2.2 M hits on a clutter of 1959 faces took 0.30 to 0.46 ms of which 0.16 to
// 0.32 went with the atomics taken out.  Blocks so add into several copies of
// the counters (tally_copies), and this kernel sums them.  Integer sums: the
// same result in any order.
constexpr int kSumCounters = 32, kSumLanes = 8;
template <class T>
__global__ void __launch_bounds__(kSumCounters* kSumLanes)
    k_tally_sum(const T* __restrict__ in, int copies, int stride, int n, T* __restrict__ out)
{
  __shared__ T part[kSumLanes][kSumCounters];
  const int x = threadIdx.x % kSumCounters, y = threadIdx.x / kSumCounters;
  const int i = blockIdx.x * kSumCounters + x;
  T sum = 0;
  if (i < n) {
#pragma unroll 8
    for (int k = y; k < copies; k += kSumLanes)
      sum += in[(size_t)k * stride + i];
  }
  part[y][x] = sum;
  __syncthreads();
  if (y == 0 && i < n) {
#pragma unroll
    for (int k = 1; k < kSumLanes; ++k)
      sum += part[k][x];
    out[i] = sum;
  }
}

// Materialises rays [0, n_rays) of a disc source (parallel_rays_cpu.cpp:88-106).
__global__ void k_emit_disc(const __grid_constant__ DiscSource src, unsigned long long n_rays, uint32_t key0,
                            uint32_t key1, uint32_t epoch, float* __restrict__ rays6)
{
  for (unsigned long long j = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; j < n_rays;
       j += (unsigned long long)gridDim.x * blockDim.x) {
    float3 o, e;
    emit_disc_ray(src, j, key0, key1, epoch, o, e);
    float* r = rays6 + 6 * j;
    r[0] = o.x; r[1] = o.y; r[2] = o.z;
    r[3] = e.x; r[4] = e.y; r[5] = e.z;
  }
}

// Advances the device-resident Philox epoch of a captured launch, so that every
// replay of a CUDA graph draws fresh rays.
__global__ void k_epoch_bump(uint32_t* epoch)
{
  if (threadIdx.x == 0 && blockIdx.x == 0)
    *epoch += 1;
}

// ---------------------------------------------------------------------------
// Ray-batch cast through the grid (the ray_caster interface): rays are
// {origin, end point} as in math::ray_t.  hit_face gets the face index or -1;
// hit_point (optional) gets the point, NaN for a miss.  Persistent warps take
// rays from a global cursor (one atomic per refill) as lanes fall idle.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kTraceThreads, FFB_MIN_BLOCKS)
    k_cast(GridView g, const float* __restrict__ rays6, long n_rays, int32_t* __restrict__ hit_face,
           float* __restrict__ hit_point, unsigned long long* __restrict__ stats,
           unsigned long long* __restrict__ cursor)
{
  __shared__ float4 s_ray[2][kTraceThreads];  // as in k_form_factors
  const int lane = threadIdx.x & 31;
  const unsigned lane_below = (1u << lane) - 1u;
  Tally<true> count;
  count.clear();
  Tracer T;
  bool active = false;
  long id = -1;
  bool exhausted = false;
  auto finish = [&](long i, int h, float3 pt) {
    hit_face[i] = h;
    if (hit_point) {
      if (h < 0)
        pt = f3(NAN, NAN, NAN);
      hit_point[3 * i + 0] = pt.x;
      hit_point[3 * i + 1] = pt.y;
      hit_point[3 * i + 2] = pt.z;
    }
    count.add(kCountRays, 1u);
    count.add(kCountHits, h >= 0);
  };
  for (;;) {
    const unsigned need = __ballot_sync(kFull, !active);
    if ((__popc(need) >= kRefillMin || need == kFull) && !exhausted) {
      unsigned long long base = 0;
      if (lane == 0)
        base = atomicAdd(cursor, (unsigned long long)__popc(need));
      base = __shfl_sync(kFull, base, 0);
      if (base >= (unsigned long long)n_rays)
        exhausted = true;
      if ((need >> lane) & 1u) {
        const unsigned long long r = base + __popc(need & lane_below);
        if (r < (unsigned long long)n_rays) {
          id = (long)r;
          const float* q = rays6 + 6 * r;
          const float3 o = f3(__ldg(q + 0), __ldg(q + 1), __ldg(q + 2));
          const float3 e = f3(__ldg(q + 3), __ldg(q + 4), __ldg(q + 5));
          const float3 dir = sub3(e, o);
          float t0;
          uint32_t n_cells = 0;
          active = tracer_begin<true>(T, g, o, dir, &t0, n_cells);
          count.add(kCountCells, n_cells);
          s_ray[0][threadIdx.x] = make_float4(o.x, o.y, o.z, dir.x);
          s_ray[1][threadIdx.x] = make_float4(dir.y, dir.z, t0, 0.f);
          if (!active)
            finish(id, -1, o);
        }
      }
    }
    if (exhausted && !__any_sync(kFull, active))
      break;
    uint32_t n_tests = 0;
    warp_tests<FFB_TEST_PER_ITER, 6, true, false>(T, g, active, s_ray, n_tests);
    count.add(kCountTests, n_tests);
    if (active && T.i >= T.en) {
      bool live = true;
      uint32_t n_cells = 0, n_jumps = 0;
#pragma unroll
      for (int k = 0; k < FFB_ADV_PER_ITER; ++k)
        if (live && T.i >= T.en)
          live = tracer_advance(T, g, n_cells, n_jumps);
      count.add(kCountCells, n_cells);
      count.add(kCountJumps, n_jumps);
      if (!live) {
        active = false;
        float3 pt = f3(0.f, 0.f, 0.f);
        if (hit_point && T.face >= 0) {  // the reference's hit point
          const float4 q = s_ray[0][threadIdx.x], r = s_ray[1][threadIdx.x];
          tri_hit(reinterpret_cast<const float4*>(g.tri + T.face), f3(q.x, q.y, q.z), f3(q.w, r.x, r.y), pt);
        }
        finish(id, T.face, pt);
      }
    }
  }
  count.flush(stats);
}

// Brute force: every ray against every face (the naive_cpu definition),
// faces staged through shared memory in tiles, in index order with a strict
// '<' as the reference scans them.
constexpr int kBruteTile = 128;

__global__ void __launch_bounds__(kTraceThreads) k_cast_brute(const TriRec* __restrict__ tri, int n_faces,
                                                               const float* __restrict__ rays6, long n_rays,
                                                               int32_t* __restrict__ hit_face,
                                                               float* __restrict__ hit_point)
{
  __shared__ TriRec tile[kBruteTile];
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const bool live = i < n_rays;
  float3 o = f3(0.f, 0.f, 0.f), e = f3(0.f, 0.f, 0.f);
  if (live) {
    const float* r = rays6 + 6 * i;
    o = f3(r[0], r[1], r[2]);
    e = f3(r[3], r[4], r[5]);
  }
  const float3 dir = sub3(e, o);
  float best = 3.40282347e+38f;
  int best_idx = -1;
  float3 best_pt = f3(NAN, NAN, NAN);
  for (int base = 0; base < n_faces; base += kBruteTile) {
    __syncthreads();
    for (int k = threadIdx.x; k < kBruteTile && base + k < n_faces; k += blockDim.x)
      tile[k] = tri[base + k];
    __syncthreads();
    const int m = min(kBruteTile, n_faces - base);
    if (live) {
      for (int k = 0; k < m; ++k) {
        float3 pt;
        if (tri_hit(reinterpret_cast<const float4*>(tile + k), o, dir, pt)) {
          const float d = dist2(pt, o);
          if (d < best) {
            best = d;
            best_idx = base + k;
            best_pt = pt;
          }
        }
      }
    }
  }
  if (live) {
    hit_face[i] = best_idx;
    if (hit_point) {
      hit_point[3 * i + 0] = best_pt.x;
      hit_point[3 * i + 1] = best_pt.y;
      hit_point[3 * i + 2] = best_pt.z;
    }
  }
}

// Materialises the emission rays (packed face by face, front then rear, as
// emission/malley_cpu.cpp:142-189 packs them).  ray_offsets[f] is the first
// ray of face f (n_faces + 1 entries).
__global__ void k_emit(const float* __restrict__ frames, const long long* __restrict__ ray_offsets,
                       const int32_t* __restrict__ front, int n_faces, long n_rays, uint32_t key0, uint32_t key1,
                       uint32_t epoch, float* __restrict__ rays6)
{
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n_rays; i += (long)gridDim.x * blockDim.x) {
    int lo = 0, hi = n_faces;  // largest f with ray_offsets[f] <= i
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (ray_offsets[mid] <= i)
        lo = mid;
      else
        hi = mid;
    }
    const int f = lo;
    const uint32_t j = (uint32_t)(i - ray_offsets[f]);
    float3 o, e;
    emit_ray(frames + 20 * (size_t)f, (uint32_t)f, j, front[f], key0, key1, epoch, o, e);
    float* r = rays6 + 6 * i;
    r[0] = o.x; r[1] = o.y; r[2] = o.z;
    r[3] = e.x; r[4] = e.y; r[5] = e.z;
  }
}

// Per-mesh normalisation of the counts (cpuFactorsCalculator/cpu_system.cpp
// :193-195): ff[m][j] = (float)count[m][j] * (1.f / (float)outgoing[m]) for
// `rows` rows of n_cols entries (outgoing indexed from the first of them).
__global__ void k_normalise(const uint32_t* __restrict__ counts, const int32_t* __restrict__ outgoing, int rows,
                            int n_cols, float* __restrict__ ff)
{
  const size_t n = (size_t)rows * n_cols;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const int m = (int)(i / n_cols);
    const float ratio = 1.f / (float)outgoing[m];
    ff[i] = (float)counts[i] * ratio;
  }
}

}  // namespace ffb
