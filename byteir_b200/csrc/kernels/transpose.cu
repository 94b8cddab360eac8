// TransposeOp for sm_100a: batched 2-D transpose  [batch, rows, cols] ->
// [batch, cols, rows], which covers the reference's 2-D kernel and its two 4-D
// NCHW <-> NHWC permutations, plus a general permutation fallback.
//
// Fast path (2- and 4-byte elements, row pitches multiples of 16 bytes): a
// persistent block walks over 128-byte x 128-byte tiles.  TMA loads a tile into
// shared memory in the 128-byte swizzled layout, the block transposes it out of
// shared memory through registers into a second swizzled tile, and TMA stores
// that tile; loads of the next tile and stores of the previous one overlap the
// shuffle.  With the swizzle both the column-wise reads and the 16-byte writes
// are free of bank conflicts.  Out-of-range parts of edge tiles are zero-filled
// on load and clipped on store by the TMA unit.
//
// Matrices with one short side, and pitches that TMA does not take, have kernels
// of plain loads and stores below.
#include <algorithm>
#include <vector>

#include "common.cuh"
#include "tma.cuh"

namespace b200 {
namespace {

// =============================================================================
// TMA path
// =============================================================================
constexpr int kMaxInStages = 6;
constexpr int kOutStages = 2;
// Input tiles a block keeps in its ring (loads run in_stages - 1 tiles ahead), blocks per SM of the
// persistent grid, and the width of a panel of the tile order; 0 = the rule in launch_tma.
// b200_transpose_tune sets them for measurements.  Measured (TB/s of bytes read + written; ring depth /
// blocks per SM): bf16 8192 x 8192: 2/6 4.3, 3/5 5.2, 4/4 5.4; f16 [32] x 128 x 4096: 2/6 4.2, 3/5 6.4,
// 4/4 6.2; f16 1000 x 30000 (panels of 16): 3/5 5.6, 4/4 5.9, row-major order 4.5 / 4.8; f32 4096 x 4096 with
// tiles of 64 rows (two output tiles per input tile): 2/6 4.3, 3/5 6.0, 4/4 6.0 (with tiles of 32 rows: 4.9 at best).
int g_in_stages = 0, g_blocks_per_sm = 0, g_panel = 0;

// byte offset of 16-byte chunk `chunk` (0..7) of tile row `row` in the 128-byte
// swizzled layout the TMA unit reads and writes
__device__ __forceinline__ uint32_t swz(int row, int chunk) {
  return (uint32_t)row * 128u + (uint32_t)((chunk ^ (row & 7)) << 4);
}

template <int ES> // element size: 2 or 4
__global__ void __launch_bounds__(256)
    transpose_tma_kernel(const __grid_constant__ CUtensorMap in_map,
                         const __grid_constant__ CUtensorMap out_map, int tiles_c, int tiles_r,
                         int64_t num_tiles, int in_stages, int panel, int64_t rows, int *error) {
  constexpr int TC = 128 / ES; // tile columns = elements per 128-byte row
  constexpr int TR = 64;       // tile rows
  constexpr int TRo = 128 / ES; // elements of an output row that one 128-byte swizzled row holds
  constexpr int H = TR / TRo;  // output tiles per input tile: TC rows of TRo elements each (1, or 2 for 4-byte elements)
  constexpr uint32_t kInBytes = TR * 128;  // TR rows of 128 bytes
  constexpr uint32_t kOutHalf = TC * 128;  // TC rows of 128 bytes
  constexpr uint32_t kOutBytes = H * kOutHalf;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  // 1024-byte alignment is what the 128-byte swizzle pattern repeats on
  unsigned char *smem = reinterpret_cast<unsigned char *>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char *in_tile = smem;
  unsigned char *out_tile = smem + in_stages * kInBytes;
  __shared__ uint64_t full[kMaxInStages];

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    prefetch_tensormap(&in_map);
    prefetch_tensormap(&out_map);
    for (int s = 0; s < in_stages; ++s)
      mbar_init(&full[s], 1);
    mbar_fence_init();
  }
  __syncthreads();

  const int64_t my_tiles = (num_tiles - blockIdx.x + gridDim.x - 1) / gridDim.x;
  // Tile order inside one matrix: panels of `panel` tile columns, row-major inside a panel.  The tiles
  // in flight at one time (a contiguous range of the order) then cover a roughly square region, so that
  // the loads AND the stores fall on a few kilobytes of every memory row they touch; in plain row-major
  // order the stores of the tiles in flight are 128-byte pieces of thousands of output rows.
  const int per_matrix = tiles_c * tiles_r;
  const int full_panels = tiles_c / panel;
  auto coords = [&](int64_t k, int &b, int &tr, int &tc) {
    const int64_t tile = blockIdx.x + k * gridDim.x;
    b = (int)(tile / per_matrix);
    const int t = (int)(tile - (int64_t)b * per_matrix);
    const int p = min(t / (panel * tiles_r), full_panels);
    const int width = p < full_panels ? panel : tiles_c - full_panels * panel;
    const int u = t - p * panel * tiles_r;
    tr = u / width;
    tc = p * panel + u - tr * width;
  };
  // Thread 0 issues the loads and thread 32 the stores.  Each works out the coordinates of its next
  // tile (a few integer divisions) while it would otherwise wait, so that no division sits between the
  // arrival of a tile and the issue of the next load.
  int nb = 0, ntr = 0, ntc = 0; // thread 0: coordinates of the next tile to load
  int64_t next_load = 0;
  int load_stage = 0; // stage of the next load (counted, not divided: the ring depth is a run-time value)
  auto issue_next = [&]() {
    mbar_arrive_expect_tx(&full[load_stage], kInBytes);
    tma_load_3d(in_tile + load_stage * kInBytes, &in_map, ntc * TC, ntr * TR, nb, &full[load_stage]);
    load_stage = load_stage + 1 == in_stages ? 0 : load_stage + 1;
    ++next_load;
    if (next_load < my_tiles)
      coords(next_load, nb, ntr, ntc);
  };

  // The first tiles of this block are hinted into L2 before the wait for the kernel in front of this
  // one (a hint returns nothing, and L2 is the point of coherence, so it is harmless even if that kernel
  // is still writing the input): the DRAM fetch then overlaps the other kernel's tail.
  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    for (int64_t k = 0; k < my_tiles && k < 2; ++k) {
      int b, tr, tc;
      coords(k, b, tr, tc);
      tma_prefetch_3d(&in_map, tc * TC, tr * TR, b);
    }
    if (my_tiles > 0)
      coords(0, nb, ntr, ntc);
  }
  pdl_wait();
  const int ahead = in_stages - 1;
  if (threadIdx.x == 0)
    for (int64_t k = 0; k < my_tiles && k < ahead; ++k)
      issue_next();

  int s = 0;          // stage of tile k
  uint32_t phase = 0; // parity of its barrier
  for (int64_t k = 0; k < my_tiles; ++k) {
    const int so = (int)(k % kOutStages);
    int sb = 0, str = 0, stc = 0; // thread 32: where tile k goes
    if (threadIdx.x == 32) {
      bulk_wait_read<kOutStages - 1>(); // the store that last read out_tile[so] is done
      coords(k, sb, str, stc);
    }
    const bool arrived = mbar_wait(&full[s], phase);
    // block-wide agreement (and the barrier after which tile k-1's input stage
    // may be refilled, which is where tile k + ahead goes): if the tile never arrived,
    // all threads leave together
    if (!__syncthreads_and(arrived)) {
      if (error)
        *error = 2;
      break;
    }
    if (threadIdx.x == 0 && next_load < my_tiles)
      issue_next();

    const unsigned char *src = in_tile + s * kInBytes;
    unsigned char *dst = out_tile + so * kOutBytes;
    if (ES == 2) {
      // thread: columns c, c+1 (c = 2 * lane) x rows 8 * warp .. 8 * warp + 7
      const int c = 2 * lane, r0 = 8 * warp;
      uint32_t w[8];
#pragma unroll
      for (int i = 0; i < 8; ++i)
        w[i] = *reinterpret_cast<const uint32_t *>(src + swz(r0 + i, c >> 3) + ((c & 7) << 1));
      uint4 even, odd; // output rows c and c + 1, elements r0 .. r0 + 7
      even.x = __byte_perm(w[0], w[1], 0x5410);
      even.y = __byte_perm(w[2], w[3], 0x5410);
      even.z = __byte_perm(w[4], w[5], 0x5410);
      even.w = __byte_perm(w[6], w[7], 0x5410);
      odd.x = __byte_perm(w[0], w[1], 0x7632);
      odd.y = __byte_perm(w[2], w[3], 0x7632);
      odd.z = __byte_perm(w[4], w[5], 0x7632);
      odd.w = __byte_perm(w[6], w[7], 0x7632);
      // half of each quarter-warp writes its odd row first, so that the eight
      // 16-byte stores of a quarter-warp fall into eight different bank groups
      if (lane & 4) {
        *reinterpret_cast<uint4 *>(dst + swz(c + 1, warp)) = odd;
        *reinterpret_cast<uint4 *>(dst + swz(c, warp)) = even;
      } else {
        *reinterpret_cast<uint4 *>(dst + swz(c, warp)) = even;
        *reinterpret_cast<uint4 *>(dst + swz(c + 1, warp)) = odd;
      }
    } else {
      // thread: column c = lane x rows 4 * warp .. 4 * warp + 3 of each 32-row half of the tile
      const int c = lane;
#pragma unroll
      for (int h = 0; h < H; ++h) {
        const int r0 = h * TRo + 4 * warp;
        uint4 v;
        v.x = *reinterpret_cast<const uint32_t *>(src + swz(r0 + 0, c >> 2) + ((c & 3) << 2));
        v.y = *reinterpret_cast<const uint32_t *>(src + swz(r0 + 1, c >> 2) + ((c & 3) << 2));
        v.z = *reinterpret_cast<const uint32_t *>(src + swz(r0 + 2, c >> 2) + ((c & 3) << 2));
        v.w = *reinterpret_cast<const uint32_t *>(src + swz(r0 + 3, c >> 2) + ((c & 3) << 2));
        *reinterpret_cast<uint4 *>(dst + h * kOutHalf + swz(c, warp)) = v;
      }
    }
    fence_proxy_async_smem();
    __syncthreads();
    if (threadIdx.x == 32) {
#pragma unroll
      for (int h = 0; h < H; ++h)
        if ((int64_t)str * TR + h * TRo < rows) // a store that would start past the end of the rows is left out
          tma_store_3d(&out_map, dst + h * kOutHalf, str * TR + h * TRo, stc * TC, sb);
      bulk_commit();
    }
    if (++s == in_stages) {
      s = 0;
      phase ^= 1u;
    }
  }
  if (threadIdx.x == 32)
    bulk_wait_all<0>();
}

template <int ES>
int launch_tma(const void *in, void *out, int64_t batch, int64_t rows, int64_t cols,
               cudaStream_t stream) {
  constexpr int TC = 128 / ES;
  constexpr int TR = 64;
  constexpr int TRo = 128 / ES;
  CUtensorMap in_map, out_map;
  const CUtensorMapDataType dt = ES == 2 ? CU_TENSOR_MAP_DATA_TYPE_UINT16 : CU_TENSOR_MAP_DATA_TYPE_UINT32;
  {
    const uint64_t dims[3] = {(uint64_t)cols, (uint64_t)rows, (uint64_t)batch};
    const uint64_t strides[2] = {(uint64_t)cols * ES, (uint64_t)rows * cols * ES};
    const uint32_t box[3] = {TC, TR, 1};
    if (int rc = make_tensor_map(&in_map, dt, 3, const_cast<void *>(in), dims, strides, box,
                                 CU_TENSOR_MAP_SWIZZLE_128B))
      return rc;
  }
  {
    const uint64_t dims[3] = {(uint64_t)rows, (uint64_t)cols, (uint64_t)batch};
    const uint64_t strides[2] = {(uint64_t)rows * ES, (uint64_t)rows * cols * ES};
    const uint32_t box[3] = {TRo, TC, 1};
    if (int rc = make_tensor_map(&out_map, dt, 3, out, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B))
      return rc;
  }
  const int tiles_c = (int)ceil_div<int64_t>(cols, TC);
  const int tiles_r = (int)ceil_div<int64_t>(rows, TR);
  const int64_t num_tiles = (int64_t)tiles_c * tiles_r * batch;
  // large matrices: four tiles in the ring and four blocks per SM; everything else three and five
  const bool deep = (int64_t)tiles_c * tiles_r >= 4096;
  const int in_stages = g_in_stages > 0 ? std::max(2, std::min(g_in_stages, kMaxInStages)) : (deep ? 4 : 3);
  const int blocks_per_sm = g_blocks_per_sm > 0 ? g_blocks_per_sm : (deep ? 4 : 5);
  const int panel = std::max(1, std::min(g_panel > 0 ? g_panel : 16, tiles_c));
  const size_t smem = (size_t)in_stages * TR * 128 + (size_t)kOutStages * TC * TR * ES + 1024;
  // the attribute belongs to the current device's context: set on every call (a host-side table write)
  if (int rc = check_cuda(cudaFuncSetAttribute(transpose_tma_kernel<ES>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)smem)))
    return rc;
  const unsigned grid = (unsigned)std::min<int64_t>(num_tiles, (int64_t)kNumSMs * blocks_per_sm);
  return launch_pdl(transpose_tma_kernel<ES>, dim3(grid), dim3(256), smem, stream, in_map, out_map, tiles_c, tiles_r,
                    num_tiles, in_stages, panel, rows, (int *)nullptr);
}

// =============================================================================
// paths for every other shape: any element size, any pitch, any alignment
// =============================================================================
template <int ES> struct Raw;
template <> struct Raw<1> { using T = uint8_t; };
template <> struct Raw<2> { using T = uint16_t; };
template <> struct Raw<4> { using T = uint32_t; };
template <> struct Raw<8> { using T = uint64_t; };

// ---- one short side ----------------------------------------------------------
// [batch, rows, cols] with at most kShort rows (or columns): the three planes of an image, a handful of heads.
// A block takes `width` positions along the long side.  On the side where the short dimension is innermost they
// are ONE contiguous run of width * short elements, which moves in 16-byte pieces; on the other side they are
// `short` runs of `width` elements.  The elements change places in shared memory, where a row of the long
// dimension has a pitch of width + 16 bytes.  A 32 x 32 tile uses 3 of 32 lanes on three planes: f32
// [32, 3, 224, 224] -> (0, 2, 3, 1) took 92 us there and takes 7.9 us here (4.9 TB/s); f16 [64, 16, 200, 200], a TMA
// tile three quarters empty before, 82 -> 35 us (4.7 TB/s).
constexpr int kShort = 40;         // longest short side (a 128-byte tile row of the TMA path is a third full there)
constexpr int kShortBytes = 16384; // bytes of one block's piece, at most

// FROM_ROWS: rows is the short side (long runs are read, the interleaved run is written); otherwise cols is.
// VEC: every long run starts on a 16-byte boundary and `len` is a multiple of 16 bytes.
template <int ES, bool FROM_ROWS, bool VEC>
__global__ void __launch_bounds__(256)
    transpose_short_kernel(const void *__restrict__ in_, void *__restrict__ out_, int64_t len, int shorts, int log_width,
                           int64_t pieces, FastDiv by_short) {
  using T = typename Raw<ES>::T;
  constexpr int N = 16 / ES;
  const T *in = static_cast<const T *>(in_);
  T *out = static_cast<T *>(out_);
  extern __shared__ __align__(16) unsigned char short_smem[];
  T *sm = reinterpret_cast<T *>(short_smem);
  const int width = 1 << log_width, pitch = width + N;
  const int64_t batch = blockIdx.x / pieces, first = (blockIdx.x - batch * pieces) << log_width;
  const int here = (int)min((int64_t)width, len - first);
  const int64_t plane = batch * len * shorts;
  const int count = here * shorts;
  pdl_launch_dependents();
  pdl_wait();
  // long runs, shared memory [short][pitch] <-> global [short][len]
  auto long_side = [&](auto &&move_vec, auto &&move_one) {
    if (VEC) {
      const int lv = log_width - (ES == 1 ? 4 : ES == 2 ? 3 : ES == 4 ? 2 : 1); // vectors per run, logarithm
      for (int i = threadIdx.x; i < shorts << lv; i += 256) {
        const int r = i >> lv, c = (i & ((1 << lv) - 1)) * N;
        if (c < here)
          move_vec(sm + r * pitch + c, plane + r * len + first + c);
      }
    } else {
      for (int i = threadIdx.x; i < shorts << log_width; i += 256) {
        const int r = i >> log_width, c = i & (width - 1);
        if (c < here)
          move_one(sm + r * pitch + c, plane + r * len + first + c);
      }
    }
  };
  // the contiguous run: elements before the first 16-byte boundary one by one, then 16 bytes at a time
  const int64_t run = plane + first * shorts;
  const uintptr_t run_addr = reinterpret_cast<uintptr_t>((FROM_ROWS ? static_cast<const T *>(out) : in) + run);
  const int head = min(count, (int)(((16 - (run_addr & 15)) & 15) / ES));
  const int vecs = (count - head) / N;
  auto at = [&](int o, int &c, int &r) {
    c = (int)by_short.quot((uint32_t)o);
    r = o - c * shorts;
  };
  if (FROM_ROWS) {
    long_side([&](T *s, int64_t g) { *reinterpret_cast<uint4 *>(s) = ld_nc_v4(in + g); }, [&](T *s, int64_t g) { *s = in[g]; });
    __syncthreads();
    for (int v = threadIdx.x; v < vecs; v += 256) {
      int c, r;
      at(head + v * N, c, r);
      union { T e[N]; uint4 q; } u;
#pragma unroll
      for (int k = 0; k < N; ++k) {
        u.e[k] = sm[r * pitch + c];
        if (++r == shorts)
          r = 0, ++c;
      }
      *reinterpret_cast<uint4 *>(out + run + head + v * N) = u.q;
    }
    const int rest = count - vecs * N; // head and tail
    for (int i = threadIdx.x; i < rest; i += 256) {
      const int o = i < head ? i : i + vecs * N;
      int c, r;
      at(o, c, r);
      out[run + o] = sm[r * pitch + c];
    }
  } else {
    for (int v = threadIdx.x; v < vecs; v += 256) {
      int c, r;
      at(head + v * N, c, r);
      union { T e[N]; uint4 q; } u;
      u.q = ld_nc_v4(in + run + head + v * N);
#pragma unroll
      for (int k = 0; k < N; ++k) {
        sm[r * pitch + c] = u.e[k];
        if (++r == shorts)
          r = 0, ++c;
      }
    }
    const int rest = count - vecs * N;
    for (int i = threadIdx.x; i < rest; i += 256) {
      const int o = i < head ? i : i + vecs * N;
      int c, r;
      at(o, c, r);
      sm[r * pitch + c] = in[run + o];
    }
    __syncthreads();
    long_side([&](T *s, int64_t g) { *reinterpret_cast<uint4 *>(out + g) = *reinterpret_cast<const uint4 *>(s); },
              [&](T *s, int64_t g) { out[g] = *s; });
  }
}

// ---- tiles of plain loads -----------------------------------------------------
// Both sides longer than kShort and a pitch that TMA does not take (not a multiple of 16 bytes).  One tile of
// 64 x 64 elements per block (64 x 32 for 8 bytes), all 16 loads of a thread in flight at once; several blocks per SM
// overlap one another's loads and stores.  Two-byte elements move in pairs on the sides whose pitch is even (PAIR_IN,
// PAIR_OUT).  The pitch of the shared tile is an odd number of 32-bit words.  Bound by memory for 4 bytes, by the number
// of load and store instructions (64 bytes each) where 2-byte elements cannot be paired.  Against 32 x 32 tiles with
// four loads in flight: f32 [5001, 7003] 74 -> 50 us (5.6 TB/s), bf16 [5002, 7004] 66 -> 31 us (4.6 TB/s), bf16
// [8191, 8193] 123 -> 65 us (4.2 TB/s).
template <int ES, bool PAIR_IN, bool PAIR_OUT>
__global__ void __launch_bounds__(256, 6)
    transpose_tile_kernel(const void *__restrict__ in_, void *__restrict__ out_, int64_t rows, int64_t cols, int tiles_c,
                          int tiles_r, int64_t batch, int panel) {
  using T = typename Raw<ES>::T;
  constexpr int TR = 64, TC = ES <= 4 ? 64 : 32;
  constexpr int WI = PAIR_IN ? 2 : 1, WO = PAIR_OUT ? 2 : 1; // elements per load / store
  using LT = typename Raw<ES * WI>::T;
  using ST = typename Raw<ES * WO>::T;
  constexpr int PITCH = ES == 8 ? TC + 1 : TC + (ES == 4 ? 1 : 4 / ES); // elements; odd in 32-bit words below 8 bytes
  constexpr int LROW = TC / WI;               // loads per tile row
  constexpr int LSTEP = 256 / LROW;           // rows between two loads of a thread
  constexpr int LOADS = TR / LSTEP;           // loads per thread
  constexpr int SROW = TR / WO;               // stores per output row
  constexpr int SSTEP = 256 / SROW;
  constexpr int STORES = TC / SSTEP;
  __shared__ __align__(16) T tile[TR * PITCH];
  const T *in = static_cast<const T *>(in_);
  T *out = static_cast<T *>(out_);
  // the panel order of the TMA path
  const int t = (int)blockIdx.x, full_panels = tiles_c / panel;
  const int p = min(t / (panel * tiles_r), full_panels);
  const int w = p < full_panels ? panel : tiles_c - full_panels * panel;
  const int u = t - p * panel * tiles_r;
  const int tr = u / w;
  const int64_t r0 = (int64_t)tr * TR, c0 = (int64_t)(p * panel + u - tr * w) * TC;
  const int nr = (int)min((int64_t)TR, rows - r0), nc = (int)min((int64_t)TC, cols - c0);
  const int lc = threadIdx.x % LROW * WI, lr = threadIdx.x / LROW;
  const int so = threadIdx.x % SROW * WO, sc = threadIdx.x / SROW;
  pdl_launch_dependents();
  pdl_wait();
  const int64_t b = blockIdx.y + (int64_t)blockIdx.z * gridDim.y;
  if (b >= batch)
    return;
  // addresses advance by addition: sixteen precomputed 64-bit addresses on either side cost 190 registers a thread
  const T *src = in + b * rows * cols + (r0 + lr) * cols + c0 + lc;
  const int64_t lstep = LSTEP * cols, sstep = SSTEP * rows;
  LT reg[LOADS];
  if (nr == TR && nc == TC) {
#pragma unroll
    for (int i = 0; i < LOADS; ++i, src += lstep)
      reg[i] = *reinterpret_cast<const LT *>(src);
  } else {
#pragma unroll
    for (int i = 0; i < LOADS; ++i, src += lstep)
      if (lr + i * LSTEP < nr && lc < nc)
        reg[i] = *reinterpret_cast<const LT *>(src);
  }
#pragma unroll
  for (int i = 0; i < LOADS; ++i)
    *reinterpret_cast<LT *>(tile + (lr + i * LSTEP) * PITCH + lc) = reg[i];
  __syncthreads();
  T *dst = out + b * rows * cols + (c0 + sc) * rows + r0 + so;
  const T *from = tile + so * PITCH + sc;
#pragma unroll
  for (int i = 0; i < STORES; ++i, dst += sstep)
    if (sc + i * SSTEP < nc && so < nr) {
      ST v;
      if (WO == 2)
        v = (ST)((uint32_t)from[i * SSTEP] | (uint32_t)from[i * SSTEP + PITCH] << 16);
      else
        v = (ST)from[i * SSTEP];
      *reinterpret_cast<ST *>(dst) = v;
    }
}

template <int ES>
int launch_tile(const void *in, void *out, int64_t batch, int64_t rows, int64_t cols, cudaStream_t stream) {
  constexpr int TR = 64, TC = ES <= 4 ? 64 : 32;
  const int64_t tiles_c = ceil_div<int64_t>(cols, TC), tiles_r = ceil_div<int64_t>(rows, TR);
  if (tiles_c * tiles_r > 0x7fffffffLL)
    return B200_ERR_UNSUPPORTED;
  const int panel = (int)std::min<int64_t>(16, tiles_c);
  const int64_t by = std::min<int64_t>(batch, 65535), bz = ceil_div<int64_t>(batch, by);
  if (bz > 65535)
    return B200_ERR_UNSUPPORTED;
  const dim3 grid((unsigned)(tiles_c * tiles_r), (unsigned)by, (unsigned)bz), block(256);
  auto go = [&](auto kernel) {
    return launch_pdl(kernel, grid, block, 0, stream, in, out, rows, cols, (int)tiles_c, (int)tiles_r, batch, panel);
  };
  if constexpr (ES == 2) {
    // pairs of 2-byte elements: the pitch is even and the matrix starts on a 4-byte boundary
    const bool pin = cols % 2 == 0 && reinterpret_cast<uintptr_t>(in) % 4 == 0;
    const bool pout = rows % 2 == 0 && reinterpret_cast<uintptr_t>(out) % 4 == 0;
    if (pin && pout)
      return go(transpose_tile_kernel<2, true, true>);
    if (pin)
      return go(transpose_tile_kernel<2, true, false>);
    if (pout)
      return go(transpose_tile_kernel<2, false, true>);
  }
  return go(transpose_tile_kernel<ES, false, false>);
}

template <int ES>
int launch_short(const void *in, void *out, int64_t batch, int64_t rows, int64_t cols, cudaStream_t stream) {
  const bool from_rows = rows <= cols;
  const int shorts = (int)(from_rows ? rows : cols);
  const int64_t len = from_rows ? cols : rows;
  // a power of two of positions, at least one vector and at most kShortBytes; fewer where that leaves SMs idle
  int lw = 4;
  while ((2ll << lw) * shorts * ES <= kShortBytes && (1ll << lw) < len && batch * ceil_div<int64_t>(len, 2ll << lw) >= 2 * kNumSMs)
    ++lw;
  const int64_t pieces = ceil_div<int64_t>(len, 1ll << lw);
  if (batch * pieces > 0x7fffffffLL) // more pieces than a grid dimension has blocks: tiles, the batch in two dimensions
    return launch_tile<ES>(in, out, batch, rows, cols, stream);
  const size_t smem = (size_t)shorts * ((1 << lw) + 16 / ES) * ES;
  const bool vec = len * ES % 16 == 0 && aligned16(from_rows ? in : out);
  const FastDiv div((uint32_t)shorts);
  const dim3 grid((unsigned)(batch * pieces)), block(256);
  if (from_rows)
    return vec ? launch_pdl(transpose_short_kernel<ES, true, true>, grid, block, smem, stream, in, out, len, shorts, lw, pieces, div)
               : launch_pdl(transpose_short_kernel<ES, true, false>, grid, block, smem, stream, in, out, len, shorts, lw, pieces, div);
  return vec ? launch_pdl(transpose_short_kernel<ES, false, true>, grid, block, smem, stream, in, out, len, shorts, lw, pieces, div)
             : launch_pdl(transpose_short_kernel<ES, false, false>, grid, block, smem, stream, in, out, len, shorts, lw, pieces, div);
}

template <int ES>
int launch_plain(const void *in, void *out, int64_t batch, int64_t rows, int64_t cols, cudaStream_t stream) {
  return std::min(rows, cols) <= kShort ? launch_short<ES>(in, out, batch, rows, cols, stream)
                                        : launch_tile<ES>(in, out, batch, rows, cols, stream);
}

// ---- general permutation --------------------------------------------------------
// One thread per unit of the output, in output order; reads through strides.  A unit is one element, or 1 to 16
// bytes of the innermost dimension where that one stays innermost ([B, S, H, D] -> [B, H, S, D]): then a row of D
// elements is copied in the widest pieces that its length and the pointers allow, kUnits of them in flight per thread:
// bf16 [8, 4096, 32, 128] -> (0, 2, 1, 3) 1074 us element by element with 64-bit divisions, 82 us here (6.6 TB/s).
struct PermuteDims {
  int rank;
  int64_t src_stride[8]; // in units
  FastDiv div[8];        // output sizes, for totals below 2^31 units
  int64_t out_shape[8];
};
constexpr int kUnits = 4;

template <typename T, typename I>
__device__ __forceinline__ int64_t permute_source(const PermuteDims &d, I i) {
  int64_t off = 0;
#pragma unroll
  for (int k = 7; k > 0; --k)
    if (k < d.rank) {
      const I q = sizeof(I) == 4 ? (I)d.div[k].quot((uint32_t)i) : (I)(i / (I)d.out_shape[k]);
      off += (int64_t)(i - q * (I)d.out_shape[k]) * d.src_stride[k];
      i = q;
    }
  return off + (int64_t)i * d.src_stride[0];
}

template <typename T, typename I>
__global__ void __launch_bounds__(256)
    permute_kernel(const T *__restrict__ in, T *__restrict__ out, const __grid_constant__ PermuteDims d, int64_t n) {
  const int64_t base = (int64_t)blockIdx.x * (256 * kUnits) + threadIdx.x;
  pdl_launch_dependents();
  int64_t src[kUnits];
#pragma unroll
  for (int u = 0; u < kUnits; ++u)
    src[u] = base + u * 256 < n ? permute_source<T, I>(d, (I)(base + u * 256)) : 0;
  pdl_wait();
  T v[kUnits];
#pragma unroll
  for (int u = 0; u < kUnits; ++u)
    if (base + u * 256 < n)
      v[u] = in[src[u]];
#pragma unroll
  for (int u = 0; u < kUnits; ++u)
    if (base + u * 256 < n)
      out[base + u * 256] = v[u];
}

template <typename T>
int launch_permute(const void *in, void *out, const PermuteDims &d, int64_t n, cudaStream_t stream) {
  const int64_t grid = ceil_div<int64_t>(n, 256 * kUnits);
  if (grid > 0x7fffffffLL)
    return B200_ERR_UNSUPPORTED;
  if (n < (1LL << 31))
    return launch_pdl(permute_kernel<T, uint32_t>, dim3((unsigned)grid), dim3(256), 0, stream, (const T *)in, (T *)out, d, n);
  return launch_pdl(permute_kernel<T, int64_t>, dim3((unsigned)grid), dim3(256), 0, stream, (const T *)in, (T *)out, d, n);
}

} // namespace
} // namespace b200

using namespace b200;

extern "C" void b200_transpose_tune(int in_stages, int blocks_per_sm, int panel) {
  g_panel = panel;
  g_in_stages = in_stages;
  g_blocks_per_sm = blocks_per_sm;
}

extern "C" int b200_transpose_batched_path(int path, int elt_bytes, const void *in, void *out,
                                           int64_t batch, int64_t rows, int64_t cols,
                                           cudaStream_t stream) {
  if (batch < 0 || rows < 0 || cols < 0)
    return B200_ERR_INVALID_ARG;
  if (batch == 0 || rows == 0 || cols == 0)
    return B200_OK;
  if (!in || !out || in == out)
    return B200_ERR_INVALID_ARG;
  if (rows == 1 || cols == 1) // a transpose that moves nothing
    return check_cuda(cudaMemcpyAsync(out, in, (size_t)batch * rows * cols * elt_bytes,
                                      cudaMemcpyDeviceToDevice, stream));
  const bool tma_ok = (elt_bytes == 2 || elt_bytes == 4) && aligned16(in) && aligned16(out) &&
                      (cols * elt_bytes) % 16 == 0 && (rows * elt_bytes) % 16 == 0 &&
                      rows < (1LL << 31) && cols < (1LL << 31) && batch < (1LL << 31) &&
                      get_encode_tiled() != nullptr;
  if (path == 1 && !tma_ok)
    return B200_ERR_ALIGNMENT;
  if ((path == 0 && tma_ok && std::min(rows, cols) > kShort) || path == 1)
    return elt_bytes == 2 ? launch_tma<2>(in, out, batch, rows, cols, stream)
                          : launch_tma<4>(in, out, batch, rows, cols, stream);
  switch (elt_bytes) {
  case 1:
    return launch_plain<1>(in, out, batch, rows, cols, stream);
  case 2:
    return launch_plain<2>(in, out, batch, rows, cols, stream);
  case 4:
    return launch_plain<4>(in, out, batch, rows, cols, stream);
  case 8:
    return launch_plain<8>(in, out, batch, rows, cols, stream);
  default:
    return B200_ERR_UNSUPPORTED;
  }
}

extern "C" int b200_transpose_batched(int elt_bytes, const void *in, void *out, int64_t batch,
                                      int64_t rows, int64_t cols, cudaStream_t stream) {
  return b200_transpose_batched_path(0, elt_bytes, in, out, batch, rows, cols, stream);
}

extern "C" int b200_permute(int elt_bytes, const void *in, void *out, int rank, const int64_t *shape,
                            const int64_t *perm, cudaStream_t stream) {
  if (rank < 1 || rank > 8 || !shape || !perm)
    return B200_ERR_INVALID_ARG;
  bool seen[8] = {false};
  int64_t n = 1;
  for (int k = 0; k < rank; ++k) {
    if (perm[k] < 0 || perm[k] >= rank || seen[perm[k]] || shape[k] < 0)
      return B200_ERR_INVALID_ARG;
    seen[perm[k]] = true;
    n *= shape[k];
  }
  if (n == 0)
    return B200_OK;
  if (!in || !out)
    return B200_ERR_INVALID_ARG;
  // Drop size-1 dims, then merge input dims that stay adjacent and in order in
  // the output.  Work in output order: entry k is input dim p[k].
  int compact[8], next_id = 0; // input dim -> its position among the kept dims
  for (int i = 0; i < rank; ++i)
    compact[i] = shape[i] != 1 ? next_id++ : -1;
  std::vector<int64_t> p, s; // permutation entry and its size, output order
  for (int k = 0; k < rank; ++k)
    if (shape[perm[k]] != 1) {
      p.push_back(compact[perm[k]]);
      s.push_back(shape[perm[k]]);
    }
  std::vector<int64_t> mp, ms;
  for (size_t k = 0; k < p.size(); ++k) {
    if (!mp.empty() && p[k] == p[k - 1] + 1) {
      ms.back() *= s[k];
      // the merged group keeps the id of its first input dim
    } else {
      mp.push_back(p[k]);
      ms.push_back(s[k]);
    }
  }
  const size_t g = mp.size();
  // rank of each group in input order
  std::vector<int> order(g);
  for (size_t k = 0; k < g; ++k) {
    int r = 0;
    for (size_t j = 0; j < g; ++j)
      if (mp[j] < mp[k])
        ++r;
    order[k] = r;
  }
  if (g <= 1)
    return check_cuda(cudaMemcpyAsync(out, in, (size_t)n * elt_bytes, cudaMemcpyDeviceToDevice, stream));
  if (g == 2) // (1, 0)
    return b200_transpose_batched(elt_bytes, in, out, 1, ms[1], ms[0], stream);
  if (g == 3 && order[0] == 0 && order[1] == 2 && order[2] == 1) // (0, 2, 1)
    return b200_transpose_batched(elt_bytes, in, out, ms[0], ms[2], ms[1], stream);
  // general case
  if (elt_bytes != 1 && elt_bytes != 2 && elt_bytes != 4 && elt_bytes != 8)
    return B200_ERR_UNSUPPORTED;
  std::vector<int64_t> in_sizes(g), in_strides(g); // of the merged input dims
  for (size_t k = 0; k < g; ++k)
    in_sizes[order[k]] = ms[k];
  int64_t st = 1;
  for (int i = (int)g - 1; i >= 0; --i) {
    in_strides[i] = st;
    st *= in_sizes[i];
  }
  // widest unit of the innermost dimension, if that stays innermost
  int unit = elt_bytes;
  if (order[g - 1] == (int)g - 1)
    while (unit < 16 && ms[g - 1] * elt_bytes % (2 * unit) == 0 &&
           ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & (2 * unit - 1)) == 0)
      unit *= 2;
  const int64_t per_unit = unit / elt_bytes;
  PermuteDims d{};
  d.rank = (int)g;
  for (size_t k = 0; k < g; ++k) {
    const bool inner = k + 1 == g;
    d.out_shape[k] = inner ? ms[k] / per_unit : ms[k];
    d.src_stride[k] = inner ? in_strides[order[k]] : in_strides[order[k]] / per_unit;
    d.div[k] = FastDiv((uint32_t)std::min<int64_t>(d.out_shape[k], 0x7fffffff));
  }
  n /= per_unit;
  switch (unit) {
  case 1:
    return launch_permute<uint8_t>(in, out, d, n, stream);
  case 2:
    return launch_permute<uint16_t>(in, out, d, n, stream);
  case 4:
    return launch_permute<uint32_t>(in, out, d, n, stream);
  case 8:
    return launch_permute<uint64_t>(in, out, d, n, stream);
  case 16:
    return launch_permute<uint4>(in, out, d, n, stream);
  default:
    return B200_ERR_UNSUPPORTED;
  }
}
