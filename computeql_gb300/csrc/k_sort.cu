// ORDER BY: an LSD radix sort of (key, position) pairs, the replacement of the reference's bitonic sorts
// (src/gpu/vulkan/shaders/bitonic_sort*.comp, the generated tiled sort query_kernel.c:2114-2267, driven by
// qe_sort_rows, src/query_exec/query_exec.c:5376-6155).
//
// The reference orders rows by up to 4 keys with ties broken by input position. Here every key is turned
// into an unsigned word whose order is the key's order (sign bits flipped, negative floats complemented,
// -0.0 taken as +0.0, complemented again for DESC), and the keys are sorted least significant first with
// a stable radix sort starting from the identity permutation, so equal keys keep their input order.
// Keys of 32-bit columns travel as 4-byte words, the others as 8-byte words.
//
//  cql_sort_keys      binding 0 source column, 1 permutation (u32), 2 key out, 3 selection (u32 rows),
//                     4 histogram [256][tiles] of the first digit, 5 digit totals [key bytes][256] (4 and 5
//                     with word 14 = 1); word 0 n, word 2 the CQL type, word 4 descending, word 6 1 = gather
//                     through the permutation, word 8 1 = the n positions are the selection's rows, word 10
//                     the column's narrow width (0 full, 1 u8 codes, 2 u16 codes, 3 the row number), word 12
//                     the narrow base (value = base + code, in 32 bits), word 14 flags: 1 = count the first
//                     digit, 2 = write no identity permutation (the first scatter takes row numbers)
//  cql_radix_count    binding 0 keys, 1 histogram [256][tiles], 2 the pass's digit totals [256] (added to);
//                     word 0 n, word 2 bit shift, word 4 key bytes
//  cql_radix_offsets  binding 0 histogram [256][tiles], 1 the pass's digit totals [256], 2 offsets out
//                     [256][tiles] (where each (digit, tile) run starts in the pass's output); word 0 n
//  cql_radix_scatter  binding 0 keys in, 1 positions in, 2 keys out, 3 positions out, 4 offsets,
//                     5 selection; word 0 n, word 2 bit shift, word 4 key bytes, word 6 1 = write the
//                     selection's row instead of the position, word 8 1 = write no keys (the last pass),
//                     word 10 1 = the positions in are the row numbers (binding 1 is not read); binding 6
//                     (optional) the pass's digit totals: one digit holding all n rows makes the pass a copy
//  cql_pairs_unpack   binding 0 records (u32 words), 1 first out, 2 second out; word 0 n, word 2 words per
//                     record, word 4 the first's word offset, word 6 the second's
//  cql_pairs_pack     binding 0 sorted positions, 1 first, 2 second, 3 pairs out (first, second); word 0 n
//                     (result pairs - join or scan output - put in order on the device by the sort above)
//
// A tile is 8 warps x 16 rounds x 32 rows = 4096 rows. The scatter ranks a row within its tile in input
// order: eight ballots or the match instruction (alternate rounds) find the lanes of a round with the same
// digit, per-warp digit counters carry the rounds, and a prefix over the warps orders the warps; the global
// base of (digit, tile) comes from the offsets kernel: the digit's place in the pass's output (the totals of the digits below it, counted
// while the histogram is made) plus the digit's counts in the tiles before.
#include "cql_internal.cuh"
#include <algorithm>

#define SORT_THREADS 256
#define SORT_WARPS (SORT_THREADS / 32)
#define SORT_ROUNDS 16
#define SORT_TILE (SORT_THREADS * SORT_ROUNDS)
#define RADIX 256

__device__ __forceinline__ unsigned long long f64_order(unsigned long long b)
{
  if ((b << 1) == 0) b = 0;  // -0.0 sorts as +0.0
  return (b & 0x8000000000000000ull) ? ~b : (b | 0x8000000000000000ull);
}

// The reference compares every numeric key as an F64 (qe_sort_rows_compare_ctx, query_exec.c:4859-4882):
// 32-bit keys convert exactly, 64-bit integers are rounded to the nearest double first so that values
// that meet in F64 tie (and fall back to their position) as they do there.
__device__ __forceinline__ unsigned long long order_bits(uint32_t type, unsigned long long raw)
{
  switch (type)
  {
    case 1: case 12: return (uint32_t)raw;
    case 7: case 9: return (uint32_t)raw ^ 0x80000000u;
    case 3:
    {
      uint32_t b = (uint32_t)raw;
      if ((b << 1) == 0) b = 0;
      return (b & 0x80000000u) ? (~b & 0xffffffffu) : (b | 0x80000000u);
    }
    case 4: return f64_order(raw);
    case 2: return f64_order(__double_as_longlong((double)raw));
    default: return f64_order(__double_as_longlong((double)(long long)raw));
  }
}

// Counts digits into a histogram a run of equal digits at a time: one shared atomic per run, so a digit
// that does not vary (the high bytes of small keys, the low bytes of whole-number doubles) costs one atomic
// per thread and tile instead of 32 lanes meeting on one counter for every row.
struct DigitRun
{
  uint32_t digit = 0xffffffffu, count = 0;
  __device__ __forceinline__ void add(uint32_t* hist, uint32_t dg)
  {
    if (dg != digit)
    {
      if (count) atomicAdd(&hist[digit], count);
      digit = dg;
      count = 0;
    }
    count += 1;
  }
  __device__ __forceinline__ void flush(uint32_t* hist)
  {
    if (count) atomicAdd(&hist[digit], count);
  }
};

// The keys of one tile in sort order; with COUNT, the first digit counted into the warp's histogram. The
// source rows are found first, then the values read (16 loads in flight a thread), then turned into keys.
template <typename K, bool PARTIAL, bool COUNT>
__device__ __forceinline__ void keys_tile(const CqlLaunch& a, uint64_t n, uint64_t src_rows, uint32_t tile, uint32_t* warp_hist)
{
  const uint32_t* src = (const uint32_t*)a.buf[0];
  uint32_t* perm = (uint32_t*)a.buf[1];
  K* keys = (K*)a.buf[2];
  const uint32_t* sel = (const uint32_t*)a.buf[3];
  uint32_t type = cql_word(a, 2);
  bool desc = cql_word(a, 4) != 0, gather = cql_word(a, 6) != 0, selected = cql_word(a, 8) != 0;
  bool write_identity = !gather && (cql_word(a, 14) & 2u) == 0;
  uint32_t width = cql_word(a, 10), base = cql_word(a, 12);
  uint32_t flip = (type == 7 || type == 9) ? 0x80000000u : 0u;
  uint64_t first = (uint64_t)tile * SORT_TILE;
  uint32_t rows = PARTIAL ? (uint32_t)(n - first) : SORT_TILE;
  uint32_t row[SORT_ROUNDS];
#pragma unroll
  for (uint32_t j = 0; j < SORT_ROUNDS; j++)
  {
    uint32_t o = j * SORT_THREADS + threadIdx.x;
    uint32_t p = (uint32_t)(first + o);
    if (gather && (!PARTIAL || o < rows)) p = perm[first + o];
    row[j] = p;
  }
  if (selected)
  {
#pragma unroll
    for (uint32_t j = 0; j < SORT_ROUNDS; j++)
      if (!PARTIAL || j * SORT_THREADS + threadIdx.x < rows) row[j] = sel[row[j]];
  }
  if (write_identity)
  {
#pragma unroll
    for (uint32_t j = 0; j < SORT_ROUNDS; j++)
    {
      uint32_t o = j * SORT_THREADS + threadIdx.x;
      if (!PARTIAL || o < rows) perm[first + o] = (uint32_t)(first + o);
    }
  }
  K raw[SORT_ROUNDS];
#pragma unroll
  for (uint32_t j = 0; j < SORT_ROUNDS; j++)
  {
    uint32_t o = j * SORT_THREADS + threadIdx.x;
    uint32_t r = row[j];
    K v = 0;
    if ((!PARTIAL || o < rows) && r < src_rows)
    {
      if (sizeof(K) == 8) v = (K)((const unsigned long long*)src)[r];
      else if (width == 0) v = (K)src[r];
      else if (width == 1) v = (K)((const uint8_t*)src)[r];
      else if (width == 2) v = (K)((const uint16_t*)src)[r];
      else v = (K)r;
    }
    raw[j] = v;
  }
  DigitRun run;
#pragma unroll
  for (uint32_t j = 0; j < SORT_ROUNDS; j++)
  {
    uint32_t o = j * SORT_THREADS + threadIdx.x;
    if (PARTIAL && o >= rows) continue;
    unsigned long long k = 0ull;
    if (row[j] < src_rows) k = width == 0 ? order_bits(type, raw[j]) : (unsigned long long)(((uint32_t)raw[j] + base) ^ flip);
    if (desc) k = ~k;
    keys[first + o] = (K)k;
    if (COUNT) run.add(warp_hist, (uint32_t)k & 0xffu);
  }
  if (COUNT) run.flush(warp_hist);
}

template <typename K, bool COUNT>
__global__ void __launch_bounds__(SORT_THREADS) k_sort_keys(CqlLaunch a, uint64_t n, uint64_t src_rows, uint32_t tiles)
{
  __shared__ uint32_t hist[COUNT ? SORT_WARPS : 1][RADIX];
  uint32_t* hist_out = (uint32_t*)a.buf[4];
  uint32_t* totals = (uint32_t*)a.buf[5];
  uint32_t warp = threadIdx.x >> 5, d = threadIdx.x;  // RADIX == SORT_THREADS: thread d sums digit d
  uint32_t full_tiles = (uint32_t)(n / SORT_TILE), cta_total = 0;
  for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x)
  {
    if (COUNT)
    {
      for (uint32_t i = threadIdx.x; i < SORT_WARPS * RADIX; i += SORT_THREADS) (&hist[0][0])[i] = 0;
      __syncthreads();
    }
    if (tile < full_tiles) keys_tile<K, false, COUNT>(a, n, src_rows, tile, hist[COUNT ? warp : 0]);
    else keys_tile<K, true, COUNT>(a, n, src_rows, tile, hist[COUNT ? warp : 0]);
    if (COUNT)
    {
      __syncthreads();
      uint32_t total = 0;
#pragma unroll
      for (uint32_t w = 0; w < SORT_WARPS; w++) total += hist[w][d];
      hist_out[(uint64_t)d * tiles + tile] = total;
      cta_total += total;
      __syncthreads();
    }
  }
  if (COUNT && cta_total) atomicAdd(&totals[d], cta_total);
}

template <typename K, bool PARTIAL>
__device__ __forceinline__ void count_tile(const K* keys, uint64_t n, uint32_t tile, uint32_t shift, uint32_t* warp_hist)
{
  uint64_t first = (uint64_t)tile * SORT_TILE;
  const K* kin = keys + first;
  uint32_t rows = PARTIAL ? (uint32_t)(n - first) : SORT_TILE;
  K k[SORT_ROUNDS];
#pragma unroll
  for (uint32_t j = 0; j < SORT_ROUNDS; j++)
  {
    uint32_t o = j * SORT_THREADS + threadIdx.x;
    k[j] = (!PARTIAL || o < rows) ? kin[o] : (K)0;
  }
  DigitRun run;
#pragma unroll
  for (uint32_t j = 0; j < SORT_ROUNDS; j++)
    if (!PARTIAL || j * SORT_THREADS + threadIdx.x < rows) run.add(warp_hist, (uint32_t)(k[j] >> shift) & 0xffu);
  run.flush(warp_hist);
}

template <typename K>
__global__ void __launch_bounds__(SORT_THREADS) k_radix_count(CqlLaunch a, uint64_t n, uint32_t tiles)
{
  // one histogram per warp (fewer lanes on one shared counter), summed at the end of the tile
  __shared__ uint32_t hist[SORT_WARPS][RADIX];
  const K* keys = (const K*)a.buf[0];
  uint32_t* out = (uint32_t*)a.buf[1];
  uint32_t* totals = (uint32_t*)a.buf[2];
  uint32_t shift = cql_word(a, 2);
  uint32_t warp = threadIdx.x >> 5, d = threadIdx.x;
  uint32_t full_tiles = (uint32_t)(n / SORT_TILE);
  uint32_t cta_total = 0;  // digit d's count over this CTA's tiles (RADIX == SORT_THREADS)
  for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x)
  {
    for (uint32_t i = threadIdx.x; i < SORT_WARPS * RADIX; i += SORT_THREADS) (&hist[0][0])[i] = 0;
    __syncthreads();
    if (tile < full_tiles) count_tile<K, false>(keys, n, tile, shift, hist[warp]);
    else count_tile<K, true>(keys, n, tile, shift, hist[warp]);
    __syncthreads();
    uint32_t total = 0;
#pragma unroll
    for (uint32_t w = 0; w < SORT_WARPS; w++) total += hist[w][d];
    out[(uint64_t)d * tiles + tile] = total;
    cta_total += total;
    __syncthreads();
  }
  if (cta_total) atomicAdd(&totals[d], cta_total);
}

// Where each (digit, tile) run starts in the pass's output: one CTA a digit, the totals of the digits below
// it plus an exclusive scan of its row of the histogram (4 counts a thread, 2048 a step).
#define OFFSETS_THREADS 512
__global__ void __launch_bounds__(OFFSETS_THREADS) k_radix_offsets(CqlLaunch a, uint32_t tiles)
{
  __shared__ uint32_t s_warp[OFFSETS_THREADS / 32];
  const uint32_t* hist = (const uint32_t*)a.buf[0];
  const uint32_t* totals = (const uint32_t*)a.buf[1];
  uint32_t* out = (uint32_t*)a.buf[2];
  uint32_t d = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t below = threadIdx.x < d ? totals[threadIdx.x] : 0u;  // d < RADIX <= OFFSETS_THREADS
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) below += __shfl_xor_sync(0xffffffffu, below, o);
  if (lane == 0) s_warp[warp] = below;
  __syncthreads();
  uint32_t carry = 0;
#pragma unroll
  for (uint32_t w = 0; w < OFFSETS_THREADS / 32; w++) carry += s_warp[w];
  __syncthreads();
  const uint32_t* row = hist + (uint64_t)d * tiles;
  uint32_t* orow = out + (uint64_t)d * tiles;
  for (uint32_t start = 0; start < tiles; start += OFFSETS_THREADS * 4)
  {
    uint32_t j0 = start + threadIdx.x * 4;
    uint32_t v[4], t = 0;
#pragma unroll
    for (uint32_t q = 0; q < 4; q++)
    {
      v[q] = j0 + q < tiles ? row[j0 + q] : 0u;
      t += v[q];
    }
    uint32_t incl = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
      uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= (uint32_t)o) incl += y;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    uint32_t before = 0, step = 0;
#pragma unroll
    for (uint32_t w = 0; w < OFFSETS_THREADS / 32; w++)
    {
      uint32_t c = s_warp[w];
      before += w < warp ? c : 0u;
      step += c;
    }
    uint32_t at = carry + before + incl - t;
#pragma unroll
    for (uint32_t q = 0; q < 4; q++)
    {
      if (j0 + q < tiles) orow[j0 + q] = at;
      at += v[q];
    }
    carry += step;
    __syncthreads();
  }
}

// The scatter of one tile: rank every key within the tile in input order (per-warp counters, lanes of
// one digit found within each 32-row round), place the tile in shared memory in digit order, then write
// it out in that order, so consecutive threads write consecutive places of each digit's run.
//
// The ranking is bound by instruction issue and the latency of its shared-memory chain, so the kernel is
// built for several resident CTAs per SM: only the keys and their ranks live in registers while a tile is
// ranked (the positions are read once the ranks are known), within the register budget of 4 CTAs (3 for
// 8-byte keys). Full tiles take a path without bounds checks; the last, partial tile the checked one.
#define SORT_SCATTER_CTAS(K) (sizeof(K) == 4 ? 4 : 3)

// Ranking forms: the lanes of a round with the same digit found by eight ballots (ALU pipe), by the match
// instruction (its own, slower pipe), or the two in alternate rounds so that both pipes share the work.
#define RANK_BALLOTS 0
#define RANK_MATCH 1
#define RANK_ALTERNATE 2
#ifndef SORT_RANK_FORM
#define SORT_RANK_FORM RANK_ALTERNATE
#endif

// The lanes of the warp whose digit equals this lane's, from one ballot per digit bit; a ninth bit marks
// the lanes past the end in the last, partial tile.
template <bool PARTIAL>
__device__ __forceinline__ uint32_t same_digit_lanes(uint32_t dg)
{
  uint32_t peers = 0xffffffffu;
#pragma unroll
  for (uint32_t b = 0; b < (PARTIAL ? 9u : 8u); b++)
  {
    uint32_t bit = (dg >> b) & 1u;
    uint32_t m = __ballot_sync(0xffffffffu, bit);
    peers &= bit ? m : ~m;
  }
  return peers;
}

template <int FORM, bool PARTIAL>
__device__ __forceinline__ uint32_t round_peers(uint32_t dg, uint32_t r)
{
  if (FORM == RANK_MATCH || (FORM == RANK_ALTERNATE && (r & 1u))) return __match_any_sync(0xffffffffu, dg);
  return same_digit_lanes<PARTIAL>(dg);
}

struct ScatterShared
{
  uint32_t warp_count[SORT_WARPS][RADIX];  // per warp and digit: ranked count, then the place of its first key
  uint32_t off[RADIX];                      // global place of tile place j of the digit: off + j (mod 2^32)
  uint32_t warp_total[SORT_WARPS];
};

template <typename K, bool PARTIAL, int FORM>
__device__ __forceinline__ void scatter_tile(const CqlLaunch& a, ScatterShared& sh, K* s_key, uint32_t* s_pos, uint64_t n, uint32_t tiles,
                                             uint32_t tile, uint32_t shift, bool map_rows, bool write_keys, bool identity)
{
  const K* keys_in = (const K*)a.buf[0];
  const uint32_t* pos_in = (const uint32_t*)a.buf[1];
  K* keys_out = (K*)a.buf[2];
  uint32_t* pos_out = (uint32_t*)a.buf[3];
  const uint32_t* base_of = (const uint32_t*)a.buf[4];
  const uint32_t* sel = (const uint32_t*)a.buf[5];
  uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, d = threadIdx.x;
  uint32_t lt = (1u << lane) - 1u;
  for (uint32_t i = threadIdx.x; i < SORT_WARPS * RADIX; i += SORT_THREADS) (&sh.warp_count[0][0])[i] = 0;
  // each warp owns 16 rounds of 32 consecutive rows; its keys are loaded up front
  uint64_t tile_first = (uint64_t)tile * SORT_TILE;
  uint32_t tile_rows = PARTIAL ? (uint32_t)min((uint64_t)SORT_TILE, n - tile_first) : SORT_TILE;
  uint32_t warp_first = warp * 32 * SORT_ROUNDS;  // within the tile
  const K* kin = keys_in + tile_first + warp_first;
  K key[SORT_ROUNDS];
#pragma unroll
  for (uint32_t r = 0; r < SORT_ROUNDS; r++)
  {
    uint32_t j = warp_first + r * 32 + lane;
    key[r] = (!PARTIAL || j < tile_rows) ? kin[r * 32 + lane] : (K)0;
  }
  uint32_t tile_base = base_of[(uint64_t)d * tiles + tile];
  __syncthreads();
  uint32_t local[SORT_ROUNDS];
#pragma unroll
  for (uint32_t r = 0; r < SORT_ROUNDS; r++)
  {
    uint32_t j = warp_first + r * 32 + lane;
    uint32_t dg = (uint32_t)(key[r] >> shift) & 0xffu;
    if (PARTIAL && j >= tile_rows) dg = RADIX;  // past the end
    uint32_t peers = round_peers<FORM, PARTIAL>(dg, r);
    uint32_t before = (!PARTIAL || dg < RADIX) ? sh.warp_count[warp][dg] : 0u;
    local[r] = before + __popc(peers & lt);
    __syncwarp();
    if ((!PARTIAL || dg < RADIX) && (peers & lt) == 0) sh.warp_count[warp][dg] = before + __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  // per digit (one per thread): the warps before each warp, and the digit's total in the tile
  uint32_t run = 0;
#pragma unroll
  for (uint32_t w = 0; w < SORT_WARPS; w++)
  {
    uint32_t c = sh.warp_count[w][d];
    sh.warp_count[w][d] = run;
    run += c;
  }
  // exclusive scan of the digit totals over the block: where each digit starts in the tile
  uint32_t incl = run;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1)
  {
    uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= (uint32_t)o) incl += y;
  }
  if (lane == 31) sh.warp_total[warp] = incl;
  __syncthreads();
  uint32_t start = incl - run;
  for (uint32_t w = 0; w < warp; w++) start += sh.warp_total[w];
  sh.off[d] = tile_base - start;
  // the place in the tile of each warp's first key of the digit
#pragma unroll
  for (uint32_t w = 0; w < SORT_WARPS; w++) sh.warp_count[w][d] += start;
  __syncthreads();
  // the tile in digit order, in shared memory: the keys, then the positions read now
#pragma unroll
  for (uint32_t r = 0; r < SORT_ROUNDS; r++)
  {
    uint32_t j = warp_first + r * 32 + lane;
    uint32_t dg = (uint32_t)(key[r] >> shift) & 0xffu;
    local[r] += sh.warp_count[warp][dg];
    if (!PARTIAL || j < tile_rows) s_key[local[r]] = key[r];
  }
  const uint32_t* pin = pos_in + tile_first + warp_first;
  uint32_t pos[SORT_ROUNDS];
#pragma unroll
  for (uint32_t r = 0; r < SORT_ROUNDS; r++)
  {
    uint32_t j = warp_first + r * 32 + lane;
    pos[r] = identity ? (uint32_t)(tile_first + j) : (!PARTIAL || j < tile_rows) ? pin[r * 32 + lane] : 0u;
  }
#pragma unroll
  for (uint32_t r = 0; r < SORT_ROUNDS; r++)
  {
    uint32_t j = warp_first + r * 32 + lane;
    if (!PARTIAL || j < tile_rows) s_pos[local[r]] = pos[r];
  }
  __syncthreads();
  // out in order: place j of the tile goes to its digit's global base plus its place in the run
#pragma unroll 4
  for (uint32_t j = threadIdx.x; j < tile_rows; j += SORT_THREADS)
  {
    K k = s_key[j];
    uint32_t dd = (uint32_t)(k >> shift) & 0xffu;
    uint64_t dst = (uint32_t)(sh.off[dd] + j);
    if (dst < n)
    {
      if (write_keys) keys_out[dst] = k;
      uint32_t p = s_pos[j];
      pos_out[dst] = map_rows ? sel[p] : p;
    }
  }
  __syncthreads();
}

// A pass whose digit is the same for every row (a byte that does not vary) leaves the order as it is: the
// keys and positions are copied through, with no ranking.
template <typename K>
__device__ __forceinline__ void pass_copy(const CqlLaunch& a, uint64_t n, bool map_rows, bool write_keys, bool identity)
{
  const K* keys_in = (const K*)a.buf[0];
  const uint32_t* pos_in = (const uint32_t*)a.buf[1];
  K* keys_out = (K*)a.buf[2];
  uint32_t* pos_out = (uint32_t*)a.buf[3];
  const uint32_t* sel = (const uint32_t*)a.buf[5];
  uint64_t stride = (uint64_t)gridDim.x * SORT_THREADS;
#pragma unroll 4
  for (uint64_t i = (uint64_t)blockIdx.x * SORT_THREADS + threadIdx.x; i < n; i += stride)
  {
    if (write_keys) keys_out[i] = keys_in[i];
    uint32_t p = identity ? (uint32_t)i : pos_in[i];
    pos_out[i] = map_rows ? sel[p] : p;
  }
}

template <typename K, int FORM>
__global__ void __launch_bounds__(SORT_THREADS, SORT_SCATTER_CTAS(K)) k_radix_scatter(CqlLaunch a, uint64_t n, uint32_t tiles, bool has_totals)
{
  __shared__ ScatterShared sh;
  __shared__ uint32_t s_one_digit;
  extern __shared__ __align__(16) unsigned char s_tile[];
  K* s_key = (K*)s_tile;
  uint32_t* s_pos = (uint32_t*)(s_tile + sizeof(K) * SORT_TILE);
  uint32_t shift = cql_word(a, 2);
  bool map_rows = cql_word(a, 6) != 0, write_keys = cql_word(a, 8) == 0, identity = cql_word(a, 10) != 0;
  if (has_totals)
  {
    // the pass's digit totals: one digit holding every row makes the pass a copy
    const uint32_t* totals = (const uint32_t*)a.buf[6];
    if (threadIdx.x == 0) s_one_digit = 0;
    __syncthreads();
    if (totals[threadIdx.x] == (uint32_t)n) s_one_digit = 1;  // RADIX == SORT_THREADS; n < 2^32
    __syncthreads();
    if (s_one_digit)
    {
      pass_copy<K>(a, n, map_rows, write_keys, identity);
      return;
    }
  }
  uint32_t full_tiles = (uint32_t)(n / SORT_TILE);
  for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x)
  {
    if (tile < full_tiles) scatter_tile<K, false, FORM>(a, sh, s_key, s_pos, n, tiles, tile, shift, map_rows, write_keys, identity);
    else scatter_tile<K, true, FORM>(a, sh, s_key, s_pos, n, tiles, tile, shift, map_rows, write_keys, identity);
  }
}

// CTAs of SORT_THREADS threads that fit on an SM (1 when the query fails): a tile loop's grid
static int resident_ctas(const void* fn, size_t smem)
{
  int per_sm = 1;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, SORT_THREADS, smem) != cudaSuccess || per_sm < 1)
  {
    cudaGetLastError();
    per_sm = 1;
  }
  return per_sm;
}

static bool sort_type_wide_host(uint32_t type)
{
  return type == 2 || type == 4 || type == 8 || type == 10 || type == 11;
}

static int sort_key_bytes(uint32_t type)
{
  switch (type)
  {
    case 1: case 3: case 7: case 9: case 12: return 4;
    case 2: case 4: case 8: case 10: case 11: return 8;
    default: return 0;
  }
}

static int launch_sort_keys(const CqlLaunch& a, uint32_t gws, uint32_t lws, cudaStream_t stream)
{
  (void)gws;
  (void)lws;
  uint64_t n = cql_word(a, 0);
  uint32_t type = cql_word(a, 2);
  int kb = sort_key_bytes(type);
  if (n == 0) return 0;
  if (!kb || a.bytes[1] < n * 4 || a.bytes[2] < n * (uint64_t)kb) return (int)cudaErrorInvalidValue;
  if (cql_word(a, 8) && a.bytes[3] < n * 4) return (int)cudaErrorInvalidValue;
  uint32_t width = cql_word(a, 10);
  if (width > 3 || (width && sort_type_wide_host(type))) return (int)cudaErrorInvalidValue;
  uint64_t src_rows = width == 3 ? ~0ull : width ? a.bytes[0] / width : a.bytes[0] / (sort_type_wide_host(type) ? 8 : 4);
  uint32_t tiles = (uint32_t)((n + SORT_TILE - 1) / SORT_TILE);
  bool count = (cql_word(a, 14) & 1u) != 0;
  if (count && ((uint64_t)tiles * RADIX * 4 > a.bytes[4] || a.bytes[5] < RADIX * 4)) return (int)cudaErrorInvalidValue;
  const void* fn = kb == 4 ? (count ? (const void*)k_sort_keys<uint32_t, true> : (const void*)k_sort_keys<uint32_t, false>)
                            : (count ? (const void*)k_sort_keys<unsigned long long, true> : (const void*)k_sort_keys<unsigned long long, false>);
  uint32_t grid = cql_stream_grid(tiles, resident_ctas(fn, 0));
  if (kb == 4)
  {
    if (count) k_sort_keys<uint32_t, true><<<grid, SORT_THREADS, 0, stream>>>(a, n, src_rows, tiles);
    else k_sort_keys<uint32_t, false><<<grid, SORT_THREADS, 0, stream>>>(a, n, src_rows, tiles);
  }
  else
  {
    if (count) k_sort_keys<unsigned long long, true><<<grid, SORT_THREADS, 0, stream>>>(a, n, src_rows, tiles);
    else k_sort_keys<unsigned long long, false><<<grid, SORT_THREADS, 0, stream>>>(a, n, src_rows, tiles);
  }
  CQL_LAUNCH_CHECK();
  return 0;
}

static int launch_radix_count(const CqlLaunch& a, uint32_t gws, uint32_t lws, cudaStream_t stream)
{
  (void)gws;
  (void)lws;
  uint64_t n = cql_word(a, 0);
  uint32_t shift = cql_word(a, 2), kb = cql_word(a, 4);
  if (n == 0) return 0;
  uint32_t tiles = (uint32_t)((n + SORT_TILE - 1) / SORT_TILE);
  if ((kb != 4 && kb != 8) || shift >= kb * 8 || a.bytes[0] < n * kb || (uint64_t)tiles * RADIX * 4 > a.bytes[1] || a.bytes[2] < RADIX * 4)
    return (int)cudaErrorInvalidValue;
  uint32_t grid = cql_stream_grid(tiles, resident_ctas(kb == 4 ? (const void*)k_radix_count<uint32_t> : (const void*)k_radix_count<unsigned long long>, 0));
  if (kb == 4) k_radix_count<uint32_t><<<grid, SORT_THREADS, 0, stream>>>(a, n, tiles);
  else k_radix_count<unsigned long long><<<grid, SORT_THREADS, 0, stream>>>(a, n, tiles);
  CQL_LAUNCH_CHECK();
  return 0;
}

static int launch_radix_offsets(const CqlLaunch& a, uint32_t gws, uint32_t lws, cudaStream_t stream)
{
  (void)gws;
  (void)lws;
  uint64_t n = cql_word(a, 0);
  if (n == 0) return 0;
  uint32_t tiles = (uint32_t)((n + SORT_TILE - 1) / SORT_TILE);
  if ((uint64_t)tiles * RADIX * 4 > a.bytes[0] || a.bytes[1] < RADIX * 4 || (uint64_t)tiles * RADIX * 4 > a.bytes[2])
    return (int)cudaErrorInvalidValue;
  k_radix_offsets<<<RADIX, OFFSETS_THREADS, 0, stream>>>(a, tiles);
  CQL_LAUNCH_CHECK();
  return 0;
}

static int launch_radix_scatter(const CqlLaunch& a, uint32_t gws, uint32_t lws, cudaStream_t stream)
{
  (void)gws;
  (void)lws;
  uint64_t n = cql_word(a, 0);
  uint32_t shift = cql_word(a, 2), kb = cql_word(a, 4);
  if (n == 0) return 0;
  uint32_t tiles = (uint32_t)((n + SORT_TILE - 1) / SORT_TILE);
  bool write_keys = cql_word(a, 8) == 0;
  if ((kb != 4 && kb != 8) || shift >= kb * 8 || a.bytes[0] < n * kb || (!cql_word(a, 10) && a.bytes[1] < n * 4) || a.bytes[3] < n * 4 ||
      (write_keys && a.bytes[2] < n * kb) || (uint64_t)tiles * RADIX * 4 > a.bytes[4] || (cql_word(a, 6) && a.bytes[5] < n * 4))
    return (int)cudaErrorInvalidValue;
  // the tile's keys and positions staged in dynamic shared memory
  size_t smem = (size_t)SORT_TILE * (kb + 4);
  const void* fn = kb == 4 ? (const void*)k_radix_scatter<uint32_t, SORT_RANK_FORM> : (const void*)k_radix_scatter<unsigned long long, SORT_RANK_FORM>;
  // dynamic plus static shared memory passes the default 48 KB for 8-byte keys: opt in
  cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
  uint32_t grid = cql_stream_grid(tiles, resident_ctas(fn, smem));
  bool has_totals = a.buf[6] != nullptr && a.bytes[6] >= RADIX * 4;
  if (kb == 4) k_radix_scatter<uint32_t, SORT_RANK_FORM><<<grid, SORT_THREADS, smem, stream>>>(a, n, tiles, has_totals);
  else k_radix_scatter<unsigned long long, SORT_RANK_FORM><<<grid, SORT_THREADS, smem, stream>>>(a, n, tiles, has_totals);
  CQL_LAUNCH_CHECK();
  return 0;
}

// ---------------------------------------------------------------------------------------------
// ORDER BY of more than 32 key bits by a 32-bit prefix (not in the reference, nor the sort above): most of a wide
// key's bits only break ties, and few rows tie in the bits that matter. Each key's smallest and largest order word are
// found first; the highest 32 bits of the keys' distances from their ends, in the keys' order, make a prefix; the rows
// are sorted by it in four passes, and the short runs of rows that share a prefix are put in order in shared memory,
// by the full keys.
//
//  cql_sort_range   binding 0..3 the key columns, 4 selection, 5 out: per key (smallest, largest) order word, u64 each
//                   (all ones and 0 before); words as below
//  cql_sort_sample  the same, 6 out: how many rows of the sample share another's prefix and differ in the rest (u32)
//  cql_sort_prefix  the same with binding 5 the prefixes out (u32), 6 the histogram [256][tiles] of their low byte, 7 its
//                   totals [256] (zero before), 8 the ranges as found
//  cql_sort_runs    the same with binding 5 the sorted prefixes, 6 their positions, 7 rows out, 8 the ranges, 9 status
//                   (bit 0: a run longer than the kernel takes is out of order)
//  words: 0 n, 2 keys, 3 1 = the positions are the selection's rows, 4 CQL types (4 bits a key), 5 descending (bits), 6
//  narrow widths (2 bits a key), slots 4 and 5 the narrow bases (32 bits a key)
//
// 64-bit integers order as themselves while they lie within 2^53 of zero, where the F64 values they are compared as are
// all different; a column with others orders by those values. Distances, and not the words' own bits: doubles from 0.1
// to 4000 differ from bit 62 down, but span 2^56, so the prefix holds 28 bits of their fractions and not 21 (20M
// lognormal rows: most rows in runs, 407 us for the runs, against 125).
//
// 20M rows by (f64 DESC, u32): twelve passes over 12- and 8-byte pairs took 2.43 ms of kernels, this form 0.89: ranges
// 61 us, sample 17, prefixes 74, the four passes 600, runs 133.
#define PREFIX_SAMPLE 2048u
#define RUN_THREADS 256
#define RUN_TILE 1024
#define RUN_HALO 128
#define WORD_SIGN 0x8000000000000000ull

struct SortPlan
{
  uint32_t keys, bits;          // bits: of the prefix
  uint32_t hi[4], take[4];      // key k gives the `take` bits below bit hi of its distance
  uint32_t rest;                // the first key with bits below its part, `keys` when there is none
  uint32_t desc, whole;         // per key: descending; 64-bit integers ordered as themselves
  unsigned long long lo[4], top[4];
};

struct SortCols
{
  const void* col[4];
  uint64_t rows[4];
  const uint32_t* sel;
  uint32_t keys, types, desc, widths;
  uint64_t bases[2];
};

__device__ __forceinline__ bool sort_wide(uint32_t type) { return type == 2 || type == 4 || type == 8 || type == 10 || type == 11; }
__device__ __forceinline__ bool sort_integer64(uint32_t type) { return sort_wide(type) && type != 4; }

__device__ __forceinline__ SortCols sort_cols(const CqlLaunch& a)
{
  SortCols c;
  c.types = cql_word(a, 4);
  c.desc = cql_word(a, 5);
  c.widths = cql_word(a, 6);
  c.keys = cql_word(a, 2);
  c.bases[0] = a.push[4];
  c.bases[1] = a.push[5];
#pragma unroll
  for (uint32_t k = 0; k < 4; k++)
  {
    uint32_t t = (c.types >> (4 * k)) & 0xfu, w = (c.widths >> (2 * k)) & 3u;
    c.col[k] = a.buf[k];
    c.rows[k] = w == 3 ? ~0ull : a.bytes[k] / (w ? w : sort_wide(t) ? 8 : 4);
  }
  c.sel = cql_word(a, 3) ? (const uint32_t*)a.buf[4] : nullptr;
  return c;
}

// one key of the columns, for a loop over rows
struct SortKey
{
  const void* col;
  uint64_t rows;
  uint32_t type, width, base;
  bool wide, whole;
};

__device__ __forceinline__ SortKey sort_key(const SortCols& c, uint32_t k, bool whole)
{
  SortKey s;
  s.col = k == 0 ? c.col[0] : k == 1 ? c.col[1] : k == 2 ? c.col[2] : c.col[3];
  s.rows = k == 0 ? c.rows[0] : k == 1 ? c.rows[1] : k == 2 ? c.rows[2] : c.rows[3];
  s.type = (c.types >> (4 * k)) & 0xfu;
  s.width = (c.widths >> (2 * k)) & 3u;
  s.base = (uint32_t)((k < 2 ? c.bases[0] : c.bases[1]) >> (32 * (k & 1u)));
  s.wide = sort_wide(s.type);
  s.whole = whole && sort_integer64(s.type);
  return s;
}

__device__ __forceinline__ unsigned long long sort_raw(const SortKey& s, uint32_t row)
{
  if (row >= s.rows) return 0;
  if (s.wide) return ((const unsigned long long*)s.col)[row];
  if (s.width == 0) return ((const uint32_t*)s.col)[row];
  return s.width == 1 ? ((const uint8_t*)s.col)[row] : s.width == 2 ? ((const uint16_t*)s.col)[row] : row;
}

// the ascending order word; a row past the column orders first (the key pass's rule)
__device__ __forceinline__ unsigned long long sort_word(const SortKey& s, uint32_t row, unsigned long long raw)
{
  if (row >= s.rows) return 0;
  if (s.whole) return s.type == 2 ? raw : raw ^ WORD_SIGN;
  if (s.wide) return order_bits(s.type, raw);
  if (s.width == 0) return order_bits(s.type, (uint32_t)raw);
  return ((uint32_t)raw + s.base) ^ ((s.type == 7 || s.type == 9) ? 0x80000000u : 0u);
}

// The forms a loop over a key's rows is compiled for: a full-width column that holds every row, by its type. The loops are
// bound by issue (the general form's tests of type, width and row are 40 instructions a value), so a switch outside them
// picks the form.
enum SortForm { FORM_ANY = 0, FORM_U32, FORM_I32, FORM_F32, FORM_F64, FORM_I64, FORM_U64 };

__device__ __forceinline__ int sort_form(const SortKey& s, bool selected, uint64_t n)
{
  if (selected || s.width != 0 || s.rows < n) return FORM_ANY;
  switch (s.type)
  {
    case 1: case 12: return FORM_U32;
    case 7: case 9: return FORM_I32;
    case 3: return FORM_F32;
    case 4: return FORM_F64;
    case 2: return s.whole ? FORM_U64 : FORM_ANY;
    default: return s.whole ? FORM_I64 : FORM_ANY;
  }
}

template <int FORM>
__device__ __forceinline__ unsigned long long form_raw(const SortKey& s, uint32_t row)
{
  if (FORM == FORM_ANY) return sort_raw(s, row);
  if (FORM <= FORM_F32) return ((const uint32_t*)s.col)[row];
  return ((const unsigned long long*)s.col)[row];
}

template <int FORM>
__device__ __forceinline__ unsigned long long form_word(const SortKey& s, uint32_t row, unsigned long long raw)
{
  switch (FORM)
  {
    case FORM_U32: return (uint32_t)raw;
    case FORM_I32: return (uint32_t)raw ^ 0x80000000u;
    case FORM_F32: return order_bits(3, (uint32_t)raw);
    case FORM_F64: return f64_order(raw);
    case FORM_I64: return raw ^ WORD_SIGN;
    case FORM_U64: return raw;
    default: return sort_word(s, row, raw);
  }
}

__device__ inline SortPlan sort_plan(const unsigned long long* range, const SortCols& c)
{
  SortPlan p;
  p.keys = c.keys;
  p.desc = c.desc;
  p.bits = p.whole = 0;
  p.rest = c.keys;
  for (uint32_t k = 0; k < 4; k++)
  {
    p.hi[k] = p.take[k] = 0;
    p.lo[k] = p.top[k] = 0;
    if (k >= c.keys) continue;
    uint32_t type = (c.types >> (4 * k)) & 0xfu;
    unsigned long long lo = range[2 * k], top = range[2 * k + 1];
    if (sort_integer64(type))
    {
      const unsigned long long near = 1ull << 53, zero = type == 2 ? 0ull : WORD_SIGN;
      if (top <= zero + near && (type == 2 || lo >= zero - near)) p.whole |= 1u << k;
      else
      {
        lo = order_bits(type, lo ^ zero);
        top = order_bits(type, top ^ zero);
      }
    }
    p.lo[k] = lo;
    p.top[k] = top;
    unsigned long long span = top - lo;
    p.hi[k] = span ? 64u - (uint32_t)__clzll((long long)span) : 0u;
    uint32_t room = 32 - p.bits;
    p.take[k] = min(p.hi[k], room);
    p.bits += p.take[k];
    if (p.take[k] < p.hi[k] && p.rest == c.keys) p.rest = k;
  }
  return p;
}

// the key's distance from its first value in the order
__device__ __forceinline__ unsigned long long sort_distance(const SortPlan& p, uint32_t k, unsigned long long word)
{
  return ((p.desc >> k) & 1u) ? p.top[k] - word : word - p.lo[k];
}

__device__ __forceinline__ uint32_t prefix_append(const SortPlan& p, uint32_t k, uint32_t v, unsigned long long distance)
{
  uint32_t take = p.take[k];
  return (take == 32 ? 0u : v << take) | (uint32_t)((distance >> (p.hi[k] - take)) & ((1ull << take) - 1ull));
}

__device__ __forceinline__ unsigned long long sort_distance_of(const SortCols& c, const SortPlan& p, uint32_t k, uint32_t row)
{
  SortKey s = sort_key(c, k, (p.whole >> k) & 1u);
  return sort_distance(p, k, sort_word(s, row, sort_raw(s, row)));
}

template <int FORM>
__device__ __forceinline__ void range_of_key(const SortKey& s, const uint32_t* sel, uint64_t n, unsigned long long* out_lo, unsigned long long* out_top)
{
  unsigned long long lo = ~0ull, top = 0ull;
  const uint32_t step = gridDim.x * SORT_THREADS, last = (uint32_t)(n - 1);
  for (uint64_t i0 = (uint64_t)blockIdx.x * SORT_THREADS + threadIdx.x; i0 < n; i0 += (uint64_t)step * 8)
  {
    uint32_t row[8];
    unsigned long long raw[8];
#pragma unroll
    for (uint32_t u = 0; u < 8; u++)
    {
      uint32_t i = (uint32_t)min(i0 + (uint64_t)u * step, (uint64_t)last);
      row[u] = FORM == FORM_ANY && sel ? sel[i] : i;
    }
#pragma unroll
    for (uint32_t u = 0; u < 8; u++) raw[u] = form_raw<FORM>(s, row[u]);
#pragma unroll
    for (uint32_t u = 0; u < 8; u++)
    {
      unsigned long long w = form_word<FORM>(s, row[u], raw[u]);
      lo = min(lo, w);
      top = max(top, w);
    }
  }
  *out_lo = lo;
  *out_top = top;
}

__global__ void __launch_bounds__(SORT_THREADS, 5) k_sort_range(CqlLaunch a, uint64_t n)
{
  const SortCols c = sort_cols(a);
  unsigned long long* out = (unsigned long long*)a.buf[5];
#pragma unroll 1
  for (uint32_t k = 0; k < c.keys; k++)
  {
    const SortKey s = sort_key(c, k, true);
    unsigned long long lo, top;
    switch (sort_form(s, c.sel != nullptr, n))
    {
      case FORM_U32: range_of_key<FORM_U32>(s, c.sel, n, &lo, &top); break;
      case FORM_I32: range_of_key<FORM_I32>(s, c.sel, n, &lo, &top); break;
      case FORM_F32: range_of_key<FORM_F32>(s, c.sel, n, &lo, &top); break;
      case FORM_F64: range_of_key<FORM_F64>(s, c.sel, n, &lo, &top); break;
      case FORM_I64: range_of_key<FORM_I64>(s, c.sel, n, &lo, &top); break;
      case FORM_U64: range_of_key<FORM_U64>(s, c.sel, n, &lo, &top); break;
      default: range_of_key<FORM_ANY>(s, c.sel, n, &lo, &top); break;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
    {
      lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
    }
    if ((threadIdx.x & 31u) == 0)
    {
      if (lo < __ldcg(&out[2 * k])) atomicMin(&out[2 * k], lo);
      if (top > __ldcg(&out[2 * k + 1])) atomicMax(&out[2 * k + 1], top);
    }
  }
}

// One CTA: the prefixes of a spread sample meet in a hash table, with a hash of the bits below them.
__global__ void __launch_bounds__(1024) k_sort_sample(CqlLaunch a, uint64_t n)
{
  __shared__ unsigned long long table[2 * PREFIX_SAMPLE];
  __shared__ uint32_t s_count;
  const SortCols c = sort_cols(a);
  const SortPlan p = sort_plan((const unsigned long long*)a.buf[5], c);
  if (threadIdx.x == 0) s_count = 0;
  for (uint32_t i = threadIdx.x; i < 2 * PREFIX_SAMPLE; i += 1024) table[i] = ~0ull;
  __syncthreads();
  uint32_t mine = 0;
  for (uint32_t i = threadIdx.x; i < PREFIX_SAMPLE; i += 1024)
  {
    uint64_t at = (uint64_t)i * n / PREFIX_SAMPLE;
    uint32_t row = c.sel ? c.sel[at] : (uint32_t)at, v = 0;
    unsigned long long rest = 0;
    for (uint32_t k = 0; k < p.keys; k++)
    {
      unsigned long long d = sort_distance_of(c, p, k, row);
      if (p.take[k]) v = prefix_append(p, k, v, d);
      if (k >= p.rest) rest = (rest ^ d) * 0x9E3779B97F4A7C15ull;
    }
    unsigned long long e = ((unsigned long long)v << 32) | (rest >> 33);   // never all ones
    uint32_t slot = (v * 0x9E3779B1u) >> 20;                              // 4096 slots, half of them used at most
    for (;;)
    {
      unsigned long long old = atomicCAS(&table[slot], ~0ull, e);
      if (old == ~0ull) break;
      if ((uint32_t)(old >> 32) == v)
      {
        mine += old != e;
        break;
      }
      slot = (slot + 1u) & (2 * PREFIX_SAMPLE - 1u);
    }
  }
  if (mine) atomicAdd(&s_count, mine);
  __syncthreads();
  if (threadIdx.x == 0) *(uint32_t*)a.buf[6] = s_count;
}

template <int FORM>
__device__ __forceinline__ void prefix_of_key(const SortKey& s, const SortPlan& p, uint32_t k, const uint32_t* row, uint32_t* v)
{
  unsigned long long raw[8];
#pragma unroll
  for (uint32_t j = 0; j < 8; j++) raw[j] = form_raw<FORM>(s, row[j]);
  const bool desc = (p.desc >> k) & 1u;
  const unsigned long long from = desc ? p.top[k] : p.lo[k], mask = (1ull << p.take[k]) - 1ull;
  const uint32_t shift = p.hi[k] - p.take[k], take = p.take[k];
#pragma unroll
  for (uint32_t j = 0; j < 8; j++)
  {
    unsigned long long w = form_word<FORM>(s, row[j], raw[j]), d = desc ? from - w : w - from;
    v[j] = (take == 32 ? 0u : v[j] << take) | (uint32_t)((d >> shift) & mask);
  }
}

__global__ void __launch_bounds__(SORT_THREADS, 4) k_sort_prefix(CqlLaunch a, uint64_t n, uint32_t tiles)
{
  __shared__ uint32_t hist[SORT_WARPS][RADIX];
  __shared__ SortPlan p;
  const SortCols c = sort_cols(a);
  uint32_t* out = (uint32_t*)a.buf[5];
  uint32_t* hist_out = (uint32_t*)a.buf[6];
  if (threadIdx.x == 0) p = sort_plan((const unsigned long long*)a.buf[8], c);
  uint32_t warp = threadIdx.x >> 5, d = threadIdx.x, cta_total = 0;
  for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x)
  {
    for (uint32_t i = threadIdx.x; i < SORT_WARPS * RADIX; i += SORT_THREADS) (&hist[0][0])[i] = 0;
    __syncthreads();
    uint64_t first = (uint64_t)tile * SORT_TILE;
    DigitRun run;
#pragma unroll 1
    for (uint32_t j0 = 0; j0 < SORT_ROUNDS; j0 += 8)
    {
      uint32_t v[8], row[8];
#pragma unroll
      for (uint32_t j = 0; j < 8; j++)
      {
        uint64_t i = min(first + (j0 + j) * SORT_THREADS + threadIdx.x, n - 1);
        row[j] = c.sel ? c.sel[i] : (uint32_t)i;
        v[j] = 0;
      }
#pragma unroll 1
      for (uint32_t k = 0; k < p.keys; k++)
      {
        if (p.take[k] == 0) continue;
        const SortKey s = sort_key(c, k, (p.whole >> k) & 1u);
        switch (sort_form(s, c.sel != nullptr, n))
        {
          case FORM_U32: prefix_of_key<FORM_U32>(s, p, k, row, v); break;
          case FORM_I32: prefix_of_key<FORM_I32>(s, p, k, row, v); break;
          case FORM_F32: prefix_of_key<FORM_F32>(s, p, k, row, v); break;
          case FORM_F64: prefix_of_key<FORM_F64>(s, p, k, row, v); break;
          case FORM_I64: prefix_of_key<FORM_I64>(s, p, k, row, v); break;
          case FORM_U64: prefix_of_key<FORM_U64>(s, p, k, row, v); break;
          default: prefix_of_key<FORM_ANY>(s, p, k, row, v); break;
        }
      }
#pragma unroll
      for (uint32_t j = 0; j < 8; j++)
      {
        uint64_t i = first + (j0 + j) * SORT_THREADS + threadIdx.x;
        if (i >= n) continue;
        out[i] = v[j];
        run.add(hist[warp], v[j] & 0xffu);
      }
    }
    run.flush(hist[warp]);
    __syncthreads();
    uint32_t total = 0;
#pragma unroll
    for (uint32_t w = 0; w < SORT_WARPS; w++) total += hist[w][d];
    hist_out[(uint64_t)d * tiles + tile] = total;
    cta_total += total;
    __syncthreads();
  }
  if (cta_total) atomicAdd(&((uint32_t*)a.buf[7])[d], cta_total);
}

// x before y among rows that share a prefix and the first unfinished key's word: by the keys after it
__device__ __noinline__ int sort_compare_rest(const SortCols* c, const SortPlan* p, uint32_t x, uint32_t y)
{
  for (uint32_t k = p->rest + 1; k < c->keys; k++)
  {
    unsigned long long wx = sort_distance_of(*c, *p, k, x), wy = sort_distance_of(*c, *p, k, y);
    if (wx != wy) return wx < wy ? -1 : 1;
  }
  return 0;
}

// whether row j of a run belongs behind the row after it, which shares its prefix
__device__ __forceinline__ bool run_out_of_order(const SortCols* c, const SortPlan* p, const uint32_t* s_row, const unsigned long long* s_word, int j)
{
  if (s_word[j] != s_word[j + 1]) return s_word[j] > s_word[j + 1];
  return p->rest + 1 < c->keys && sort_compare_rest(c, p, s_row[j], s_row[j + 1]) > 0;
}

// A row of a run: where it belongs, by counting the rows of the run before it. Runs longer than RUN_HALO are only checked.
__device__ __noinline__ int run_place(const SortCols* c, const SortPlan* p, const uint32_t* s_prefix, const uint32_t* s_row, const unsigned long long* s_word,
                                      int j, int lo, int hi, bool* unsorted)
{
  uint32_t v = s_prefix[j];
  bool more = p->rest + 1 < c->keys;
  int left = j, right = j;
  while (left > lo && j - left < RUN_HALO && s_prefix[left - 1] == v) left--;
  while (right + 1 < hi && right - j < RUN_HALO && s_prefix[right + 1] == v) right++;
  if (right - left + 1 > RUN_HALO)
  {
    // too long to rank (every row of the run finds so): fine when it is in order as it is
    if (j + 1 < hi && s_prefix[j + 1] == v && run_out_of_order(c, p, s_row, s_word, j)) *unsorted = true;
    return j;
  }
  unsigned long long w = s_word[j];
  int at = left;
  for (int m = left; m <= right; m++)
  {
    unsigned long long x = s_word[m];
    bool before = x < w;
    if (x == w && m != j)
    {
      int r = more ? sort_compare_rest(c, p, s_row[m], s_row[j]) : 0;
      before = r < 0 || (r == 0 && m < j);
    }
    at += before ? 1 : 0;
  }
  return at;
}

__global__ void __launch_bounds__(RUN_THREADS) k_sort_runs(CqlLaunch a, uint64_t n)
{
  __shared__ uint32_t s_prefix[RUN_TILE + 2 * RUN_HALO], s_row[RUN_TILE + 2 * RUN_HALO];
  __shared__ unsigned long long s_word[RUN_TILE + 2 * RUN_HALO];
  __shared__ SortPlan p;
  __shared__ SortCols c;
  const uint32_t* prefix = (const uint32_t*)a.buf[5];
  const uint32_t* pos = (const uint32_t*)a.buf[6];
  const uint32_t* sel = cql_word(a, 3) ? (const uint32_t*)a.buf[4] : nullptr;
  uint32_t* out = (uint32_t*)a.buf[7];
  if (threadIdx.x == 0)
  {
    c = sort_cols(a);
    p = sort_plan((const unsigned long long*)a.buf[8], c);
  }
  bool unsorted = false;
  const int per = RUN_TILE / RUN_THREADS;
  for (uint64_t tile = (uint64_t)blockIdx.x * RUN_TILE; tile < n; tile += (uint64_t)gridDim.x * RUN_TILE)
  {
    // place j of the shared arrays is position tile - RUN_HALO + j; lo and hi bound those that are there. A thread holds
    // `per` rows of the tile and, of the first 2 x RUN_HALO threads, one of the halo.
    int lo = tile < RUN_HALO ? RUN_HALO - (int)tile : 0, hi = (int)min((uint64_t)(RUN_TILE + 2 * RUN_HALO), n - tile + RUN_HALO);
    int halo = (int)threadIdx.x < RUN_HALO ? (int)threadIdx.x : (int)threadIdx.x < 2 * RUN_HALO ? RUN_TILE + (int)threadIdx.x : -1;
    if (halo < lo || halo >= hi) halo = -1;
    uint32_t v[per + 1], row[per + 1];
#pragma unroll
    for (int u = 0; u <= per; u++)
    {
      int j = u < per ? RUN_HALO + u * RUN_THREADS + (int)threadIdx.x : halo;
      bool there = j >= 0 && j < hi;
      v[u] = there ? __ldcs(prefix + (tile + (uint64_t)j - RUN_HALO)) : 0u;
      row[u] = there ? __ldcs(pos + (tile + (uint64_t)j - RUN_HALO)) : 0u;
    }
    if (sel)
    {
#pragma unroll
      for (int u = 0; u <= per; u++)
        if (u < per ? RUN_HALO + u * RUN_THREADS + (int)threadIdx.x < hi : halo >= 0) row[u] = sel[row[u]];
    }
    __syncthreads();   // the tile before is done with the arrays; the first time, the plan is there
#pragma unroll
    for (int u = 0; u <= per; u++)
    {
      int j = u < per ? RUN_HALO + u * RUN_THREADS + (int)threadIdx.x : halo;
      if (j < 0 || j >= hi) continue;
      s_prefix[j] = v[u];
      s_row[j] = row[u];
    }
    __syncthreads();
    uint32_t in_run = 0;
#pragma unroll
    for (int u = 0; u <= per; u++)
    {
      int j = u < per ? RUN_HALO + u * RUN_THREADS + (int)threadIdx.x : halo;
      if (j < 0 || j >= hi) continue;
      if ((j > lo && s_prefix[j - 1] == v[u]) || (j + 1 < hi && s_prefix[j + 1] == v[u])) in_run |= 1u << u;
      else if (u < per) out[tile + (uint64_t)j - RUN_HALO] = row[u];
    }
    // most tiles have a few rows in runs: their words are read now, all rows' loads in flight together
    const int runners = __syncthreads_count(in_run != 0);   // threads that hold such a row
    if (runners == 0) continue;
    for (uint32_t left = in_run; left; left &= left - 1u)
    {
      int u = __ffs(left) - 1, j = u < per ? RUN_HALO + u * RUN_THREADS + (int)threadIdx.x : halo;
      s_word[j] = sort_distance_of(c, p, p.rest, s_row[j]);
    }
    __syncthreads();
    // Runs of equal keys, in order as the passes left them, are most of what a column of few values has: when no row of the tile
    // and its halo comes before the one ahead of it, each stays (5M rows of 300 values: the kernel 298 us without this). Looked
    // for where nearly every thread holds such a row
    bool off = false;
    for (uint32_t left = runners >= RUN_THREADS - 6 ? in_run : 0u; left && !off; left &= left - 1u)
    {
      int u = __ffs(left) - 1, j = u < per ? RUN_HALO + u * RUN_THREADS + (int)threadIdx.x : halo;
      off = j + 1 < hi && s_prefix[j + 1] == s_prefix[j] && run_out_of_order(&c, &p, s_row, s_word, j);
    }
    if (runners >= RUN_THREADS - 6 && !__syncthreads_or(off))
    {
      for (uint32_t left = in_run & ((1u << per) - 1u); left; left &= left - 1u)
      {
        int j = RUN_HALO + (__ffs(left) - 1) * RUN_THREADS + (int)threadIdx.x;
        out[tile + (uint64_t)j - RUN_HALO] = s_row[j];
      }
      continue;
    }
    for (uint32_t left = in_run & ((1u << per) - 1u); left; left &= left - 1u)
    {
      int j = RUN_HALO + (__ffs(left) - 1) * RUN_THREADS + (int)threadIdx.x;
      int at = run_place(&c, &p, s_prefix, s_row, s_word, j, lo, hi, &unsorted);
      out[tile + (uint64_t)at - RUN_HALO] = s_row[j];
    }
  }
  if (__syncthreads_or(unsorted) && threadIdx.x == 0) atomicOr((uint32_t*)a.buf[9], 1u);
}

static int sort_cols_check(const CqlLaunch& a, uint64_t n)
{
  uint32_t keys = cql_word(a, 2), types = cql_word(a, 4);
  if (n == 0 || n > 0xffffffffull || keys == 0 || keys > 4 || (cql_word(a, 3) && a.bytes[4] < n * 4)) return 0;
  for (uint32_t k = 0; k < keys; k++)
    if (!sort_key_bytes((types >> (4 * k)) & 0xfu)) return 0;
  return 1;
}

static int launch_sort_range(const CqlLaunch& a, uint32_t gws, uint32_t lws, cudaStream_t stream)
{
  (void)gws;
  (void)lws;
  uint64_t n = a.push[0];
  if (n == 0) return 0;
  if (!sort_cols_check(a, n) || a.bytes[5] < 64) return (int)cudaErrorInvalidValue;
  k_sort_range<<<cql_stream_grid((n + SORT_THREADS * 8 - 1) / (SORT_THREADS * 8), 5), SORT_THREADS, 0, stream>>>(a, n);
  CQL_LAUNCH_CHECK();
  return 0;
}

static int launch_sort_sample(const CqlLaunch& a, uint32_t gws, uint32_t lws, cudaStream_t stream)
{
  (void)gws;
  (void)lws;
  uint64_t n = a.push[0];
  if (n == 0) return 0;
  if (!sort_cols_check(a, n) || a.bytes[5] < 64 || a.bytes[6] < 4) return (int)cudaErrorInvalidValue;
  k_sort_sample<<<1, 1024, 0, stream>>>(a, n);
  CQL_LAUNCH_CHECK();
  return 0;
}

static int launch_sort_prefix(const CqlLaunch& a, uint32_t gws, uint32_t lws, cudaStream_t stream)
{
  (void)gws;
  (void)lws;
  uint64_t n = a.push[0];
  if (n == 0) return 0;
  uint32_t tiles = (uint32_t)((n + SORT_TILE - 1) / SORT_TILE);
  if (!sort_cols_check(a, n) || a.bytes[5] < n * 4 || a.bytes[6] < (uint64_t)tiles * RADIX * 4 || a.bytes[7] < RADIX * 4 || a.bytes[8] < 64)
    return (int)cudaErrorInvalidValue;
  uint32_t grid = cql_stream_grid(tiles, resident_ctas((const void*)k_sort_prefix, 0));
  k_sort_prefix<<<grid, SORT_THREADS, 0, stream>>>(a, n, tiles);
  CQL_LAUNCH_CHECK();
  return 0;
}

static int launch_sort_runs(const CqlLaunch& a, uint32_t gws, uint32_t lws, cudaStream_t stream)
{
  (void)gws;
  (void)lws;
  uint64_t n = a.push[0];
  if (n == 0) return 0;
  if (!sort_cols_check(a, n) || a.bytes[5] < n * 4 || a.bytes[6] < n * 4 || a.bytes[7] < n * 4 || a.bytes[8] < 64 || a.bytes[9] < 4 || a.buf[6] == a.buf[7])
    return (int)cudaErrorInvalidValue;
  k_sort_runs<<<cql_stream_grid((n + RUN_TILE - 1) / RUN_TILE, resident_ctas((const void*)k_sort_runs, 0)), RUN_THREADS, 0, stream>>>(a, n);
  CQL_LAUNCH_CHECK();
  return 0;
}

__global__ void k_pairs_unpack(CqlLaunch a, uint64_t n, uint32_t stride, uint32_t fa, uint32_t fb)
{
  const uint32_t* rec = (const uint32_t*)a.buf[0];
  uint32_t* first = (uint32_t*)a.buf[1];
  uint32_t* second = (uint32_t*)a.buf[2];
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
  {
    first[i] = rec[i * stride + fa];
    second[i] = rec[i * stride + fb];
  }
}

__global__ void k_pairs_pack(CqlLaunch a, uint64_t n)
{
  const uint32_t* order = (const uint32_t*)a.buf[0];
  const uint32_t* first = (const uint32_t*)a.buf[1];
  const uint32_t* second = (const uint32_t*)a.buf[2];
  uint2* out = (uint2*)a.buf[3];
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
  {
    uint32_t p = order[i];
    out[i] = make_uint2(first[p], second[p]);
  }
}

static int launch_pairs_unpack(const CqlLaunch& a, uint32_t gws, uint32_t lws, cudaStream_t stream)
{
  (void)gws;
  (void)lws;
  uint64_t n = cql_word(a, 0);
  uint32_t stride = cql_word(a, 2), fa = cql_word(a, 4), fb = cql_word(a, 6);
  if (n == 0) return 0;
  if (stride == 0 || fa >= stride || fb >= stride || a.bytes[0] < n * stride * 4 || a.bytes[1] < n * 4 || a.bytes[2] < n * 4)
    return (int)cudaErrorInvalidValue;
  k_pairs_unpack<<<cql_stream_grid((n + SORT_THREADS - 1) / SORT_THREADS, 8), SORT_THREADS, 0, stream>>>(a, n, stride, fa, fb);
  CQL_LAUNCH_CHECK();
  return 0;
}

static int launch_pairs_pack(const CqlLaunch& a, uint32_t gws, uint32_t lws, cudaStream_t stream)
{
  (void)gws;
  (void)lws;
  uint64_t n = cql_word(a, 0);
  if (n == 0) return 0;
  if (a.bytes[0] < n * 4 || a.bytes[1] < n * 4 || a.bytes[2] < n * 4 || a.bytes[3] < n * 8) return (int)cudaErrorInvalidValue;
  k_pairs_pack<<<cql_stream_grid((n + SORT_THREADS - 1) / SORT_THREADS, 8), SORT_THREADS, 0, stream>>>(a, n);
  CQL_LAUNCH_CHECK();
  return 0;
}

const CqlKernelDesc cql_kernels_sort[] = {
  { "cql_pairs_unpack", launch_pairs_unpack },
  { "cql_pairs_pack", launch_pairs_pack },
  { "cql_sort_keys", launch_sort_keys },
  { "cql_radix_count", launch_radix_count },
  { "cql_radix_offsets", launch_radix_offsets },
  { "cql_radix_scatter", launch_radix_scatter },
  { "cql_sort_range", launch_sort_range },
  { "cql_sort_sample", launch_sort_sample },
  { "cql_sort_prefix", launch_sort_prefix },
  { "cql_sort_runs", launch_sort_runs },
  { nullptr, nullptr },
};
