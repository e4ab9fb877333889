// GROUP BY forms of GB300's own, beside the reference's hash path in k_hash.cu.
#include "cql_bits.cuh"
#include "cql_fixed.cuh"
#include "../host/cql_group_plan.h"
#include <algorithm>

#define GROUP_THREADS 256

// ---------------------------------------------------------------------------------------------
// cql_hll_rows: the HyperLogLog registers of whole columns, for a table or per value of a small-range key:
// binding 0 the key (u32 words; the first column again without a key), 1..8 the columns, 9 the registers
// (u32, zero before) [key value][column][2^10]; word 0 rows, 2 the columns, 4 their CQL types (4 bits each),
// 6 the key's values (at most 64; 0: no key), 8 its smallest (bits). A row whose key lies outside the values is left out.
//
// The update is one max per row on few registers, so the only traffic it needs is the column itself. Without a
// key a CTA keeps the 1024 registers in shared memory and merges them once (the member reduce read and wrote them
// in L2, where one table's 4 KB lie in a few slices and every row of the grid meets there: 329 us for 10M
// rows, after a widening pass of 32 us; this form 37 us with its launch). With a key the registers of all groups are spread over
// many slices, and a read that shows the register large enough saves nearly every atomic; a table in
// shared memory would be filled and flushed more often than it is hit (50 groups x 1024 registers against 66k
// rows an SM). Eight rows a thread are loaded before any is used.
#define HLL_P 10
#define HLL_REGS (1u << HLL_P)
#define HLL_ROWS 8
#define HLL_VALUES 64   // what the operators number by a small-range key

template <int TYPE>
__device__ __forceinline__ unsigned long long value_bits(unsigned long long raw)
{
  if (TYPE == 1) return cql_int_bits((long long)raw);
  if (TYPE == 7) return cql_int_bits((long long)(int)(uint32_t)raw);
  if (TYPE == 3) return (unsigned long long)__double_as_longlong((double)__uint_as_float((uint32_t)raw));
  if (TYPE == 2) return (unsigned long long)__double_as_longlong((double)raw);
  if (TYPE == 8) return (unsigned long long)__double_as_longlong((double)(long long)raw);
  return raw;
}

template <int TYPE>
__device__ __forceinline__ unsigned long long value_raw(const void* col, uint64_t row)
{
  if (TYPE == 1 || TYPE == 7 || TYPE == 3) return __ldcs((const uint32_t*)col + row);
  return __ldcs((const unsigned long long*)col + row);
}

template <int TYPE>
__global__ void __launch_bounds__(GROUP_THREADS) k_hll_table(const void* col, uint64_t rows, uint32_t* out)
{
  __shared__ uint32_t regs[HLL_REGS];
  for (uint32_t i = threadIdx.x; i < HLL_REGS; i += blockDim.x) regs[i] = 0;
  __syncthreads();
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t r0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; r0 < rows; r0 += step * HLL_ROWS)
  {
    unsigned long long raw[HLL_ROWS];
#pragma unroll
    for (uint32_t i = 0; i < HLL_ROWS; i++) raw[i] = r0 + i * step < rows ? value_raw<TYPE>(col, r0 + i * step) : 0ull;
#pragma unroll
    for (uint32_t i = 0; i < HLL_ROWS; i++)
    {
      if (r0 + i * step >= rows) continue;
      uint32_t bucket, rho;
      cql_hll_place(value_bits<TYPE>(raw[i]), HLL_P, &bucket, &rho);
      if (regs[bucket] < rho) atomicMax(&regs[bucket], rho);
    }
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < HLL_REGS; i += blockDim.x)
    if (regs[i] && __ldcg(&out[i]) < regs[i]) atomicMax(&out[i], regs[i]);
}

template <int TYPE>
__global__ void __launch_bounds__(GROUP_THREADS) k_hll_keyed(const uint32_t* key, const void* col, uint64_t rows, uint32_t kmin, uint32_t values,
                                                             uint32_t columns, uint32_t column, uint32_t* out)
{
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t r0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; r0 < rows; r0 += step * HLL_ROWS)
  {
    uint32_t at[HLL_ROWS], rho[HLL_ROWS], held[HLL_ROWS];
    unsigned long long raw[HLL_ROWS];
#pragma unroll
    for (uint32_t i = 0; i < HLL_ROWS; i++)
    {
      uint64_t r = r0 + i * step;
      at[i] = r < rows ? __ldcs(key + r) - kmin : 0xffffffffu;
      raw[i] = r < rows ? value_raw<TYPE>(col, r) : 0ull;
    }
#pragma unroll
    for (uint32_t i = 0; i < HLL_ROWS; i++)
    {
      uint32_t bucket;
      cql_hll_place(value_bits<TYPE>(raw[i]), HLL_P, &bucket, &rho[i]);
      at[i] = at[i] < values ? (at[i] * columns + column) * HLL_REGS + bucket : 0xffffffffu;   // values x columns <= 2^9
    }
#pragma unroll
    for (uint32_t i = 0; i < HLL_ROWS; i++) held[i] = at[i] != 0xffffffffu ? __ldcg(&out[at[i]]) : 0xffffffffu;
#pragma unroll
    for (uint32_t i = 0; i < HLL_ROWS; i++)
      if (held[i] < rho[i]) atomicMax(&out[at[i]], rho[i]);
  }
}

template <int TYPE>
static void launch_hll_column(const CqlLaunch& a, uint64_t rows, uint32_t j, uint32_t columns, uint32_t values, uint32_t kmin, cudaStream_t stream)
{
  uint32_t grid = cql_stream_grid((rows + GROUP_THREADS * HLL_ROWS - 1) / (GROUP_THREADS * HLL_ROWS), 8);
  if (values)
    k_hll_keyed<TYPE><<<grid, GROUP_THREADS, 0, stream>>>((const uint32_t*)a.buf[0], a.buf[1 + j], rows, kmin, values, columns, j, (uint32_t*)a.buf[9]);
  else
    k_hll_table<TYPE><<<grid, GROUP_THREADS, 0, stream>>>(a.buf[1 + j], rows, (uint32_t*)a.buf[9] + (uint64_t)j * HLL_REGS);
}

static int launch_hll_rows(const CqlLaunch& a, uint32_t gws, uint32_t lws, cudaStream_t stream)
{
  (void)gws;
  (void)lws;
  uint64_t rows = a.push[0];
  uint32_t columns = cql_word(a, 2), types = cql_word(a, 4), values = cql_word(a, 6), kmin = cql_word(a, 8);
  if (rows == 0 || columns == 0) return 0;
  if (columns > 8 || rows > 0xffffffffull || values > HLL_VALUES || a.bytes[9] < (uint64_t)(values ? values : 1) * columns * HLL_REGS * 4 ||
      (values && a.bytes[0] < rows * 4))
    return (int)cudaErrorInvalidValue;
  for (uint32_t j = 0; j < columns; j++)
  {
    uint32_t t = (types >> (4 * j)) & 0xfu;
    bool wide = t == 2 || t == 4 || t == 8;
    if (!(wide || t == 1 || t == 3 || t == 7) || a.bytes[1 + j] < rows * (wide ? 8 : 4)) return (int)cudaErrorInvalidValue;
    switch (t)
    {
      case 1: launch_hll_column<1>(a, rows, j, columns, values, kmin, stream); break;
      case 2: launch_hll_column<2>(a, rows, j, columns, values, kmin, stream); break;
      case 3: launch_hll_column<3>(a, rows, j, columns, values, kmin, stream); break;
      case 4: launch_hll_column<4>(a, rows, j, columns, values, kmin, stream); break;
      case 7: launch_hll_column<7>(a, rows, j, columns, values, kmin, stream); break;
      default: launch_hll_column<8>(a, rows, j, columns, values, kmin, stream); break;
    }
    CQL_LAUNCH_CHECK();
  }
  return 0;
}

// ---------------------------------------------------------------------------------------------
// cql_group_exact: GROUP BY up to 4 numeric keys with COUNT/SUM/AVG/MIN/MAX of up to 8 columns in one pass over
// them, the SUMs exact. Bindings 0..3 the keys, 4..11 the columns, 12 the plan (cql_group_plan.h), 13 the table, 14
// the status word (zero before); word 0 rows. cql_group_exact_emit lists the groups: binding 0 the table, 1 the
// plan, 2 status, 3 header out (u32 groups), 4 representative rows out (u64), 5 counts out (u64), 6 results
// out (f64 [group][expr]), 7 the slots of the groups in order (with word 2 = 1; their number in binding 8), word
// 0 the most groups the outputs take.
//
// The group's number is the keys' digits in mixed radix (value - smallest, by the columns' ranges; bits for
// floats), so a key is compared and claimed with one 64-bit word. A small number range indexes the table (direct); else
// the table is open-addressed by it. With few groups each CTA first groups its rows in a table of its own in shared
// memory (the same two forms) and merges it at the end: shared atomics take a row's updates at several a clock an
// SM, where global ones of a thousand groups meet on the same L2 lines.
//
// A SUM is exact: a double's 53 bits are added at their place in a number of 126 bits whose top is the column's
// largest exponent (4 words of 32 bits in shared memory, carries passed up; 3 signed 64-bit parts at bits 0, L
// and 63 in the table, L = log2 rows + 1, wide enough that the rows' pieces add without a carry), and rounded
// once when the group is listed. The sum does not depend on the order of the rows. A value outside that window
// (over 48 binades below the column's largest for 10M rows) sets the status, and the caller takes the member
// lists; the other CTAs meet the status a round later and leave too, so that such data costs little beside the lists.
// Two of the three parts hold any value within 2^(62 - 2L) of the largest, so a row mostly costs two 64-bit
// reductions; f64 reductions would cost one but round per row.
//
// What it replaced, per 10M rows: member lists (assign 640 us, scatter 575, reduce 460, prefix sums and ranges 100)
// for 1000 groups of two keys, this form 155 and the listing 10. For 1M groups of one key, assign 337, scatter 143, reduce
// 122, ranges, sums and compaction 230, this form 209 and the listing of the groups 70.
#define EXACT_ROWS 4
#define EXACT_EMPTY 0xffffffffffffffffull
#define EXACT_LOCAL_PROBES 64
// The slots tried for a group in the table, a constant of the kernel (as a value it cost a hashed table of 333k groups 202 -> 380
// us): in a half-full table the longest chain stays well below. A row that finds no room tries them one after another, some
// 0.4 us each, so that a first table, whose size is a guess, takes few.
#define EXACT_PROBES 256
#define EXACT_GUESS_PROBES 64

struct ExactTable
{
  unsigned long long* key;
  unsigned long long* mn;
  uint32_t* row;
  unsigned long long* part;
  unsigned long long* mx;
  uint32_t* cnt;
  uint32_t* flags;
};

__host__ __device__ inline ExactTable exact_table(const CqlGroupPlan& p, void* base)
{
  ExactTable t;
  char* at = (char*)base;
  t.key = (unsigned long long*)at;
  if (!p.direct) at += 8ull * p.slots;
  t.mn = (unsigned long long*)at;
  at += 8ull * p.slots * p.mins;
  t.row = (uint32_t*)at;
  at = (char*)base + cql_exact_ones_bytes(&p);
  t.part = (unsigned long long*)at;
  at += 24ull * p.slots * p.sums;
  t.mx = (unsigned long long*)at;
  at += 8ull * p.slots * p.maxs;
  t.cnt = (uint32_t*)at;
  at += 4ull * p.slots;
  t.flags = (uint32_t*)at;
  return t;
}

__device__ __forceinline__ uint32_t exact_hash(unsigned long long id, uint32_t slots)
{
  // slots is a power of two: the product's top bits
  id ^= id >> 32;
  return (uint32_t)((id * 0x9E3779B97F4A7C15ull) >> 32) >> (__clz(slots) + 1);
}

// A key of a thread's rows: its digits appended to the groups' numbers; `bad` gets the rows whose key the numbering
// does not hold. The key's type is fixed (8 for both 64-bit integers).
template <int TYPE>
__device__ __forceinline__ void exact_key(const void* col, unsigned long long kmin, unsigned long long range, const uint32_t (&row)[EXACT_ROWS],
                                          unsigned long long (&id)[EXACT_ROWS], uint32_t* bad)
{
  constexpr bool WIDE = !(TYPE == 1 || TYPE == 3 || TYPE == 7);
  unsigned long long raw[EXACT_ROWS];
#pragma unroll
  for (uint32_t i = 0; i < EXACT_ROWS; i++)
    raw[i] = WIDE ? __ldcs((const unsigned long long*)col + row[i]) : (unsigned long long)__ldcs((const uint32_t*)col + row[i]);
#pragma unroll
  for (uint32_t i = 0; i < EXACT_ROWS; i++)
  {
    unsigned long long v = raw[i];
    bool off = false;
    if (TYPE == 7) v = (unsigned long long)(long long)(int)(uint32_t)v;
    if (TYPE == CQL_EXACT_KEY_U64_AS_F64) v = (unsigned long long)__double_as_longlong((double)v);
    if (TYPE == CQL_EXACT_KEY_I64_AS_F64) v = (unsigned long long)__double_as_longlong((double)(long long)v);
    if (TYPE == 3) off = (v & 0x7fffffffull) > 0x7f800000ull || v == 0x80000000ull;
    if (TYPE == 4) off = (v & 0x7fffffffffffffffull) > 0x7ff0000000000000ull || v == 0x8000000000000000ull;
    v -= kmin;
    if (off || (range && v >= range)) *bad |= 1u << i;
    id[i] = id[i] * range + v;
  }
}

// Adds (or subtracts) m * 2^pos, m < 2^53, to a 128-bit two's-complement number of four words `stride` apart that
// threads share.
__device__ __forceinline__ void exact_add_local(uint32_t* word, uint32_t stride, unsigned long long m, uint32_t pos, bool negative)
{
  const uint32_t j = pos >> 5, sh = pos & 31u, keep = negative ? 0u : 0xffffffffu;
  const unsigned long long low = m << sh;
  const uint32_t piece[3] = { (uint32_t)low, (uint32_t)(low >> 32), (uint32_t)((m >> 32) >> (32u - sh)) };   // a shift by 32 gives 0
  uint32_t* at = word + j * stride;
  uint32_t carry = 0;
#pragma unroll
  for (uint32_t k = 0; k < 4; k++)
  {
    if (k >= 2 && piece[2] == 0 && carry == 0) break;   // the second word may hold nothing yet, the third mostly does not
    if (j + k > 3) break;
    uint32_t add = (k < 3 ? piece[k] : 0u) + carry;
    carry = add < carry ? 1u : 0u;
    // the word's old value, or its complement, below what is subtracted or added: a borrow or a carry
    if (add) carry += (atomicAdd(at, negative ? 0u - add : add) ^ keep) < add ? 1u : 0u;
    at += stride;
  }
}

// the same into the table's three signed parts
__device__ __forceinline__ void exact_add_parts(unsigned long long* part, uint64_t stride, uint32_t low_bits, unsigned __int128 v, bool negative)
{
  unsigned long long lo = (unsigned long long)v & ((1ull << low_bits) - 1ull);
  unsigned long long mid = (unsigned long long)(v >> low_bits) & ((1ull << (63u - low_bits)) - 1ull);
  unsigned long long hi = (unsigned long long)(v >> 63);
  if (lo) atomicAdd(part, negative ? 0ull - lo : lo);
  if (mid) atomicAdd(part + stride, negative ? 0ull - mid : mid);
  if (hi) atomicAdd(part + 2 * stride, negative ? 0ull - hi : hi);
}

// The slot of a group's number, claimed where the group is new (*claimed); slots when the probes run out.
__device__ __forceinline__ uint32_t exact_slot(unsigned long long* key, uint32_t slots, uint32_t probes, unsigned long long id, bool* claimed)
{
  uint32_t h = exact_hash(id, slots);
  for (uint32_t p = 0; p < probes; p++)
  {
    unsigned long long k = *(volatile unsigned long long*)&key[h];
    if (k == EXACT_EMPTY)
    {
      k = atomicCAS(&key[h], EXACT_EMPTY, id);
      if (k == EXACT_EMPTY)
      {
        *claimed = true;
        return h;
      }
    }
    if (k == id) return h;
    h = (h + 1) & (slots - 1);
  }
  return slots;
}

struct ExactColumn
{
  const void* data;
  uint32_t type, what;
  int base, scale;
  uint32_t low_bits, number;
};

// One column of a thread's rows into their slots (0xffffffff: none). KIND: 0 whole numbers and decimals, 4 f64, 3
// f32, 8 64-bit integers met as doubles.
template <bool LOCAL, int KIND>
__device__ __forceinline__ void exact_column(const ExactColumn& v, const uint32_t (&row)[EXACT_ROWS], const uint32_t (&sl)[EXACT_ROWS], uint32_t* words, uint32_t S,
                                             unsigned long long* part, uint32_t T, unsigned long long* mn, unsigned long long* mx, uint32_t* flags,
                                             uint32_t pos_max, uint32_t* wrong)
{
  const uint32_t type = v.type, what = v.what;
  const bool wide = KIND == 4 || KIND == 8 || (KIND == 0 && (type == 2 || type == 4 || type == 8));
  unsigned long long raw[EXACT_ROWS];
#pragma unroll
  for (uint32_t i = 0; i < EXACT_ROWS; i++)
    raw[i] = wide ? __ldcs((const unsigned long long*)v.data + row[i]) : (unsigned long long)__ldcs((const uint32_t*)v.data + row[i]);
#pragma unroll
  for (uint32_t i = 0; i < EXACT_ROWS; i++)
  {
    const uint32_t s = sl[i];
    if (s == 0xffffffffu) continue;
    // the value's magnitude and place, and its double's bits
    unsigned long long m, b;
    bool negative, finite = true;
    uint32_t pos = 0;
    if (KIND == 0)
    {
      const long long q = (what & CQL_EXACT_DECIMAL) ? (long long)fix_scaled(fix_decode_f64(raw[i]), v.scale)
                                                     : type == 7 ? (long long)(int)(uint32_t)raw[i] : (long long)raw[i];
      negative = q < 0;
      m = (unsigned long long)(negative ? -q : q);
      b = (what & (CQL_EXACT_MIN | CQL_EXACT_MAX)) ? cql_int_bits(q) : 0ull;
    }
    else
    {
      b = KIND == 3 ? cql_f32_bits((uint32_t)raw[i])
                    : KIND == 4 ? raw[i] : (unsigned long long)__double_as_longlong(type == 8 ? (double)(long long)raw[i] : (double)raw[i]);
      const uint32_t top = (uint32_t)(b >> 32);
      const int e = (int)((top >> 20) & 0x7ffu);
      finite = e != 0x7ff;
      negative = (b >> 63) != 0;
      m = ((unsigned long long)((top & 0xfffffu) | (e ? 0x100000u : 0u)) << 32) | (uint32_t)b;
      int at = max(e, 1) - 1075 - v.base;
      if ((what & CQL_EXACT_SUM) && (uint32_t)at > pos_max && finite && m)
      {
        // below the window's last bit: exact only where those bits are zero
        if (at >= 0 || at <= -53 || (m & ((1ull << -at) - 1ull))) *wrong |= CQL_EXACT_RANGE;
        else m >>= -at;
        at = 0;
      }
      pos = (uint32_t)at;
    }
    if (what & CQL_EXACT_SUM)
    {
      if (!finite)
        atomicOr(&flags[s], ((b & 0xfffffffffffffull) ? 1u : negative ? 4u : 2u) << (3 * v.number));
      else if (m)
      {
        if (LOCAL) exact_add_local(words + s, S, m, pos, negative);
        else if (KIND == 0) atomicAdd(&part[s], negative ? 0ull - m : m);
        else exact_add_parts(part + s, T, v.low_bits, (unsigned __int128)m << pos, negative);
      }
    }
    if (what & (CQL_EXACT_MIN | CQL_EXACT_MAX))
    {
      // NaN is left out; -0.0 compares equal to +0.0
      unsigned long long o = (b >> 63) ? ~b : (b | 0x8000000000000000ull);
      const bool nan = KIND != 0 && (b << 1) > 0xffe0000000000000ull;
      if ((b << 1) == 0) o = 0x8000000000000000ull;
      if (LOCAL)
      {
        if ((what & CQL_EXACT_MIN) && o < mn[s] && !nan) atomicMin(&mn[s], o);
        if ((what & CQL_EXACT_MAX) && o > mx[s] && !nan) atomicMax(&mx[s], o);
      }
      else if (!nan)
      {
        if (what & CQL_EXACT_MIN) atomicMin(&mn[s], o);
        if (what & CQL_EXACT_MAX) atomicMax(&mx[s], o);
      }
    }
  }
}

template <bool LOCAL, bool DIRECT, int THREADS, uint32_t PROBES = EXACT_PROBES>
__global__ void __launch_bounds__(THREADS, 1024 / THREADS) k_group_exact(CqlLaunch a, uint64_t rows)
{
  extern __shared__ __align__(16) unsigned char local_mem[];
  __shared__ CqlGroupPlan p;
  __shared__ uint32_t s_stop;
  for (uint32_t i = threadIdx.x; i < sizeof(CqlGroupPlan) / 4; i += THREADS) ((uint32_t*)&p)[i] = ((const uint32_t*)a.buf[12])[i];
  if (threadIdx.x == 0) s_stop = 0;
  __syncthreads();
  ExactTable t = exact_table(p, a.buf[13]);
  uint32_t* status = (uint32_t*)a.buf[14];
  const uint32_t S = p.local_slots, T = p.slots;
  // the CTA's own table
  unsigned long long* lkey = (unsigned long long*)local_mem;
  unsigned long long* lmn = lkey + (DIRECT ? 0 : S);
  unsigned long long* lmx = lmn + S * p.mins;
  uint32_t* lsum = (uint32_t*)(lmx + S * p.maxs);
  uint32_t* lrow = lsum + 4 * S * p.sums;
  uint32_t* lcnt = lrow + S;
  uint32_t* lflags = lcnt + S;
  if (LOCAL)
  {
    uint32_t ones = S * ((DIRECT ? 0 : 1) + p.mins);
    for (uint32_t i = threadIdx.x; i < ones; i += THREADS) lkey[i] = ~0ull;
    for (uint32_t i = threadIdx.x; i < S * p.maxs; i += THREADS) lmx[i] = 0ull;
    for (uint32_t i = threadIdx.x; i < S * (4 * p.sums + 3); i += THREADS) lsum[i] = (i >= 4 * S * p.sums && i < S * (4 * p.sums + 1)) ? 0xffffffffu : 0u;
    __syncthreads();
  }
  const uint32_t copies_log2 = p.copies_log2, copy = threadIdx.x & ((1u << copies_log2) - 1u);
  const uint32_t pos_max = 73u - p.low_bits;
  const uint64_t step = (uint64_t)gridDim.x * THREADS;
  uint32_t wrong = 0;
  for (uint64_t r0 = (uint64_t)blockIdx.x * THREADS + threadIdx.x; r0 < rows; r0 += step * EXACT_ROWS)
  {
    if (*(volatile uint32_t*)&s_stop) break;
    const uint32_t stopped = threadIdx.x == 0 ? *(volatile uint32_t*)status : 0u;   // another CTA's; needed at the round's end
    unsigned long long id[EXACT_ROWS];
    uint32_t bad = 0, row[EXACT_ROWS];   // a row past the end reads the last one and is left out below
#pragma unroll
    for (uint32_t i = 0; i < EXACT_ROWS; i++)
    {
      id[i] = 0;
      row[i] = (uint32_t)min(r0 + i * step, rows - 1);
    }
#pragma unroll 1
    for (uint32_t k = 0; k < p.key_count; k++)
    {
      const unsigned long long kmin = p.key_min[k], range = p.key_range[k];
      switch (p.key_type[k])
      {
        case 1: exact_key<1>(a.buf[k], kmin, range, row, id, &bad); break;
        case 3: exact_key<3>(a.buf[k], kmin, range, row, id, &bad); break;
        case 4: exact_key<4>(a.buf[k], kmin, range, row, id, &bad); break;
        case 7: exact_key<7>(a.buf[k], kmin, range, row, id, &bad); break;
        case CQL_EXACT_KEY_U64_AS_F64: exact_key<CQL_EXACT_KEY_U64_AS_F64>(a.buf[k], kmin, range, row, id, &bad); break;
        case CQL_EXACT_KEY_I64_AS_F64: exact_key<CQL_EXACT_KEY_I64_AS_F64>(a.buf[k], kmin, range, row, id, &bad); break;
        default: exact_key<8>(a.buf[k], kmin, range, row, id, &bad); break;
      }
    }
    uint32_t sl[EXACT_ROWS];
#pragma unroll
    for (uint32_t i = 0; i < EXACT_ROWS; i++) sl[i] = 0xffffffffu;
#pragma unroll
    for (uint32_t i = 0; i < EXACT_ROWS; i++)
    {
      uint64_t r = r0 + i * step;
      if (r >= rows || wrong) continue;   // (once a row found no room, the next would look as long)
      if (((bad >> i) & 1u) || (!DIRECT && id[i] == EXACT_EMPTY))
      {
        wrong |= CQL_EXACT_KEY;
        continue;
      }
      if (LOCAL)
      {
        unsigned long long lid = (id[i] << copies_log2) + copy;
        bool claimed = false;
        uint32_t s = DIRECT ? (uint32_t)lid : exact_slot(lkey, S, EXACT_LOCAL_PROBES, lid, &claimed);
        if (s >= S)
        {
          wrong |= CQL_EXACT_OVERFLOW;
          continue;
        }
        if (DIRECT ? (uint32_t)r < lrow[s] : claimed) atomicMin(&lrow[s], (uint32_t)r);
        atomicAdd(&lcnt[s], 1u);
        sl[i] = s;
      }
      else
      {
        bool claimed = false;
        uint32_t s = DIRECT ? (uint32_t)id[i] : exact_slot(t.key, T, PROBES, id[i], &claimed);
        if (s >= T)
        {
          wrong |= CQL_EXACT_OVERFLOW;
          continue;
        }
        if (DIRECT || claimed) atomicMin(&t.row[s], (uint32_t)r);
        atomicAdd(&t.cnt[s], 1u);
        sl[i] = s;
      }
    }
    if (wrong) *(volatile uint32_t*)&s_stop = 1;
#pragma unroll 1
    for (uint32_t c = 0; c < p.column_count; c++)
    {
      const ExactColumn v = { a.buf[4 + c], p.col_type[c], p.col_what[c], p.col_base[c], (int)p.col_scale[c], p.low_bits, c };
      unsigned long long* part = t.part + (uint64_t)p.col_sum[c] * 3 * T;
      unsigned long long* mn = LOCAL ? lmn + p.col_min[c] * S : t.mn + (uint64_t)p.col_min[c] * T;
      unsigned long long* mx = LOCAL ? lmx + p.col_max[c] * S : t.mx + (uint64_t)p.col_max[c] * T;
      uint32_t* flags = LOCAL ? lflags : t.flags;
      uint32_t* words = lsum + (uint64_t)p.col_sum[c] * 4 * S;
      if (v.what & (CQL_EXACT_WHOLE | CQL_EXACT_DECIMAL)) exact_column<LOCAL, 0>(v, row, sl, words, S, part, T, mn, mx, flags, pos_max, &wrong);
      else if (v.type == 4) exact_column<LOCAL, 4>(v, row, sl, words, S, part, T, mn, mx, flags, pos_max, &wrong);
      else if (v.type == 3) exact_column<LOCAL, 3>(v, row, sl, words, S, part, T, mn, mx, flags, pos_max, &wrong);
      else exact_column<LOCAL, 8>(v, row, sl, words, S, part, T, mn, mx, flags, pos_max, &wrong);
    }
    if (wrong | stopped) *(volatile uint32_t*)&s_stop = 1;
  }
  if (wrong) atomicOr(status, wrong);
  if (!LOCAL) return;
  __syncthreads();
  if (s_stop) return;   // the caller starts over in another form
  // the CTA's groups merged into the table, each CTA from another slot on
  uint32_t from = (uint32_t)((uint64_t)blockIdx.x * S / gridDim.x);
  for (uint32_t i = threadIdx.x; i < S; i += THREADS)
  {
    uint32_t s = i + from < S ? i + from : i + from - S;
    uint32_t n = lcnt[s];
    if (n == 0) continue;
    bool claimed = false;
    uint32_t g = DIRECT ? s >> copies_log2 : exact_slot(t.key, T, EXACT_PROBES, lkey[s] >> copies_log2, &claimed);
    if (g >= T)
    {
      *(volatile uint32_t*)&s_stop = 1;
      atomicOr(status, CQL_EXACT_OVERFLOW);
    }
    if (*(volatile uint32_t*)&s_stop) break;   // no room: its other groups would each try every slot again
    atomicAdd(&t.cnt[g], n);
    atomicMin(&t.row[g], lrow[s]);
    if (lflags[s]) atomicOr(&t.flags[g], lflags[s]);
    for (uint32_t j = 0; j < p.sums; j++)
    {
      const uint32_t* w = lsum + (uint64_t)j * 4 * S + s;
      __int128 v = (__int128)(((unsigned __int128)(((unsigned long long)w[3 * S] << 32) | w[2 * S]) << 64) | (((unsigned long long)w[S] << 32) | w[0]));
      bool negative = v < 0;
      exact_add_parts(t.part + (uint64_t)j * 3 * T + g, T, p.low_bits, (unsigned __int128)(negative ? -v : v), negative);
    }
    for (uint32_t j = 0; j < p.mins; j++)
      if (lmn[j * S + s] != ~0ull) atomicMin(&t.mn[(uint64_t)j * T + g], lmn[j * S + s]);
    for (uint32_t j = 0; j < p.maxs; j++)
      if (lmx[j * S + s] != 0ull) atomicMax(&t.mx[(uint64_t)j * T + g], lmx[j * S + s]);
  }
}

// T * 2^base rounded once to a double: the top 64 bits with the rest as a sticky bit convert with the one
// rounding; the scaling is exact (base >= -1074, so a subnormal result has no bits to lose).
__device__ __forceinline__ double exact_double(__int128 total, int base)
{
  bool negative = total < 0;
  unsigned __int128 u = (unsigned __int128)(negative ? -total : total);
  unsigned long long hi = (unsigned long long)(u >> 64), lo = (unsigned long long)u;
  double d;
  if (hi == 0) d = (double)lo;
  else
  {
    int z = __clzll((long long)hi), sh = 64 - z;
    unsigned long long top = (unsigned long long)(u >> sh);
    if ((unsigned __int128)top << sh != u) top |= 1ull;
    d = (double)top;
    base += sh;
  }
  d = scalbn(d, base);
  return negative ? -d : d;
}

__device__ __forceinline__ void exact_write(const CqlGroupPlan& p, const ExactTable& t, uint32_t s, uint64_t g, unsigned long long* repr,
                                            unsigned long long* counts, double* results)
{
  const uint32_t T = p.slots;
  uint32_t n = t.cnt[s], flags = t.flags[s];
  repr[g] = t.row[s];
  counts[g] = n;
  const double pow10[7] = { 1.0, 10.0, 100.0, 1000.0, 10000.0, 100000.0, 1000000.0 };
#pragma unroll 1
  for (uint32_t e = 0; e < p.expr_count; e++)
  {
    uint32_t f = p.expr_func[e], c = p.expr_col[e];
    double r = (double)n;
    if (f == 1 || f == 2)
    {
      const unsigned long long* part = t.part + (uint64_t)p.col_sum[c] * 3 * T + s;
      __int128 total = (__int128)(long long)part[0] + ((__int128)(long long)part[T] << p.low_bits) + ((__int128)(long long)part[2ull * T] << 63);
      uint32_t fl = (flags >> (3 * c)) & 7u;
      double sum = exact_double(total, p.col_base[c]);
      if (p.decimals) sum = __ddiv_rn(sum, pow10[p.col_scale[c]]);
      if ((fl & 1u) || (fl & 6u) == 6u) sum = __longlong_as_double(0x7ff8000000000000ll);
      else if (fl & 2u) sum = __longlong_as_double(0x7ff0000000000000ll);
      else if (fl & 4u) sum = __longlong_as_double((long long)0xfff0000000000000ull);
      r = f == 2 ? __ddiv_rn(sum, (double)n) : sum;
    }
    else if (f == 3 || f == 4)
    {
      // a member reduce starts at 1e300 and -1e300
      unsigned long long o = f == 3 ? t.mn[(uint64_t)p.col_min[c] * T + s] : t.mx[(uint64_t)p.col_max[c] * T + s];
      bool none = f == 3 ? o == ~0ull : o == 0ull;
      double v = cql_f64_from_order_key(o);
      if (f == 3) r = none || v > 1.0e300 ? 1.0e300 : v;
      else r = none || v < -1.0e300 ? -1.0e300 : v;
      if (p.decimals) r = __ddiv_rn(r, pow10[p.col_scale[c]]);
    }
    results[g * p.expr_count + e] = r;
  }
}

// Small tables (word 2 = 0): CTA b takes slots [256 b, 256 b + 256), after the groups of the slots before, which it
// counts itself. Large ones: the slots listed in order by the caller (the bitmap's rows).
#define EXACT_EMIT_SLOTS 65536u

__global__ void __launch_bounds__(GROUP_THREADS) k_group_exact_emit(CqlLaunch a, uint64_t cap, bool listed)
{
  __shared__ CqlGroupPlan p;
  __shared__ uint32_t s_warp[GROUP_THREADS / 32], s_before;
  for (uint32_t i = threadIdx.x; i < sizeof(CqlGroupPlan) / 4; i += GROUP_THREADS) ((uint32_t*)&p)[i] = ((const uint32_t*)a.buf[1])[i];
  if (threadIdx.x == 0) s_before = 0;
  __syncthreads();
  if (*(const uint32_t*)a.buf[2]) return;
  ExactTable t = exact_table(p, a.buf[0]);
  uint32_t* header = (uint32_t*)a.buf[3];
  unsigned long long* repr = (unsigned long long*)a.buf[4];
  unsigned long long* counts = (unsigned long long*)a.buf[5];
  double* results = (double*)a.buf[6];
  if (listed)
  {
    const uint32_t* list = (const uint32_t*)a.buf[7];
    uint32_t groups = *(const uint32_t*)a.buf[8];
    if (blockIdx.x == 0 && threadIdx.x == 0) header[0] = groups;
    uint64_t n = min((uint64_t)groups, cap);
    for (uint64_t g = (uint64_t)blockIdx.x * GROUP_THREADS + threadIdx.x; g < n; g += (uint64_t)gridDim.x * GROUP_THREADS)
      if (list[g] < p.slots) exact_write(p, t, list[g], g, repr, counts, results);
    return;
  }
  uint32_t first = blockIdx.x * GROUP_THREADS, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, mine = 0;
#pragma unroll 8
  for (uint32_t s = threadIdx.x; s < first; s += GROUP_THREADS) mine += t.cnt[s] != 0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, o);
  if (lane == 0 && mine) atomicAdd(&s_before, mine);
  uint32_t s = first + threadIdx.x;
  bool there = s < p.slots && t.cnt[s] != 0;
  uint32_t m = __ballot_sync(0xffffffffu, there);
  if (lane == 0) s_warp[warp] = (uint32_t)__popc(m);
  __syncthreads();
  uint32_t g = s_before + (uint32_t)__popc(m & ((1u << lane) - 1u)), all = s_before;
  for (uint32_t w = 0; w < GROUP_THREADS / 32; w++)
  {
    if (w < warp) g += s_warp[w];
    all += s_warp[w];
  }
  if (there && g < cap) exact_write(p, t, s, g, repr, counts, results);
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) header[0] = all;
}

// The launchers read the plan on the host: the operator layer puts the same plan in binding 12 (1) on the device and
// names its shape in the words: word 2 local slots, 3 local bytes, word 4 direct, 5 the table is a guess, word 6 its slots.
template <bool LOCAL, bool DIRECT, int THREADS, uint32_t PROBES = EXACT_PROBES>
static int launch_exact_as(const CqlLaunch& a, uint64_t rows, size_t smem, int per_sm, cudaStream_t stream)
{
  const void* fn = (const void*)k_group_exact<LOCAL, DIRECT, THREADS, PROBES>;
  if (LOCAL && smem > 40 * 1024)
  {
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
  }
  uint32_t grid = cql_stream_grid((rows + THREADS * EXACT_ROWS - 1) / (THREADS * EXACT_ROWS), per_sm);
  k_group_exact<LOCAL, DIRECT, THREADS, PROBES><<<grid, THREADS, smem, stream>>>(a, rows);
  CQL_LAUNCH_CHECK();
  return 0;
}

static int launch_group_exact(const CqlLaunch& a, uint32_t gws, uint32_t lws, cudaStream_t stream)
{
  (void)gws;
  (void)lws;
  uint64_t rows = a.push[0];
  uint32_t local_slots = cql_word(a, 2), local_bytes = cql_word(a, 3), slots = cql_word(a, 6);
  bool direct = cql_word(a, 4) != 0;
  if (rows == 0) return 0;
  if (rows > 0x7fffffffull || slots == 0 || a.bytes[12] < sizeof(CqlGroupPlan) || a.bytes[14] < 4 || a.bytes[13] < a.push[4]) return (int)cudaErrorInvalidValue;
  if (local_slots == 0 && !direct && cql_word(a, 5)) return launch_exact_as<false, false, 256, EXACT_GUESS_PROBES>(a, rows, 0, 4, stream);
  if (local_slots == 0)
    return direct ? launch_exact_as<false, true, 256>(a, rows, 0, 4, stream) : launch_exact_as<false, false, 256>(a, rows, 0, 4, stream);
  if (local_bytes > (uint32_t)g_cql_max_smem_optin - 2048) return (int)cudaErrorInvalidValue;
  if (local_bytes <= 48 * 1024)
    return direct ? launch_exact_as<true, true, 256>(a, rows, local_bytes, 4, stream) : launch_exact_as<true, false, 256>(a, rows, local_bytes, 4, stream);
  if (local_bytes <= 104 * 1024)
    return direct ? launch_exact_as<true, true, 512>(a, rows, local_bytes, 2, stream) : launch_exact_as<true, false, 512>(a, rows, local_bytes, 2, stream);
  return direct ? launch_exact_as<true, true, 1024>(a, rows, local_bytes, 1, stream) : launch_exact_as<true, false, 1024>(a, rows, local_bytes, 1, stream);
}

static int launch_group_exact_emit(const CqlLaunch& a, uint32_t gws, uint32_t lws, cudaStream_t stream)
{
  (void)gws;
  (void)lws;
  uint64_t cap = a.push[0];
  bool listed = cql_word(a, 2) != 0;
  uint32_t slots = cql_word(a, 6), exprs = cql_word(a, 4);
  if (slots == 0 || exprs == 0 || exprs > 8 || a.bytes[3] < 4 || a.bytes[4] < cap * 8 || a.bytes[5] < cap * 8 || a.bytes[6] < cap * 8 * exprs)
    return (int)cudaErrorInvalidValue;
  if (!listed && slots > EXACT_EMIT_SLOTS) return (int)cudaErrorInvalidValue;
  if (listed && (a.bytes[7] < cap * 4 || a.bytes[8] < 4)) return (int)cudaErrorInvalidValue;
  uint64_t most = listed ? std::min<uint64_t>(cap, slots) : slots;
  uint64_t blocks = (most + GROUP_THREADS - 1) / GROUP_THREADS;
  uint32_t grid = listed ? cql_stream_grid(blocks, 8) : (uint32_t)blocks;
  k_group_exact_emit<<<grid, GROUP_THREADS, 0, stream>>>(a, cap, listed);
  CQL_LAUNCH_CHECK();
  return 0;
}

const CqlKernelDesc cql_kernels_group[] = {
  { "cql_hll_rows", launch_hll_rows },
  { "cql_group_exact", launch_group_exact },
  { "cql_group_exact_emit", launch_group_exact_emit },
  { nullptr, nullptr },
};
