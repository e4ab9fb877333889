/*
 * cql_ops_sort.c - ORDER BY up to 4 numeric keys, ties by input position (qe_sort_rows,
 * src/query_exec/query_exec.c:5376-6155; the tie rule of the generated sort, query_kernel.c:2156-2177),
 * as a stable LSD radix sort on the GPU: the last key first, each key 8 bits per pass. Keys of more than
 * 32 bits together are sorted by a 32-bit prefix of them, then within the runs that share it.
 */
#include "cqlops.h"
#include "cql_ops_internal.h"

#include <math.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#define SORT_TILE 4096
#define QE_GPU_WORKGROUP_SIZE 256

static int refuse(const char* why)
{
  cqlops_note_error(why);
  return 0;
}

static CqlBuffer* pooled(const char* name, uint64_t size, uint32_t flags)
{
  return cqlcuda_buffer_alloc_pooled(name, (uint64_t)strlen(name), size ? size : 8, flags, NULL);
}

static int key_bytes(uint32_t type)
{
  switch (type)
  {
    case CQLOPS_TYPE_U32: case CQLOPS_TYPE_I32: case CQLOPS_TYPE_F32: case 9: case 12: return 4;
    case CQLOPS_TYPE_U64: case CQLOPS_TYPE_I64: case CQLOPS_TYPE_F64: case 10: case 11: return 8;
    default: return 0;
  }
}

/* The sort's checks and scratch; 0 (with the reason noted) when the keys cannot be sorted. */
static int sort_check(const CqlColumn* keys, uint32_t key_count, CqlBuffer* selection, uint64_t selection_count, uint64_t* out_n)
{
  if (key_count == 0 || key_count > 4) return refuse("1 to 4 sort keys");
  uint64_t rows = keys[0].rows;
  uint64_t n = selection ? selection_count : rows;
  if (!cqlops_rows_fit(rows) || !cqlops_rows_fit(n)) return 0;
  for (uint32_t k = 0; k < key_count; k++)
  {
    int narrow_ok = keys[k].width == 0 || (keys[k].width <= 3 && key_bytes(keys[k].type) == 4 && keys[k].type != CQLOPS_TYPE_F32);
    if (keys[k].rows != rows || (!keys[k].buffer && keys[k].width != 3) || !narrow_ok || !key_bytes(keys[k].type))
      return refuse("sort keys are numeric columns of the same length (narrow encodings only for 32-bit integers)");
  }
  if (selection && cqlcuda_buffer_size(selection) < n * 4) return refuse("selection buffer smaller than its count");
  *out_n = n;
  return 1;
}

/* One 8-bit pass: digit p of the keys in kbuf[cur] counted (`count`; else it is already), its runs' places, and the keys and
   positions scattered to the other buffers. `map`: the selection's rows are written instead of positions; `last`: no keys
   are written; `identity`: the positions in are the row numbers. */
static void digit_pass(CqlBatch* b, CqlKernel* kcount, CqlKernel* koffsets, CqlKernel* kscatter, CqlBuffer* const* kbuf, CqlBuffer* const* perm,
                       CqlBuffer* hist, CqlBuffer* offsets, CqlBuffer* totals, CqlBuffer* sel, uint64_t n, uint64_t tiles, int kb, uint32_t p, int count,
                       int map, int last, int identity, int cur)
{
  uint64_t pass_totals = (uint64_t)p * 256 * 4;
  if (count)
  {
    cqlcuda_kernel_set_arg_buffer(kcount, 0, kbuf[cur]);
    cqlcuda_kernel_set_arg_buffer(kcount, 1, hist);
    cqlcuda_kernel_set_arg_buffer_range(kcount, 2, totals, pass_totals, 256 * 4);
    cqlcuda_kernel_set_arg_u64(kcount, 0, n);
    cqlcuda_kernel_set_arg_u64(kcount, 1, (uint64_t)(8 * p));
    cqlcuda_kernel_set_arg_u64(kcount, 2, (uint64_t)kb);
    cqlcuda_batch_kernel_execute(b, kcount, (uint32_t)(tiles * 256), 256);
  }
  cqlcuda_kernel_set_arg_buffer(koffsets, 0, hist);
  cqlcuda_kernel_set_arg_buffer_range(koffsets, 1, totals, pass_totals, 256 * 4);
  cqlcuda_kernel_set_arg_buffer(koffsets, 2, offsets);
  cqlcuda_kernel_set_arg_u64(koffsets, 0, n);
  cqlcuda_batch_kernel_execute(b, koffsets, 256u * 512u, 512);
  cqlcuda_kernel_set_arg_buffer(kscatter, 0, kbuf[cur]);
  cqlcuda_kernel_set_arg_buffer(kscatter, 1, perm[cur]);
  cqlcuda_kernel_set_arg_buffer(kscatter, 2, kbuf[cur ^ 1]);
  cqlcuda_kernel_set_arg_buffer(kscatter, 3, perm[cur ^ 1]);
  cqlcuda_kernel_set_arg_buffer(kscatter, 4, offsets);
  cqlcuda_kernel_set_arg_buffer(kscatter, 5, sel);
  cqlcuda_kernel_set_arg_buffer_range(kscatter, 6, totals, pass_totals, 256 * 4);
  cqlcuda_kernel_set_arg_u64(kscatter, 0, n);
  cqlcuda_kernel_set_arg_u64(kscatter, 1, (uint64_t)(8 * p));
  cqlcuda_kernel_set_arg_u64(kscatter, 2, (uint64_t)kb);
  cqlcuda_kernel_set_arg_u64(kscatter, 3, map ? 1 : 0);
  cqlcuda_kernel_set_arg_u64(kscatter, 4, last ? 1 : 0);
  cqlcuda_kernel_set_arg_u64(kscatter, 5, identity ? 1 : 0);
  cqlcuda_batch_kernel_execute(b, kscatter, (uint32_t)(tiles * 256), 256);
}

/* Queues the stable LSD radix sort of n > 0 rows into batch b; *out_sorted receives the buffer that holds
   the row numbers in sorted order when the batch has run. top_bits (optional): below which bit each key varies. */
static int sort_enqueue(CqlBatch* b, const CqlColumn* keys, uint32_t key_count, const uint32_t* desc, CqlBuffer* selection, uint64_t n,
                        const uint32_t* top_bits, CqlBuffer** out_sorted)
{
  uint32_t widest = 4;
  for (uint32_t k = 0; k < key_count; k++)
    if (key_bytes(keys[k].type) > (int)widest) widest = 8;
  uint64_t tiles = (n + SORT_TILE - 1) / SORT_TILE;
  uint64_t hist_n = tiles * 256;
  CqlBuffer* perm[2] = { pooled("sort_perm_a", n * 4, CQLCUDA_BUFFER_READ_WRITE), pooled("sort_perm_b", n * 4, CQLCUDA_BUFFER_READ_WRITE) };
  CqlBuffer* kbuf[2] = { pooled("sort_keys_a", n * widest, CQLCUDA_BUFFER_READ_WRITE), pooled("sort_keys_b", n * widest, CQLCUDA_BUFFER_READ_WRITE) };
  CqlBuffer* hist = pooled("sort_hist", hist_n * 4, CQLCUDA_BUFFER_READ_WRITE);
  CqlBuffer* offsets = pooled("sort_offsets", hist_n * 4, CQLCUDA_BUFFER_READ_WRITE);
  CqlBuffer* totals = pooled("sort_digit_totals", 8 * 256 * 4, CQLCUDA_BUFFER_READ_WRITE);
  CqlKernel* kkeys = cqlcuda_kernel_alloc("cql_sort_keys", 13);
  CqlKernel* kcount = cqlcuda_kernel_alloc("cql_radix_count", 15);
  CqlKernel* koffsets = cqlcuda_kernel_alloc("cql_radix_offsets", 17);
  CqlKernel* kscatter = cqlcuda_kernel_alloc("cql_radix_scatter", 17);
  if (!perm[0] || !perm[1] || !kbuf[0] || !kbuf[1] || !hist || !offsets || !totals || !kkeys || !kcount || !koffsets || !kscatter)
    return 0;
  CqlBuffer* sel = selection ? selection : perm[0];
  /* a key's passes: its bytes, or those below the bit it varies under (top_bits); a key that does not vary has none */
  int passes[4] = { 0, 0, 0, 0 }, first_sorted = -1, last_key = -1, cur = 0;
  for (int k = (int)key_count - 1; k >= 0; k--)
  {
    passes[k] = top_bits ? (int)(top_bits[k] + 7) / 8 : key_bytes(keys[k].type);
    if (k == 0 && first_sorted < 0 && passes[0] == 0) passes[0] = 1;   /* nothing varies: one pass that copies */
    if (passes[k] && first_sorted < 0) first_sorted = k;
    if (passes[k]) last_key = k;
  }
  for (int k = (int)key_count - 1; k >= 0; k--)
  {
    int kb = key_bytes(keys[k].type);
    int first_key = k == first_sorted;
    if (passes[k] == 0) continue;
    /* each pass's digit totals start at zero: the key pass counts the first digit, the count kernels the rest */
    cqlcuda_batch_fill_range(b, totals, 0, (uint64_t)kb * 256 * 4, 0);
    /* the key in the current order, with its first digit counted (the first key sorted starts from the
       identity permutation, which the first scatter takes as row numbers) */
    cqlcuda_kernel_set_arg_buffer(kkeys, 0, keys[k].buffer ? keys[k].buffer : perm[cur]);
    cqlcuda_kernel_set_arg_buffer(kkeys, 1, perm[cur]);
    cqlcuda_kernel_set_arg_buffer(kkeys, 2, kbuf[cur]);
    cqlcuda_kernel_set_arg_buffer(kkeys, 3, sel);
    cqlcuda_kernel_set_arg_buffer(kkeys, 4, hist);
    cqlcuda_kernel_set_arg_buffer(kkeys, 5, totals);
    cqlcuda_kernel_set_arg_u64(kkeys, 0, n);
    cqlcuda_kernel_set_arg_u64(kkeys, 1, keys[k].type);
    cqlcuda_kernel_set_arg_u64(kkeys, 2, desc && desc[k] ? 1 : 0);
    cqlcuda_kernel_set_arg_u64(kkeys, 3, first_key ? 0 : 1);
    cqlcuda_kernel_set_arg_u64(kkeys, 4, selection ? 1 : 0);
    cqlcuda_kernel_set_arg_u64(kkeys, 5, keys[k].width);
    cqlcuda_kernel_set_arg_u64(kkeys, 6, keys[k].base);
    cqlcuda_kernel_set_arg_u64(kkeys, 7, first_key ? 3 : 1);
    cqlcuda_batch_kernel_execute(b, kkeys, (uint32_t)n, QE_GPU_WORKGROUP_SIZE);
    for (int p = 0; p < passes[k]; p++)
    {
      int last = k == last_key && p == passes[k] - 1;
      digit_pass(b, kcount, koffsets, kscatter, kbuf, perm, hist, offsets, totals, sel, n, tiles, kb, (uint32_t)p, p > 0, last && selection != NULL, last,
                 first_key && p == 0, cur);
      cur ^= 1;
    }
  }
  *out_sorted = perm[cur];
  return 1;
}

/* ---- more than 32 key bits: by a prefix of the bits that vary, then the short runs that share one (cql_sort_range ...
   cql_sort_runs, csrc/k_sort.cu) ----
   -1: the keys' rows share prefixes too often (a sample says so, or the runs pass found a long run out of order), and the
   passes over every digit sort them; top_bits then says below which bit each key varies. From SORT_PREFIX_MIN_ROWS rows
   on: the ranges are read back before the passes are queued, a wait of some 15 us, against four passes saved or more (17000 rows
   by one f64 key 172 to 145 us, by f64 and u32 250 to 146; 2M rows 348 and 479 to 276 and 293). Where the sample sends the rows
   back to the passes, those 20 to 45 us are lost: 300k rows by a price and a u32 252 to 282, 5M rows 735 to 767. */
#define SORT_PREFIX_MIN_ROWS 16384u
#define SORT_SAMPLE 2048ull
#define SORT_RUN_ROWS 16.0   /* the runs pass takes up to 128 rows; 20M rows that share a prefix by 40: 2.5 ms, the passes 3.7 */

static uint32_t bits_of(uint64_t v)
{
  uint32_t n = 0;
  for (; v; v >>= 1) n++;
  return n;
}

static uint64_t f64_order_word(double x)
{
  uint64_t b;
  memcpy(&b, &x, 8);
  if ((b << 1) == 0) b = 0;
  return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}

/* A key's (smallest, largest) order words, as cql_sort_range finds them, in the order the kernels sort by: 64-bit integers as
   themselves within 2^53 of zero, else as doubles. *out_span: the bits of its distances; *out_top: the bit below which the
   key pass's words vary. */
static void key_range_bits(const CqlColumn* key, const uint64_t* range, uint32_t* out_span, uint32_t* out_top)
{
  uint64_t lo = range[0], top = range[1];
  int wide = key_bytes(key->type) == 8;
  if (wide && key->type != CQLOPS_TYPE_F64)
  {
    int is_signed = key->type != CQLOPS_TYPE_U64;
    uint64_t zero = is_signed ? 0x8000000000000000ull : 0, near = 1ull << 53;
    uint64_t flo = f64_order_word(is_signed ? (double)(int64_t)(lo ^ zero) : (double)lo);
    uint64_t ftop = f64_order_word(is_signed ? (double)(int64_t)(top ^ zero) : (double)top);
    *out_top = bits_of(flo ^ ftop);
    if (!(top <= zero + near && (!is_signed || lo >= zero - near)))
    {
      lo = flo;
      top = ftop;
    }
  }
  else *out_top = bits_of(lo ^ top);
  *out_span = bits_of(top - lo);
}

static void sort_bind(CqlKernel* kn, const CqlColumn* keys, uint32_t key_count, const uint32_t* desc, CqlBuffer* selection, CqlBuffer* filler, uint64_t n)
{
  uint64_t types = 0, widths = 0, down = 0, bases[2] = { 0, 0 };
  for (uint32_t k = 0; k < 4; k++)
  {
    cqlcuda_kernel_set_arg_buffer(kn, k, k < key_count && keys[k].buffer ? keys[k].buffer : filler);
    if (k >= key_count) continue;
    types |= (uint64_t)(keys[k].type & 0xfu) << (4 * k);
    widths |= (uint64_t)(keys[k].width & 3u) << (2 * k);
    if (desc && desc[k]) down |= 1ull << k;
    bases[k / 2] |= (uint64_t)keys[k].base << (32 * (k % 2));
  }
  cqlcuda_kernel_set_arg_buffer(kn, 4, selection ? selection : filler);
  cqlcuda_kernel_set_arg_u64(kn, 0, n);
  cqlcuda_kernel_set_arg_u64(kn, 1, (uint64_t)key_count | (uint64_t)(selection != NULL) << 32);
  cqlcuda_kernel_set_arg_u64(kn, 2, types | down << 32);
  cqlcuda_kernel_set_arg_u64(kn, 3, widths);
  cqlcuda_kernel_set_arg_u64(kn, 4, bases[0]);
  cqlcuda_kernel_set_arg_u64(kn, 5, bases[1]);
}

static int sort_by_prefix(const CqlColumn* keys, uint32_t key_count, const uint32_t* desc, CqlBuffer* selection, uint64_t n, uint32_t* out_rows,
                          uint64_t m, uint32_t* top_bits)
{
  uint64_t tiles = (n + SORT_TILE - 1) / SORT_TILE, hist_n = tiles * 256;
  CqlBuffer* perm[2] = { pooled("sort_perm_a", n * 4, CQLCUDA_BUFFER_READ_WRITE), pooled("sort_perm_b", n * 4, CQLCUDA_BUFFER_READ_WRITE) };
  CqlBuffer* kbuf[2] = { pooled("sort_keys_a", n * 4, CQLCUDA_BUFFER_READ_WRITE), pooled("sort_keys_b", n * 4, CQLCUDA_BUFFER_READ_WRITE) };
  CqlBuffer* hist = pooled("sort_hist", hist_n * 4, CQLCUDA_BUFFER_READ_WRITE);
  CqlBuffer* offsets = pooled("sort_offsets", hist_n * 4, CQLCUDA_BUFFER_READ_WRITE);
  CqlBuffer* totals = pooled("sort_digit_totals", 8 * 256 * 4, CQLCUDA_BUFFER_READ_WRITE);
  CqlBuffer* facts = pooled("sort_prefix_facts", 96, CQLCUDA_BUFFER_READ_WRITE);   /* (smallest, largest) per key, sample, status */
  CqlKernel* krange = cqlcuda_kernel_alloc("cql_sort_range", 14);
  CqlKernel* ksample = cqlcuda_kernel_alloc("cql_sort_sample", 15);
  CqlKernel* kprefix = cqlcuda_kernel_alloc("cql_sort_prefix", 15);
  CqlKernel* kruns = cqlcuda_kernel_alloc("cql_sort_runs", 13);
  CqlKernel* kcount = cqlcuda_kernel_alloc("cql_radix_count", 15);
  CqlKernel* koffsets = cqlcuda_kernel_alloc("cql_radix_offsets", 17);
  CqlKernel* kscatter = cqlcuda_kernel_alloc("cql_radix_scatter", 17);
  if (!perm[0] || !perm[1] || !kbuf[0] || !kbuf[1] || !hist || !offsets || !totals || !facts || !krange || !ksample || !kprefix || !kruns || !kcount ||
      !koffsets || !kscatter)
    return 0;
  uint64_t host[12] = { ~0ull, 0, ~0ull, 0, ~0ull, 0, ~0ull, 0, 0, 0, 0, 0 };
  sort_bind(krange, keys, key_count, desc, selection, perm[0], n);
  cqlcuda_kernel_set_arg_buffer_range(krange, 5, facts, 0, 64);
  sort_bind(ksample, keys, key_count, desc, selection, perm[0], n);
  cqlcuda_kernel_set_arg_buffer_range(ksample, 5, facts, 0, 64);
  cqlcuda_kernel_set_arg_buffer_range(ksample, 6, facts, 64, 4);
  CqlBatch* b = cqlcuda_batch_begin(96, 96);
  cqlcuda_batch_buffer_write(b, facts, host, 96);
  cqlcuda_batch_kernel_execute(b, krange, (uint32_t)n, QE_GPU_WORKGROUP_SIZE);
  cqlcuda_batch_kernel_execute(b, ksample, 1024, 1024);
  cqlcuda_batch_buffer_read(b, facts, host, 96);
  if (!cqlcuda_batch_end(b)) return 0;
  uint32_t bits = 0, rest = 0;
  for (uint32_t k = 0; k < key_count; k++)
  {
    uint32_t span;
    key_range_bits(&keys[k], host + 2 * k, &span, &top_bits[k]);
    bits += span;
  }
  if (bits > 32)
  {
    bits = 32;
    rest = 1;
    /* rows of the sample that share another's prefix and no more: as many as runs of SORT_RUN_ROWS rows would give, all
       but one of each of the n / SORT_RUN_ROWS runs that the sample meets */
    double runs = (double)n / SORT_RUN_ROWS, limit = (double)SORT_SAMPLE + runs * expm1(-(double)SORT_SAMPLE / runs);
    if ((double)(uint32_t)host[8] > (limit < 4.0 ? 4.0 : limit)) return -1;
  }
  uint32_t passes = bits ? (bits + 7) / 8 : 1;
  sort_bind(kprefix, keys, key_count, desc, selection, perm[0], n);
  cqlcuda_kernel_set_arg_buffer(kprefix, 5, kbuf[0]);
  cqlcuda_kernel_set_arg_buffer(kprefix, 6, hist);
  cqlcuda_kernel_set_arg_buffer_range(kprefix, 7, totals, 0, 256 * 4);
  cqlcuda_kernel_set_arg_buffer_range(kprefix, 8, facts, 0, 64);
  b = cqlcuda_batch_begin(0, 64);
  cqlcuda_batch_fill_range(b, totals, 0, (uint64_t)passes * 256 * 4, 0);
  cqlcuda_batch_kernel_execute(b, kprefix, (uint32_t)n, QE_GPU_WORKGROUP_SIZE);
  int cur = 0;
  for (uint32_t p = 0; p < passes; p++)
  {
    int last = p + 1 == passes;
    digit_pass(b, kcount, koffsets, kscatter, kbuf, perm, hist, offsets, totals, selection ? selection : perm[0], n, tiles, 4, p, p > 0,
               last && !rest && selection != NULL, last && !rest, p == 0, cur);
    cur ^= 1;
  }
  uint32_t status = 0;
  if (rest)
  {
    sort_bind(kruns, keys, key_count, desc, selection, perm[cur], n);
    cqlcuda_kernel_set_arg_buffer(kruns, 5, kbuf[cur]);
    cqlcuda_kernel_set_arg_buffer(kruns, 6, perm[cur]);
    cqlcuda_kernel_set_arg_buffer(kruns, 7, perm[cur ^ 1]);
    cqlcuda_kernel_set_arg_buffer_range(kruns, 8, facts, 0, 64);
    cqlcuda_kernel_set_arg_buffer_range(kruns, 9, facts, 80, 4);
    cqlcuda_batch_kernel_execute(b, kruns, (uint32_t)n, QE_GPU_WORKGROUP_SIZE);
    cqlcuda_batch_buffer_read_at(b, facts, 80, &status, 4);
    cur ^= 1;
  }
  if (out_rows && m) cqlcuda_batch_buffer_read(b, perm[cur], out_rows, m * 4);
  if (!cqlcuda_batch_end(b)) return 0;
  return status ? -1 : 1;
}

int cqlops_sort_rows(const CqlColumn* keys, uint32_t key_count, const uint32_t* desc, CqlBuffer* selection,
                     uint64_t selection_count, uint32_t* out_rows, uint64_t out_capacity)
{
  cqlops_note_error("");
  uint64_t n = 0;
  if (!sort_check(keys, key_count, selection, selection_count, &n)) return 0;
  if (n == 0) return 1;
  uint64_t m = n < out_capacity ? n : out_capacity;
  uint32_t bytes = 0, top_bits[4] = { 0, 0, 0, 0 };
  for (uint32_t k = 0; k < key_count; k++) bytes += (uint32_t)key_bytes(keys[k].type);
  int prefixed = bytes > 4 && n >= SORT_PREFIX_MIN_ROWS;
  if (prefixed)
  {
    int r = sort_by_prefix(keys, key_count, desc, selection, n, out_rows, m, top_bits);
    if (r >= 0) return r;
  }
  CqlBatch* b = cqlcuda_batch_begin(0, n * 4);
  CqlBuffer* sorted = NULL;
  if (!sort_enqueue(b, keys, key_count, desc, selection, n, prefixed ? top_bits : NULL, &sorted))
  {
    cqlcuda_batch_end(b);
    return 0;
  }
  if (out_rows && m) cqlcuda_batch_buffer_read(b, sorted, out_rows, m * 4);
  return cqlcuda_batch_end(b);
}

/* Result pairs put in order on the device (the join's pair output, the scan's rows with their scores): n
   records of stride_words u32 words in `records`; the pair (word first_word, word second_word) of each,
   sorted by the first word then the second (by_second) or by the first alone (ties by position) with the
   radix sort above, and up to out_capacity sorted pairs (first, second) read into out. first_bits and second_bits: below
   which bit each word orders (32: all of it), so that row numbers are sorted by the bytes they have. */
int cqlops_sort_pairs(CqlBuffer* records, uint64_t n, uint32_t stride_words, uint32_t first_word, uint32_t second_word, int by_second,
                      uint32_t first_bits, uint32_t second_bits, uint32_t* out, uint64_t out_capacity)
{
  if (n == 0 || out_capacity == 0) return 1;
  if (!cqlops_rows_fit(n)) return 0;
  CqlBuffer* first = pooled("pairs_first", n * 4, CQLCUDA_BUFFER_READ_WRITE);
  CqlBuffer* second = pooled("pairs_second", n * 4, CQLCUDA_BUFFER_READ_WRITE);
  CqlBuffer* packed = pooled("pairs_sorted", n * 8, CQLCUDA_BUFFER_READ_WRITE);
  CqlKernel* unpack = cqlcuda_kernel_alloc("cql_pairs_unpack", 16);
  CqlKernel* pack = cqlcuda_kernel_alloc("cql_pairs_pack", 14);
  if (!first || !second || !packed || !unpack || !pack) return 0;
  CqlColumn keys[2];
  memset(keys, 0, sizeof(keys));
  for (int k = 0; k < 2; k++)
  {
    keys[k].type = CQLOPS_TYPE_U32;
    keys[k].rows = n;
    keys[k].buffer = k ? second : first;
  }
  uint64_t m = n < out_capacity ? n : out_capacity;
  CqlBatch* b = cqlcuda_batch_begin(0, m * 8);
  cqlcuda_kernel_set_arg_buffer(unpack, 0, records);
  cqlcuda_kernel_set_arg_buffer(unpack, 1, first);
  cqlcuda_kernel_set_arg_buffer(unpack, 2, second);
  cqlcuda_kernel_set_arg_u64(unpack, 0, n);
  cqlcuda_kernel_set_arg_u64(unpack, 1, stride_words);
  cqlcuda_kernel_set_arg_u64(unpack, 2, first_word);
  cqlcuda_kernel_set_arg_u64(unpack, 3, second_word);
  cqlcuda_batch_kernel_execute(b, unpack, (uint32_t)n, QE_GPU_WORKGROUP_SIZE);
  CqlBuffer* sorted = NULL;
  uint32_t top_bits[4] = { first_bits, second_bits, 0, 0 };
  if (!sort_enqueue(b, keys, by_second ? 2u : 1u, NULL, NULL, n, top_bits, &sorted))
  {
    cqlcuda_batch_end(b);
    return 0;
  }
  cqlcuda_kernel_set_arg_buffer(pack, 0, sorted);
  cqlcuda_kernel_set_arg_buffer(pack, 1, first);
  cqlcuda_kernel_set_arg_buffer(pack, 2, second);
  cqlcuda_kernel_set_arg_buffer(pack, 3, packed);
  cqlcuda_kernel_set_arg_u64(pack, 0, n);
  cqlcuda_batch_kernel_execute(b, pack, (uint32_t)n, QE_GPU_WORKGROUP_SIZE);
  cqlcuda_batch_buffer_read(b, packed, out, m * 8);
  return cqlcuda_batch_end(b);
}

/* ROW_NUMBER, RANK and DENSE_RANK (qe_window_rank_gpu, src/query_exec/query_exec.c:6155-6540): the rows
   sorted by (partition keys, order keys) with the sort above, then per sorted position whether it starts a
   partition or a peer group (keys compared as F64 with !=, window_rank_flags.comp), then the three ranks by
   one scan over the positions - all in one batch. */
#define WIN_TILE 2048u
#define WIN_AGG_BYTES 24u

int cqlops_window_rank(const CqlColumn* keys, uint32_t key_count, const uint32_t* desc, uint32_t partition_key_count, CqlBuffer* selection,
                       uint64_t selection_count, uint32_t* out_rows, uint32_t* out_row_number, uint32_t* out_rank, uint32_t* out_dense_rank,
                       uint64_t out_capacity)
{
  cqlops_note_error("");
  uint64_t n = 0;
  if (partition_key_count > key_count) return refuse("more partition keys than keys");
  if (!sort_check(keys, key_count, selection, selection_count, &n)) return 0;
  if (n == 0) return 1;
  if (out_capacity < n) return refuse("the outputs must hold every row");
  uint64_t tiles = (n + WIN_TILE - 1) / WIN_TILE;
  CqlBuffer* flags = pooled("window_flags", n, CQLCUDA_BUFFER_READ_WRITE);
  CqlBuffer* agg = pooled("window_tiles", tiles * WIN_AGG_BYTES, CQLCUDA_BUFFER_READ_WRITE);
  CqlBuffer* carry = pooled("window_carry", tiles * WIN_AGG_BYTES, CQLCUDA_BUFFER_READ_WRITE);
  CqlBuffer* ranks = pooled("window_ranks", n * 12, CQLCUDA_BUFFER_READ_WRITE);
  CqlKernel* kflags = cqlcuda_kernel_alloc("cql_window_flags", 16);
  CqlKernel* ktiles = cqlcuda_kernel_alloc("cql_window_tiles", 16);
  CqlKernel* kcarry = cqlcuda_kernel_alloc("cql_window_carry", 16);
  CqlKernel* kapply = cqlcuda_kernel_alloc("cql_window_apply", 16);
  if (!flags || !agg || !carry || !ranks || !kflags || !ktiles || !kcarry || !kapply) return 0;
  CqlBatch* b = cqlcuda_batch_begin(0, n * 16);
  CqlBuffer* sorted = NULL;
  if (!sort_enqueue(b, keys, key_count, desc, selection, n, NULL, &sorted))
  {
    cqlcuda_batch_end(b);
    return 0;
  }
  uint32_t types = 0, widths = 0;
  for (uint32_t k = 0; k < key_count; k++)
  {
    types |= (keys[k].type & 0xffu) << (8 * k);
    widths |= (keys[k].width & 0xffu) << (8 * k);
  }
  cqlcuda_kernel_set_arg_buffer(kflags, 0, sorted);
  cqlcuda_kernel_set_arg_buffer(kflags, 1, flags);
  for (uint32_t k = 0; k < 4; k++)
    cqlcuda_kernel_set_arg_buffer(kflags, 2 + k, k < key_count && keys[k].buffer ? keys[k].buffer : sorted);
  cqlcuda_kernel_set_arg_u64(kflags, 0, n);
  cqlcuda_kernel_set_arg_u64(kflags, 1, (uint64_t)key_count | (uint64_t)partition_key_count << 32);
  cqlcuda_kernel_set_arg_u64(kflags, 2, (uint64_t)types | (uint64_t)widths << 32);
  cqlcuda_kernel_set_arg_u64(kflags, 3, (uint64_t)(key_count > 0 ? keys[0].base : 0) | (uint64_t)(key_count > 1 ? keys[1].base : 0) << 32);
  cqlcuda_kernel_set_arg_u64(kflags, 4, (uint64_t)(key_count > 2 ? keys[2].base : 0) | (uint64_t)(key_count > 3 ? keys[3].base : 0) << 32);
  cqlcuda_batch_kernel_execute(b, kflags, (uint32_t)n, QE_GPU_WORKGROUP_SIZE);
  cqlcuda_kernel_set_arg_buffer(ktiles, 0, flags);
  cqlcuda_kernel_set_arg_buffer(ktiles, 1, agg);
  cqlcuda_kernel_set_arg_u64(ktiles, 0, n);
  cqlcuda_batch_kernel_execute(b, ktiles, (uint32_t)(tiles * QE_GPU_WORKGROUP_SIZE), QE_GPU_WORKGROUP_SIZE);
  cqlcuda_kernel_set_arg_buffer(kcarry, 0, agg);
  cqlcuda_kernel_set_arg_buffer(kcarry, 1, carry);
  cqlcuda_kernel_set_arg_u64(kcarry, 0, tiles);
  cqlcuda_batch_kernel_execute(b, kcarry, QE_GPU_WORKGROUP_SIZE, QE_GPU_WORKGROUP_SIZE);
  cqlcuda_kernel_set_arg_buffer(kapply, 0, flags);
  cqlcuda_kernel_set_arg_buffer(kapply, 1, carry);
  cqlcuda_kernel_set_arg_buffer_range(kapply, 2, ranks, 0, n * 4);
  cqlcuda_kernel_set_arg_buffer_range(kapply, 3, ranks, n * 4, n * 4);
  cqlcuda_kernel_set_arg_buffer_range(kapply, 4, ranks, n * 8, n * 4);
  cqlcuda_kernel_set_arg_u64(kapply, 0, n);
  cqlcuda_batch_kernel_execute(b, kapply, (uint32_t)(tiles * QE_GPU_WORKGROUP_SIZE), QE_GPU_WORKGROUP_SIZE);
  if (out_rows) cqlcuda_batch_buffer_read(b, sorted, out_rows, n * 4);
  if (out_row_number) cqlcuda_batch_buffer_read_at(b, ranks, 0, out_row_number, n * 4);
  if (out_rank) cqlcuda_batch_buffer_read_at(b, ranks, n * 4, out_rank, n * 4);
  if (out_dense_rank) cqlcuda_batch_buffer_read_at(b, ranks, n * 8, out_dense_rank, n * 4);
  return cqlcuda_batch_end(b);
}
