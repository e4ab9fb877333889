/*
 * cql_group_plan.h - the plan of an exact GROUP BY (cql_group_exact, csrc/k_group.cu), written by the operator
 * layer (cql_ops_hash.c) and read by the kernels.
 */
#ifndef CQL_GROUP_PLAN_H
#define CQL_GROUP_PLAN_H

#include <stdint.h>

#ifdef __CUDACC__
#define CQL_PLAN_FN __host__ __device__ static inline
#else
#define CQL_PLAN_FN static inline
#endif

#define CQL_EXACT_KEYS 4
#define CQL_EXACT_COLUMNS 8
#define CQL_EXACT_EXPRS 8

/* how a key's value becomes a digit of the group's number (besides the CQL types U32, U64, F32, F64, I32, I64):
   64-bit integers of a range in which doubles repeat, as their doubles' bits */
#define CQL_EXACT_KEY_U64_AS_F64 9
#define CQL_EXACT_KEY_I64_AS_F64 10

/* what is kept of a column */
#define CQL_EXACT_SUM 1u
#define CQL_EXACT_MIN 2u
#define CQL_EXACT_MAX 4u
#define CQL_EXACT_WHOLE 8u    /* whole numbers below 2^32 in magnitude: a sum in units of 1 */
#define CQL_EXACT_DECIMAL 16u /* f64 decimals summed as the whole number round(x * 10^scale), below 2^31 */

/* why the tables cannot be used (the status word) */
#define CQL_EXACT_OVERFLOW 1u /* more groups than the table takes */
#define CQL_EXACT_RANGE 2u    /* a value whose bits lie outside the sums' window */
#define CQL_EXACT_KEY 4u      /* a key that is NaN, -0.0 or outside its column's range */

typedef struct CqlGroupPlan
{
  uint32_t key_count, column_count, expr_count, decimals;
  uint32_t key_type[CQL_EXACT_KEYS];
  uint64_t key_min[CQL_EXACT_KEYS];    /* subtracted from the value (or the bits) */
  uint64_t key_range[CQL_EXACT_KEYS];  /* its digits: below this; 0 = all 64 bits (a single key) */
  uint32_t col_type[CQL_EXACT_COLUMNS];
  uint32_t col_what[CQL_EXACT_COLUMNS];
  int32_t col_base[CQL_EXACT_COLUMNS];  /* a sum is in units of 2^base */
  uint32_t col_scale[CQL_EXACT_COLUMNS];
  uint32_t col_sum[CQL_EXACT_COLUMNS], col_min[CQL_EXACT_COLUMNS], col_max[CQL_EXACT_COLUMNS];  /* which sum, minimum, maximum it is */
  uint32_t expr_func[CQL_EXACT_EXPRS], expr_col[CQL_EXACT_EXPRS];
  uint32_t sums, mins, maxs, low_bits;  /* low_bits: the bits of a sum's lowest part, ceil(log2(rows)) + 1 */
  uint32_t direct;                      /* 1: the table is indexed by the group's number */
  uint32_t slots;                       /* the table's slots (a power of two unless direct) */
  uint32_t local_slots, copies_log2;    /* a CTA's own table in shared memory (0: none), copies of each group in it */
} CqlGroupPlan;

/* the table: parts in this order, each `slots` long. The first region starts as all ones, the second as zeros. */
CQL_PLAN_FN uint64_t cql_exact_ones_bytes(const CqlGroupPlan* p)
{
  uint64_t b = (uint64_t)p->slots * ((p->direct ? 0 : 8) + 8ull * p->mins + 4);
  return (b + 15) & ~15ull;
}
CQL_PLAN_FN uint64_t cql_exact_zero_bytes(const CqlGroupPlan* p)
{
  return (uint64_t)p->slots * (24ull * p->sums + 8ull * p->maxs + 4 + 4);
}

#endif
