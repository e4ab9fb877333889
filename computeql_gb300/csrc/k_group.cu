// GROUP BY forms of GB300's own, beside the reference's hash path in k_hash.cu.
#include "cql_bits.cuh"

#define GROUP_THREADS 256

// ---------------------------------------------------------------------------------------------
// cql_hll_rows: the HyperLogLog registers of whole columns, for a table or per value of a small-range key:
// binding 0 the key (u32 words; the first column again without a key), 1..8 the columns, 9 the registers
// (u32, zero before) [key value][column][2^10]; word 0 rows, 2 the columns, 4 their CQL types (4 bits each),
// 6 the key's values (0: no key), 8 its smallest (bits). A row whose key lies outside the values is left out.
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
      at[i] = at[i] < values ? (at[i] * columns + column) * HLL_REGS + bucket : 0xffffffffu;   // values x columns <= 2^16
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
  if (columns > 8 || rows > 0xffffffffull || values > 8192 || a.bytes[9] < (uint64_t)(values ? values : 1) * columns * HLL_REGS * 4 ||
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

const CqlKernelDesc cql_kernels_group[] = {
  { "cql_hll_rows", launch_hll_rows },
  { nullptr, nullptr },
};
