/*
 * fake_backend.c - the backend ABI over host memory, without a device: the operator layer's host code runs against it
 * on the CPU, and a test reads what it queued.
 *
 * Writes into a batch take their bytes when the batch ends, as late as a device may; kernels do nothing, so buffers
 * hold what was written, filled or zeroed. Kernel executions and compiled images are logged by name; fake_fail_name
 * makes the allocation of a pooled buffer fail.
 */
#include "cqlcuda.h"

#include <stdio.h>
#include <stdlib.h>
#include <string.h>

struct CqlBuffer
{
  char name[64];
  uint64_t size, capacity;
  unsigned char* data;
};

struct CqlKernel
{
  char name[96];
};

typedef struct
{
  CqlBuffer* buffer;
  uint64_t at, size;
  const void* from;   /* NULL: fill with `value` */
  void* to;           /* a read */
  uint32_t value;
} Op;

struct CqlBatch
{
  Op ops[4096];
  uint32_t count;
};

#define LOG 4096
static CqlBuffer* g_pool[512];
static uint32_t g_pooled;
static CqlKernel g_kernels[512];
static uint32_t g_kernel_count;
static char g_log[LOG][96];
static uint32_t g_logged;
static char g_fail_name[64];
static char g_error[256];

static void note(const char* what, const char* name)
{
  if (g_logged < LOG) snprintf(g_log[g_logged++], sizeof(g_log[0]), "%s %s", what, name);
}

/* ---- what a test uses ---- */
void fake_reset(void)
{
  g_logged = 0;
  g_fail_name[0] = 0;
  for (uint32_t i = 0; i < g_kernel_count; i++)   /* the generated kernels are compiled anew */
    if (!strncmp(g_kernels[i].name, "qk_", 3)) g_kernels[i].name[0] = 0;
}
void fake_clear_log(void) { g_logged = 0; }
void fake_fail_name(const char* name) { snprintf(g_fail_name, sizeof(g_fail_name), "%s", name); }
uint32_t fake_log_count(void) { return g_logged; }
const char* fake_log(uint32_t i) { return i < g_logged ? g_log[i] : ""; }
const void* fake_pooled_data(const char* name)
{
  for (uint32_t i = 0; i < g_pooled; i++)
    if (!strcmp(g_pool[i]->name, name)) return g_pool[i]->data;
  return NULL;
}

/* ---- the ABI ---- */
int cqlcuda_init(void) { return 1; }
uint32_t cqlcuda_sm_count(void) { return 152; }
uint64_t cqlcuda_device_total_memory(void) { return 1ull << 38; }
uint64_t cqlcuda_device_free_memory(void) { return 1ull << 38; }
uint32_t cqlcuda_kernel_launch_count(void) { return 0; }
const char* cqlcuda_last_error(void) { return g_error; }
void cqlcuda_clear_error(void) { g_error[0] = 0; }
int cqlcuda_thread_lane_begin(const char* tag)
{
  (void)tag;
  return 1;
}
void cqlcuda_thread_lane_end(void) {}
void cqlcuda_set_evict_hook(CqlEvictHook hook) { (void)hook; }

CqlBuffer* cqlcuda_buffer_alloc(uint64_t size, uint32_t flags, const void* data)
{
  (void)flags;
  CqlBuffer* b = (CqlBuffer*)calloc(1, sizeof(CqlBuffer));
  b->size = b->capacity = size;
  b->data = (unsigned char*)calloc(1, size ? size : 1);
  if (data) memcpy(b->data, data, size);
  return b;
}
void cqlcuda_buffer_release(CqlBuffer* b)
{
  if (!b) return;
  free(b->data);
  free(b);
}
CqlBuffer* cqlcuda_buffer_alloc_pooled(const char* name, uint64_t name_len, uint64_t size, uint32_t flags, const void* data)
{
  char key[64];
  (void)flags;
  (void)data;
  snprintf(key, sizeof(key), "%.*s", (int)name_len, name);
  if (!strcmp(key, g_fail_name))
  {
    note("refused", key);
    snprintf(g_error, sizeof(g_error), "fake: no room for %s", key);
    return NULL;
  }
  CqlBuffer* b = NULL;
  for (uint32_t i = 0; i < g_pooled && !b; i++)
    if (!strcmp(g_pool[i]->name, key)) b = g_pool[i];
  if (!b)
  {
    if (g_pooled == 512) return NULL;
    b = g_pool[g_pooled++] = (CqlBuffer*)calloc(1, sizeof(CqlBuffer));
    memcpy(b->name, key, sizeof(key));
  }
  if (size > b->capacity || !b->data)
  {
    free(b->data);
    b->data = (unsigned char*)calloc(1, size ? size : 1);
    b->capacity = size;
  }
  b->size = size;
  return b;
}
void cqlcuda_pool_idle(const char* name, uint64_t name_len)
{
  char key[64];
  snprintf(key, sizeof(key), "%.*s", (int)name_len, name);
  note("idle", key);
}
CqlBuffer* cqlcuda_buffer_alloc_host_mapped(uint64_t size, void** out_host)
{
  CqlBuffer* b = cqlcuda_buffer_alloc(size, 0, NULL);
  *out_host = b->data;
  return b;
}
uint64_t cqlcuda_buffer_size(const CqlBuffer* b) { return b ? b->size : 0; }
void* cqlcuda_buffer_device_pointer(const CqlBuffer* b) { return b ? b->data : NULL; }
void cqlcuda_buffer_write(CqlBuffer* b, const void* data, uint64_t size) { memcpy(b->data, data, size); }
void cqlcuda_buffer_read(CqlBuffer* b, void* data, uint64_t size) { memcpy(data, b->data, size); }
int cqlcuda_fill_sequence_u32(CqlBuffer* b, uint64_t rows, uint32_t first)
{
  for (uint64_t r = 0; r < rows; r++) ((uint32_t*)b->data)[r] = first + (uint32_t)r;
  return 1;
}

static CqlKernel* kernel_named(const char* name, uint64_t n)
{
  for (uint32_t i = 0; i < g_kernel_count; i++)
    if (strlen(g_kernels[i].name) == n && !strncmp(g_kernels[i].name, name, n)) return &g_kernels[i];
  return NULL;
}
static CqlKernel* kernel_new(const char* name, uint64_t n)
{
  if (g_kernel_count == 512) return NULL;
  snprintf(g_kernels[g_kernel_count].name, sizeof(g_kernels[0].name), "%.*s", (int)n, name);
  return &g_kernels[g_kernel_count++];
}
/* generated kernels (qk_*) are there once their image was given; every other name is built in */
CqlKernel* cqlcuda_kernel_alloc(const char* name, uint64_t n)
{
  CqlKernel* k = kernel_named(name, n);
  return k || !strncmp(name, "qk_", 3) ? k : kernel_new(name, n);
}
CqlKernel* cqlcuda_kernel_alloc_from_image(const char* name, uint64_t n, const void* image, uint64_t image_len)
{
  (void)image;
  CqlKernel* k = kernel_named(name, n);
  if (k || image_len == 0) return k;
  k = kernel_new(name, n);
  if (k) note("compile", k->name);
  return k;
}
void cqlcuda_kernel_release(CqlKernel* k) { (void)k; }
void cqlcuda_kernel_set_arg_buffer(CqlKernel* k, uint32_t i, CqlBuffer* b) { (void)k, (void)i, (void)b; }
void cqlcuda_kernel_set_arg_buffer_range(CqlKernel* k, uint32_t i, CqlBuffer* b, uint64_t at, uint64_t n) { (void)k, (void)i, (void)b, (void)at, (void)n; }
void cqlcuda_kernel_set_arg_u64(CqlKernel* k, uint32_t i, uint64_t v) { (void)k, (void)i, (void)v; }

CqlBatch* cqlcuda_batch_begin(uint64_t up, uint64_t down)
{
  (void)up;
  (void)down;
  return (CqlBatch*)calloc(1, sizeof(CqlBatch));
}
CqlBatch* cqlcuda_batch_begin_graph(uint64_t up, uint64_t down, uint64_t key)
{
  (void)key;
  return cqlcuda_batch_begin(up, down);
}
static void put(CqlBatch* b, CqlBuffer* buffer, uint64_t at, uint64_t size, const void* from, void* to, uint32_t value)
{
  if (!buffer || at > buffer->size || b->count == 4096) return;
  if (size > buffer->size - at) size = buffer->size - at;
  Op o = { buffer, at, size, from, to, value };
  b->ops[b->count++] = o;
}
void cqlcuda_batch_buffer_write(CqlBatch* b, CqlBuffer* buffer, const void* data, uint64_t size) { put(b, buffer, 0, size, data, NULL, 0); }
void cqlcuda_batch_buffer_zero(CqlBatch* b, CqlBuffer* buffer, uint64_t size) { put(b, buffer, 0, size, NULL, NULL, 0); }
void cqlcuda_batch_buffer_fill(CqlBatch* b, CqlBuffer* buffer, uint64_t size, uint32_t v) { put(b, buffer, 0, size, NULL, NULL, v); }
void cqlcuda_batch_fill_range(CqlBatch* b, CqlBuffer* buffer, uint64_t at, uint64_t size, uint32_t v) { put(b, buffer, at, size, NULL, NULL, v); }
void cqlcuda_batch_buffer_read(CqlBatch* b, CqlBuffer* buffer, void* out, uint64_t size) { put(b, buffer, 0, size, NULL, out, 0); }
void cqlcuda_batch_buffer_read_at(CqlBatch* b, CqlBuffer* buffer, uint64_t at, void* out, uint64_t size) { put(b, buffer, at, size, NULL, out, 0); }
void cqlcuda_batch_kernel_execute(CqlBatch* b, CqlKernel* k, uint32_t global, uint32_t local)
{
  (void)b;
  (void)global;
  (void)local;
  note("run", k->name);
}
/* what calls before this one left below the caller's frame is gone by the time a device copies it */
static void __attribute__((noinline)) scribble(void)
{
  volatile unsigned char below[192 * 1024];
  for (uint32_t i = 0; i < sizeof(below); i++) below[i] = 0xa5;
}
int cqlcuda_batch_end(CqlBatch* b)
{
  scribble();
  for (uint32_t i = 0; i < b->count; i++)
  {
    Op* o = &b->ops[i];
    unsigned char* at = o->buffer->data + o->at;
    if (o->to) memcpy(o->to, at, o->size);
    else if (o->from) memcpy(at, o->from, o->size);
    else
      for (uint64_t j = 0; j + 4 <= o->size; j += 4) memcpy(at + j, &o->value, 4);
  }
  free(b);
  return 1;
}

int cqlcuda_persistent_launch(CqlPersistent* p, uint32_t ctas, CqlBuffer* zero, uint64_t zero_bytes)
{
  (void)p, (void)ctas, (void)zero, (void)zero_bytes;
  return 0;
}
CqlPersistent* cqlcuda_persistent_create(CqlKernel* k, const char* entry)
{
  (void)k, (void)entry;
  return NULL;
}
uint32_t cqlcuda_persistent_ctas(CqlPersistent* p)
{
  (void)p;
  return 0;
}
int cqlcuda_persistent_running(CqlPersistent* p)
{
  (void)p;
  return 0;
}
int cqlcuda_persistent_copy(CqlPersistent* p, CqlBuffer* b, uint64_t at, const void* data, uint64_t size)
{
  (void)p, (void)b, (void)at, (void)data, (void)size;
  return 0;
}
int cqlcuda_persistent_destroy(CqlPersistent* p, uint32_t ms)
{
  (void)p, (void)ms;
  return 1;
}
