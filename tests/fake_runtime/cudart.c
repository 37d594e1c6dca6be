/* A stand-in for the CUDA runtime with which the engine's host side runs without a GPU: nothing is
 * computed, every call is written down, and a call can be made to fail. Built with the runtime's own
 * library name and symbol version, so the engine library binds to it in a process that loads it first. */
#include <cuda.h>
#include <cuda_runtime_api.h>
#include <stdarg.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#define API __attribute__((visibility("default")))

static char *log_text;
static size_t log_len, log_cap;
static uintptr_t next_handle = 0x1000;
static uint64_t next_address = 0x7f0000000000ull;
static cudaError_t last_error;
static char fail_name[64];
static int fail_after = -1;

static void note(const char* fmt, ...) {
  va_list ap;
  if (log_cap - log_len < 4096) log_text = realloc(log_text, log_cap += 1 << 16);
  va_start(ap, fmt);
  log_len += (size_t)vsnprintf(log_text + log_len, 4000, fmt, ap);
  va_end(ap);
  log_text[log_len++] = '\n';
  log_text[log_len] = 0;
}
/* The calls so far, one a line; forgets them. */
API const char* fake_take(void) {
  static char* out;
  free(out);
  out = log_text ? log_text : strdup("");
  log_text = NULL;
  log_len = log_cap = 0;
  return out;
}
/* The (after + 1)-th call of `name` from now on returns an error, once. */
API void fake_fail(const char* name, int after) {
  snprintf(fail_name, sizeof fail_name, "%s", name);
  fail_after = after;
}
static cudaError_t done(const char* name) {
  if (fail_after >= 0 && !strcmp(name, fail_name) && fail_after-- == 0) {
    note("FAILED %s", name);
    return cudaErrorInvalidResourceHandle;
  }
  return cudaSuccess;
}

/* kernels: the host stub's address and its (mangled) name */
struct fun { const void* host; const char* name; };
static struct fun* funs;
static int nfuns;
API void** __cudaRegisterFatBinary(void* bin) { static void* h; (void)bin; return &h; }
API void __cudaRegisterFatBinaryEnd(void** h) { (void)h; }
API void __cudaUnregisterFatBinary(void** h) { (void)h; }
API void __cudaRegisterVar(void** h, char* var, char* dev, const char* name, int ext, size_t n, int c, int g) {
  (void)h; (void)var; (void)dev; (void)name; (void)ext; (void)n; (void)c; (void)g;
}
API void __cudaRegisterFunction(void** h, const char* host, char* dev, const char* name, int limit, uint3* tid,
                                uint3* bid, dim3* bdim, dim3* gdim, int* wsize) {
  (void)h; (void)dev; (void)limit; (void)tid; (void)bid; (void)bdim; (void)gdim; (void)wsize;
  funs = realloc(funs, sizeof *funs * (size_t)(nfuns + 1));
  funs[nfuns].host = host;
  funs[nfuns++].name = strdup(name);
}
static const char* name_of(const void* host) {
  for (int i = 0; i < nfuns; ++i)
    if (funs[i].host == host) return funs[i].name;
  return "?";
}

static __thread struct { dim3 grid, block; size_t smem; void* stream; } call;
API unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, void* stream) {
  call.grid = grid; call.block = block; call.smem = smem; call.stream = stream;
  return 0;
}
API cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
  *grid = call.grid; *block = call.block; *smem = call.smem; *(void**)stream = call.stream;
  return cudaSuccess;
}
static cudaError_t launch(const void* f, dim3 g, dim3 b, size_t smem, cudaStream_t s, const char* more) {
  const uint64_t threads = (uint64_t)b.x * b.y * b.z;
  if (!g.x || !g.y || !g.z || !threads || g.x > 0x7fffffffu || g.y > 65535 || g.z > 65535 || threads > 1024 ||
      smem > 232448) {
    note("REFUSED %s grid %u %u %u", name_of(f), g.x, g.y, g.z);
    return last_error = cudaErrorInvalidConfiguration;
  }
  note("launch %s grid %u %u %u stream %p%s", name_of(f), g.x, g.y, g.z, (void*)s, more);
  const cudaError_t e = done("cudaLaunchKernel");
  if (e) last_error = e;  /* the one a launch is checked by; other calls' errors are their results */
  return e;
}
API cudaError_t cudaLaunchKernel(const void* f, dim3 g, dim3 b, void** args, size_t smem, cudaStream_t s) {
  (void)args;
  return launch(f, g, b, smem, s, "");
}
API cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args) {
  char more[64] = "";
  (void)args;
  for (unsigned i = 0; i < c->numAttrs; ++i)
    if (c->attrs[i].id == cudaLaunchAttributePreferredSharedMemoryCarveout)
      snprintf(more, sizeof more, " carveout %u", c->attrs[i].val.sharedMemCarveout);
  return launch(f, c->gridDim, c->blockDim, c->dynamicSmemBytes, c->stream, more);
}
API cudaError_t cudaFuncSetAttribute(const void* f, enum cudaFuncAttribute a, int v) {
  note("attribute %s %d = %d", name_of(f), (int)a, v);
  return done("cudaFuncSetAttribute");
}
API cudaError_t cudaFuncGetAttributes(struct cudaFuncAttributes* a, const void* f) {
  (void)f;
  memset(a, 0, sizeof *a);
  return cudaSuccess;
}
API cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* f, int t, size_t s,
                                                                       unsigned fl) {
  (void)f; (void)t; (void)s; (void)fl;
  *n = 4;
  return cudaSuccess;
}

/* streams and events */
API cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned fl) {
  (void)fl;
  *s = (cudaStream_t)(next_handle += 16);
  note("stream %p", (void*)*s);
  return done("cudaStreamCreateWithFlags");
}
API cudaError_t cudaStreamDestroy(cudaStream_t s) { note("destroy stream %p", (void*)s); return cudaSuccess; }
API cudaError_t cudaStreamSynchronize(cudaStream_t s) { (void)s; return done("cudaStreamSynchronize"); }
API cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned fl) {
  (void)fl;
  note("wait %p on %p", (void*)e, (void*)s);
  return done("cudaStreamWaitEvent");
}
API cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned fl) {
  (void)fl;
  *e = (cudaEvent_t)(next_handle += 16);
  return done("cudaEventCreateWithFlags");
}
API cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
API cudaError_t cudaEventDestroy(cudaEvent_t e) { (void)e; return cudaSuccess; }
API cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  note("record %p on %p", (void*)e, (void*)s);
  return done("cudaEventRecord");
}
API cudaError_t cudaEventQuery(cudaEvent_t e) { (void)e; return cudaSuccess; }
API cudaError_t cudaEventSynchronize(cudaEvent_t e) { (void)e; return cudaSuccess; }
API cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t a, cudaEvent_t b) { (void)a; (void)b; *ms = 0; return cudaSuccess; }

/* graphs */
API cudaError_t cudaStreamBeginCapture(cudaStream_t s, enum cudaStreamCaptureMode m) {
  (void)m;
  note("capture %p", (void*)s);
  return done("cudaStreamBeginCapture");
}
API cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g) {
  *g = (cudaGraph_t)(next_handle += 16);
  note("end capture %p", (void*)s);
  return done("cudaStreamEndCapture");
}
API cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t g, unsigned long long fl) {
  (void)g; (void)fl;
  *x = (cudaGraphExec_t)(next_handle += 16);
  return done("cudaGraphInstantiate");
}
API cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t s) {
  note("graph %p on %p", (void*)x, (void*)s);
  return done("cudaGraphLaunch");
}
API cudaError_t cudaGraphDestroy(cudaGraph_t g) { (void)g; return cudaSuccess; }
API cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { (void)x; return cudaSuccess; }

/* memory: addresses that nothing reads */
API cudaError_t cudaMalloc(void** p, size_t n) {
  *p = (void*)next_address;
  next_address += (n + 0xffff) & ~0xffffull;
  return done("cudaMalloc");
}
API cudaError_t cudaFree(void* p) { (void)p; return cudaSuccess; }
API cudaError_t cudaHostAlloc(void** p, size_t n, unsigned fl) { (void)fl; *p = calloc(n, 1); return cudaSuccess; }
API cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
API cudaError_t cudaMemcpy(void* d, const void* s, size_t n, enum cudaMemcpyKind k) {
  (void)d; (void)s; (void)n; (void)k;
  return done("cudaMemcpy");
}
API cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, enum cudaMemcpyKind k, cudaStream_t st) {
  (void)d; (void)s; (void)n; (void)k; (void)st;
  return done("cudaMemcpyAsync");
}
API cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t s) {
  (void)d; (void)v; (void)n; (void)s;
  return done("cudaMemsetAsync");
}
API cudaError_t cudaMemcpyFromSymbol(void* d, const void* s, size_t n, size_t o, enum cudaMemcpyKind k) {
  (void)s; (void)o; (void)k;
  memset(d, 0, n);
  return cudaSuccess;
}
API cudaError_t cudaMemcpyToSymbol(const void* d, const void* s, size_t n, size_t o, enum cudaMemcpyKind k) {
  (void)d; (void)s; (void)n; (void)o; (void)k;
  return cudaSuccess;
}
API cudaError_t cudaGetSymbolAddress(void** p, const void* s) { (void)s; return cudaMalloc(p, 64); }

/* device, errors, driver */
API cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
API cudaError_t cudaDeviceSynchronize(void) { return cudaSuccess; }
API cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr a, int d) {
  (void)d;
  *v = a == cudaDevAttrMultiProcessorCount ? 148 : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 232448 : 0;
  return cudaSuccess;
}
API cudaError_t cudaGetLastError(void) { const cudaError_t e = last_error; last_error = cudaSuccess; return e; }
API cudaError_t cudaPeekAtLastError(void) { return last_error; }
API const char* cudaGetErrorString(cudaError_t e) { return e ? "error of the fake runtime" : "no error"; }
static CUresult encode(CUtensorMap* m, CUtensorMapDataType t, cuuint32_t rank, void* base, const cuuint64_t* dims,
                       const cuuint64_t* strides, const cuuint32_t* box, const cuuint32_t* es, CUtensorMapInterleave i,
                       CUtensorMapSwizzle s, CUtensorMapL2promotion l, CUtensorMapFloatOOBfill f) {
  (void)m; (void)t; (void)base; (void)es; (void)i; (void)s; (void)l; (void)f;
  note("map box %u %u of %llu %llu", box[0], box[1], (unsigned long long)dims[0], (unsigned long long)dims[1]);
  for (cuuint32_t k = 0; k < rank; ++k)
    if (!dims[k] || dims[k] > (1ull << 32) || !box[k] || box[k] > 256) return CUDA_ERROR_INVALID_VALUE;
  for (cuuint32_t k = 0; k + 1 < rank; ++k)
    if (strides[k] % 16 || strides[k] >= (1ull << 40)) return CUDA_ERROR_INVALID_VALUE;
  return CUDA_SUCCESS;
}
API cudaError_t cudaGetDriverEntryPointByVersion(const char* name, void** p, unsigned v, unsigned long long fl,
                                                 enum cudaDriverEntryPointQueryResult* q) {
  (void)name; (void)v; (void)fl;
  *p = (void*)encode;
  *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
