/* A CUDA runtime without a GPU for tests of the library's launch code on the
 * CPU: two devices, memory that is only addresses, copies that give zeros,
 * and a record of every launch (cudaLaunchKernelExC) and of the shared memory
 * that each kernel has been granted on each device. */
#include <cuda_runtime_api.h>
#include <string.h>

enum { MAX_LAUNCH = 65536, MAX_GRANT = 4096 };
static int device, sms = 152;
static struct { unsigned grid[3], block[3]; size_t smem; int device, granted, programmatic; const void *func; } launch[MAX_LAUNCH];
static int launches;
static struct { const void *func; int device, bytes; } grant[MAX_GRANT];
static int grants;
static char *next_address = (char *) 0x100000000;

void fake_reset(void) { launches = 0; }
void fake_set_device(int d) { device = d; }
int fake_launches(void) { return launches; }
/* out: grid x, y, z, block x, y, z, dynamic shared memory, device, whether the kernel may have that much there,
 * whether the launch is programmatic, a number of the kernel */
void fake_launch(int i, long *out) {
  for (int k = 0; k < 3; k++) { out[k] = launch[i].grid[k]; out[3 + k] = launch[i].block[k]; }
  out[6] = (long) launch[i].smem; out[7] = launch[i].device; out[8] = launch[i].granted; out[9] = launch[i].programmatic;
  out[10] = (long) launch[i].func;
}

cudaError_t cudaGetDevice(int *d) { *d = device; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { device = d; return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n) { *n = 2; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(struct cudaDeviceProp *p, int d) {
  (void) d;
  memset(p, 0, sizeof(*p));
  p->multiProcessorCount = sms;
  p->sharedMemPerBlockOptin = 232448;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, enum cudaDeviceAttr a, int d) {
  (void) d;
  *v = a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 232448 : a == cudaDevAttrMultiProcessorCount ? sms : 0;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *f, enum cudaFuncAttribute a, int v) {
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize && grants < MAX_GRANT) {
    grant[grants].func = f; grant[grants].device = device; grant[grants++].bytes = v;
  }
  return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(struct cudaFuncAttributes *a, const void *f) { (void) f; memset(a, 0, sizeof(*a)); return cudaSuccess; }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **args) {
  (void) args;
  if (launches == MAX_LAUNCH) return cudaErrorUnknown;
  const dim3 g = c->gridDim, b = c->blockDim;
  launch[launches].grid[0] = g.x; launch[launches].grid[1] = g.y; launch[launches].grid[2] = g.z;
  launch[launches].block[0] = b.x; launch[launches].block[1] = b.y; launch[launches].block[2] = b.z;
  launch[launches].smem = c->dynamicSmemBytes;
  launch[launches].device = device;
  launch[launches].func = f;
  launch[launches].granted = c->dynamicSmemBytes <= 48 * 1024;
  for (int i = 0; i < grants; i++)
    if (grant[i].func == f && grant[i].device == device && grant[i].bytes >= (int) c->dynamicSmemBytes) launch[launches].granted = 1;
  launch[launches].programmatic = 0;
  for (unsigned i = 0; i < c->numAttrs; i++)
    if (c->attrs[i].id == cudaLaunchAttributeProgrammaticStreamSerialization)
      launch[launches].programmatic = c->attrs[i].val.programmaticStreamSerializationAllowed;
  launches++;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *f, int t, size_t s, unsigned fl) {
  (void) f; (void) t; (void) s; (void) fl;
  *n = 2;
  return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t n) { *p = next_address; next_address += (n + 255) / 256 * 256; return cudaSuccess; }
cudaError_t cudaFree(void *p) { (void) p; return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void **p, const void *s) { (void) s; return cudaMalloc(p, 64 << 20); }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, enum cudaMemcpyKind k) {
  (void) s;
  if (k == cudaMemcpyDeviceToHost) memset(d, 0, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, enum cudaMemcpyKind k, cudaStream_t t) { (void) t; return cudaMemcpy(d, s, n, k); }
cudaError_t cudaMemset(void *d, int v, size_t n) { (void) d; (void) v; (void) n; return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t t) { (void) d; (void) v; (void) n; (void) t; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize(void) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { (void) s; return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned f) { (void) f; return cudaMalloc((void **) s, 1); }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned f) { (void) s; (void) e; (void) f; return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t s, enum cudaStreamCaptureStatus *c) { (void) s; *c = cudaStreamCaptureStatusNone; return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return cudaMalloc((void **) e, 1); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned f) { (void) f; return cudaMalloc((void **) e, 1); }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { (void) e; (void) s; return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaPeekAtLastError(void) { return cudaSuccess; }
cudaError_t cudaGetDriverEntryPointByVersion(const char *n, void **p, unsigned v, unsigned long long f, enum cudaDriverEntryPointQueryResult *q) {
  (void) n; (void) v; (void) f; (void) q;
  *p = 0;
  return cudaErrorUnknown;
}
