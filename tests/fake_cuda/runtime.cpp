// A CUDA runtime without a GPU, to be linked with the objects of the kernel library in place of the real one: it keeps the rules
// that launchers depend on (a stream belongs to a device, more than 48 KB of dynamic shared memory are allowed per kernel and
// device, what a tensor map may look like) and records every launch.  Devices, streams and events are numbers; nothing runs.
#include <cuda.h>
#include <cuda_runtime.h>
#include <string.h>
#include <map>
#include <set>
#include <string>
#include <vector>

namespace {

struct Launch {
  std::string kernel;
  int device, threads, smem, cluster;
  long long grid;
};
struct Call {
  dim3 grid, block;
  size_t smem;
  cudaStream_t stream;
};

thread_local int g_device = 0;
thread_local std::vector<Call> g_calls;
std::map<const void*, std::string> g_names;
std::map<std::pair<int, const void*>, int> g_smem;     // dynamic shared memory that a kernel may have on a device
std::vector<Launch> g_log;
long long g_attributes = 0;

// Streams and events of device d: (d + 1) << 32 and above.  The null stream is the current device's.
int device_of(const void* handle) { return handle == nullptr ? g_device : (int)(((uintptr_t)handle >> 32) - 1); }

cudaError_t launch(const void* f, dim3 grid, dim3 block, size_t smem, cudaStream_t stream, int cluster) {
  if (device_of(stream) != g_device) return cudaErrorInvalidResourceHandle;
  const auto it = g_smem.find({g_device, f});
  if ((long long)smem > (it == g_smem.end() ? 48 * 1024 : it->second)) return cudaErrorInvalidValue;
  if (grid.x == 0 || grid.y == 0 || grid.z == 0 || grid.y > 65535 || grid.z > 65535 || block.x * block.y * block.z > 1024 || block.x == 0) return cudaErrorInvalidConfiguration;
  if (cluster < 1 || cluster > 8 || grid.x % cluster) return cudaErrorInvalidClusterSize;
  g_log.push_back({g_names.count(f) ? g_names[f] : "?", g_device, (int)(block.x * block.y * block.z), (int)smem, cluster, (long long)grid.x * grid.y * grid.z});
  return cudaSuccess;
}

int element_bytes(CUtensorMapDataType t) { return t == CU_TENSOR_MAP_DATA_TYPE_FLOAT32 ? 4 : t == CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 ? 2 : 0; }

// The rules for a tiled map with a 128-byte swizzle.
CUresult encode(CUtensorMap*, CUtensorMapDataType type, cuuint32_t rank, void* base, const cuuint64_t* dims, const cuuint64_t* strides,
                const cuuint32_t* box, const cuuint32_t* element_strides, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                CUtensorMapFloatOOBfill) {
  const int es = element_bytes(type);
  if (es == 0 || rank < 1 || rank > 5 || ((uintptr_t)base & 15)) return CUDA_ERROR_INVALID_VALUE;
  for (cuuint32_t i = 0; i < rank; ++i) {
    if (dims[i] < 1 || dims[i] > (1ull << 32) || box[i] < 1 || box[i] > 256 || element_strides[i] < 1 || element_strides[i] > 8) return CUDA_ERROR_INVALID_VALUE;
    if (i + 1 < rank && (strides[i] % 16 || strides[i] >= (1ull << 40))) return CUDA_ERROR_INVALID_VALUE;
  }
  if (box[0] * es % 16 || box[0] * es > 128) return CUDA_ERROR_INVALID_VALUE;
  return CUDA_SUCCESS;
}

}  // namespace

extern "C" {

// ---- what the tests ask for
void fake_device(int device) { g_device = device; }
int fake_current_device() { return g_device; }
void* fake_stream(int device) { return (void*)((uintptr_t)(device + 1) << 32 | 64); }
int fake_launches() { return (int)g_log.size(); }
long long fake_attributes() { return g_attributes; }
const char* fake_launch(int i, int* out) {     // device, threads, dynamic shared memory, cluster, blocks
  const Launch& l = g_log[i];
  out[0] = l.device; out[1] = l.threads; out[2] = l.smem; out[3] = l.cluster; out[4] = (int)l.grid;
  return l.kernel.c_str();
}
void fake_clear() { g_log.clear(); }

// ---- registration and launches
void** __cudaRegisterFatBinary(void*) { static void* handle; return &handle; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) { g_names[host] = name; }
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, struct CUstream_st* stream) {
  g_calls.push_back({grid, block, smem, stream});
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
  const Call c = g_calls.back();
  g_calls.pop_back();
  *grid = c.grid; *block = c.block; *smem = c.smem; *(cudaStream_t*)stream = c.stream;
  return cudaSuccess;
}

thread_local cudaError_t g_last = cudaSuccess;
static cudaError_t said(cudaError_t e) {
  if (e != cudaSuccess) g_last = e;
  return e;
}
cudaError_t cudaLaunchKernel(const void* f, dim3 grid, dim3 block, void**, size_t smem, cudaStream_t s) { return said(launch(f, grid, block, smem, s, 1)); }
cudaError_t cudaLaunchCooperativeKernel(const void* f, dim3 grid, dim3 block, void**, size_t smem, cudaStream_t s) { return said(launch(f, grid, block, smem, s, 1)); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
  int cluster = 1;
  for (unsigned i = 0; i < c->numAttrs; ++i)
    if (c->attrs[i].id == cudaLaunchAttributeClusterDimension) cluster = (int)c->attrs[i].val.clusterDim.x;
  return said(launch(f, c->gridDim, c->blockDim, c->dynamicSmemBytes, c->stream, cluster));
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int value) {
  ++g_attributes;
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) {
    if (value > 227 * 1024) return said(cudaErrorInvalidValue);
    g_smem[{g_device, f}] = value;
  }
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) { *n = 2; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t* c) {
  const int size = (int)c->attrs[0].val.clusterDim.x;
  *n = size >= 7 ? 15 : 148 / size;                   // a B200's
  return cudaSuccess;
}

// ---- devices
cudaError_t cudaGetDevice(int* d) { *d = g_device; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { g_device = d; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) { *v = a == cudaDevAttrMultiProcessorCount ? 148 : 0; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaDeviceCanAccessPeer(int* can, int, int) { *can = 1; return cudaSuccess; }
cudaError_t cudaDeviceEnablePeerAccess(int, unsigned) { return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = g_last; g_last = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaGetDriverEntryPoint(const char*, void** f, unsigned long long, cudaDriverEntryPointQueryResult* q) {
  *f = (void*)&encode;
  *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void* symbol) { *p = const_cast<void*>(symbol); return cudaSuccess; }

// ---- streams and events: copies and waits may come from any device, an event is recorded on a stream of its own
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)((uintptr_t)(g_device + 1) << 32 | 128); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { return said(device_of(e) == device_of(s) ? cudaSuccess : cudaErrorInvalidResourceHandle); }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }

// ---- memory: addresses that nobody follows
static uintptr_t g_next = (uintptr_t)1 << 44;
cudaError_t cudaMalloc(void** p, size_t n) { *p = (void*)g_next; g_next += (n + 511) / 512 * 512; return cudaSuccess; }
cudaError_t cudaFree(void*) { return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { *p = new char[n](); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { delete[] (char*)p; return cudaSuccess; }
cudaError_t cudaMemset(void*, int, size_t) { return cudaSuccess; }
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void*, const void*, size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaIpcGetMemHandle(cudaIpcMemHandle_t*, void*) { return cudaSuccess; }
cudaError_t cudaIpcOpenMemHandle(void**, cudaIpcMemHandle_t, unsigned) { return cudaErrorNotSupported; }
cudaError_t cudaIpcCloseMemHandle(void*) { return cudaSuccess; }

}  // extern "C"
