// A CUDA runtime without a GPU, for tests of the engine's host code: device memory is host memory,
// kernels do nothing, and two devices exist.  Loaded with RTLD_GLOBAL before libscopi_gpu.so, whose
// undefined runtime symbols then bind to it.  It keeps the runtime's rules that the engine's launches
// depend on: the attributes of a kernel are those of the device they were set on, a cluster of more
// than 8 CTAs and more than 48 KB of dynamic shared memory need them.
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <string>
#include <utility>

#include <cuda_runtime_api.h>

namespace {
int g_dev = 0, g_error = 0;
long long g_mallocs = 0, g_fail_malloc = -1;  // allocations so far; number of good ones until one fails
int g_contacts = 0;                           // what detection "finds"
int g_superellipsoids = 0;                    // what an upload's census counts
int g_refuse_clusters = 0;
std::map<std::string, long long> g_by_name;
std::set<std::string> g_loaded;               // kernels launched or asked about so far
long long g_late = 0;                         // first launches since the "late_loads" count was reset
long long g_refused = 0;                      // launches that broke a rule
long long g_cluster_launches = 0, g_launches = 0;
std::map<void*, size_t> g_blocks;
size_t g_bytes = 0;
std::map<const void*, std::string> g_names;
std::set<std::pair<int, const void*>> g_nonportable;
std::map<std::pair<int, const void*>, int> g_smem;
cudaError_t fail(cudaError_t e) {
    if (e != cudaSuccess) g_error = e;
    return e;
}
cudaError_t launch(const void* f, void** args, size_t smem) {
    if (smem > 48 * 1024 && g_smem[{g_dev, f}] < (int)smem) {
        ++g_refused;
        return fail(cudaErrorInvalidValue);
    }
    ++g_launches;
    ++g_by_name[g_names[f]];
    if (g_loaded.insert(g_names[f]).second) ++g_late;
    // k_sizes(totals, sizes, cap): the number of contacts is the struct's first field
    if (g_names[f].find("k_sizes") != std::string::npos) **(int**)args[1] = g_contacts;
    // k_shape_census(shape, worm, n, nin, dim, out)
    if (g_names[f].find("k_shape_census") != std::string::npos) **(int**)args[5] = g_superellipsoids;
    return cudaSuccess;
}
}  // namespace

extern "C" {
void fake_set(const char* what, long long v) {
    const std::string w = what;
    if (w == "device") g_dev = (int)v;
    if (w == "fail_malloc") g_fail_malloc = v;
    if (w == "contacts") g_contacts = (int)v;
    if (w == "superellipsoids") g_superellipsoids = (int)v;
    if (w == "late_loads") g_late = v;
    if (w == "refuse_clusters") g_refuse_clusters = (int)v;
}
long long fake_get(const char* what) {
    const std::string w = what;
    if (w == "mallocs") return g_mallocs;
    if (w == "bytes") return (long long)g_bytes;
    if (w == "late_loads") return g_late;
    if (w == "refused") return g_refused;
    if (w == "launches") return g_launches;
    if (w == "cluster_launches") return g_cluster_launches;
    return -1;
}

// launches of the kernels whose (mangled) name contains `part`
long long fake_launches_of(const char* part) {
    long long n = 0;
    for (const auto& k : g_by_name)
        if (k.first.find(part) != std::string::npos) n += k.second;
    return n;
}

void** __cudaRegisterFatBinary(void*) {
    static void* h;
    return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
    g_names[host] = name;
}
static dim3 g_grid, g_block;
static size_t g_shared;
static void* g_stream;
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, void* s) {
    g_grid = grid;
    g_block = block;
    g_shared = smem;
    g_stream = s;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void** s) {
    *grid = g_grid;
    *block = g_block;
    *smem = g_shared;
    *s = g_stream;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void** args, size_t smem, cudaStream_t) {
    return launch(f, args, smem);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* cfg, const void* f, void** args) {
    for (unsigned i = 0; i < cfg->numAttrs; ++i) {
        const cudaLaunchAttribute& a = cfg->attrs[i];
        if (a.id != cudaLaunchAttributeClusterDimension) continue;
        if (g_refuse_clusters) return fail(cudaErrorLaunchOutOfResources);
        if (a.val.clusterDim.x > 8 && !g_nonportable.count({g_dev, f})) return fail(cudaErrorInvalidValue);
        ++g_cluster_launches;
    }
    return launch(f, args, cfg->dynamicSmemBytes);
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute attr, int v) {
    if (attr == cudaFuncAttributeNonPortableClusterSizeAllowed && v) g_nonportable.insert({g_dev, f});
    if (attr == cudaFuncAttributeMaxDynamicSharedMemorySize) g_smem[{g_dev, f}] = v;
    return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void* f) {
    memset(a, 0, sizeof(*a));
    g_loaded.insert(g_names[f]);
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t* cfg) {
    *n = 148 / (int)cfg->attrs[0].val.clusterDim.x;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceCount(int* n) {
    *n = 2;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
    *d = g_dev;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int d) {
    g_dev = d;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? 148 : 0;
    return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t n) {
    if (g_fail_malloc == 0) {
        g_fail_malloc = -1;
        return fail(cudaErrorMemoryAllocation);
    }
    if (g_fail_malloc > 0) --g_fail_malloc;
    ++g_mallocs;
    *p = calloc(n, 1);
    g_blocks[*p] = n;
    g_bytes += n;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    auto it = g_blocks.find(p);
    if (it != g_blocks.end()) {
        g_bytes -= it->second;
        g_blocks.erase(it);
    }
    free(p);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
    *p = calloc(n, 1);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
    free(p);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) {
    memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
    memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
    static void* m[2];
    if (!m[g_dev]) m[g_dev] = calloc(8 << 20, 1);
    *p = m[g_dev];
    return cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t) { return "from the test's CUDA runtime"; }
cudaError_t cudaGetLastError() {
    const int e = g_error;
    g_error = 0;
    return (cudaError_t)e;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    *s = (cudaStream_t)malloc(1);
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
    free(s);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
    *g = (cudaGraph_t)malloc(1);
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) {
    *x = (cudaGraphExec_t)malloc(1);
    return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) {
    free(g);
    return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) {
    free(x);
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) {
    *e = (cudaEvent_t)malloc(1);
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    free(e);
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
    *ms = 0;
    return cudaSuccess;
}
}
