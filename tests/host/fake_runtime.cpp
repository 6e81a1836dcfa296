// The library's host objects (abi.cu, batch.cu) against a fake CUDA runtime, so
// that what they ask of the runtime can be checked without a GPU.  Work of a
// stream is queued and done when the stream is waited for: a call that returns
// too early, a copy whose source dies with the call, a kernel's store to another
// GPU's memory and work on a stream that nothing orders are then seen as such.
// usage: fake_runtime <scenario>; exit code 0 = as it has to be.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <map>
#include <string>
#include <vector>

#include "rfx_internal.cuh"

namespace {

struct Op {
    std::function<void()> run;
    const void* reads_host;  // pageable source of a queued copy
};
struct Range {
    size_t bytes;
    cudaMemoryType type;
    int device;
};
std::map<void*, std::deque<Op>> g_queue;  // per stream; key nullptr: the legacy default stream
std::map<const char*, Range> g_mem;
std::vector<std::string> g_faults;
int g_copies = 0;
bool g_running = false;  // within main
rfx_status g_route_status = RFX_OK;

Range where(const void* p) {
    auto it = g_mem.upper_bound((const char*)p);
    if (it != g_mem.begin()) {
        --it;
        if ((const char*)p < it->first + it->second.bytes) return it->second;
    }
    return {0, cudaMemoryTypeUnregistered, 0};
}

void* make(size_t bytes, cudaMemoryType type, int device) {
    void* p = std::malloc(bytes ? bytes : 1);
    std::memset(p, 0xCD, bytes);
    g_mem[(const char*)p] = {bytes, type, device};
    return p;
}

void flush(void* s) {
    while (!g_queue[s].empty()) {
        Op op = g_queue[s].front();
        g_queue[s].pop_front();
        op.run();
    }
}

// a kernel of the context's device stores `v`
void kernel_store(rfx::Ctx* c, void* dst, size_t words, int32_t v) {
    const Range r = where(dst);
    const bool ok = r.type == cudaMemoryTypeManaged || (r.type == cudaMemoryTypeDevice && r.device == c->device);
    if (!ok) {
        g_faults.push_back("a kernel stores outside its device");
        return;
    }
    g_queue[c->stream].push_back({[=]() {
                                      for (size_t i = 0; i < words; ++i) ((int32_t*)dst)[i] = v;
                                  },
                                  nullptr});
}

// whether a queued copy still has to read from p
bool source_of_a_copy(const void* p) {
    for (auto& q : g_queue)
        for (auto& op : q.second)
            if (p && op.reads_host == p) return true;
    return false;
}

int fail(const char* what) {
    std::printf("%s\n", what);
    return 1;
}

}  // namespace

// Host memory given back while a queued copy still reads it.
void operator delete(void* p) noexcept {
    if (g_running && source_of_a_copy(p)) {
        std::fprintf(stderr, "host memory freed under a copy\n");
        std::_Exit(1);
    }
    std::free(p);
}
void operator delete(void* p, size_t) noexcept { operator delete(p); }

extern "C" {
void** __cudaRegisterFatBinary(void*) { static void* h = nullptr; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}

cudaError_t cudaGetDeviceCount(int* n) { *n = 2; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaMalloc(void** p, size_t bytes) { *p = make(bytes, cudaMemoryTypeDevice, 0); return cudaSuccess; }
cudaError_t cudaFree(void* p) {
    for (auto& q : g_queue) flush(q.first); g_mem.erase((const char*)p); std::free(p); return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    const Range r = where(p);
    std::memset(a, 0, sizeof(*a));
    a->type = r.type;
    a->device = r.device;
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)std::malloc(1); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { flush(s); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st) {
    ++g_copies;
    g_queue[st].push_back({[=]() { std::memcpy(d, s, n); }, where(s).type == cudaMemoryTypeUnregistered ? s : nullptr});
    return cudaSuccess;
}
// between two device buffers the host does not wait
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind kind) {
    cudaMemcpyAsync(d, s, n, kind, nullptr);
    if (where(d).type != cudaMemoryTypeDevice || where(s).type != cudaMemoryTypeDevice) flush(nullptr);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st) {
    g_queue[st].push_back({[=]() { std::memset(d, v, n); }, nullptr});
    return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) { return cudaMemsetAsync(d, v, n, nullptr); }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)std::malloc(1); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { *g = nullptr; return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaGraphGetNodes(cudaGraph_t, cudaGraphNode_t*, size_t* n) { *n = 0; return cudaSuccess; }
}

namespace rfx {
rfx_status launch_route(Ctx* c, int32_t* votes_out, int32_t* nout_out) {
    if (g_route_status != RFX_OK) return g_route_status;
    kernel_store(c, c->d_votes, (size_t)c->n * c->nclass, 5);
    kernel_store(c, c->d_nout, c->n, 4);
    if (votes_out) kernel_store(c, votes_out, (size_t)c->n * c->nclass, 5);
    if (nout_out) kernel_store(c, nout_out, c->n, 4);
    return RFX_OK;
}
rfx_status launch_route_leaf(Ctx* c, int32_t* leaf, int32_t* votes_out, int32_t* nout_out) {
    kernel_store(c, leaf, (size_t)c->n * c->T, 0);
    return launch_route(c, votes_out, nout_out);
}
rfx_status launch_oob_summary(Ctx* c, float* err, int32_t* pred, float* proba) {
    if (err) kernel_store(c, err, 1, 0);
    if (pred) kernel_store(c, pred, c->n, 3);
    if (proba) kernel_store(c, proba, (size_t)c->n * c->nclass, 0);
    return RFX_OK;
}
rfx_status launch_oob_summary_f32(Ctx* c, const float*, float* err, int32_t* pred, float* proba) {
    return launch_oob_summary(c, err, pred, proba);
}
rfx_status launch_tnodewt(Ctx*) { return RFX_OK; }
rfx_status launch_casewise_votes(Ctx* c, const int32_t*, float* q) {
    kernel_store(c, q, (size_t)c->n * c->nclass, 7);
    return RFX_OK;
}
rfx_status launch_factor_operator(Ctx* c, const float*, int, const double* V, double* W, int) {
    for (int e = 0; e < 16 * c->n; ++e) W[e] = V[e];
    return RFX_OK;
}
rfx_status launch_build_csr(Ctx*) { return RFX_OK; }
rfx_status launch_gap_keys(Ctx*, const int32_t*, int32_t*) { return RFX_OK; }
rfx_status launch_build_csr_raw(cudaStream_t, int, const int32_t*, int, int, const int64_t*, int32_t*, int32_t*, int,
                                uint32_t*) {
    return RFX_OK;
}
rfx_status launch_weighted_rows(Ctx* c, int, const int32_t*, const int64_t*, const int32_t*, const int32_t*, int64_t,
                                double* out) {
    kernel_store(c, out, (size_t)c->n * (c->n + 1), 9);  // (words)
    return RFX_OK;
}
}  // namespace rfx

// A context with a forest of one split-free tree, as far as the host code looks at it.
static rfx::Ctx* context(bool casewise) {
    rfx_config cfg{};
    cfg.use_casewise = casewise;
    rfx_ctx* h = nullptr;
    if (rfx_ctx_create(&cfg, &h) != RFX_OK) std::exit(9);
    auto* c = reinterpret_cast<rfx::Ctx*>(h);
    c->loaded = true;
    c->n = 3;
    c->nclass = 2;
    c->T = 2;
    c->h_nnode = {1, 1};
    c->max_nnode = 1;
    c->h_segbase = {0, 3, 6};
    rfx::dalloc(c, &c->d_votes, 6);
    rfx::dalloc(c, &c->d_nout, 3);
    return c;
}

static rfx_ctx* handle(rfx::Ctx* c) { return reinterpret_cast<rfx_ctx*>(c); }
static int32_t* dev_int(size_t n, int device) { return (int32_t*)make(4 * n, cudaMemoryTypeDevice, device); }

// Votes and counts for another GPU's memory arrive by copies; the device's own
// memory (and managed memory) is written without one.
static int other_gpu() {
    for (int device = 0; device < 2; ++device) {
        rfx::Ctx* c = context(false);
        int32_t *q = dev_int(6, device), *nout = dev_int(3, device);
        g_copies = 0;
        if (rfx_route_oob(handle(c), q, nout, nullptr) != RFX_OK) return fail("rfx_route_oob");
        if (g_copies != (device ? 2 : 0)) return fail("copies of votes and counts");
        if (g_queue[c->stream].empty()) return fail("device outputs: waited");
        flush(c->stream);
        if (q[5] != 5 || nout[2] != 4) return fail("votes and counts did not arrive");
        int32_t *bq = dev_int(6, device), *bn = dev_int(3, device);
        rfx_batch_item it{};
        it.ctx = handle(c);
        it.votes = bq;
        it.nout = bn;
        rfx_graph* g = nullptr;
        if (rfx_graph_capture_batch(&it, 1, &g, nullptr) != RFX_OK) return fail("rfx_graph_capture_batch");
        flush(c->stream);
        if (bq[5] != 5 || bn[2] != 4) return fail("a batch's votes and counts did not arrive");
    }
    rfx::Ctx* c = context(false);
    auto* q = (int32_t*)make(24, cudaMemoryTypeManaged, 1);
    if (rfx_route_oob(handle(c), q, nullptr, nullptr) != RFX_OK) return fail("managed votes");
    flush(c->stream);
    int32_t host[3];
    if (rfx_route_oob(handle(c), nullptr, host, nullptr) != RFX_OK || host[2] != 4) return fail("host counts");
    return q[5] == 5 ? 0 : fail("managed votes did not arrive");
}

// The error word and the counters are cleared in the order of the context's
// stream: nothing may be left to a stream that does not order it.
static int clears() {
    rfx::Ctx* c = context(false);
    if (!g_queue[nullptr].empty()) return fail("a new context leaves work on the default stream");
    flush(c->stream);
    if (*c->d_err || c->d_pairs[0] || c->d_pairs[1] || c->d_pairs[2]) return fail("a new context's words are not zero");
    *c->d_err = 1;
    if (rfx_synchronize(handle(c)) == RFX_OK) return fail("the error word was not read");
    if (!g_queue[nullptr].empty() || !g_queue[c->stream].empty()) return fail("the clear is still to come");
    return *c->d_err ? fail("the error word was not cleared") : 0;
}

// Calls that return their results complete, also in device memory.
static int complete() {
    rfx::Ctx* c = context(false);
    auto* err = (float*)dev_int(1, 0);
    int32_t* pred = dev_int(3, 0);
    auto* d = (double*)dev_int(12, 0);
    if (rfx_oob_summary(handle(c), err, pred, nullptr) != RFX_OK || pred[2] != 3) return fail("rfx_oob_summary");
    if (rfx_proximity_upper_f64(handle(c), d, 6) != RFX_OK || ((int32_t*)d)[11] != 9) return fail("rfx_proximity_upper_f64");
    d = (double*)dev_int(12, 0);
    if (rfx_proximity_rfgap(handle(c), d, 6) != RFX_OK || ((int32_t*)d)[11] != 9) return fail("rfx_proximity_rfgap");
    if (!g_queue[c->stream].empty()) return fail("work is left on the stream");
    rfx::Ctx* cw = context(true);
    int32_t *q = dev_int(6, 0), *nout = dev_int(3, 0), *pred2 = dev_int(3, 0);
    if (rfx_casewise_votes(handle(cw), (float*)q, nout) != RFX_OK || q[5] != 7 || nout[2] != 4)
        return fail("rfx_casewise_votes");
    if (rfx_oob_summary(handle(cw), nullptr, pred2, nullptr) != RFX_OK || pred2[2] != 3)
        return fail("rfx_oob_summary (case-wise)");
    return g_queue[cw->stream].empty() ? 0 : fail("work is left on the stream");
}

// The key table of RF-GAP outlives its copy, also where a launch fails.
static int tables() {
    rfx::Ctx* c = context(false);
    auto* d = (double*)dev_int(12, 0);
    if (rfx_proximity_rfgap(handle(c), d, 6) != RFX_OK) return fail("rfx_proximity_rfgap");
    g_route_status = RFX_ERR_CUDA;
    if (rfx_proximity_rfgap(handle(c), d, 6) != RFX_ERR_CUDA) return fail("rfx_proximity_rfgap hides an error");
    return 0;
}

// The factor operator's block arrives before its kernels read it.
static int operator_block() {
    rfx::Ctx* c = context(false);
    c->lr_rank = 1;
    rfx::dalloc(c, &c->d_lrA, 3);
    auto *V = (double*)dev_int(96, 0), *W = (double*)dev_int(96, 0);
    for (int e = 0; e < 48; ++e) V[e] = e;
    if (rfx_factor_mds_operator(handle(c), 0, 0, V, W) != RFX_OK) return fail("rfx_factor_mds_operator");
    if (!g_queue[nullptr].empty() || W[47] != 47) return fail("the product of another block, or not there on return");
    return 0;
}

int main(int argc, char** argv) {
    const std::map<std::string, int (*)()> all = {{"other_gpu", other_gpu}, {"clears", clears}, {"complete", complete},
                                                  {"tables", tables}, {"operator_block", operator_block}};
    g_running = true;
    const int rc = all.at(argv[argc - 1])();
    g_running = false;
    for (auto& f : g_faults) std::printf("%s\n", f.c_str());
    return g_faults.empty() ? rc : 1;
}
