// A device made of host memory, for checks of the C ABI's host side without a
// GPU: the library's own objects (api, builder, geometry) link against the
// runtime calls and kernel launchers of this file.  Work of a stream runs at
// once, or is recorded while the stream is capturing.  A level's populations
// are a model: how many steps it took, whether its ghosts repeat their sources,
// whether a ghost exchange is due, and whether a kernel ever ran on a state that
// it cannot read ("wrong").
#include <algorithm>
#include <cmath>

// what the launchers' header names of device code (never called here)
template <class T> static T __ldg(const T* p) { return *p; }
template <class T> static T __ldcg(const T* p) { return *p; }
static struct { unsigned x, y, z; } blockIdx, threadIdx;

#include "../../lbm3_b200/csrc/builder.h"
#include "../../lbm3_b200/csrc/energy_noalloc.h"
#include "../../lbm3_b200/csrc/step_launch.h"

#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <memory>
#include <mutex>
#include <unistd.h>
#include <vector>

namespace {

using Ops = std::vector<std::function<void()>>;
struct Stream {
    std::shared_ptr<Ops> graph;  // not null: capturing
};
struct Event {
    std::shared_ptr<Ops> graph;
};
struct Model {
    int order = 0, steps = 0;
    bool ghosts = false, due = false, wrong = false;
};

std::recursive_mutex lock;
std::map<const void*, Model> models;
std::map<cudaStream_t, Stream> streams;
bool initialGhosts = true;
int launches = 0, instantiateLeft = -1, uploadsLeft = -1, copyDelayUs = 0;
size_t pitchLimit = 0x7fffffff;

cudaError_t run(cudaStream_t s, std::function<void()> op) {
    std::unique_lock<std::recursive_mutex> hold(lock);
    if (auto g = streams[s].graph) g->push_back(op);
    else op();
    return cudaSuccess;
}
// one kernel launch
void launch(cudaStream_t s, std::function<void()> op) {
    run(s, [op] { ++launches; op(); });
}
Model& of(const lbm::DevLevel& g) { return models[g.f]; }
void collide(Model& m) {
    m.wrong = m.wrong || m.due;
    m.ghosts = false;
    ++m.steps;
}
void copyGhosts(Model& m) { m.ghosts = true; }
void reads(Model& m) { m.wrong = m.wrong || m.due; }

}  // namespace

extern "C" {
void host_device_reset(int ghosts) {
    models.clear();
    streams.clear();
    initialGhosts = ghosts != 0;
    launches = 0;
    instantiateLeft = uploadsLeft = -1;
    copyDelayUs = 0;
    pitchLimit = 0x7fffffff;
}
int host_device_launches() { return launches; }
// graph instantiations and copies to the device that succeed from now on (-1: all)
void host_device_instantiations(int n) { instantiateLeft = n; }
void host_device_uploads(int n) { uploadsLeft = n; }
void host_device_copy_delay(int us) { copyDelayUs = us; }
void host_device_pitch_limit(size_t bytes) { pitchLimit = bytes; }
// {steps, ghosts, due, wrong} of the order-th level built
int host_device_level(int order, int* out) {
    for (auto& [f, m] : models)
        if (m.order == order) {
            out[0] = m.steps; out[1] = m.ghosts; out[2] = m.due; out[3] = m.wrong;
            return 0;
        }
    return 1;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void** __cudaRegisterFatBinary(void*) { return nullptr; }
void __cudaUnregisterFatBinary(void**) {}
}

// ---- the runtime -------------------------------------------------------------
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    if (a != cudaDevAttrMaxPitch) return cudaErrorInvalidValue;
    *v = static_cast<int>(pitchLimit);
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "host device"; }
cudaError_t cudaMalloc(void** p, size_t n) { *p = std::calloc(n ? n : 1, 1); return *p ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFree(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = reinterpret_cast<cudaStream_t>(new char); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { delete reinterpret_cast<char*>(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    std::unique_lock<std::recursive_mutex> hold(lock);
    return streams[s].graph ? cudaErrorStreamCaptureUnsupported : cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = reinterpret_cast<cudaEvent_t>(new Event); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete reinterpret_cast<Event*>(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { reinterpret_cast<Event*>(e)->graph = streams[s].graph; return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0.f; return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
    if (auto g = reinterpret_cast<Event*>(e)->graph) streams[s].graph = g;
    return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus* st) {
    *st = streams[s].graph ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) {
    streams[s].graph = std::make_shared<Ops>();
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g) {
    const auto graph = streams[s].graph;
    for (auto& [k, v] : streams)
        if (v.graph == graph) v.graph = nullptr;
    *g = reinterpret_cast<cudaGraph_t>(new Ops(*graph));
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t g, unsigned long long) {
    if (instantiateLeft == 0) return cudaErrorMemoryAllocation;
    if (instantiateLeft > 0) --instantiateLeft;
    *e = reinterpret_cast<cudaGraphExec_t>(new Ops(*reinterpret_cast<Ops*>(g)));
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { delete reinterpret_cast<Ops*>(g); return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { delete reinterpret_cast<Ops*>(e); return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t s) {
    if (streams[s].graph) return cudaErrorStreamCaptureUnsupported;
    for (auto& op : *reinterpret_cast<Ops*>(e)) op();
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t s) { return run(s, [=] { std::memset(p, v, n); }); }
cudaError_t cudaMemcpyAsync(void* to, const void* from, size_t n, cudaMemcpyKind kind, cudaStream_t s) {
    if (kind == cudaMemcpyDeviceToHost && copyDelayUs) usleep(copyDelayUs);
    if (kind == cudaMemcpyHostToDevice && uploadsLeft == 0) return cudaErrorUnknown;
    if (kind == cudaMemcpyHostToDevice && uploadsLeft > 0) --uploadsLeft;
    return run(s, [=] { std::memcpy(to, from, n); });
}
cudaError_t cudaMemcpy2DAsync(void* to, size_t toPitch, const void* from, size_t fromPitch, size_t width, size_t rows,
                              cudaMemcpyKind kind, cudaStream_t s) {
    if (toPitch > pitchLimit || fromPitch > pitchLimit) return cudaErrorInvalidPitchValue;
    for (size_t r = 0; r < rows; ++r)
        cudaMemcpyAsync(static_cast<char*>(to) + r * toPitch, static_cast<const char*>(from) + r * fromPitch, width, kind, s);
    return cudaSuccess;
}

// ---- the launchers -----------------------------------------------------------
namespace lbm {

CollideVariant collideVariant() { return CollideVariant::Pair; }
int stepLaunchCount(const DevLevel&) { return 0; }
void launchInit(const DevLevel& g, bool, cudaStream_t, const float4*, float4) {
    Model& m = of(g);
    m = Model{};
    m.order = static_cast<int>(models.size()) - 1;
    m.ghosts = initialGhosts;
}
void launchOpenBoundaryInit(const DevLevel&, bool, cudaStream_t) {}
void launchCollideStream(const DevLevel& g, bool, cudaStream_t s) { launch(s, [&m = of(g)] { collide(m); }); }
void launchPeriodic(const DevLevel& g, bool, cudaStream_t s) { launch(s, [&m = of(g)] { copyGhosts(m); }); }
void launchRotorCells(const DevLevel&, bool, cudaStream_t) {}
void launchOpenBoundary(const DevLevel&, bool, cudaStream_t) {}
void launchWrapped(const DevLevel* const* levels, int count, bool, cudaStream_t s) {
    for (int first = 0; first < count; first += kWrapDomains) {
        std::vector<Model*> step;
        for (int q = first; q < std::min(count, first + kWrapDomains); ++q) step.push_back(&of(*levels[q]));
        launch(s, [step] {
            for (Model* m : step) {
                m->wrong = m->wrong || !m->ghosts;
                m->due = true;
                ++m->steps;
            }
        });
    }
}
void launchWrappedFlush(const DevLevel* const* levels, int count, bool, cudaStream_t s) {
    for (int first = 0; first < count; first += kWrapDomains) {
        std::vector<Model*> flush;
        for (int q = first; q < std::min(count, first + kWrapDomains); ++q) flush.push_back(&of(*levels[q]));
        launch(s, [flush] {
            for (Model* m : flush) m->due = false;
        });
    }
}
void launchGhostsDiffer(const DevLevel& g, bool, cudaStream_t s, int* differ) {
    launch(s, [&m = of(g), differ] { reads(m); *differ = !m.ghosts; });
}
void launchPackedStep(const DevBatch& b, int, bool, cudaStream_t s) {
    launch(s, [b] {
        for (int q = 0; q < b.domainCount; ++q)
            if (b.itemStart[q + 1] > b.itemStart[q]) collide(of(b.levels[q]));
    });
    if (b.periodicCount > 0)
        launch(s, [b] {
            for (int q = 0; q < b.domainCount; ++q)
                if (b.periodicStart[q + 1] > b.periodicStart[q]) copyGhosts(of(b.levels[q]));
        });
}
// what a reader of a level finds: fields and populations tell level, quantity and cell apart
void launchMacro(const DevLevel& g, bool, cudaStream_t s, int first, int count, float* out) {
    launch(s, [&m = of(g), first, count, out] {
        reads(m);
        for (int q = 0; q < 4; ++q)
            for (int i = 0; i < count; ++i) out[size_t(q) * count + i] = float(first + i) * 16 + q * 4 + m.order;
    });
}
void launchGatherF(const DevLevel& g, cudaStream_t s, long long first, int count, float* out) {
    launch(s, [&m = of(g), first, count, out] {
        reads(m);
        for (int i = 0; i < count; ++i) out[i] = -float((first + i) % (1 << 20)) * 8 - m.order;
    });
}
void launchScatterF(const DevLevel& g, cudaStream_t s, long long, int, const float*) {
    launch(s, [&m = of(g)] { m.ghosts = false; });
}
void launchInterface(const DevLevel&, const DevLevel&, const DevInterface&, bool, bool, cudaStream_t) {}
void launchKineticEnergy(const DevLevel& g, bool, cudaStream_t s, double*) { launch(s, [&m = of(g)] { reads(m); }); }
void launchGlobalSums(const DevLevel& g, bool, cudaStream_t s, double*) { launch(s, [&m = of(g)] { reads(m); }); }
void launchWallForce(const DevLevel&, int, cudaStream_t, double*) {}
void launchFlowReport(const DevLevel&, bool, cudaStream_t, int, int, int, int, int, int, double*) {}
void launchRotorForce(const DevRotor&, const int*, cudaStream_t, double*) {}
void launchOpenFlow(const DevLevel&, int, float, cudaStream_t, double*) {}
void launchCollideBatch(float*, int, const CollisionConsts&, float, float, float, cudaStream_t) {}
void launchFlowImageClear(float*, long long, cudaStream_t) {}
void launchFlowImage(const DevLevel&, bool, cudaStream_t, const FlowImagePass&, float*) {}
void launchFlowImageSum(const float*, long long, cudaStream_t, double*) {}
cudaError_t kineticEnergyNoAlloc(const DevLevel&, bool, cudaStream_t, double* sum) { *sum = 0.0; return cudaSuccess; }

}  // namespace lbm
