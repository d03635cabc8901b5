// batch.cu - ensembles of contexts advanced together (athad_batch_* of include/athad_gpu.h).
//
// A batch owns no field memory: its members are ordinary mixed-precision contexts, each
// with its own grid and parameters.  One batched model iteration forks up to 32 of the members'
// own streams (lanes) from the batch's stream, enqueues each member's iteration on one of them -
// the column physics at the member's own cadence (pressure sweep every 4th iteration, saturation
// adjustment + moist convection + densities every 2nd), the level mean, the four RK4 stages
// with the time-level copy fused into the last - and joins the lanes in a tiny launch that
// advances the members' device-side iteration counters.
//
// The members depend on one another nowhere, so a lane never waits for another: a member's
// column kernels, which fill only part of the GPU (one thread per column, latency-bound
// recurrences), run beside other members' RK4 stages, which are bound by memory traffic.
// One persistent launch per stage over the tiles of all members, behind a join of all
// column physics, was 1.56 times slower per point than the single-grid stage kernels (a
// member's arguments in shared memory, neighbouring planes read at unrelated times).  Four
// iterations, persistent -> lanes: the 64 members of the largest ensemble (60.1 M points) 273 ->
// 128 ms, 64 of 15x61x109 31.9 -> 14.7, 64 of 11x21x41 6.0 -> 3.5, six of 0.4 to 2.4 M points
// 19.1 -> 13.8, one of 27x99x151 2.44 -> 1.42.  Without a graph, where the host issues each
// launch: 64 of 15x61x109 33.1 -> 16.0, 64 of 11x21x41 6.9 -> 6.8.
//
// Step scalars live on the device: every member's buoyancy ramp min(1, n / ramp_iters) is
// in its step record, kept with its iteration counter, so one captured CUDA graph of an
// iteration stays valid from step to step.  Graphs are keyed by what changes the launch
// list: each member's cadence (pressure sweep? column physics?), its pressure ceiling (above
// 300 iterations) and the tile shape; a batch replays at most a handful.
#include <algorithm>
#include <cstring>
#include <map>
#include <new>
#include <string>
#include <vector>

#include "ctx.cuh"

namespace athad {

// the buoyancy prefactor of a member's iteration, ramp min(1, iter / ramp_iters)
__host__ __device__ inline float batch_buoyancy(const BatchStep& st)
{
    const double x = (double)st.iter / (double)st.ramp_iters;
    const double ramp = (x < 1.0) ? x : 1.0;
    return (float)(ramp * st.g * st.dt / st.u_0);
}

__global__ void batch_advance_kernel(BatchStep* step, int n)
{
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= n || !step[m].active) return;
    step[m].iter += 1;
    step[m].buoy_pref = batch_buoyancy(step[m]);
}

}  // namespace athad

namespace {

// a cadence pattern: how often it ran without a graph, then its graph
struct GraphEntry {
    int uses = 0;
    cudaGraphExec_t exec = nullptr;
};

}  // namespace

// Lanes of a batched iteration.  Four iterations with 4, 8, 16, 32 lanes: 32 members of
// 11x21x41 3.73, 2.53, 2.00, 1.76 ms; 16 of 15x61x109 4.52, 4.14, 3.81, 3.80; twelve of
// 27x99x151 11.6, 11.2, 10.9, 11.0.  More members than lanes, replayed, with 8, 16, 32 lanes:
// 64 of 11x21x41 5.01, 4.19, 3.62.
constexpr int kSideStreams = 32;

// A pattern is captured when it comes for the kCaptureAt-th time.  The graph of an iteration of
// 33 or more members takes 2 ms to instantiate and 2 to end (60 us a lane each), a batch has three
// or four of them, and a server drops them whenever its members change: every twenty iterations
// or so with 64 runs of a thousand.  A replay saves 0.5 ms per iteration of 33 members of
// 11x21x41.  A batch of them made, run and closed, for kCaptureAt = 1, 2, 4, 8: 4 iterations 15,
// 8.3, 4.9 and 4.7 ms, 8 iterations 17, 18, 12 and 8.2, 16 iterations 26, 22, 28 and 19, 40
// iterations 33, 35, 38 and 41, 120 iterations 72, 71, 74 and 99.  Members of 27x99x151 and more
// keep the GPU busy while the host captures.
constexpr int kCaptureAt = 8;

struct athad_batch {
    std::vector<athad_ctx*> m;
    std::vector<cudaStream_t> side;     // member q's iteration runs on side[q % size], streams of the members
    cudaEvent_t fork = nullptr;
    std::vector<cudaEvent_t> join;
    std::vector<RK4MArgs> args;         // the members' stage arguments (stage buffer A in Yout, B in Ybnd)
    std::vector<int32_t> iter;          // host mirror of each member's next iteration number
    std::vector<uint8_t> active;
    cudaStream_t own_stream = nullptr;
    cudaStream_t stream = nullptr;
    BatchStep* d_step = nullptr;        // [n] step records on the device
    int shape = 0;                      // tile shape of the RK4 stages
    std::map<std::vector<uint8_t>, GraphEntry> graphs;
    std::string err;
};

static athad_status bfail(athad_batch* b, athad_status s, const std::string& msg)
{
    if (b) b->err = msg;
    return s;
}

static athad_status bcuda(athad_batch* b, cudaError_t e, const char* what)
{
    if (e == cudaSuccess) return ATHAD_OK;
    if (b) b->err = std::string(what) + ": " + cudaGetErrorString(e);
    return (e == cudaErrorMemoryAllocation) ? ATHAD_ERR_OOM : ATHAD_ERR_CUDA;
}

static void drop_graphs(athad_batch* b)
{
    for (auto& kv : b->graphs)
        if (kv.second.exec) cudaGraphExecDestroy(kv.second.exec);
    b->graphs.clear();
}

// A member's column physics at its cadence, on its context's stream.
static athad_status enqueue_columns(athad_ctx* c, int it)
{
    athad_status s = ATHAD_OK;
    if (it % 4 == 0) s = athad_pressure_sweep(c, 1, it);
    if (s == ATHAD_OK && it % 2 == 0) {
        s = athad_saturation_adjust(c);
        if (s == ATHAD_OK) s = athad_moist_convection(c, it);
        if (s == ATHAD_OK) s = athad_densities(c, 0);
    }
    return s;
}

// The level mean (single-grid kernels) and an RK4 stage of member q on its context's stream.
static athad_status enqueue_level_mean(athad_ctx* c)
{
    launch_level_mean(c->L.d, c->field[ATHAD_T], c->sin_w, c->prof[ATHAD_PROF_T_REF_LEVEL], c->row_sum, c->stream, nullptr);
    return cuda_check(c, cudaGetLastError(), "batch level mean");
}

static athad_status enqueue_stage(athad_batch* b, int q, int stage, int shape)
{
    athad_ctx* c = b->m[q];
    RK4MArgs& a = b->args[q];
    for (int f = 0; f < kMixedGroups; f++) {
        a.Yin[f] = (stage == 3) ? c->mB[f] : c->mA[f];
        a.Yout[f] = (stage == 1 || stage == 3) ? c->mA[f] : c->mB[f];
    }
    launch_rk4m_member_stage(stage, shape, a, b->d_step + q, c->stream);
    return cuda_check(c, cudaGetLastError(), "batch rk4 stage");
}

// Runs enqueue(q) for every active member with its context's stream on the member's lane,
// between a fork of the lanes from b->stream and their join to it (also under capture).  The
// lanes that have forked join, whatever failed.
template <class F> static athad_status on_lanes(athad_batch* b, F enqueue)
{
    const int n = (int)b->m.size(), ns = (int)b->side.size();
    athad_status s = bcuda(b, cudaEventRecord(b->fork, b->stream), "batch fork");
    int forked = 0;
    for (; forked < ns && s == ATHAD_OK; forked++) s = bcuda(b, cudaStreamWaitEvent(b->side[forked], b->fork, 0), "batch fork");
    for (int q = 0; q < n && s == ATHAD_OK; q++) {
        if (!b->active[q]) continue;
        athad_ctx* c = b->m[q];
        cudaStream_t saved = c->stream;
        c->stream = b->side[q % ns];
        s = enqueue(q);
        c->stream = saved;
        if (s != ATHAD_OK) bfail(b, s, std::string("member ") + std::to_string(q) + ": " + c->err);
    }
    for (int q = 0; q < forked; q++) {
        cudaError_t e = cudaEventRecord(b->join[q], b->side[q]);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(b->stream, b->join[q], 0);
        if (s == ATHAD_OK) s = bcuda(b, e, "batch join");
    }
    return s;
}

// Enqueue one iteration of every active member on b->stream (also used under capture).
static athad_status enqueue_iteration(athad_batch* b)
{
    const int n = (int)b->m.size();
    athad_status s = on_lanes(b, [b](int q) {
        athad_status r = enqueue_columns(b->m[q], b->iter[q]);
        if (r == ATHAD_OK) r = enqueue_level_mean(b->m[q]);
        for (int stage = 1; stage <= 4 && r == ATHAD_OK; stage++) r = enqueue_stage(b, q, stage, b->shape);
        return r;
    });
    if (s != ATHAD_OK) return s;
    batch_advance_kernel<<<(n + 127) / 128, 128, 0, b->stream>>>(b->d_step, n);
    return bcuda(b, cudaGetLastError(), "batch advance");
}

// Whether the batch's stream can be captured: not while a caller captures it, and not the legacy
// stream.
static bool capturable(const athad_batch* b)
{
    if (b->stream == cudaStreamLegacy) return false;
    cudaStreamCaptureStatus c = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(b->stream, &c) != cudaSuccess) { cudaGetLastError(); return false; }
    return c == cudaStreamCaptureStatusNone;
}

// What enqueue() puts on b->stream, as a graph.
template <class F> static athad_status capture(athad_batch* b, F enqueue, cudaGraphExec_t* exec)
{
    cudaGraph_t graph = nullptr;
    athad_status s = bcuda(b, cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal), "begin capture");
    if (s != ATHAD_OK) { cudaGetLastError(); return s; }   // the next launch's check must not see it
    s = enqueue();
    const cudaError_t e = cudaStreamEndCapture(b->stream, &graph);
    if (s == ATHAD_OK) s = bcuda(b, e, "end capture");
    if (s == ATHAD_OK) s = bcuda(b, cudaGraphInstantiate(exec, graph, 0), "instantiate");
    if (s != ATHAD_OK) { cudaGetLastError(); *exec = nullptr; }
    if (graph) cudaGraphDestroy(graph);
    return s;
}

static std::vector<uint8_t> graph_key(const athad_batch* b)
{
    std::vector<uint8_t> key;
    key.reserve(b->m.size() + 1);
    key.push_back((uint8_t)b->shape);
    for (size_t q = 0; q < b->m.size(); q++) {
        const int it = b->iter[q];
        uint8_t k = 0;
        if (b->active[q]) {
            k |= 1;
            if (it % 4 == 0) k |= 2;
            if (it % 2 == 0) k |= 4;
            if (it > 300) k |= 8;     // pressure ceiling 3 instead of 10
        }
        key.push_back(k);
    }
    return key;
}

static void advance_host(athad_batch* b)
{
    for (size_t q = 0; q < b->m.size(); q++)
        if (b->active[q]) b->iter[q] += 1;
}

extern "C" {

athad_status athad_batch_create(athad_ctx* const* members, int32_t n_members, const athad_batch_step* step,
                                const int32_t* first_iter, athad_batch** out)
{
    if (!out) return ATHAD_ERR_INVALID;
    *out = nullptr;
    if (!members || n_members < 1 || !step || step->dt <= 0.0 || step->buoyancy_ramp_iters < 1)
        return ATHAD_ERR_INVALID;
    for (int q = 0; q < n_members; q++) {
        if (!members[q]) return ATHAD_ERR_INVALID;
        if (members[q]->p.precision != ATHAD_PRECISION_MIXED) return ATHAD_ERR_UNSUPPORTED;
        for (int r = 0; r < q; r++)
            if (members[r] == members[q]) return ATHAD_ERR_INVALID;
    }
    // the batch runs the members on its own streams: what is queued on theirs (an initial
    // state, an upload) must be complete first
    for (int q = 0; q < n_members; q++)
        if (cudaStreamSynchronize(members[q]->stream) != cudaSuccess) { cudaGetLastError(); return ATHAD_ERR_CUDA; }
    athad_batch* b = new (std::nothrow) athad_batch();
    if (!b) return ATHAD_ERR_OOM;
    b->m.assign(members, members + n_members);
    b->iter.resize(n_members);
    b->active.assign(n_members, 1);
    for (int q = 0; q < n_members; q++) b->iter[q] = first_iter ? first_iter[q] : 1;
    const int n = n_members;

    b->args.resize(n);
    std::vector<BatchStep> steps(n);
    for (int q = 0; q < n; q++) {
        athad_ctx* c = members[q];
        RK4MArgs& a = b->args[q];
        // the time-level copy fused; the buoyancy ramp of the scalars is not used (MEMBER kernels)
        const athad_step_scalars sc{step->dt, step->diffusion_ramp, 1.0, 0, 1};
        mixed_args(c, &sc, a);
        for (int f = 0; f < kMixedGroups; f++) a.Ybnd[f] = c->mB[f];
        BatchStep& s = steps[q];
        std::memset(&s, 0, sizeof s);
        s.g = c->p.g; s.dt = step->dt; s.u_0 = c->p.u_0;
        s.iter = b->iter[q];
        s.ramp_iters = step->buoyancy_ramp_iters;
        s.active = 1;
        s.buoy_pref = batch_buoyancy(s);
    }

    athad_status st = ATHAD_OK;
    if (cudaStreamCreateWithFlags(&b->own_stream, cudaStreamNonBlocking) != cudaSuccess) {
        cudaGetLastError(); delete b; return ATHAD_ERR_CUDA;
    }
    b->stream = b->own_stream;
    if (cudaMalloc((void**)&b->d_step, sizeof(BatchStep) * n) != cudaSuccess) {
        cudaGetLastError(); cudaStreamDestroy(b->own_stream); delete b; return ATHAD_ERR_OOM;
    }
    st = bcuda(b, cudaMemcpyAsync(b->d_step, steps.data(), sizeof(BatchStep) * n, cudaMemcpyHostToDevice, b->stream), "steps");
    if (st == ATHAD_OK) st = bcuda(b, cudaStreamSynchronize(b->stream), "batch create sync");
    // The lanes are the streams that the first members own (made with each context), and the
    // events of their fork and join.  Streams of the batch's own cost a batch of 64 members of
    // 11x21x41 1.2 ms more at creation and 1.3 ms more at its end, and a server makes a batch
    // whenever its members change.
    if (st == ATHAD_OK) st = bcuda(b, cudaEventCreateWithFlags(&b->fork, cudaEventDisableTiming), "batch events");
    const int ns = std::min(n, kSideStreams);
    for (int q = 0; q < ns && st == ATHAD_OK; q++) {
        cudaEvent_t e = nullptr;
        st = bcuda(b, cudaEventCreateWithFlags(&e, cudaEventDisableTiming), "batch events");
        if (st == ATHAD_OK) { b->join.push_back(e); b->side.push_back(members[q]->own_stream); }
    }
    if (st != ATHAD_OK) {
        for (cudaEvent_t e : b->join) cudaEventDestroy(e);
        if (b->fork) cudaEventDestroy(b->fork);
        cudaFree(b->d_step); cudaStreamDestroy(b->own_stream); delete b;
        return st;
    }
    *out = b;
    return ATHAD_OK;
}

athad_status athad_batch_destroy(athad_batch* b)
{
    if (!b) return ATHAD_ERR_INVALID;
    cudaStreamSynchronize(b->stream);   // the lanes have joined it (the members may be gone)
    drop_graphs(b);
    for (cudaEvent_t e : b->join) cudaEventDestroy(e);
    if (b->fork) cudaEventDestroy(b->fork);
    cudaFree(b->d_step);
    cudaStreamDestroy(b->own_stream);
    delete b;
    return ATHAD_OK;
}

const char* athad_batch_last_error(const athad_batch* b)
{
    return b ? b->err.c_str() : "null batch";
}

athad_status athad_batch_set_stream(athad_batch* b, void* s)
{
    if (!b) return ATHAD_ERR_INVALID;
    cudaStream_t ns = s ? (cudaStream_t)s : b->own_stream;
    if (ns != b->stream) drop_graphs(b);
    b->stream = ns;
    return ATHAD_OK;
}

athad_status athad_batch_synchronize(athad_batch* b)
{
    if (!b) return ATHAD_ERR_INVALID;
    return bcuda(b, cudaStreamSynchronize(b->stream), "batch synchronize");
}

athad_status athad_batch_member_iter(const athad_batch* b, int32_t member, int32_t* next_iter)
{
    if (!b || !next_iter || member < 0 || member >= (int32_t)b->m.size()) return ATHAD_ERR_INVALID;
    *next_iter = b->iter[member];
    return ATHAD_OK;
}

athad_status athad_batch_set_active(athad_batch* b, int32_t member, int32_t active)
{
    if (!b || member < 0 || member >= (int32_t)b->m.size()) return ATHAD_ERR_INVALID;
    const uint8_t a = active ? 1 : 0;
    if (b->active[member] == a) return ATHAD_OK;
    b->active[member] = a;
    const int32_t v = a;
    return bcuda(b, cudaMemcpyAsync(&b->d_step[member].active, &v, sizeof v, cudaMemcpyHostToDevice, b->stream),
                 "set active");
}

athad_status athad_batch_iteration(athad_batch* b)
{
    if (!b) return ATHAD_ERR_INVALID;
    athad_status s = enqueue_iteration(b);
    if (s == ATHAD_OK) advance_host(b);
    return s;
}

athad_status athad_batch_iteration_graph(athad_batch* b)
{
    if (!b) return ATHAD_ERR_INVALID;
    const std::vector<uint8_t> key = graph_key(b);
    auto it = b->graphs.find(key);
    if (it == b->graphs.end()) {
        if (b->graphs.size() >= 16) drop_graphs(b);
        it = b->graphs.emplace(key, GraphEntry()).first;
    }
    GraphEntry& g = it->second;
    // a stream that cannot be captured is refused from the first use on
    if (!g.exec && ++g.uses < kCaptureAt && capturable(b)) return athad_batch_iteration(b);
    athad_status s = ATHAD_OK;
    if (!g.exec) s = capture(b, [b] { return enqueue_iteration(b); }, &g.exec);
    if (s == ATHAD_OK) s = bcuda(b, cudaGraphLaunch(g.exec, b->stream), "graph launch");
    if (s == ATHAD_OK) advance_host(b);
    return s;
}

int32_t athad_batch_shape_count(void) { return batch_shape_count(); }

athad_status athad_batch_set_shape(athad_batch* b, int32_t shape)
{
    if (!b || shape < 0 || shape >= batch_shape_count()) return ATHAD_ERR_INVALID;
    if (shape != b->shape) drop_graphs(b);
    b->shape = shape;
    return ATHAD_OK;
}

athad_status athad_batch_autotune(athad_batch* b, int32_t reps, int32_t* best_shape, float* ms_per_shape)
{
    if (!b || reps < 1) return ATHAD_ERR_INVALID;
    cudaEvent_t e0, e1;
    if (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess) {
        cudaGetLastError(); return bfail(b, ATHAD_ERR_CUDA, "autotune events");
    }
    float best = 3.4e38f;
    int best_id = b->shape;
    athad_status s = ATHAD_OK;
    for (int sh = 0; sh < batch_shape_count() && s == ATHAD_OK; sh++) {
        // stages 1-3 write only the members' private FP32 buffers, which the next
        // iteration's stage 1 rewrites, so timing them leaves the model state unchanged
        auto stages = [b, sh] {
            return on_lanes(b, [b, sh](int q) {
                athad_status r = ATHAD_OK;
                for (int stage = 1; stage <= 3 && r == ATHAD_OK; stage++) r = enqueue_stage(b, q, stage, sh);
                return r;
            });
        };
        // Replays of a graph, as iterations run: launched one by one, the stages of many small
        // members take the host longer than the GPU, whatever the shape.
        // A stream that cannot be captured (the legacy one) runs them one by one.
        cudaGraphExec_t exec = nullptr;
        (void)capture(b, stages, &exec);
        auto once = [&] { return exec ? bcuda(b, cudaGraphLaunch(exec, b->stream), "autotune") : stages(); };
        s = once();
        cudaEventRecord(e0, b->stream);
        for (int r = 0; r < reps && s == ATHAD_OK; r++) s = once();
        cudaEventRecord(e1, b->stream);
        if (s == ATHAD_OK) s = bcuda(b, cudaEventSynchronize(e1), "autotune");
        if (exec) cudaGraphExecDestroy(exec);
        float ms = 0.0f;
        if (s == ATHAD_OK) s = bcuda(b, cudaEventElapsedTime(&ms, e0, e1), "autotune time");
        ms /= (float)reps;
        if (ms_per_shape) ms_per_shape[sh] = ms;
        if (s == ATHAD_OK && ms < best) { best = ms; best_id = sh; }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (s != ATHAD_OK) return s;
    if (best_id != b->shape) drop_graphs(b);
    b->shape = best_id;
    if (best_shape) *best_shape = best_id;
    return ATHAD_OK;
}

}  // extern "C"
