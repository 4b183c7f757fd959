// Device memory, stream order and ray order of the render entry points (ftb_api.cpp) on a CUDA
// runtime made of host memory (test infrastructure, built and run by
// tests/test_render_memory.py).  cudaMalloc fails past a limit, launches of the wave buffers
// are recorded instead of run, and the runtime knows which launches each stream, event and
// synchronization is ordered after, so a render that runs out of memory can be looked at
// without a device: what it launched, what is still in flight when it returns, and whether a
// CUDA error is left on the thread.
#include <cstdio>
#include <cstdlib>
#include <map>
#include <set>

#include "../goodphotons_b200/csrc/ftb_api.cpp"

// ---- the runtime ------------------------------------------------------------------------
namespace fake {
struct Launch { const char *lo, *hi; int64_t photons; ftb::RayOrder order; };
std::vector<Launch> launches;
std::map<cudaStream_t, std::set<int>> after;         // launches a stream's next work runs after
std::map<cudaEvent_t, std::set<int>> recorded;
std::set<int> done;                                  // known to the host to have ended
std::map<void*, size_t> blocks;
size_t live = 0, peak = 0, limit = SIZE_MAX;
int events = 0, overlaps = 0, launch_fails_at = -1;
uintptr_t handles = 0;
bool order_pays = true;
cudaError_t last = cudaSuccess;

cudaError_t err(cudaError_t e) { if (e != cudaSuccess) last = e; return e; }
cudaError_t take(void** p, size_t n) {
    if (live + n > limit) return err(cudaErrorMemoryAllocation);
    *p = std::calloc(1, n ? n : 1);
    blocks[*p] = n;
    live += n;
    peak = std::max(peak, live);
    return cudaSuccess;
}
void give(void* p) {
    if (!p) return;
    live -= blocks[p];
    blocks.erase(p);
    std::free(p);
}
void sync(cudaStream_t s) { done.insert(after[s].begin(), after[s].end()); }
cudaError_t launch(const ftb::Wave& w, int64_t photons, const ftb::WaveKind& kind, cudaStream_t st) {
    if ((int)launches.size() == launch_fails_at) return err(cudaErrorLaunchFailure);
    const Launch l{(const char*)w.block, (const char*)w.block + w.bytes, photons, kind.order};
    for (int k = 0; k < (int)launches.size(); ++k)
        if (launches[k].lo < l.hi && l.lo < launches[k].hi && !done.count(k) && !after[st].count(k)) ++overlaps;
    after[st].insert((int)launches.size());
    launches.push_back(l);
    return cudaSuccess;
}
// launches that neither the host nor work issued next to `user` is ordered after
int in_flight(cudaStream_t user) {
    int n = 0;
    for (int k = 0; k < (int)launches.size(); ++k) n += !done.count(k) && !after[user].count(k);
    return n;
}
void reset() {
    launches.clear(); after.clear(); recorded.clear(); done.clear();
    overlaps = 0; launch_fails_at = -1; last = cudaSuccess; limit = SIZE_MAX; peak = live;
}
}  // namespace fake

extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) { return fake::take(p, n); }
cudaError_t cudaFree(void* p) {   // waits for the device
    for (int k = 0; k < (int)fake::launches.size(); ++k) fake::done.insert(k);
    fake::give(p);
    return cudaSuccess;
}
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return fake::take(p, n); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { fake::give(p); return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { *p = std::calloc(1, n); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) { *f = *t = 0; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) { std::memset(p, 0, sizeof *p); return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaGetLastError() { cudaError_t e = fake::last; fake::last = cudaSuccess; return e; }
cudaError_t cudaPeekAtLastError() { return fake::last; }
cudaError_t cudaDeviceSynchronize() {
    for (int k = 0; k < (int)fake::launches.size(); ++k) fake::done.insert(k);
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)(++fake::handles); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { fake::sync(s); return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
    fake::after[s].insert(fake::recorded[e].begin(), fake::recorded[e].end());
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { ++fake::events; *e = (cudaEvent_t)(++fake::handles); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { --fake::events; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { fake::recorded[e] = fake::after[s]; return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    fake::done.insert(fake::recorded[e].begin(), fake::recorded[e].end());
    return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float* t, cudaEvent_t, cudaEvent_t) {   // ordered rays take half the time, or twice
    const bool ordered = !fake::launches.empty() && fake::launches.back().order.rays;
    *t = ordered == fake::order_pays ? 1.0f : 2.0f;
    return cudaSuccess;
}
}

namespace ftb {
void wave_carve(Wave& w, void* block, int32_t W, bool log, int32_t hero) {
    w = Wave{};
    w.W = W;
    w.hero = hero > 1 ? hero : 1;
    w.bytes = wave_bytes(W, log, hero);
    w.block = block;
    w.jobs = (DevJob*)block;
    w.params = (int32_t*)((char*)block + sizeof(DevJob) * kWaveJobs);
}
cudaError_t wave_alloc(Wave& w, int32_t W, bool log, int32_t hero) {
    void* block = nullptr;
    cudaError_t e = cudaMalloc(&block, wave_bytes(W, log, hero));
    if (e != cudaSuccess) { w = Wave{}; return e; }
    wave_carve(w, block, W, log, hero);
    return cudaSuccess;
}
void wave_free(Wave& w) {
    if (w.block) cudaFree(w.block);
    w.block = nullptr;
}
struct WaveGraphs {};
WaveGraphs* wave_graphs_create() { return new WaveGraphs(); }
void wave_graphs_destroy(WaveGraphs* g) { delete g; }
int32_t trace_limit(int32_t) { return 75776; }
// as the real ones: launches without a graph end in a look at the thread's last error
cudaError_t launch_stream(Wave& w, int64_t photons, int32_t, const WaveKind& kind, const Frame&, int32_t,
                          const LaunchShape& shape, cudaStream_t st, LaunchSink*, WaveGraphs*) {
    cudaError_t e = fake::launch(w, photons, kind, st);
    return e != cudaSuccess || shape.graph ? e : cudaGetLastError();
}
cudaError_t launch_wave(Wave& w, int32_t, const WaveKind& kind, const Frame&, int32_t, const LaunchShape& shape,
                        cudaStream_t st, LaunchSink*, WaveGraphs*, bool) {
    cudaError_t e = fake::launch(w, w.params[1], kind, st);
    return e != cudaSuccess || shape.graph ? e : cudaGetLastError();
}
bool build_wide_lbvh_device(const std::vector<Box>&, int, int, WideBvh&, std::string& err) {
    err = "no device";
    return false;
}
}  // namespace ftb

// ---- renders ----------------------------------------------------------------------------
namespace {
constexpr int32_t kSlots = 4096;
int failures = 0;
void check(bool ok, const char* what, const std::string& where) {
    if (!ok) { std::printf("%s: %s\n", where.c_str(), what); ++failures; }
}

struct Host {   // a scene without geometry: nothing is launched for real
    ftb_scene* s = new ftb_scene();
    ftb_camera cam{};
    std::vector<int64_t> film = std::vector<int64_t>(4 * 4 * 4);
    Host(int regenerate, int graphs, int32_t slots = kSlots, int sort_rays = 2) {
        ftb_tuning t{};
        t.wave_slots = slots; t.sort_rays = sort_rays; t.grid_mult = 16; t.use_graphs = graphs; t.regenerate = regenerate;
        ftb_set_tuning(0, &t);
        s->eng = engine_for(0);
        s->tables = std::make_shared<DevBlock>();
        s->power = 1.0;
        cam.res_x = cam.res_y = 4;
    }
    ~Host() { delete s; }
    ftb_status batch(const std::vector<int>& heroes, int64_t n, cudaStream_t user) {
        std::vector<ftb_job> jobs;
        for (int h : heroes) {
            ftb_job j{};
            j.scene = s; j.cam = cam; j.d_film = film.data(); j.n_photons = n; j.max_bounce = 4; j.hero_c = h;
            jobs.push_back(j);
        }
        return ftb_render_batch(jobs.data(), (int32_t)jobs.size(), nullptr, nullptr, user);
    }
};
int64_t photons_launched(size_t from) {
    int64_t n = 0;
    for (size_t k = from; k < fake::launches.size(); ++k) n += fake::launches[k].photons;
    return n;
}

// A buffer of twice the slots does not fit, one of the slots does: the render is whole and
// leaves no error on the thread; and where neither fits, the error is the call's alone.
void error_left_behind() {
    for (int graphs : {1, 0})
        for (bool fits : {true, false}) {
            fake::reset();
            Host h(1, graphs);
            fake::limit = fake::live + 4096 + ftb::wave_bytes(kSlots, false) * (fits ? 3 : 1) / 2;
            const std::string where = "graphs " + std::to_string(graphs) + (fits ? " fits" : " too large");
            const ftb_status st = h.batch({1, 1}, 3 * kSlots, nullptr);
            check(st == (fits ? FTB_OK : FTB_ERR_OOM), "status", where + " " + ftb_last_error());
            check(photons_launched(0) == (fits ? 6 * kSlots : 0), "photons launched", where);
            check(fake::last == cudaSuccess, "a CUDA error is left on the thread", where);
        }
}

// Memory limits from nothing to plenty under renders of one and of several passes or waves:
// the render is whole, or it fails with nothing in flight.
void second_buffer() {
    for (int regenerate : {1, 0})
        for (int graphs : {1, 0})
            for (const std::vector<int>& heroes : {std::vector<int>{1, 1}, std::vector<int>{1, 4, 1}}) {
                int whole = 0, refused = 0;
                const size_t step = ftb::wave_bytes(kSlots, false, 4) / 3;
                for (size_t limit = 0; limit <= 12 * step; limit += step) {
                    fake::reset();
                    Host h(regenerate, graphs);
                    fake::limit = fake::live + 4096 + limit;
                    const cudaStream_t user = (cudaStream_t)(uintptr_t)77777;
                    const ftb_status st = h.batch(heroes, 3 * kSlots, user);
                    const std::string where = "regenerate " + std::to_string(regenerate) + " graphs " +
                                              std::to_string(graphs) + " jobs " + std::to_string(heroes.size()) +
                                              " limit " + std::to_string(limit);
                    check(fake::overlaps == 0, "a buffer is used by two launches at once", where);
                    check(fake::in_flight(user) == 0, "launches are in flight beside the caller's stream", where);
                    if (st == FTB_OK) {
                        ++whole;
                        check(photons_launched(0) == (int64_t)heroes.size() * 3 * kSlots, "photons are missing", where);
                    } else {
                        ++refused;
                        check(st == FTB_ERR_OOM, "another error than out of memory", where);
                        check(fake::launches.empty(), "launches before the render was refused", where);
                    }
                }
                check(whole > 0 && refused > 0, "limits that do not bite", std::to_string(whole));
            }
    // a launch that fails after others: nothing stays in flight, and the event is given back
    for (int regenerate : {1, 0}) {
        fake::reset();
        Host h(regenerate, 1);
        const cudaStream_t user = (cudaStream_t)(uintptr_t)77777;
        check(h.batch({1, 4, 1}, 3 * kSlots, user) == FTB_OK, "render", "warm");
        fake::reset();
        const int events = fake::events;
        fake::launch_fails_at = 2;
        check(h.batch({1, 4, 1}, 3 * kSlots, user) == FTB_ERR_CUDA, "no error", "failing launch");
        for (int k = 0; k < (int)fake::launches.size(); ++k)
            check(fake::done.count(k) == 1, "a launch is in flight after the error", "failing launch");
        check(fake::events == events, "an event is lost", "failing launch");
    }
}

// Renders of one and of several passes in turn, from streams that do not wait for one another:
// the device's buffers stay within the footprint the library states, and no launch uses a
// buffer that another may still be using.
void stated_memory() {
    for (int regenerate : {1, 0})
        for (bool several_first : {true, false}) {
            fake::reset();
            Host h(regenerate, 1);
            const std::vector<int> one{1, 1}, several(300, 1);
            ftb_footprint fp;
            check(ftb_scene_footprint(h.s, 4, 4, &fp) == FTB_OK, "footprint", "");
            const size_t before = fake::live, small = 300 * 64 + 4096;   // tallies, status
            for (int k = 0; k < 4; ++k) {
                const bool sev = (k & 1) == (several_first ? 0 : 1);
                const std::string where = "regenerate " + std::to_string(regenerate) + " render " + std::to_string(k);
                const size_t from = fake::launches.size();
                const ftb_status st = h.batch(sev ? several : one, sev ? 100 : 3 * kSlots, (cudaStream_t)(uintptr_t)(90000 + k));
                check(st == FTB_OK, ftb_last_error(), where);
                check(!sev || fake::launches.size() - from > 1, "one pass only", where);
                check(fake::live - before <= fp.wave_bytes + small, "more than the stated buffers", where);
                check(fake::overlaps == 0, "a buffer is used by two launches at once", where);
            }
        }
}

// Rays are ordered where the tuning says so: never, always, or where the scene is large and the
// paths in flight are many.
void ray_order() {
    struct Row { int nodes; bool shapes; int32_t slots; bool rays, connections; };   // for sort_rays 2
    const Row rows[] = {
        {100000, false, 1 << 19, false, false}, {100000, false, 1 << 20, false, true},
        {100000, false, 1 << 21, false, true},  {100000, false, 1 << 22, true, true},
        {100000, true, 1 << 18, false, false},  {100000, true, 1 << 19, true, false},
        {100000, true, 1 << 20, true, true},    {100, false, 1 << 22, false, false},
        {100, true, 1 << 22, false, false}};
    for (int regenerate : {1, 0})
        for (const Row& r : rows)
            for (int sort_rays : {0, 1, 2}) {
                fake::reset();
                Host h(regenerate, 1, 1 << 22, sort_rays);
                h.s->dev.max_nodes = r.nodes;
                h.s->dev.n_recs = r.shapes;
                const std::string where = "sort_rays " + std::to_string(sort_rays) + " nodes " + std::to_string(r.nodes) +
                                          " paths " + std::to_string(r.slots) + (r.shapes ? " shapes" : "");
                check(h.batch({1}, r.slots, nullptr) == FTB_OK && fake::launches.size() == 1, ftb_last_error(), where);
                const ftb::RayOrder o = fake::launches.empty() ? ftb::RayOrder{} : fake::launches[0].order;
                check(o.rays == (sort_rays == 2 ? r.rays : sort_rays == 1), "closest-hit rays", where);
                check(o.connections == (sort_rays == 2 ? r.connections : sort_rays == 1 && r.nodes > 10000),
                      "connections", where);
            }
    // the autotuner's choice: by its times, and in a large scene one that leaves small scenes alone
    for (int nodes : {100000, 100})
        for (bool pays : {true, false}) {
            fake::reset();
            fake::order_pays = pays;
            Host h(1, 1, 1 << 22);
            h.s->dev.max_nodes = nodes;
            ftb_tuning t{};
            check(ftb_autotune(h.s, &h.cam, 1 << 22, 4, &t) == FTB_OK, ftb_last_error(), "autotune");
            check(t.sort_rays == (pays ? (nodes > 10000 ? 2 : 1) : 0), "sort_rays",
                  "autotune nodes " + std::to_string(nodes) + (pays ? " pays" : "") + " " + std::to_string(t.sort_rays));
        }
}
}  // namespace

int main(int argc, char** argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    if (what == "error_left_behind") error_left_behind();
    else if (what == "second_buffer") second_buffer();
    else if (what == "stated_memory") stated_memory();
    else if (what == "ray_order") ray_order();
    else return 2;
    std::printf("%s: %s\n", what.c_str(), failures ? "wrong" : "ok");
    return failures ? 1 : 0;
}
