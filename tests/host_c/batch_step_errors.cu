// fb_batch_submit on the host: batch_step.cu with fakes of the CUDA runtime
// (fake_cudart.cpp) and of the session functions it calls, which note every call and can refuse
// one.  Prints "<check> <runs> <failures>" per check.
#include "../../fusion_b200/csrc/batch_step.cu"

#include <cstdio>
#include <set>

// ------------------------------------------------------------------- fakes

static std::vector<fb_session*> pop;          // the sessions of the scenario
extern std::set<cudaStream_t> busy;           // fake_cudart.cpp: streams with work the host has not waited for
extern const void* device_memory;             // fake_cudart.cpp: the address that is device memory
extern int refuse_graph;                      // fake_cudart.cpp: no graph is instantiated
static std::vector<int> copied, launched, finished;   // calls per session
static int refuse_copy, refuse_frame;         // the session whose call is refused, -1: none
static bool finished_early;                   // a result was taken while its stream was busy

static int index_of(const fb_session* s) {
    for (size_t i = 0; i < pop.size(); ++i)
        if (pop[i] == s) return (int)i;
    return -1;
}

namespace fb {
bool cuda_ok(cudaError_t e) { return e == cudaSuccess; }
int check_launch() { return FB_OK; }
LaunchRecorder*& launch_recorder() {
    static LaunchRecorder* r = nullptr;
    return r;
}
int copy_frame_in(fb_session* s, const uint16_t*, size_t, const uint8_t*, size_t, int, cudaStream_t st) {
    const int i = index_of(s);
    busy.insert(st);   // the depth image is on its way even where the colour is refused
    if (i == refuse_copy) return FB_ECUDA;
    ++copied[i];
    return FB_OK;
}
FramePlan plan_frame(fb_session* s) {
    FramePlan p{};
    std::swap(s->state, s->last_state);
    p.state = s->state;
    p.track = true;
    p.mode = 1;
    return p;
}
void unplan_frame(fb_session* s) { std::swap(s->state, s->last_state); }
int enqueue_frame(fb_session* s, const FramePlan&, cudaStream_t st, unsigned*) {
    const int i = index_of(s);
    if (i == refuse_frame) return FB_ECUDA;
    busy.insert(st);
    ++launched[i];
    return FB_OK;
}
int fetch_result(fb_session*, cudaStream_t) { return FB_OK; }
// a frame that records no launch: a fused step refuses it
int issue_frame(fb_session*, bool, bool, bool, bool, unsigned*, int, const double*) { return 1; }
void finish_frame(fb_session* s, const FramePlan&, fb_frame_result*) {
    if (!busy.empty()) finished_early = true;
    s->last_state = 0;
    ++finished[index_of(s)];
}
}  // namespace fb
void fb_set_error_text(const char*) {}

// ---------------------------------------------------------------- scenarios

static int runs, failures;
static void check(bool ok) {
    ++runs;
    failures += !ok;
}
static void report(const char* name) {
    std::printf("%s %d %d\n", name, runs, failures);
    runs = failures = 0;
}

static std::vector<fb_frame_input> inputs;
static uint64_t last_id;
static uint16_t depth, depth_k;
static uint8_t rgb;
static void reset(int n) {
    for (fb_session* s : pop) delete s;
    pop.clear();
    for (int i = 0; i < n; ++i) {
        fb_session* s = new fb_session();
        s->id = ++last_id;
        s->W[0] = 16;
        s->H[0] = 16;
        s->state = 3;        // told apart from the last state by value only
        s->last_state = 4;
        s->h_out_dev = (FrameOut*)16;
        pop.push_back(s);
    }
    inputs.assign(n, fb_frame_input{&depth, 32, &rgb, 48, 0});
    copied.assign(n, 0);
    launched.assign(n, 0);
    finished.assign(n, 0);
    busy.clear();
    finished_early = false;
    refuse_copy = refuse_frame = -1;
    refuse_graph = 0;
    device_memory = nullptr;
}

static bool untouched(int i) {
    return pop[i]->state == 3 && pop[i]->last_state == 4 && !pop[i]->shared_gpu && !finished[i];
}

static bool good_step(fb_batch* b, int n) {
    refuse_copy = refuse_frame = -1;
    refuse_graph = 0;
    std::vector<fb_frame_result> out(n);
    const std::vector<int> before = finished;
    if (fb_batch_step(b, pop.data(), n, inputs.data(), out.data()) != FB_OK) return false;
    for (int i = 0; i < n; ++i)
        if (finished[i] != before[i] + 1 || pop[i]->shared_gpu) return false;
    return !finished_early;
}

int main() {
    fb_batch* b = nullptr;
    if (fb_batch_create(nullptr, &b) != FB_OK) return 1;
    for (int n : {1, 3, 5, 32, 34, 70})
        for (int k : {0, n / 2, n - 1}) {
            // mode 0: an input that is refused leaves every session as it was
            // (host memory that is said to be on the device, and the reverse)
            reset(n);
            refuse_copy = k;
            inputs[k].on_device = k & 1;
            device_memory = k & 1 ? nullptr : &depth_k;
            inputs[k].depth = &depth_k;
            check(fb_batch_submit(b, pop.data(), n, inputs.data()) == FB_ECUDA);
            for (int i = 0; i < n; ++i) check(untouched(i) && !launched[i]);
            check(busy.empty());
            // taken after all: copied once, and the step runs
            check(good_step(b, n));
            for (int i = 0; i < n; ++i) check(pop[i]->state == 4 && launched[i] == 1 && copied[i] >= 1);
            check(copied[k] == 1);
        }
    report("refused_input");
    for (int n : {1, 3, 5, 34})
        for (int k : {0, n / 2, n - 1, n + n / 2}) {
            // mode 0: frames before a launch (or a copy that looked right) that
            // fails are finished, the others never planned
            reset(n);
            if (k < n) {
                refuse_frame = k;
            } else {
                k -= n;
                refuse_copy = k;
            }
            check(fb_batch_submit(b, pop.data(), n, inputs.data()) == FB_ECUDA);
            check(busy.empty() && !finished_early);
            for (int i = 0; i < n; ++i)
                check(i < k ? finished[i] == 1 && pop[i]->state == 4 && !pop[i]->shared_gpu : untouched(i));
            check(good_step(b, n));
        }
    report("failed_launch");
    for (int mode : {1, 2})
        for (int n : {2, 5}) {
            // the other modes: a refused input, a graph that is not made, a frame that is not recorded
            check(fb_batch_set_mode(b, mode) == FB_OK);
            for (int what = 0; what < 2; ++what) {
                reset(n);
                refuse_copy = what == 0 ? n - 1 : -1;
                refuse_graph = 1;
                check(fb_batch_submit(b, pop.data(), n, inputs.data()) != FB_OK);
                for (int i = 0; i < n; ++i) check(untouched(i));
                check(busy.empty());
            }
        }
    report("other_modes");
    {
        // a session made where a destroyed one was takes no graph of it
        uint64_t steps, before, again, other;
        check(fb_batch_set_mode(b, 1) == FB_OK);
        reset(2);
        check(good_step(b, 2));
        fb_batch_stats(b, &steps, &before);
        check(good_step(b, 2));
        fb_batch_stats(b, &steps, &again);
        check(again == before);
        pop[0]->id = ++last_id;
        check(good_step(b, 2));
        fb_batch_stats(b, &steps, &other);
        check(other == before + 1);
    }
    report("same_address");
    return 0;
}
