// Checks of csrc/devmem.cu, of the handle's release and of csrc/small.cu's launch on a host-side
// CUDA runtime: one check per name, exit code 0 when it holds.
#include "cudart.hpp"

#include "handle.cuh"

#include <thread>

namespace btc200 {
void note_cuda_error(cudaError_t, const char*, const char*, int) {}
int device_sm_count() { return 148; }
}  // namespace btc200

using namespace btc200;

static int failures = 0;
#define EXPECT(c)                                                            \
    do {                                                                     \
        if (!(c)) {                                                          \
            std::printf("%s:%d: %s\n", __FILE__, __LINE__, #c);              \
            ++failures;                                                      \
        }                                                                    \
    } while (0)

// Every free on device `dev` comes after a wait for that device.
static void expect_waited(int dev)
{
    bool waited = false, freed = false;
    for (const std::string& l : fake::log) {
        waited |= l == "wait@" + std::to_string(dev);
        if (l == "free@" + std::to_string(dev)) {
            freed = true;
            EXPECT(waited);
        }
    }
    EXPECT(freed);
}

// A handle on device 1 released while device 0 is current.
static void handle_of_another_device()
{
    cudaSetDevice(1);
    btc_bitbsr g;
    g.device = 1;
    g.h_meta = host_slot_alloc(&g.h_context);
    EXPECT(g.indptr.reserve(100) == 0 && g.blocks.reserve(1000) == 0);
    EXPECT(g.policy.dev.reserve(24) == 0);
    g.policy.host = host_slot_alloc(&g.policy.host_context);
    cudaSetDevice(0);
    fake::log.clear();
    g.release_all();
    expect_waited(1);
    EXPECT(fake::current == 0 && fake::device_of.empty());
}

// A buffer alone, and one that grows.
static void buffer_of_another_device()
{
    cudaSetDevice(1);
    DevBuf a, b;
    EXPECT(a.reserve(64) == 0 && b.reserve(64) == 0);
    cudaSetDevice(0);
    fake::log.clear();
    a.release();
    expect_waited(1);
    fake::log.clear();
    EXPECT(b.reserve(4096) == 0);  // the old memory is device 1's, the new one device 0's
    expect_waited(1);
    EXPECT(fake::device_of.at(b.ptr) == 0);
    fake::log.clear();
    b.release();
    expect_waited(0);
    EXPECT(fake::current == 0);
}

// The arrays of a reference-shaped struct.
static void arrays_of_another_device()
{
    cudaSetDevice(1);
    void* p[3] = {nullptr, nullptr, nullptr};
    EXPECT(dev_alloc(&p[1], 64) == cudaSuccess && dev_alloc(&p[2], 64) == cudaSuccess);
    cudaSetDevice(0);
    fake::log.clear();
    free_arrays(p, 3);
    expect_waited(1);
    EXPECT(fake::current == 0 && fake::device_of.empty());
    free_arrays(p, 1);  // nothing held
}

// A program that builds from a new thread each time keeps one block of host slots.
static void slots_of_many_threads()
{
    fake::devices = 1;
    for (int i = 0; i < 20; ++i)
        std::thread([] {
            unsigned long long context = 0;
            unsigned long long* s = host_slot_alloc(&context);
            EXPECT(s && context == fake::context_id[0]);
            host_slot_free(s, context);
        }).join();
    EXPECT(fake::pinned_made == 1);
}

// A slot freed after its context's end is not handed out again; the slots of the new context are.
static void slots_across_a_reset()
{
    cudaSetDevice(0);
    unsigned long long ca = 0, cb = 0, cc = 0;
    unsigned long long* a = host_slot_alloc(&ca);
    fake::reset(0);
    unsigned long long* b = host_slot_alloc(&cb);
    EXPECT(ca != cb && fake::pinned_made == 2);
    host_slot_free(a, ca);
    unsigned long long* c = host_slot_alloc(&cc);
    EXPECT(cc == cb && c != a && c != b);
    EXPECT(*reinterpret_cast<unsigned char*>(a) == 0xEE);  // nothing wrote to the dead memory
    host_slot_free(b, cb);
    EXPECT(host_slot_alloc(&cc) == b);
}

// Two contexts of one device in turn: one pool and one block each, and none more.
static void contexts_in_turn()
{
    fake::devices = 1;
    const unsigned long long first = fake::context_id[0];
    for (int i = 0; i < 6; ++i) {
        fake::context_id[0] = first + i % 2;
        cudaSetDevice(0);
        void* p = nullptr;
        EXPECT(dev_alloc(&p, 64) == cudaSuccess);
        dev_free(p);
        unsigned long long context = 0;
        unsigned long long* s = host_slot_alloc(&context);
        EXPECT(context == first + i % 2);
        host_slot_free(s, context);
    }
    EXPECT(fake::pools_made == 2 && fake::pinned_made == 2);
}

// A kernel's shared-memory opt-in is made once per context of each device.
static void opt_ins()
{
    std::atomic<unsigned long long> done[kMaxDevices] = {};
    int kernel = 0;
    fake::log.clear();
    for (int dev : {0, 0, 1, 0, 1}) {
        cudaSetDevice(dev);
        EXPECT(allow_dynamic_smem(&kernel, 100000, done));
    }
    EXPECT((fake::log == std::vector<std::string>{"attribute100000@0", "attribute100000@1"}));
    fake::reset(0);
    for (int dev : {0, 1, 0}) {
        cudaSetDevice(dev);
        EXPECT(allow_dynamic_smem(&kernel, 100000, done));
    }
    EXPECT(fake::log.size() == 3 && fake::log.back() == "attribute100000@0");
}

// The kept memory is given back on the current device, down to what is asked for.
static void trim()
{
    void* p = nullptr;
    cudaSetDevice(1);
    EXPECT(dev_alloc(&p, 64) == cudaSuccess);
    dev_free(p);
    fake::log.clear();
    EXPECT(btc_trim_memory(4096) == BTC_OK && btc_trim_memory(0) == BTC_OK);
    EXPECT((fake::log == std::vector<std::string>{"trim1to4096@1", "trim1to0@1"}));
}

// A refused cooperative launch is told apart from an error, and leaves none behind.
static void refused_launch()
{
    SmallBuild b{};
    b.m = 100000;
    b.n = 1000;
    fake::cooperative = cudaErrorCooperativeLaunchTooLarge;
    EXPECT(launch_build_small(b, nullptr) == kNotLaunched);
    EXPECT(fake::last_error == cudaSuccess);
    fake::cooperative = cudaErrorLaunchFailure;
    EXPECT(launch_build_small(b, nullptr) == BTC_E_CUDA);
    fake::cooperative = cudaSuccess;
    EXPECT(launch_build_small(b, nullptr) == BTC_OK);
}

int main(int argc, char** argv)
{
    const std::string name = argc > 1 ? argv[1] : "";
    if (name == "handle_of_another_device") handle_of_another_device();
    else if (name == "buffer_of_another_device") buffer_of_another_device();
    else if (name == "arrays_of_another_device") arrays_of_another_device();
    else if (name == "slots_of_many_threads") slots_of_many_threads();
    else if (name == "slots_across_a_reset") slots_across_a_reset();
    else if (name == "contexts_in_turn") contexts_in_turn();
    else if (name == "opt_ins") opt_ins();
    else if (name == "refused_launch") refused_launch();
    else if (name == "trim") trim();
    else return 2;
    return failures ? 1 : 0;
}
