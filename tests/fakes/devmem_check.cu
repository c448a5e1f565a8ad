// Checks of csrc/devmem.cu and of the handle's release on a host-side CUDA runtime: one check
// per name, exit code 0 when it holds.
#include "cudart.hpp"

#include "handle.cuh"

namespace btc200 {
void note_cuda_error(cudaError_t, const char*, const char*, int) {}
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
    g.h_meta = host_slot_alloc();
    EXPECT(g.indptr.reserve(100) == 0 && g.blocks.reserve(1000) == 0);
    EXPECT(g.policy.dev.reserve(24) == 0);
    g.policy.host = host_slot_alloc();
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

int main(int argc, char** argv)
{
    const std::string name = argc > 1 ? argv[1] : "";
    if (name == "handle_of_another_device") handle_of_another_device();
    else if (name == "buffer_of_another_device") buffer_of_another_device();
    else if (name == "arrays_of_another_device") arrays_of_another_device();
    else return 2;
    return failures ? 1 : 0;
}
