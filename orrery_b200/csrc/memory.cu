// Device blocks kept from destroyed objects for the next ones.
//
// Device allocations above 1 MB take new memory from the driver, 0.35 ms each
// here, and give it back when freed, 0.3 ms (small ones 1 and 2 us): several times
// the work of a small evaluation, and a program that makes a solver per call
// (compute_accelerations does) pays them every time. Blocks of destroyed objects
// are therefore kept, at most kKeptBytes and kKeptBlocks of them in the process, and
// given back to the device when that is exceeded, when an allocation fails or when
// the caller asks (ob_release_kept_memory).
//
// Nothing here waits: an owner keeps a block once its own streams have finished
// with it, and frees (cudaFree, which waits by itself) what a caller's stream or
// pointer may still use. A wait for the whole device in a destructor would
// invalidate every graph capture under way in other threads.
#include <algorithm>
#include <mutex>
#include <vector>

#include "runtime.hpp"

namespace ob {
namespace {

constexpr size_t kKeptBytes = size_t{256} << 20;
constexpr size_t kKeptBlocks = 256;
// Larger blocks are allocated as they are asked for and freed at once.
constexpr size_t kLargestKept = kKeptBytes / 4;

struct Block {
    void *ptr;
    size_t bytes;
    int device;
};

struct Kept {
    std::mutex mutex;
    std::vector<Block> blocks; // oldest first
    size_t bytes = 0;
};

// Never destroyed: objects may outlive static destruction, and the driver
// reclaims the memory at exit.
Kept &kept() {
    static Kept *k = new Kept;
    return *k;
}

// Frees the blocks of `device` (-1: of every device); cudaFree takes a pointer
// of any device.
void give_back(int device) {
    std::vector<Block> out;
    {
        Kept &k = kept();
        std::lock_guard<std::mutex> lock(k.mutex);
        const auto split = std::stable_partition(
            k.blocks.begin(), k.blocks.end(),
            [device](const Block &b) { return device >= 0 && b.device != device; });
        out.assign(split, k.blocks.end());
        k.blocks.erase(split, k.blocks.end());
        for (const Block &b : out) {
            k.bytes -= b.bytes;
        }
    }
    for (const Block &b : out) {
        cudaFree(b.ptr);
    }
}

} // namespace

void *take_device_block(size_t bytes, size_t &got, int &device) {
    check(cudaGetDevice(&device), "cudaGetDevice");
    // Sizes in steps of an eighth, so that blocks fit the next object of about
    // the same size.
    size_t want = bytes;
    if (bytes <= kLargestKept) {
        size_t step = 512;
        while (step * 8 < bytes) {
            step *= 2;
        }
        want = (bytes + step - 1) / step * step;
        Kept &k = kept();
        std::lock_guard<std::mutex> lock(k.mutex);
        auto best = k.blocks.end();
        for (auto it = k.blocks.begin(); it != k.blocks.end(); ++it) {
            if (it->device == device && it->bytes >= want && it->bytes <= want + want / 2 &&
                (best == k.blocks.end() || it->bytes < best->bytes)) {
                best = it;
            }
        }
        if (best != k.blocks.end()) {
            void *p = best->ptr;
            got = best->bytes;
            k.bytes -= got;
            k.blocks.erase(best);
            return p;
        }
    }
    void *p = nullptr;
    cudaError_t err = cudaMalloc(&p, want);
    if (err == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        give_back(device);
        err = cudaMalloc(&p, want);
    }
    check(err, "device allocation");
    got = want;
    return p;
}

void release_kept_blocks() { give_back(-1); }

void keep_device_block(void *ptr, size_t bytes, int device) noexcept {
    if (bytes > kLargestKept) {
        cudaFree(ptr);
        return;
    }
    std::vector<Block> over;
    try {
        Kept &k = kept();
        std::lock_guard<std::mutex> lock(k.mutex);
        k.blocks.push_back(Block{ptr, bytes, device});
        k.bytes += bytes;
        ptr = nullptr;
        while (k.bytes > kKeptBytes || k.blocks.size() > kKeptBlocks) {
            over.push_back(k.blocks.front());
            k.bytes -= k.blocks.front().bytes;
            k.blocks.erase(k.blocks.begin());
        }
    } catch (...) { // no host memory for the list: give the block back at once
    }
    if (ptr != nullptr) {
        cudaFree(ptr);
    }
    for (const Block &b : over) {
        cudaFree(b.ptr);
    }
}

} // namespace ob
