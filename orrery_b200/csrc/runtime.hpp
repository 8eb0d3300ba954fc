// Host-side runtime pieces shared by the C ABI: errors, device buffers.
#pragma once

#include <atomic>
#include <cstdint>
#include <cstdio>
#include <stdexcept>
#include <string>
#include <utility>

#include <cuda_runtime.h>

#include "orrery_b200.h"

namespace ob {

// An error that crosses no ABI boundary: caught in the extern "C" layer and
// turned into a status code plus ob_last_error() text.
class Error : public std::runtime_error {
public:
    Error(int code, const std::string &message) : std::runtime_error(message), code_(code) {}
    [[nodiscard]] int code() const noexcept { return code_; }

private:
    int code_;
};

inline void check(cudaError_t err, const char *what) {
    if (err != cudaSuccess) {
        const int code = err == cudaErrorMemoryAllocation ? OB_ERROR_OUT_OF_MEMORY : OB_ERROR_CUDA;
        throw Error(code, std::string(what) + ": " + cudaGetErrorName(err) + " (" +
                              cudaGetErrorString(err) + ")");
    }
}

// Raises `kernel`'s dynamic shared-memory limit to `bytes` on the current
// device. The attribute belongs to each device's context, so it is set once
// per device: `configured` is the caller's per-kernel set of devices done
// (bit d for device d; devices from 64 on are set on every call).
inline cudaError_t set_smem_limit_once(const void *kernel, int bytes,
                                       std::atomic<uint64_t> &configured) {
    int device = 0;
    cudaError_t err = cudaGetDevice(&device);
    if (err != cudaSuccess) {
        return err;
    }
    const uint64_t bit = device >= 0 && device < 64 ? (1ull << device) : 0ull;
    if (bit != 0 && (configured.load(std::memory_order_acquire) & bit) != 0) {
        return cudaSuccess;
    }
    err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (err == cudaSuccess && bit != 0) {
        configured.fetch_or(bit, std::memory_order_acq_rel);
    }
    return err;
}

// Sets the calling thread's last-error text and returns `code`.
int set_error(int code, const std::string &message);

// A device block of at least `bytes` on the current device: one kept from a
// destroyed object, or newly allocated (memory.cu). Its contents are undefined.
void *take_device_block(size_t bytes, size_t &got, int &device);
// Keeps a block for the next object (bounded; else frees it). Nothing enqueued
// on the device may still use it.
void keep_device_block(void *ptr, size_t bytes, int device) noexcept;
// Frees every kept block.
void release_kept_blocks();

// Owning device allocation that grows on demand and never shrinks, the
// capacity policy of the reference's CUDA solvers
// (src/solvers/cuda_direct_solver.cpp:120-137).
template <typename T> class DeviceArray {
public:
    DeviceArray() = default;
    DeviceArray(const DeviceArray &) = delete;
    DeviceArray &operator=(const DeviceArray &) = delete;
    DeviceArray(DeviceArray &&o) noexcept { swap(o); }
    DeviceArray &operator=(DeviceArray &&o) noexcept {
        if (this != &o) {
            release();
            swap(o);
        }
        return *this;
    }
    ~DeviceArray() { release(); }

    // Returns true when the storage moved (callers holding the old pointer,
    // such as captured graphs, must refresh).
    bool reserve(size_t count) {
        if (count <= count_) {
            return false;
        }
        release();
        ptr_ = static_cast<T *>(take_device_block(count * sizeof(T), block_bytes_, device_));
        count_ = count;
        return true;
    }
    void release() noexcept {
        if (ptr_ != nullptr) {
            cudaFree(ptr_);
        }
        ptr_ = nullptr;
        count_ = 0;
    }
    // Releases the storage to the next object's use: for owners that know that
    // nothing enqueued on the device may still use it.
    void keep() noexcept {
        if (ptr_ != nullptr) {
            keep_device_block(ptr_, block_bytes_, device_);
        }
        ptr_ = nullptr;
        count_ = 0;
    }
    [[nodiscard]] T *data() const noexcept { return ptr_; }
    [[nodiscard]] size_t size() const noexcept { return count_; }
    [[nodiscard]] size_t bytes() const noexcept { return count_ * sizeof(T); }

private:
    void swap(DeviceArray &o) noexcept {
        std::swap(ptr_, o.ptr_);
        std::swap(count_, o.count_);
        std::swap(block_bytes_, o.block_bytes_);
        std::swap(device_, o.device_);
    }

    T *ptr_ = nullptr;
    size_t count_ = 0;
    size_t block_bytes_ = 0; // of the whole block, which may exceed count_ values
    int device_ = 0;
};

// True once all work enqueued on `stream` has finished.
inline bool finished(cudaStream_t stream) noexcept {
    if (cudaStreamSynchronize(stream) == cudaSuccess) {
        return true;
    }
    cudaGetLastError();
    return false;
}

// Records `event` on `stream`; `external` makes it a real event-record node
// when the stream is being captured into a graph.
inline void record(cudaEvent_t event, cudaStream_t stream, bool external) {
    check(external ? cudaEventRecordWithFlags(event, stream, cudaEventRecordExternal)
                   : cudaEventRecord(event, stream),
          "recording an event");
}

// Device status word of one solver; see common.cuh for the bits.
unsigned read_and_clear_status(unsigned *device_word, cudaStream_t stream);

} // namespace ob
