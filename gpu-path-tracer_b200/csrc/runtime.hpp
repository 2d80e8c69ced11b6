// Host runtime pieces shared by the frame renderer (renderer.cu) and the job engine (engine.cu):
// status values, RAII device buffers, texture objects and device-resident scenes.
#pragma once
#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>

#include <atomic>
#include <condition_variable>
#include <cstdint>
#include <cstring>
#include <memory>
#include <mutex>
#include <string>
#include <thread>
#include <utility>
#include <vector>

#include "../../include/gpt_b200.h"
#include "kernels.h"
#include "pt_internal.h"

namespace pt
{
    struct Status
    {
        int code = GPT_OK;
        std::string message;
        static Status Ok() { return {}; }
        static Status Err(int c, std::string m) { return Status{c, std::move(m)}; }
        bool ok() const { return code == GPT_OK; }
    };

    inline Status CudaStatus(const char* op, cudaError_t e)
    {
        if (e == cudaSuccess) return Status::Ok();
        cudaGetLastError();  // reported here; left as the thread's last error, the next launch would report it as its own
        // Error text format of the reference (Cuda/Utils/Error.cpp:22-25).
        std::string msg = std::string(op) + " failed: " + cudaGetErrorName(e) + ": " + cudaGetErrorString(e);
        return Status::Err(e == cudaErrorMemoryAllocation ? GPT_ERR_OUT_OF_MEMORY : GPT_ERR_CUDA, msg);
    }

#define PT_TRY(expr)                      \
    do                                    \
    {                                     \
        Status _s = (expr);               \
        if (!_s.ok()) return _s;          \
    } while (0)
#define PT_CUDA(op, expr) PT_TRY(CudaStatus(op, (expr)))

    // A named host range on the calling thread's NVTX stack (scene upload and its stages, frames,
    // the autotuner, job-server slices), so a profiler's timeline shows which host step issued the
    // kernels under it (ncu: --nvtx --nvtx-include "gpt render frame/"). NVTX is header-only: with
    // no tool attached a push or pop is one predictable branch. end() closes the range early; the
    // destructor closes it on every return path otherwise.
    class NvtxRange
    {
    public:
        explicit NvtxRange(const char* name) { nvtxRangePushA(name); }
        ~NvtxRange() { end(); }
        NvtxRange(const NvtxRange&) = delete;
        NvtxRange& operator=(const NvtxRange&) = delete;
        void end()
        {
            if (open_) nvtxRangePop();
            open_ = false;
        }

    private:
        bool open_ = true;
    };

    // True when this device allocation is the one gpt_inject_allocation_failure chose to fail.
    bool InjectedAllocationFailure();

    // RAII device allocation (the reference's DeviceBuffer1D, Runtime/Memory/DeviceBuffer1D.cpp:33-80).
    class DeviceBuffer
    {
    public:
        DeviceBuffer() = default;
        DeviceBuffer(const DeviceBuffer&) = delete;
        DeviceBuffer& operator=(const DeviceBuffer&) = delete;
        ~DeviceBuffer() { reset(); }
        // Grows the buffer to at least `bytes` (contents are not kept). The new allocation is made before
        // the old one is freed, so a failed call leaves the buffer as it was.
        Status allocate(size_t bytes)
        {
            if (bytes <= bytes_ && ptr_) return Status::Ok();
            if (bytes == 0) return Status::Ok();
            if (InjectedAllocationFailure())
                return Status::Err(GPT_ERR_OUT_OF_MEMORY, "cudaMalloc failed: out of memory (injected by gpt_inject_allocation_failure)");
            void* fresh = nullptr;
            PT_CUDA("cudaMalloc", cudaMalloc(&fresh, bytes));
            reset();
            ptr_ = fresh;
            bytes_ = bytes;
            return Status::Ok();
        }
        void reset()
        {
            if (ptr_) cudaFree(ptr_);
            ptr_ = nullptr;
            bytes_ = 0;
        }
        void swap(DeviceBuffer& other)
        {
            std::swap(ptr_, other.ptr_);
            std::swap(bytes_, other.bytes_);
        }
        template <typename T>
        T* get() const { return static_cast<T*>(ptr_); }
        size_t bytes() const { return bytes_; }

    private:
        void* ptr_ = nullptr;
        size_t bytes_ = 0;
    };

    // Several device arrays in one allocation: add() every array, then allocate(). A cudaMalloc and a cudaFree
    // cost 0.1 to 0.3 ms each, whatever their size, and the free waits for the device.
    class DeviceArena
    {
    public:
        template <typename T>
        void add(T*& array, size_t count)
        {
            parts_.push_back({reinterpret_cast<void**>(&array), bytes_});
            bytes_ += (count * sizeof(T) + 255) / 256 * 256;
        }
        Status allocate()
        {
            PT_TRY(buffer_.allocate(bytes_));
            for (const Part& p : parts_) *p.array = buffer_.get<char>() + p.offset;
            return Status::Ok();
        }

    private:
        struct Part
        {
            void** array;
            size_t offset;
        };
        DeviceBuffer buffer_;
        std::vector<Part> parts_;
        size_t bytes_ = 0;
    };

    // Uploads of large pageable arrays through pinned memory by several threads. One cudaMemcpyAsync of pageable
    // memory moves 11 GB/s and blocks its caller, and several at once are not faster; four threads that copy
    // into pinned chunks and send those move 25 to 35 GB/s (200 MB: 5.5 to 9 ms instead of 18.5) while the
    // caller works on. The 8 MB of pinned memory, the streams and the events live as long as the object (a
    // renderer's or a server's). Pinning takes about 1 ms per MB, so it waits for an upload that pays for it.
    class PinnedUpload
    {
    public:
        struct Item
        {
            void* device;
            const void* host;
            size_t bytes;
        };

        PinnedUpload() = default;
        PinnedUpload(const PinnedUpload&) = delete;
        PinnedUpload& operator=(const PinnedUpload&) = delete;
        ~PinnedUpload()
        {
            for (Lane& l : lanes_)
            {
                for (cudaEvent_t e : l.sent)
                    if (e) cudaEventDestroy(e);
                if (l.stream) cudaStreamDestroy(l.stream);
            }
            if (pinned_) cudaFreeHost(pinned_);
        }

        // A running upload; wait() (or the destructor) ends it, and everything is on the device then.
        class Job
        {
        public:
            Job() = default;
            Job(const Job&) = delete;
            Job& operator=(const Job&) = delete;
            ~Job() { wait(); }
            Status wait()
            {
                for (std::thread& t : threads_) t.join();
                threads_.clear();
                if (lock_.owns_lock()) lock_.unlock();
                const cudaError_t e = static_cast<cudaError_t>(error_.exchange(cudaSuccess));
                return CudaStatus("cudaMemcpyAsync", e);
            }

        private:
            friend class PinnedUpload;
            std::vector<Item> items_;
            std::vector<std::thread> threads_;
            std::unique_lock<std::mutex> lock_;
            std::atomic<size_t> next_{0};
            std::atomic<int> error_{cudaSuccess};
        };

        // Starts copying the items (to the current device). Small uploads, and ones without pinned memory or
        // threads, are copied on `stream` by the caller.
        Status start(Job& job, std::vector<Item> items, cudaStream_t stream)
        {
            size_t bytes = 0;
            for (const Item& i : items) bytes += i.bytes;
            int device = 0;
            PT_CUDA("cudaGetDevice", cudaGetDevice(&device));
            if (bytes >= (ready_ ? kSmallest : kSmallestFirst))
            {
                job.lock_ = std::unique_lock<std::mutex>(mutex_);
                if (!prepare())
                    cudaGetLastError();  // copied without it; a later launch must not report this error as its own
                else
                {
                    job.items_ = std::move(items);
                    job.next_ = 0;
                    try
                    {
                        for (Lane& l : lanes_) job.threads_.emplace_back([&job, &l, device] { send(job, l, device); });
                    }
                    catch (const std::exception&)
                    {
                        if (job.threads_.empty()) send(job, lanes_[0], device);
                    }
                    return Status::Ok();
                }
                job.lock_.unlock();
            }
            for (const Item& i : items) PT_CUDA("cudaMemcpyAsync", cudaMemcpyAsync(i.device, i.host, i.bytes, cudaMemcpyHostToDevice, stream));
            return Status::Ok();
        }

    private:
        static constexpr size_t kSmallest = 4u << 20, kSmallestFirst = 32u << 20, kChunk = 512u << 10;
        static constexpr int kLanes = 4, kSlots = 4;
        struct Lane
        {
            cudaStream_t stream = nullptr;
            cudaEvent_t sent[kSlots] = {};
            char* slots = nullptr;
        };

        bool prepare()
        {
            if (ready_) return true;
            if (!pinned_ && cudaHostAlloc(&pinned_, kLanes * kSlots * kChunk, cudaHostAllocPortable) != cudaSuccess)
            {
                pinned_ = nullptr;
                return false;
            }
            for (int k = 0; k < kLanes; k++)
            {
                Lane& l = lanes_[k];
                l.slots = static_cast<char*>(pinned_) + static_cast<size_t>(k) * kSlots * kChunk;
                if (!l.stream && cudaStreamCreateWithFlags(&l.stream, cudaStreamNonBlocking) != cudaSuccess) return false;
                for (cudaEvent_t& e : l.sent)
                    if (!e && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) return false;
            }
            ready_ = true;
            return true;
        }

        // One thread: takes chunks of the items (numbered through) until none is left, through its slots in turn.
        static void send(Job& job, Lane& lane, int device)
        {
            cudaError_t e = cudaSetDevice(device);
            for (int slot = 0; e == cudaSuccess; slot = (slot + 1) % kSlots)
            {
                size_t chunk = job.next_.fetch_add(1);
                size_t i = 0;
                for (; i < job.items_.size(); i++)
                {
                    const size_t chunks = (job.items_[i].bytes + kChunk - 1) / kChunk;
                    if (chunk < chunks) break;
                    chunk -= chunks;
                }
                if (i == job.items_.size()) break;
                const Item& item = job.items_[i];
                const size_t at = chunk * kChunk, bytes = item.bytes - at < kChunk ? item.bytes - at : kChunk;
                char* pinned = lane.slots + static_cast<size_t>(slot) * kChunk;
                e = cudaEventSynchronize(lane.sent[slot]);  // (an event not recorded yet is done)
                if (e != cudaSuccess) break;
                std::memcpy(pinned, static_cast<const char*>(item.host) + at, bytes);
                e = cudaMemcpyAsync(static_cast<char*>(item.device) + at, pinned, bytes, cudaMemcpyHostToDevice, lane.stream);
                if (e == cudaSuccess) e = cudaEventRecord(lane.sent[slot], lane.stream);
            }
            const cudaError_t done = cudaStreamSynchronize(lane.stream);
            if (e == cudaSuccess) e = done;
            if (e != cudaSuccess) job.error_.store(e);
        }

        std::mutex mutex_;
        void* pinned_ = nullptr;
        Lane lanes_[kLanes];
        std::atomic<bool> ready_{false};
    };

    // The states of a renderer's ray batches, one for each call in flight: callers on several threads get different ones,
    // and a call beyond kCount waits for one of them. A batch's last block leaves its state all zero. A call that failed
    // between its launches may have left something in it, so a state whose last call did not end well is cleared before
    // the next one's launch.
    class BatchStates
    {
    public:
        static constexpr uint32_t kCount = 16;

        // errors, errorsDevice: a host-mapped word per state.
        Status create(volatile uint32_t* errors, uint32_t* errorsDevice, cudaStream_t stream)
        {
            errors_ = errors;
            errorsDevice_ = errorsDevice;
            PT_TRY(states_.allocate(kCount * sizeof(BatchState)));
            PT_CUDA("cudaMemsetAsync", cudaMemsetAsync(states_.get<void>(), 0, kCount * sizeof(BatchState), stream));
            PT_CUDA("cudaStreamSynchronize", cudaStreamSynchronize(stream));
            return Status::Ok();
        }

        // One call: begin(), the launches, end().
        class Call
        {
        public:
            explicit Call(BatchStates& all) : all_(all)
            {
                std::unique_lock lock(all_.mutex_);
                all_.freed_.wait(lock, [&] { return all_.free_ != 0; });
                index_ = static_cast<uint32_t>(__builtin_ctz(all_.free_));
                all_.free_ &= all_.free_ - 1u;
            }
            ~Call()
            {
                {
                    std::scoped_lock lock(all_.mutex_);
                    all_.free_ |= 1u << index_;
                }
                all_.freed_.notify_one();
            }
            Call(const Call&) = delete;
            Call& operator=(const Call&) = delete;

            BatchState* state() const { return all_.states_.get<BatchState>() + index_; }
            uint32_t* errorsDevice() const { return all_.errorsDevice_ + index_; }

            Status begin(cudaStream_t stream)
            {
                all_.errors_[index_] = 0u;
                if (all_.unclean_[index_]) PT_CUDA("cudaMemsetAsync", cudaMemsetAsync(state(), 0, sizeof(BatchState), stream));
                all_.unclean_[index_] = true;
                return Status::Ok();
            }
            // Waits for what was launched, whether or not all of it was.
            Status end(cudaError_t launched, cudaStream_t stream)
            {
                const cudaError_t done = cudaStreamSynchronize(stream);
                PT_CUDA("intersect", launched);
                PT_CUDA("cudaStreamSynchronize", done);
                all_.unclean_[index_] = false;
                const uint32_t errors = all_.errors_[index_];
                if (errors) return Status::Err(GPT_ERR_DEVICE_FAULT, "Traversal reported error flags " + std::to_string(errors));
                return Status::Ok();
            }

        private:
            BatchStates& all_;
            uint32_t index_;
        };

    private:
        DeviceBuffer states_;
        volatile uint32_t* errors_ = nullptr;
        uint32_t* errorsDevice_ = nullptr;
        std::mutex mutex_;
        std::condition_variable freed_;
        uint32_t free_ = (1u << kCount) - 1u;
        bool unclean_[kCount] = {};  // (only the call that holds a state touches its entry)
    };

    // An image texture with the reference's descriptors (Texture.cpp:65-189).
    struct TextureObject
    {
        cudaArray_t array = nullptr;
        cudaTextureObject_t object = 0;
        TextureObject() = default;
        TextureObject(const TextureObject&) = delete;
        TextureObject& operator=(const TextureObject&) = delete;
        ~TextureObject()
        {
            if (object) cudaDestroyTextureObject(object);
            if (array) cudaFreeArray(array);
        }
    };

    struct SceneGpu
    {
        DeviceBuffer blocks, blockMasks, shading, materials, lights, bins, binsPower, materialTextures, entry, nodes2;
        std::vector<std::unique_ptr<TextureObject>> textures;
        uint32_t nodeCount = 0, blockCount = 0, triangleCount = 0, depth = 0, lightCount = 0, materialCount = 0;
        uint32_t nodeCount2 = 0, depth2 = 0;  // binary FP32 BVH, built when the scene is uploaded with it
        bool modelPresent[kModelCount] = {};
        uint64_t version = 0;
        double bvhSeconds = 0.0, uploadSeconds = 0.0;  // BVH build (host or device); whole upload (wall clock)
        bool deviceBvh = false;                         // the BVH8 was built on the device
        SceneView view() const
        {
            SceneView v{};
            v.records = blocks.get<Record8>();
            v.shading = shading.get<float4>();
            v.materials = materials.get<MaterialDev>();
            v.textures = textures.empty() ? nullptr : materialTextures.get<MaterialTextures>();
            v.lights = lights.get<float4>();
            v.bins = bins.get<uint4>();
            v.binsPower = binsPower.get<uint4>();
            v.lightCount = lightCount;
            v.triangleCount = triangleCount;
            v.depth = depth;
            v.nodes2 = nodeCount2 ? nodes2.get<Node2>() : nullptr;
            v.depth2 = depth2;
            return v;
        }
    };

    // Minimal PNG writer (zlib deflate) for SaveRenderedFrame (Renderer.cpp:649-675): RGBA8, rows
    // flipped vertically like Import::FlipVertically.
    // Validates a scene description and builds its device copy: image textures, BVH8, shading records,
    // light list and alias table. The BVH8 is built on the host (binned SAH), with `withBinary` also the
    // binary FP32 BVH, or with `deviceBvh` on the device (clustering; no binary BVH). The vertex arrays go
    // through `upload`, the attributes while the BVH is built.
    Status BuildScene(const gpt_scene_desc& d, cudaStream_t stream, PinnedUpload& upload, std::unique_ptr<SceneGpu>& out, bool withBinary = false,
                      bool deviceBvh = false);
}
