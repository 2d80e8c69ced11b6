// Host runtime pieces (csrc/runtime.hpp) against a fake CUDA runtime in which calls can be made to fail: device memory
// is host memory, copies happen at once. Usage: runtime_kat <case>; prints what is wrong and exits with 1, or exits with 0.
#include <dlfcn.h>
#include <pthread.h>

#include <cstdio>
#include <cstdlib>
#include <string>

#include "runtime.hpp"

namespace
{
    std::string g_failing;         // name of the call that fails
    std::atomic<int> g_before{0};  // how many of these calls succeed first
    std::atomic<int> g_streamCopies{0}, g_laneCopies{0}, g_memsets{0};
    thread_local cudaError_t t_last = cudaSuccess;
    int g_wrong = 0;
    const cudaStream_t kCallersStream = reinterpret_cast<cudaStream_t>(1);

    bool fails(const char* name) { return g_failing == name && g_before.fetch_sub(1) <= 0; }
    cudaError_t result(const char* name, cudaError_t e)
    {
        if (!fails(name)) return cudaSuccess;
        t_last = e;
        return e;
    }
    void expect(bool ok, const char* what)
    {
        if (ok) return;
        std::printf("wrong: %s\n", what);
        g_wrong++;
    }
}

extern "C"
{
    cudaError_t cudaGetLastError() { return std::exchange(t_last, cudaSuccess); }
    const char* cudaGetErrorName(cudaError_t) { return "cudaErrorFake"; }
    const char* cudaGetErrorString(cudaError_t) { return "made to fail"; }
    cudaError_t cudaSetDevice(int) { return cudaSuccess; }
    cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
    cudaError_t cudaMalloc(void** p, size_t n) { return *p = std::malloc(n), cudaSuccess; }
    cudaError_t cudaFree(void* p) { return std::free(p), cudaSuccess; }
    cudaError_t cudaHostAlloc(void** p, size_t n, unsigned)
    {
        const cudaError_t e = result("cudaHostAlloc", cudaErrorMemoryAllocation);
        if (e == cudaSuccess) *p = std::malloc(n);
        return e;
    }
    cudaError_t cudaFreeHost(void* p) { return std::free(p), cudaSuccess; }
    cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned)
    {
        const cudaError_t e = result("cudaStreamCreateWithFlags", cudaErrorMemoryAllocation);
        if (e == cudaSuccess) *s = reinterpret_cast<cudaStream_t>(2);
        return e;
    }
    cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
    cudaError_t cudaStreamSynchronize(cudaStream_t) { return result("cudaStreamSynchronize", cudaErrorStreamCaptureUnsupported); }
    cudaError_t cudaMemsetAsync(void* p, int value, size_t n, cudaStream_t)
    {
        g_memsets++;
        std::memset(p, value, n);
        return cudaSuccess;
    }
    cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned)
    {
        const cudaError_t r = result("cudaEventCreateWithFlags", cudaErrorMemoryAllocation);
        if (r == cudaSuccess) *e = reinterpret_cast<cudaEvent_t>(3);
        return r;
    }
    cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
    cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
    cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
    cudaError_t cudaMemcpyAsync(void* to, const void* from, size_t n, cudaMemcpyKind, cudaStream_t s)
    {
        (s == kCallersStream ? g_streamCopies : g_laneCopies)++;
        const cudaError_t e = result("cudaMemcpyAsync", cudaErrorInvalidValue);
        if (e == cudaSuccess) std::memcpy(to, from, n);
        return e;
    }
    int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* x)
    {
        if (fails("pthread_create")) return EAGAIN;
        using Create = int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
        static const Create real = reinterpret_cast<Create>(dlsym(RTLD_NEXT, "pthread_create"));
        return real(t, a, f, x);
    }
}

namespace pt
{
    bool InjectedAllocationFailure() { return false; }
}

namespace
{
    std::vector<char> bytes(size_t n, unsigned seed)
    {
        std::vector<char> v(n);
        for (size_t i = 0; i < n; i++) v[i] = static_cast<char>((i * 2654435761u + seed) >> 13);
        return v;
    }

    // Arrays of an upload that is large enough for pinned memory, with sizes around those of its 512 KB chunks.
    void upload(pt::PinnedUpload& through, unsigned seed)
    {
        const std::vector<char> a = bytes((33u << 20) + 1u, seed), b = bytes(512u << 10, seed + 1u), c = bytes(7, seed + 2u);
        std::vector<char> da(a.size()), db(b.size()), dc(c.size());
        pt::PinnedUpload::Job job;
        const pt::Status started = through.start(job, {{da.data(), a.data(), a.size()}, {db.data(), b.data(), b.size()}, {dc.data(), c.data(), c.size()}},
                                                 kCallersStream);
        const pt::Status done = job.wait();
        expect(started.ok() && done.ok(), "the upload reports success");
        expect(da == a && db == b && dc == c, "the arrays arrive");
        expect(cudaGetLastError() == cudaSuccess, "no error is left for the next launch");
    }

    // `call` fails from its (before + 1)-th time on.
    void upload_without(const char* call, int before, bool copiedByCaller)
    {
        g_failing = call;
        g_before = before;
        pt::PinnedUpload through;
        upload(through, 1u);
        expect((g_streamCopies > 0) == copiedByCaller, "the expected copies");
        g_failing.clear();  // and with everything working again
        g_streamCopies = 0;
        upload(through, 2u);
        expect(g_streamCopies == 0 && g_laneCopies > 0, "pinned copies once they can be had");
    }

    // A batch that took `rays` rays; it leaves its state clear unless its last launch was not made.
    pt::Status batch(pt::BatchStates& states, uint32_t rays, cudaError_t launched)
    {
        pt::BatchStates::Call call(states);
        const pt::Status begun = call.begin(kCallersStream);
        if (!begun.ok()) return begun;
        pt::BatchState* s = call.state();
        expect(s->cursor == 0 && s->errors == 0 && s->left == 0, "a batch starts from a clear state");
        s->cursor = rays;
        if (launched == cudaSuccess) *s = pt::BatchState{};
        return call.end(launched, kCallersStream);
    }

    void batches(cudaError_t launched, const char* failing)
    {
        uint32_t errors[pt::BatchStates::kCount] = {};
        pt::BatchStates states;
        expect(states.create(errors, errors, kCallersStream).ok(), "the states");
        g_memsets = 0;
        for (uint32_t k = 0; k < 3; k++) expect(batch(states, 100u, cudaSuccess).ok(), "a batch");
        expect(g_memsets == 0, "batches that ended well are not cleared again");
        g_failing = failing;
        expect(!batch(states, 100u, launched).ok(), "the failure is reported");
        expect(cudaGetLastError() == cudaSuccess, "no error is left for the next launch");
        g_failing.clear();
        for (uint32_t k = 0; k < 3; k++) expect(batch(states, 100u, cudaSuccess).ok(), "a batch behind the failure");
        expect(g_memsets == 1, "cleared once");
        // as many failures as there are states use none of them up
        for (uint32_t k = 0; k < 2 * pt::BatchStates::kCount; k++) expect(!batch(states, 7u, cudaErrorLaunchOutOfResources).ok(), "the failure is reported");
        expect(batch(states, 100u, cudaSuccess).ok(), "a batch behind many failures");
    }

    // Callers on more threads than there are states: each has a state to itself.
    void batches_of_threads()
    {
        uint32_t errors[pt::BatchStates::kCount] = {};
        pt::BatchStates states;
        expect(states.create(errors, errors, kCallersStream).ok(), "the states");
        std::vector<std::thread> callers;
        for (uint32_t t = 0; t < 2 * pt::BatchStates::kCount; t++)
            callers.emplace_back([&states, t] { for (uint32_t k = 0; k < 200; k++) batch(states, t + 1u, k % 5 ? cudaSuccess : cudaErrorLaunchOutOfResources); });
        for (std::thread& t : callers) t.join();
    }
}

int main(int argc, char** argv)
{
    const std::string name = argc > 1 ? argv[1] : "";
    if (name == "upload")
        upload_without("", 0, false);
    else if (name == "upload without pinned memory")
        upload_without("cudaHostAlloc", 0, true);
    else if (name == "upload without streams")
        upload_without("cudaStreamCreateWithFlags", 0, true);
    else if (name == "upload without the last stream")
        upload_without("cudaStreamCreateWithFlags", 3, true);
    else if (name == "upload without events")
        upload_without("cudaEventCreateWithFlags", 5, true);
    else if (name == "upload without threads")
        upload_without("pthread_create", 0, false);
    else if (name == "upload with two threads")
        upload_without("pthread_create", 2, false);
    else if (name == "upload that fails")
    {
        g_failing = "cudaMemcpyAsync";
        g_before = 9;
        pt::PinnedUpload through;
        const std::vector<char> a = bytes(40u << 20, 1u);
        std::vector<char> to(a.size());
        pt::PinnedUpload::Job job;
        expect(through.start(job, {{to.data(), a.data(), a.size()}}, kCallersStream).ok(), "the upload starts");
        expect(!job.wait().ok(), "its end reports the failure");
        g_failing.clear();
        upload(through, 2u);
    }
    else if (name == "a batch whose second launch fails")
        batches(cudaErrorLaunchOutOfResources, "");
    else if (name == "a batch that cannot be waited for")
        batches(cudaSuccess, "cudaStreamSynchronize");
    else if (name == "batches of many threads")
        batches_of_threads();
    else if (name == "two uploads at once")
    {
        pt::PinnedUpload through;
        std::vector<std::thread> callers;
        for (unsigned t = 0; t < 2; t++)
            callers.emplace_back([&through, t] { for (unsigned k = 0; k < 3; k++) upload(through, 10u * t + k); });
        for (std::thread& t : callers) t.join();
    }
    else
        expect(false, "a case of this name");
    return g_wrong ? 1 : 0;
}
