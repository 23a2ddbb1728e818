// fwi_stage.cu -- see fwi_stage.h
#include "fwi_stage.h"

#include <algorithm>
#include <condition_variable>
#include <cstring>
#include <deque>
#include <memory>
#include <mutex>
#include <thread>

namespace fwi {
namespace {

constexpr size_t PIECE = (size_t)1 << 20;      // bytes of a piece and of a page-locked buffer
constexpr size_t THRESHOLD = (size_t)24 << 20;  // smaller jobs are not worth waking the threads (fwi_stage.h)
constexpr int MOST_THREADS = 4;

struct Job {
    std::vector<HostCopy> pieces;
    bool to_device = true;
    int device = 0;
    cudaStream_t st = nullptr;
    size_t next = 0, done = 0;  // under the pool's mutex
    cudaError_t err = cudaSuccess;
};

class Pool {
public:
    Pool()
    {
        const int n = std::min<int>(MOST_THREADS, std::max<int>(1, (int)std::thread::hardware_concurrency() / 2));
        try {
            for (int i = 0; i < n; i++) threads_.emplace_back([this] { work(); });
        } catch (...) {  // the threads that started are enough; none: the caller copies
        }
    }
    ~Pool()
    {
        {
            std::lock_guard<std::mutex> lk(mu_);
            stop_ = true;
        }
        cv_.notify_all();
        for (auto &t : threads_) t.join();
    }
    bool usable() const { return !threads_.empty(); }

    // every piece handed to the device (or arrived on the host) when it returns
    cudaError_t run(const std::shared_ptr<Job> &j)
    {
        std::unique_lock<std::mutex> lk(mu_);
        jobs_.push_back(j);
        cv_.notify_all();
        done_.wait(lk, [&] { return j->done == j->pieces.size(); });
        return j->err;
    }

private:
    struct Buffer {
        void *p = nullptr;
        cudaEvent_t ev = nullptr;
        int device = -1;
        bool used = false;
    };
    // a piece whose device copy is under way into a buffer (to the host)
    struct Pending {
        std::shared_ptr<Job> j;
        size_t i = 0;
    };

    static cudaError_t ready(Buffer &b, int device)
    {
        cudaError_t e = cudaSetDevice(device);
        if (e == cudaSuccess && !b.p) e = cudaHostAlloc(&b.p, PIECE, cudaHostAllocPortable);
        if (e == cudaSuccess && b.used) e = cudaEventSynchronize(b.ev);
        b.used = false;
        if (e == cudaSuccess && b.device != device) {
            if (b.ev) cudaEventDestroy(b.ev);
            b.ev = nullptr;
            e = cudaEventCreateWithFlags(&b.ev, cudaEventDisableTiming);
            b.device = e == cudaSuccess ? device : -1;
        }
        return e;
    }
    void finish(const std::shared_ptr<Job> &j, cudaError_t e)
    {
        std::lock_guard<std::mutex> lk(mu_);
        if (e != cudaSuccess && j->err == cudaSuccess) j->err = e;
        if (++j->done == j->pieces.size()) done_.notify_all();
    }
    void arrive(Buffer &b, Pending &p)
    {
        if (!p.j) return;
        const HostCopy &c = p.j->pieces[p.i];
        const cudaError_t e = cudaEventSynchronize(b.ev);
        b.used = false;
        if (e == cudaSuccess) memcpy(c.dst, b.p, c.bytes);
        finish(p.j, e);
        p.j.reset();
    }
    void work()
    {
        Buffer buf[2];
        Pending pend[2];
        int k = 0;
        for (;;) {
            std::shared_ptr<Job> j;
            size_t i = 0;
            {
                std::unique_lock<std::mutex> lk(mu_);
                while (!jobs_.empty() && jobs_.front()->next == jobs_.front()->pieces.size()) jobs_.pop_front();
                if (jobs_.empty() && !pend[0].j && !pend[1].j) {
                    cv_.wait(lk, [&] { return stop_ || !jobs_.empty(); });
                    if (stop_) break;
                    continue;
                }
                if (!jobs_.empty()) {
                    j = jobs_.front();
                    i = j->next++;
                }
            }
            if (!j) {  // nothing new: let what is under way arrive, oldest first
                arrive(buf[k], pend[k]);
                arrive(buf[k ^ 1], pend[k ^ 1]);
                continue;
            }
            Buffer &b = buf[k];
            arrive(b, pend[k]);
            const HostCopy &c = j->pieces[i];
            cudaError_t e = ready(b, j->device);
            if (e == cudaSuccess && j->to_device) memcpy(b.p, c.src, c.bytes);
            if (e == cudaSuccess)
                e = j->to_device ? cudaMemcpyAsync(c.dst, b.p, c.bytes, cudaMemcpyHostToDevice, j->st)
                                 : cudaMemcpyAsync(b.p, c.src, c.bytes, cudaMemcpyDeviceToHost, j->st);
            if (e == cudaSuccess) e = cudaEventRecord(b.ev, j->st);
            b.used = e == cudaSuccess;
            if (e == cudaSuccess && !j->to_device) pend[k] = {j, i};
            else finish(j, e);
            k ^= 1;
        }
        for (Buffer &b : buf) {
            if (b.used) cudaEventSynchronize(b.ev);
            if (b.ev) cudaEventDestroy(b.ev);
            if (b.p) cudaFreeHost(b.p);
        }
    }

    std::mutex mu_;
    std::condition_variable cv_, done_;
    std::deque<std::shared_ptr<Job>> jobs_;
    bool stop_ = false;
    std::vector<std::thread> threads_;
};

Pool *pool()
{
    static Pool p;
    return p.usable() ? &p : nullptr;
}

bool pinned(const void *p)
{
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type != cudaMemoryTypeUnregistered;
}

cudaError_t stage(const std::vector<HostCopy> &copies, cudaStream_t st, bool to_device)
{
    const cudaMemcpyKind kind = to_device ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost;
    std::vector<HostCopy> direct = copies;
    cudaError_t e = cudaSuccess;
    try {
        size_t total = 0;
        auto j = std::make_shared<Job>();
        direct.clear();
        for (const HostCopy &c : copies) {
            if (pinned(to_device ? c.src : c.dst)) {
                direct.push_back(c);
                continue;
            }
            total += c.bytes;
            for (size_t o = 0; o < c.bytes; o += PIECE)
                j->pieces.push_back({(char *)c.dst + o, (const char *)c.src + o, std::min(PIECE, c.bytes - o)});
        }
        Pool *p = total >= THRESHOLD ? pool() : nullptr;
        if (p) {
            j->to_device = to_device;
            j->st = st;
            e = cudaGetDevice(&j->device);
            // The threads serve every caller in turn, so the caller waits here for what its stream still
            // holds: a thread then only ever waits for copies of its own, not for another caller's run.
            if (e == cudaSuccess) e = cudaStreamSynchronize(st);
            if (e == cudaSuccess) e = p->run(j);
        } else {
            direct = copies;
        }
    } catch (...) {  // no memory for the pieces: the plain copies
        direct = copies;
    }
    for (const HostCopy &c : direct)
        if (e == cudaSuccess) e = cudaMemcpyAsync(c.dst, c.src, c.bytes, kind, st);
    return e;
}

}  // namespace

cudaError_t stage_to_device(const std::vector<HostCopy> &copies, cudaStream_t st) { return stage(copies, st, true); }

cudaError_t stage_to_host(const std::vector<HostCopy> &copies, cudaStream_t st)
{
    const cudaError_t e = stage(copies, st, false);
    return e == cudaSuccess ? cudaStreamSynchronize(st) : e;
}

}  // namespace fwi
