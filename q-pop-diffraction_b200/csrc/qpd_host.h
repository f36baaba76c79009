// Host side of qpd_run_host: worker threads that pack the reference's float64 host arrays into the
// kernel input layout, so only the packed bytes cross PCIe.
//
// The reference hands diffraction() float64 planes (src/python/diffraction.py:62-74): 8 bytes per
// value, 72 bytes per cell with two phases and a region.  The kernels read P and u in the plan
// precision, an int8 phase index and one weight per cell: 29 bytes per cell in float32.  Packing on
// the host, chunk by chunk into a pinned ring while earlier chunks are copied, moves 2.5x fewer
// bytes over the link.  The arithmetic is the GPU pack kernel's (pack_kernel): every packed value
// is bit-identical to what qpd_pack_device would write.
#pragma once

#include <atomic>
#include <condition_variable>
#include <cstdint>
#include <functional>
#include <memory>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

namespace qpd {

// A fixed set of threads running one parallel-for at a time.
//
// Every job is an object of its own, with its own indices and its own count of unfinished ones: a worker that is late
// out of one job still holds that job, whose indices are used up, and cannot take or count an index of the next.
class Workers {
   public:
    // n threads, or as many of them as the system gives: the calling thread takes the rest of every job
    explicit Workers(int n) {
        th_.reserve(n > 0 ? n : 0);
        try {
            for (int i = 0; i < n; i++) th_.emplace_back([this] { loop(); });
        } catch (const std::system_error&) {
        }
    }
    ~Workers() {
        {
            std::lock_guard<std::mutex> g(m_);
            stop_ = true;
        }
        cv_.notify_all();
        for (auto& t : th_) t.join();
    }
    int size() const { return (int)th_.size(); }

    // f(i) for i in [0, count), spread over the workers and the calling thread; returns when done.
    void parallel(int count, const std::function<void(int)>& f) {
        if (count <= 0) return;
        const auto job = std::make_shared<Job>(f, count);
        {
            std::lock_guard<std::mutex> g(m_);
            job_ = job;
        }
        cv_.notify_all();
        work(*job);
        std::unique_lock<std::mutex> g(m_);
        done_.wait(g, [&] { return job->left.load() == 0; });
        job_.reset();
    }

   private:
    struct Job {
        const std::function<void(int)>& f;  // alive while left > 0: called for indices below count only
        const int count;
        std::atomic<int> next{0}, left;
        Job(const std::function<void(int)>& fn, int n) : f(fn), count(n), left(n) {}
    };
    void work(Job& job) {
        for (;;) {
            const int i = job.next.fetch_add(1);
            if (i >= job.count) return;
            job.f(i);
            if (job.left.fetch_sub(1) == 1) {
                std::lock_guard<std::mutex> g(m_);  // the caller is waiting, or has yet to look at `left`
                done_.notify_all();
            }
        }
    }
    void loop() {
        std::shared_ptr<Job> job;  // the last one worked on, kept so that its address is not used again meanwhile
        for (;;) {
            {
                std::unique_lock<std::mutex> g(m_);
                cv_.wait(g, [&] { return stop_ || (job_ && job_ != job); });
                if (stop_) return;
                job = job_;
            }
            work(*job);
        }
    }
    std::vector<std::thread> th_;
    std::mutex m_;
    std::condition_variable cv_, done_;
    std::shared_ptr<Job> job_;  // the job that workers join (under m_)
    bool stop_ = false;
};

// Planes of one packed chunk in a pinned slot: P[3], U[3], weight, then either the phase index
// (single mode) or nPhase dense weight planes (dense mode) in the space after the weight.
template <typename T> struct HostChunk {
    T* P;
    T* U;
    T* W;
    int8_t* ph;
    T* WD;       // nPhase planes, dense mode only
    int64_t cap;  // cells per plane
    static size_t bytes(int64_t cap, int nPhase, bool dense) {
        return (sizeof(T) * 7 + 1) * (size_t)cap + (dense ? sizeof(T) * nPhase * (size_t)cap : 0) + 64;
    }
    static HostChunk at(void* base, int64_t cap) {
        HostChunk h;
        h.cap = cap;
        h.P = static_cast<T*>(base);
        h.U = h.P + 3 * cap;
        h.W = h.U + 3 * cap;
        h.WD = h.W + cap;
        h.ph = reinterpret_cast<int8_t*>(h.WD);
        return h;
    }
};

// Pack cells [g0 + i0, g0 + i1) of the float64 planes into chunk slot positions [i0, i1); returns
// the pack flags (bit 0: a cell has several phases with weight, bit 1: a weight other than 0, 1).
// Same arithmetic as pack_kernel: T(value), weight = T(oPhase_p * region) in double.
template <typename T>
uint32_t host_pack(const HostChunk<T>& h, int64_t n, int64_t g0, int64_t i0, int64_t i1, int nStruc, int nPhase,
                   const double* oPhase, const double* oStruc, const double* u, const double* region, bool dense) {
    uint32_t f = 0;
    for (int k = 0; k < 3; k++) {
        T* dp = h.P + k * h.cap;
        T* du = h.U + k * h.cap;
        const double* sp = k < nStruc ? oStruc + k * n + g0 : nullptr;
        const double* su = u + k * n + g0;
        for (int64_t i = i0; i < i1; i++) {
            dp[i] = sp ? T(sp[i]) : T(0);
            du[i] = T(su[i]);
        }
    }
    if (dense) {
        for (int p = 0; p < nPhase; p++) {
            const double* op = oPhase + p * n + g0;
            T* dw = h.WD + p * h.cap;
            for (int64_t i = i0; i < i1; i++) dw[i] = T(op[i] * (region ? region[g0 + i] : 1.0));
        }
        return 0;
    }
    for (int64_t i = i0; i < i1; i++) {
        const double r = region ? region[g0 + i] : 1.0;
        int which = -1;
        double w = 0.0;
        for (int p = 0; p < nPhase; p++) {
            const double wp = oPhase[p * n + g0 + i] * r;
            if (wp != 0.0) {
                if (which >= 0) f |= 1u;
                else {
                    which = p;
                    w = wp;
                }
            }
        }
        if (which >= 0 && w != 1.0) f |= 2u;
        h.ph[i] = (int8_t)which;
        h.W[i] = T(w);
    }
    return f;
}

}  // namespace qpd
