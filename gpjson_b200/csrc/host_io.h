// Host-side I/O of the C ABI: parallel file reads into pinned staging and
// the host buffers of query results.  Plain C++ (POSIX), no CUDA, so the
// test suite exercises it on the CPU.
#pragma once

#include <fcntl.h>
#include <sys/types.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <cerrno>
#include <condition_variable>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <new>
#include <thread>
#include <vector>

namespace gpj {

// Reads a file with up to `threads` threads, the caller's among them.  A
// file load is bound by the copy out of the page cache, which one thread
// does at a fraction of host memory bandwidth.  The workers live for one
// load.
class SliceReader {
  public:
    SliceReader(int fd, int threads) : fd_(fd) {
        try {
            for (int i = 1; i < threads; i++) workers_.emplace_back([this] { work(); });
        } catch (const std::exception&) {
            // fewer threads than asked
        }
    }

    ~SliceReader() {
        {
            std::lock_guard<std::mutex> g(mu_);
            quit_ = true;
        }
        go_.notify_all();
        for (auto& t : workers_) t.join();
    }

    // Calls fn(i) once for each i in [0, count), numbers taken in order by
    // whichever thread is free; false when one of them returned false (no
    // more are taken then).
    template <class Fn>
    bool for_each(int64_t count, const Fn& fn) {
        {
            std::lock_guard<std::mutex> g(mu_);
            fn_ = &fn;
            call_ = [](const void* f, int64_t i) { return (*static_cast<const Fn*>(f))(i); };
            count_ = count;
            next_ = 0;
            ok_ = true;
            pending_ = static_cast<int>(workers_.size());
            ++round_;
        }
        go_.notify_all();
        take();
        std::unique_lock<std::mutex> g(mu_);
        done_.wait(g, [this] { return pending_ == 0; });
        return ok_;
    }

    // Bytes [pos, pos + len) into dst, a slice per thread; false on an I/O
    // error or a short read (the file shrank).
    bool read(uint8_t* dst, int64_t pos, size_t len) {
        const size_t parts = workers_.size() + 1;
        const size_t slice = (len + parts - 1) / parts;
        return for_each(static_cast<int64_t>(parts), [&](int64_t i) {
            const size_t off = std::min(len, slice * static_cast<size_t>(i));
            return read_here(dst + off, pos + static_cast<int64_t>(off), std::min(slice, len - off));
        });
    }

    // The same on the calling thread alone (from any thread).
    bool read_here(uint8_t* dst, int64_t pos, size_t len) const {
        size_t got = 0;
        while (got < len) {
            const ssize_t r = ::pread(fd_, dst + got, len - got, static_cast<off_t>(pos + got));
            if (r < 0 && errno == EINTR) continue;
            if (r <= 0) return false;
            got += static_cast<size_t>(r);
        }
        return true;
    }

    bool failed() const { return !ok_; }

  private:
    void take() {
        for (int64_t i = next_++; i < count_ && ok_; i = next_++)
            if (!call_(fn_, i)) ok_ = false;
    }

    void work() {
        uint64_t seen = 0;
        for (;;) {
            {
                std::unique_lock<std::mutex> g(mu_);
                go_.wait(g, [&] { return quit_ || round_ != seen; });
                if (quit_) return;
                seen = round_;
            }
            take();
            {
                std::lock_guard<std::mutex> g(mu_);
                --pending_;
            }
            done_.notify_one();
        }
    }

    const int fd_;
    std::vector<std::thread> workers_;
    std::mutex mu_;
    std::condition_variable go_, done_;
    uint64_t round_ = 0;
    int pending_ = 0;
    bool quit_ = false;
    // the current call of for_each
    const void* fn_ = nullptr;
    bool (*call_)(const void*, int64_t) = nullptr;
    int64_t count_ = 0;
    std::atomic<int64_t> next_{0};
    std::atomic<bool> ok_{true};
};

// Host memory for results.  A new buffer's first touch (page faults) costs
// several times the device-to-host copy into it, and a copy that faults in
// its own pages is slower still, so the largest released buffer (up to
// kKeepElems) is kept for the next result of the process, and a new one is
// touched once before the copy.
class ResultBuffers {
  public:
    static constexpr size_t kKeepElems = size_t(64) << 20;  // 512 MiB

    int64_t* take(size_t count, size_t* cap) {
        {
            std::lock_guard<std::mutex> g(mu_);
            if (kept_ && kept_cap_ >= count) {
                int64_t* p = kept_;
                *cap = kept_cap_;
                kept_ = nullptr;
                kept_cap_ = 0;
                return p;
            }
        }
        int64_t* p = new (std::nothrow) int64_t[count];
        if (p) std::memset(p, 0, count * sizeof(int64_t));
        *cap = count;
        return p;
    }

    void give(int64_t* p, size_t cap) {
        if (!p) return;
        {
            std::lock_guard<std::mutex> g(mu_);
            if (cap <= kKeepElems && cap > kept_cap_) {
                std::swap(p, kept_);
                std::swap(cap, kept_cap_);
            }
        }
        delete[] p;
    }

    ResultBuffers() = default;
    ResultBuffers(const ResultBuffers&) = delete;
    ResultBuffers& operator=(const ResultBuffers&) = delete;
    ~ResultBuffers() { delete[] kept_; }

  private:
    std::mutex mu_;
    int64_t* kept_ = nullptr;
    size_t kept_cap_ = 0;
};

// Never destroyed, so that results released during process exit find it.
inline ResultBuffers& result_buffers() {
    static ResultBuffers* b = new ResultBuffers;
    return *b;
}

}  // namespace gpj
