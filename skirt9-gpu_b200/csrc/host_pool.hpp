// Worker threads of a context for its host-side copies and additions (host side only).
#pragma once

#include <algorithm>
#include <condition_variable>
#include <exception>
#include <functional>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>
#include <unistd.h>

namespace skg {

// At most 16 host cores, started with the first large array and joined with the context. Starting
// threads for every chunk of a read-back took as long as adding one (16 threads, 0.3 ms).
// A process forked later has a copy of the pool but none of its threads: it takes no part of it (destroying
// the condition variables would wait for those threads for ever), and works alone.
class HostPool
{
public:
    HostPool() = default;
    HostPool(const HostPool&) = delete;
    HostPool& operator=(const HostPool&) = delete;
    ~HostPool()
    {
        if (!_shared) return;
        if (_shared->process != getpid())
        {
            _shared.release();
            return;
        }
        {
            std::lock_guard<std::mutex> lock(_shared->mutex);
            _shared->stop = true;
        }
        _shared->wake.notify_all();
        for (std::thread& t : _shared->threads) t.join();
    }

    // runs f(begin, end) over shares of [0, n) on up to one thread per `grain` items; returns when done
    void run(size_t n, size_t grain, const std::function<void(size_t, size_t)>& f)
    {
        const size_t cores = std::max(1u, std::min(std::thread::hardware_concurrency(), 16u));
        size_t parts = std::max<size_t>(1, std::min(cores, (n + grain - 1) / grain));
        if (parts > 1 && _shared && _shared->process != getpid()) parts = 1;
        if (parts > 1)
        {
            try
            {
                if (!_shared) _shared = std::make_unique<Shared>();
                std::lock_guard<std::mutex> lock(_shared->mutex);
                auto& threads = _shared->threads;
                while (threads.size() + 1 < parts) threads.emplace_back([s = _shared.get(), me = threads.size()] { s->work(me); });
            }
            catch (const std::exception&)
            {
                parts = _shared ? _shared->threads.size() + 1 : 1;  // no further thread to be had: the work goes to those there are
            }
        }
        if (parts == 1)
        {
            f(0, n);
            return;
        }
        Shared& s = *_shared;
        {
            std::lock_guard<std::mutex> lock(s.mutex);
            s.job = &f;
            s.n = n;
            s.parts = parts;
            s.open = parts - 1;
            ++s.round;
        }
        s.wake.notify_all();
        f(0, n / parts);
        std::unique_lock<std::mutex> lock(s.mutex);
        s.done.wait(lock, [&s] { return s.open == 0; });
    }

private:
    // what the caller and the workers share
    struct Shared
    {
        std::mutex mutex;
        std::condition_variable wake, done;
        std::vector<std::thread> threads;
        const std::function<void(size_t, size_t)>* job = nullptr;
        size_t n = 0, parts = 0, open = 0, round = 0;
        bool stop = false;
        const pid_t process = getpid();

        void work(size_t me)
        {
            std::unique_lock<std::mutex> lock(mutex);
            size_t seen = 0;  // a thread started for a round takes part in it: the round ends only with its part
            for (;;)
            {
                wake.wait(lock, [&] { return stop || round != seen; });
                if (stop) return;
                seen = round;
                const size_t part = me + 1;
                if (part >= parts) continue;
                const auto* f = job;
                const size_t total = n, shares = parts;
                lock.unlock();
                (*f)(total / shares * part, part + 1 == shares ? total : total / shares * (part + 1));
                lock.lock();
                if (--open == 0) done.notify_one();
            }
        }
    };
    std::unique_ptr<Shared> _shared;
};

}  // namespace skg
