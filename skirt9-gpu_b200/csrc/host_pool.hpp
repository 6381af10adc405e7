// Worker threads of a context for its host-side copies and additions (host side only).
#pragma once

#include <algorithm>
#include <condition_variable>
#include <exception>
#include <functional>
#include <mutex>
#include <thread>
#include <vector>

namespace skg {

// At most 16 host cores, started with the first large array and joined with the context. Starting
// threads for every chunk of a read-back took as long as adding one (16 threads, 0.3 ms).
class HostPool
{
public:
    HostPool() = default;
    HostPool(const HostPool&) = delete;
    HostPool& operator=(const HostPool&) = delete;
    ~HostPool()
    {
        {
            std::lock_guard<std::mutex> lock(_mutex);
            _stop = true;
        }
        _wake.notify_all();
        for (std::thread& t : _threads) t.join();
    }

    // runs f(begin, end) over shares of [0, n) on up to one thread per `grain` items; returns when done
    void run(size_t n, size_t grain, const std::function<void(size_t, size_t)>& f)
    {
        const size_t cores = std::max(1u, std::min(std::thread::hardware_concurrency(), 16u));
        size_t parts = std::max<size_t>(1, std::min(cores, (n + grain - 1) / grain));
        if (parts > 1)
        {
            std::lock_guard<std::mutex> lock(_mutex);
            try
            {
                while (_threads.size() + 1 < parts) _threads.emplace_back([this, me = _threads.size()] { work(me); });
            }
            catch (const std::exception&)
            {
                parts = _threads.size() + 1;  // no further thread to be had: the work goes to those there are
            }
        }
        if (parts == 1)
        {
            f(0, n);
            return;
        }
        {
            std::lock_guard<std::mutex> lock(_mutex);
            _job = &f;
            _n = n;
            _parts = parts;
            _open = parts - 1;
            ++_round;
        }
        _wake.notify_all();
        f(0, n / parts);
        std::unique_lock<std::mutex> lock(_mutex);
        _done.wait(lock, [this] { return _open == 0; });
    }

private:
    void work(size_t me)
    {
        std::unique_lock<std::mutex> lock(_mutex);
        size_t seen = 0;  // a thread started for a round takes part in it: the round ends only with its part
        for (;;)
        {
            _wake.wait(lock, [&] { return _stop || _round != seen; });
            if (_stop) return;
            seen = _round;
            const size_t part = me + 1;
            if (part >= _parts) continue;
            const auto* f = _job;
            const size_t n = _n, parts = _parts;
            lock.unlock();
            (*f)(n / parts * part, part + 1 == parts ? n : n / parts * (part + 1));
            lock.lock();
            if (--_open == 0) _done.notify_one();
        }
    }

    std::mutex _mutex;
    std::condition_variable _wake, _done;
    std::vector<std::thread> _threads;
    const std::function<void(size_t, size_t)>* _job = nullptr;
    size_t _n = 0, _parts = 0, _open = 0, _round = 0;
    bool _stop = false;
};

}  // namespace skg
