// Threads that stay, for work that is worth sharing but too short to make threads for: made at the first use, asleep between uses,
// joined with the pool. One caller at a time.
#pragma once
#include <algorithm>
#include <condition_variable>
#include <functional>
#include <mutex>
#include <exception>
#include <thread>
#include <vector>

namespace sp {

class CopyPool {
  public:
    CopyPool() = default;
    CopyPool(const CopyPool&) = delete;
    CopyPool& operator=(const CopyPool&) = delete;
    ~CopyPool() {
        {
            std::lock_guard<std::mutex> l(m_);
            stop_ = true;
        }
        wake_.notify_all();
        for (std::thread& t : threads_) t.join();
    }
    // work() here and on up to `helpers` threads at once; returns when all that began it have come back. Those that have not woken by
    // then are not waited for, and where no thread can be made the caller does it all. work must not throw.
    void run(int helpers, const std::function<void()>& work) {
        {
            std::lock_guard<std::mutex> l(m_);
            while ((int)threads_.size() < helpers && !refused_) {
                try {
                    threads_.emplace_back([this] { loop(); });
                } catch (const std::exception&) {  // no thread, or no memory for one: not tried again
                    refused_ = true;
                }
            }
            work_ = &work;
            wanted_ = std::min(helpers, (int)threads_.size());
        }
        wake_.notify_all();
        work();
        std::unique_lock<std::mutex> l(m_);
        wanted_ = 0;
        idle_.wait(l, [this] { return busy_ == 0; });
        work_ = nullptr;
    }
    int size() const { return (int)threads_.size(); }

  private:
    void loop() {
        std::unique_lock<std::mutex> l(m_);
        for (;;) {
            wake_.wait(l, [this] { return stop_ || wanted_ > 0; });
            if (stop_) return;
            --wanted_;
            ++busy_;
            const std::function<void()>* work = work_;
            l.unlock();
            (*work)();
            l.lock();
            if (--busy_ == 0) idle_.notify_one();
        }
    }
    std::mutex m_;
    std::condition_variable wake_, idle_;
    std::vector<std::thread> threads_;
    const std::function<void()>* work_ = nullptr;
    int wanted_ = 0, busy_ = 0;
    bool stop_ = false, refused_ = false;
};

}  // namespace sp
