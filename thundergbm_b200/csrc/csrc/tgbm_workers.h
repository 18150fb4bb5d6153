// Standing host threads that share the tasks of any number of callers.  Plain C++: no CUDA.
#pragma once
#include <condition_variable>
#include <functional>
#include <list>
#include <mutex>
#include <thread>

namespace tgbm {

// `Worker` is what a thread keeps between tasks.  Threads are started when tasks wait, at most `most` of them; a call that
// finds all of them busy waits.  Where no thread can be started the tasks go to those that exist, and with none at all the
// caller does them itself.
template <typename Worker>
class WorkerPool {
public:
    typedef std::function<void(std::function<void()>)> Start;   // runs the argument on a new thread, or throws
    explicit WorkerPool(int most, Start start = [](std::function<void()> f) { std::thread(std::move(f)).detach(); })
        : most_(most), start_(std::move(start)) {}

    // runs f(worker, t) for t = 0 .. n - 1 on the workers and returns when all have returned; f must not throw
    void run(int n, const std::function<void(Worker &, int)> &f) {
        Job job{&f, n};
        std::list<Task> tasks;
        for (int t = 0; t < n; ++t) tasks.push_back({&job, t});
        std::unique_lock<std::mutex> lock(mutex_);
        queue_.splice(queue_.end(), tasks);   // all of them or none: they point into this call
        try {
            for (; started_ < most_ && idle_ + starting_ < (int)queue_.size(); ++started_, ++starting_) start_([this] { loop(); });
        } catch (...) {
        }
        wake_.notify_all();
        if (started_ == 0) {
            Worker w;
            while (!queue_.empty()) one(w, lock);
        }
        done_.wait(lock, [&] { return job.left == 0; });
    }

private:
    struct Job { const std::function<void(Worker &, int)> *f; int left; };
    struct Task { Job *job; int t; };
    void one(Worker &w, std::unique_lock<std::mutex> &lock) {
        const Task task = queue_.front();
        queue_.pop_front();
        lock.unlock();
        (*task.job->f)(w, task.t);
        lock.lock();
        if (--task.job->left == 0) done_.notify_all();
    }
    void loop() {
        Worker w;
        std::unique_lock<std::mutex> lock(mutex_);
        --starting_;
        for (;;) {
            ++idle_;
            wake_.wait(lock, [&] { return !queue_.empty(); });
            --idle_;
            one(w, lock);
        }
    }
    const int most_;
    const Start start_;
    std::mutex mutex_;
    std::condition_variable wake_, done_;
    std::list<Task> queue_;
    int started_ = 0, starting_ = 0, idle_ = 0;
};

}  // namespace tgbm
