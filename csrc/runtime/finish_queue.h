// Queue of finished task names, drained whole by the poller (the reference's FinishQueue:
// a mutex around a std::queue of tensor names, ref hp_cuda.h:81-96, hp_cuda.cpp:135-151).
// Plain C++ (no torch) so that the host runtime can be built and stress-tested under
// ThreadSanitizer / AddressSanitizer without a GPU.
#pragma once
#include <chrono>
#include <condition_variable>
#include <mutex>
#include <string>
#include <vector>

namespace hipress {
namespace runtime {

class FinishQueue {
 public:
  void push(const std::string& key) {
    {
      std::lock_guard<std::mutex> lk(mu_);
      keys_.push_back(key);
    }
    cv_.notify_all();
  }
  // Ends the waits in progress without a name: something else that a poller looks at has changed.
  void wake() {
    {
      std::lock_guard<std::mutex> lk(mu_);
      ++wakes_;
    }
    cv_.notify_all();
  }
  // drain(), after waiting until there is a name, a wake(), or the time is up.  `seen`: the wakes() that
  // the caller had read before it last looked at that something else.
  std::vector<std::string> wait_drain(double timeout_s, unsigned long long seen) {
    std::unique_lock<std::mutex> lk(mu_);
    cv_.wait_for(lk, std::chrono::duration<double>(timeout_s), [&] { return !keys_.empty() || wakes_ != seen; });
    std::vector<std::string> out;
    out.swap(keys_);
    return out;
  }
  unsigned long long wakes() {
    std::lock_guard<std::mutex> lk(mu_);
    return wakes_;
  }
  std::vector<std::string> drain() {
    std::lock_guard<std::mutex> lk(mu_);
    std::vector<std::string> out;
    out.swap(keys_);
    return out;
  }

 private:
  std::mutex mu_;
  std::condition_variable cv_;
  std::vector<std::string> keys_;
  unsigned long long wakes_ = 0;
};

}  // namespace runtime
}  // namespace hipress
