// handle_pool.hpp -- free lists of CUDA objects (streams, events), one list per device.
//
// A stream or event works on the device it was made on only: a launch or a record on it while another
// device is current is refused. So an object is handed out on its own device alone, and goes back
// to that device's list whichever device is current when it is given back. Host code without CUDA
// headers, so that the keying can be checked without a GPU.
#pragma once

#include <map>
#include <mutex>
#include <unordered_map>
#include <vector>

namespace sov {

template <class H>
class HandlePool {
 public:
  // a free object of `device`, or make() when its list is empty
  template <class Make>
  H take(int device, Make make) {
    {
      std::lock_guard<std::mutex> g(mu_);
      std::vector<H>& v = free_[device];
      if (!v.empty()) {
        H h = v.back();
        v.pop_back();
        return h;
      }
    }
    H h = make();
    std::lock_guard<std::mutex> g(mu_);
    device_of_[h] = device;
    return h;
  }
  void give(H h) {
    std::lock_guard<std::mutex> g(mu_);
    free_[device_of_.at(h)].push_back(h);
  }

 private:
  std::mutex mu_;
  std::map<int, std::vector<H>> free_;
  std::unordered_map<H, int> device_of_;  // of every object made here (they live as long as the process)
};

}  // namespace sov
