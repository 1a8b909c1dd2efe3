// deo_once.h -- a value found once per device: a kernel's resident grid together with the
// function attributes set on the way (they belong to one device's context).  Plain C++.
#pragma once
#include <map>
#include <mutex>

namespace deo {

template <typename V>
class PerDevice {
    std::mutex mu_;
    std::map<int, V> found_;

  public:
    // The device's value in out; find(out) finds it and returns an error code.  No other
    // thread sees the value before find has returned 0; an error is not kept.
    template <typename Find>
    int get(int device, V& out, Find find) {
        std::lock_guard<std::mutex> lk(mu_);
        const auto it = found_.find(device);
        if (it != found_.end()) {
            out = it->second;
            return 0;
        }
        const int e = find(out);
        if (!e) found_[device] = out;
        return e;
    }
};

}  // namespace deo
