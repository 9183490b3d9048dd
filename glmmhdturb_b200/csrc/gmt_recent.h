// gmt_recent.h -- what was made for the last few keys, shared by threads (host code without CUDA).
#pragma once
#include <mutex>

namespace gmt {

// Values of the last N keys.  A value is copied in and out whole under a lock: a step of another thread never
// sees one that is half written.
template <class Key, class Value, int N> class Recent {
public:
    bool find(const Key& k, Value* v) const {
        std::lock_guard<std::mutex> lk(mu_);
        for (int i = 0; i < used_; ++i)
            if (key_[i] == k) {
                *v = value_[i];
                return true;
            }
        return false;
    }
    void keep(const Key& k, const Value& v) {
        std::lock_guard<std::mutex> lk(mu_);
        key_[next_] = k;
        value_[next_] = v;
        next_ = (next_ + 1) % N;
        if (used_ < N) ++used_;
    }

private:
    mutable std::mutex mu_;
    Key key_[N];
    Value value_[N];
    int used_ = 0, next_ = 0;
};

}  // namespace gmt
