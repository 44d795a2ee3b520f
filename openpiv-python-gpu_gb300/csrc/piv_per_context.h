// One object of a kind per context: the library's scratch pools and set-up
// streams (host code; Api holds the runtime's calls, so that the bookkeeping can
// be tested without a GPU).
#pragma once

#include <mutex>

namespace piv {

// An object belongs to the context in which it was made: a device reset ends
// that context and the object with it, and leaves a handle that must not be
// used. The objects are therefore found by the context's id, which no later
// context takes, and kept for the life of the process.
template <class Api>
class PerContext {
 public:
  using Value = typename Api::Value;

  // The current context's object, created on first use; Value() where there is none.
  Value get() {
    const unsigned long long id = Api::context();
    if (!id) return Value();
    std::lock_guard<std::mutex> lock(mu_);
    const Entry* e = find(id);
    if (e) return e->value;
    Value value{};
    if (used_ == kMax || !Api::create(&value)) return Value();
    entries_[used_++] = Entry{id, value};
    return value;
  }

  // f(object) for the context of device `dev`, whichever device is current; nothing where there is none.
  template <class F>
  void with(int dev, F f) {
    std::lock_guard<std::mutex> lock(mu_);
    if (!used_) return;
    typename Api::OnDevice there(dev);
    const Entry* e = find(Api::context());
    if (e) f(e->value);
  }

 private:
  struct Entry {
    unsigned long long id;
    Value value;
  };
  const Entry* find(unsigned long long id) const {
    for (int k = used_ - 1; k >= 0; --k)
      if (entries_[k].id == id) return &entries_[k];
    return nullptr;
  }
  static constexpr int kMax = 64;
  std::mutex mu_;
  Entry entries_[kMax] = {};
  int used_ = 0;
};

}  // namespace piv
