// The library's scratch pools, one per context (host code; Api holds the
// runtime's calls, so that the bookkeeping can be tested without a GPU).
#pragma once

#include <mutex>

namespace piv {

// A pool belongs to the context in which it was made: a device reset ends that
// context and the pool with it, and leaves a handle that must not be used. The
// pools are therefore found by the context's id, which no later context takes.
template <class Api>
class ScratchPools {
 public:
  // The pool of the current context, created on first use; Pool() where there is none.
  typename Api::Pool get() {
    const unsigned long long id = Api::context();
    if (!id) return typename Api::Pool();
    std::lock_guard<std::mutex> lock(mu_);
    Entry* e = find(id);
    if (e) return e->pool;
    typename Api::Pool pool{};
    if (used_ == kMax || !Api::create(&pool)) return typename Api::Pool();
    entries_[used_++] = Entry{id, pool};
    return pool;
  }

  // Gives back the idle memory of the pool of device `dev`, whichever device is current.
  void trim(int dev) {
    std::lock_guard<std::mutex> lock(mu_);
    if (!used_) return;
    typename Api::OnDevice there(dev);
    Entry* e = find(Api::context());
    if (e) Api::trim(e->pool);
  }

 private:
  struct Entry {
    unsigned long long id;
    typename Api::Pool pool;
  };
  Entry* find(unsigned long long id) {
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
