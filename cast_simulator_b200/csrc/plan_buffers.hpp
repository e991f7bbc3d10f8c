// Device copies of a plan's matrices: one a device the plan has run on, in buffers
// that go back to a pool and are handed on once nothing reads them any more.  Written
// against an Api of the runtime calls it makes, so that it runs without a device.
//
// Api: types Event and Stream, and
//   bool done(Event), bool record(Event, Stream), bool create(Event &), void destroy(Event)
//   bool id(Stream, unsigned long long &)     a stream's own, never used again
//   bool allocate(size_t, char *&), void release(char *)      on the current device
#pragma once

#include <cstddef>
#include <mutex>
#include <utility>
#include <vector>

namespace cb2 {

template <class Api> struct PlanBuffer {
  int device = 0;
  char *ptr = nullptr;
  size_t bytes = 0;
  // One event a stream, behind the last launch there that reads the buffer.  Streams
  // are told apart by id: a handle may come back as another stream while the work of
  // the one that had it is still in flight.
  struct Reader {
    unsigned long long stream;
    typename Api::Event event;
  };
  std::vector<Reader> readers;

  // Records that launches on `s` up to here read the buffer.  A new stream takes over
  // the event of one whose work is done, so there are at most as many as streams ever
  // had such work in flight at once, however many runs are queued on each.
  bool mark(Api &api, typename Api::Stream s) {
    unsigned long long id = 0;
    if (!api.id(s, id)) return false;
    Reader *at = nullptr;
    for (Reader &r : readers)
      if (r.stream == id) at = &r;
    for (size_t i = 0; i < readers.size() && !at; ++i)
      if (api.done(readers[i].event)) at = &readers[i];
    if (!at) {
      typename Api::Event e{};
      if (!api.create(e)) return false;
      readers.push_back(Reader{id, e});
      at = &readers.back();
    }
    at->stream = id;
    return api.record(at->event, s);
  }

  // True once every launch that reads the buffer has completed.
  bool settled(Api &api) {
    while (!readers.empty()) {
      if (!api.done(readers.back().event)) return false;
      api.destroy(readers.back().event);
      readers.pop_back();
    }
    return true;
  }
};

// Buffers given back, waiting for their readers and then for the next plan: at most
// `limit` bytes; a buffer beyond that is released, which waits for its device.
template <class Api> class PlanBufferPool {
 public:
  explicit PlanBufferPool(size_t limit) : limit_(limit) {}

  // A buffer of at least `bytes` on `device`, which is current.
  bool take(Api &api, int device, size_t bytes, PlanBuffer<Api> &out) {
    size_t cap = size_t(64) << 10;
    while (cap < bytes) cap <<= 1;
    {
      std::lock_guard<std::mutex> lock(mu_);
      for (size_t i = 0; i < idle_.size(); ++i)
        if (idle_[i].device == device && idle_[i].bytes == cap && idle_[i].settled(api)) {
          out = std::move(idle_[i]);
          total_ -= cap;
          idle_.erase(idle_.begin() + (std::ptrdiff_t)i);
          return true;
        }
    }
    out = PlanBuffer<Api>{};
    out.device = device;
    out.bytes = cap;
    return api.allocate(cap, out.ptr);
  }

  void give(Api &api, PlanBuffer<Api> &&b) {
    if (!b.ptr) return;
    {
      std::lock_guard<std::mutex> lock(mu_);
      if (total_ + b.bytes <= limit_) {
        total_ += b.bytes;
        idle_.push_back(std::move(b));
        return;
      }
    }
    api.release(b.ptr);
    for (auto &r : b.readers) api.destroy(r.event);
  }

 private:
  std::mutex mu_;
  std::vector<PlanBuffer<Api>> idle_;
  size_t total_ = 0;
  const size_t limit_;
};

// A plan's buffers, one a device: a kernel must read the copy of the device it runs
// on, and a program may be run on one device after another.
template <class Api> class PlanCopies {
 public:
  PlanBuffer<Api> *on(int device) {
    for (auto &b : copies_)
      if (b.device == device) return &b;
    return nullptr;
  }
  void add(PlanBuffer<Api> &&b) { copies_.push_back(std::move(b)); }
  void give_all(Api &api, PlanBufferPool<Api> &pool) {
    for (auto &b : copies_) pool.give(api, std::move(b));
    copies_.clear();
  }

 private:
  std::vector<PlanBuffer<Api>> copies_;
};

}  // namespace cb2
