// Drives plan_buffers.hpp with a fake of the runtime: argv[1] names the check; prints
// what went wrong and returns 1, or returns 0.
#include "plan_buffers.hpp"

#include <cstdio>
#include <cstring>
#include <map>
#include <set>
#include <string>

struct Fake {
  using Event = int;
  using Stream = int;
  int device = 0, made = 0, next_ptr = 0;
  std::set<Event> live;
  std::map<Event, bool> pending;      // recorded and not yet reached
  std::map<Event, Stream> on;         // stream of the last record
  std::map<char *, int> owner;        // allocation -> device
  std::map<Stream, unsigned long long> ids;  // of handles that were used before
  char arena[64] = {};
  bool done(Event e) { return !pending[e]; }
  bool record(Event e, Stream s) {
    pending[e] = true;
    on[e] = s;
    return true;
  }
  bool create(Event &e) {
    e = ++made;
    live.insert(e);
    return true;
  }
  void destroy(Event e) { live.erase(e); }
  bool id(Stream s, unsigned long long &out) {
    out = 100 * (unsigned long long)s + ids[s];
    return true;
  }
  bool allocate(size_t, char *&p) {
    p = &arena[next_ptr++];
    owner[p] = device;
    return true;
  }
  void release(char *p) { owner.erase(p); }
  void finish(Stream s) {  // everything queued on s completes
    for (auto &x : on)
      if (x.second == s) pending[x.first] = false;
  }
};

#define CHECK(x)                          \
  do {                                    \
    if (!(x)) {                           \
      std::printf("failed: %s\n", #x);    \
      return 1;                           \
    }                                     \
  } while (0)

using Buffer = cb2::PlanBuffer<Fake>;

// A plan run on two devices reads each device's own copy.
int devices() {
  Fake api;
  cb2::PlanBufferPool<Fake> pool(1 << 20);
  cb2::PlanCopies<Fake> copies;
  for (int round = 0; round < 2; ++round)
    for (int d = 0; d < 2; ++d) {
      api.device = d;
      if (!copies.on(d)) {
        Buffer b;
        CHECK(pool.take(api, d, 1000, b));
        copies.add(std::move(b));
      }
      CHECK(api.owner[copies.on(d)->ptr] == d);
    }
  CHECK(api.next_ptr == 2);
  copies.give_all(api, pool);
  CHECK(!copies.on(0) && !copies.on(1));
  // and a buffer given back is handed to its own device only
  for (int d = 1; d >= 0; --d) {
    Buffer b;
    CHECK(pool.take(api, d, 1000, b));
    CHECK(api.owner[b.ptr] == d);
    copies.add(std::move(b));
  }
  CHECK(api.next_ptr == 2);
  return 0;
}

// A buffer is not handed on while a launch that reads it is in flight.
int readers() {
  Fake api;
  cb2::PlanBufferPool<Fake> pool(1 << 20);
  Buffer a, b, c;
  CHECK(pool.take(api, 0, 1000, a));
  char *const first = a.ptr;
  CHECK(a.mark(api, 1) && a.mark(api, 2) && a.mark(api, 1));
  pool.give(api, std::move(a));
  api.finish(1);
  CHECK(pool.take(api, 0, 1000, b) && b.ptr != first);
  api.finish(2);
  CHECK(pool.take(api, 0, 1000, c) && c.ptr == first);
  CHECK(c.readers.empty() && api.live.empty());
  // over the pool's limit a buffer is released (which waits), with its events
  cb2::PlanBufferPool<Fake> none(0);
  CHECK(c.mark(api, 3));
  none.give(api, std::move(c));
  CHECK(!api.owner.count(first) && api.live.empty());
  return 0;
}

// Runs queued by the hundred, between waits, on a few streams: as many events as
// streams; and a stream handle that comes back while its old work runs gets its own.
int events() {
  Fake api;
  cb2::PlanBufferPool<Fake> pool(1 << 20);
  Buffer b, c;
  CHECK(pool.take(api, 0, 1000, b));
  for (int loop = 0; loop < 50; ++loop) {
    for (int run = 0; run < 20; ++run)
      for (int s = 1; s <= 3; ++s) CHECK(b.mark(api, s));
    for (int s = 1; s <= 3; ++s) api.finish(s);
  }
  CHECK(b.readers.size() == 3 && api.made == 3);
  CHECK(b.mark(api, 7) && api.made == 3);  // takes over the event of a finished one
  ++api.ids[7];                            // destroyed with work in flight, handle reused
  const Fake::Event old = b.readers[0].event;
  CHECK(api.pending[old] && api.on[old] == 7);
  CHECK(b.mark(api, 7) && b.readers[0].event == old);
  int in_flight = 0;
  for (auto &r : b.readers) in_flight += !api.done(r.event);
  CHECK(in_flight == 2);
  pool.give(api, std::move(b));
  CHECK(pool.take(api, 0, 1000, c) && c.readers.empty());
  return 0;
}

int main(int, char **argv) {
  const std::string what = argv[1];
  if (what == "devices") return devices();
  if (what == "readers") return readers();
  if (what == "events") return events();
  return 2;
}
