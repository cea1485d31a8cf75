// Device buffers kept between solves.  A solve has 20 to 80 of them, and a
// cudaMalloc / cudaFree pair takes 0.7 ms and more (2 MB: 0.4 + 0.3, 1 GB: 0.7 +
// 1.0): 8 of 10 ms of a host-array solve at o = 8, v = 64.  At most KEEP_BYTES
// (1.1 % of the device's memory) are kept of each context, the rest given up,
// and all of the context's when an allocation of the library fails or the
// caller asks for them.  A buffer comes back only after the stream that used it
// has been waited for, so any thread and stream may take it next.  Buffers
// belong to the context they were made in (its process-wide id): they are
// handed out, counted and given up in that context only, so solves on several
// GPUs do not lose each other's.  A destroyed context (a reset device comes back
// with a new id) takes its buffers' memory with it; what stays here is their
// list, which nothing asks for again.
// A CUDA memory pool was measured instead: it maps and unmaps at 5 ms per GB
// each way whenever the buffers of two solves do not fit its free space alike
// (FP32 upt 12/120/11/122: 58 to 200 ms a call).
//
// Bookkeeping only; standard library only.
#pragma once

#include <cstddef>
#include <cstdint>
#include <list>
#include <map>
#include <mutex>
#include <new>

namespace ptb {

constexpr size_t KEEP_BYTES = (size_t)2 << 30;
constexpr size_t KEEP_BUFFER = (size_t)1280 << 20;   // larger ones are not kept

class BufferCache {
 public:
  typedef void (*Free)(void *);   // frees a buffer of the current context
  explicit BufferCache(Free f) : free_(f) {}

  // whole 64 KiB (2 MiB from there on), so that sizes of like solves meet
  static size_t rounded(size_t n) {
    const size_t g = n <= ((size_t)2 << 20) ? (size_t)64 << 10 : (size_t)2 << 20;
    return (n + g - 1) & ~(g - 1);
  }

  // The smallest kept buffer of n bytes or little more, or null.
  void *take(uint64_t ctx, size_t n, size_t *size) {
    std::lock_guard<std::mutex> g(mu_);
    const auto of = of_.find(ctx);
    if (of == of_.end()) return nullptr;
    std::list<Kept> &kept = of->second.kept;
    auto best = kept.end();
    for (auto it = kept.begin(); it != kept.end(); ++it)
      if (it->n >= n && it->n <= n + n / 4 + ((size_t)1 << 20) &&
          (best == kept.end() || it->n < best->n))
        best = it;
    if (best == kept.end()) return nullptr;
    void *p = best->p;
    *size = best->n;
    of->second.bytes -= best->n;
    kept.erase(best);
    return p;
  }

  // Keeps a buffer nothing on the device uses any more (of the current
  // context, ctx).  Beyond KEEP_BYTES the largest ones go, so that a solve that
  // outgrows the cache allocates few buffers anew, but first the oldest if it
  // has lain unused for long.
  void give(uint64_t ctx, void *p, size_t n) {
    std::list<Kept> drop;
    if (n <= KEEP_BUFFER) {
      try {
        std::lock_guard<std::mutex> g(mu_);
        Context &c = of_[ctx];
        c.kept.push_front({p, n, ++c.gives});
        p = nullptr;
        c.bytes += n;
        while (c.bytes > KEEP_BYTES) {
          auto out = std::prev(c.kept.end());
          if (c.gives - out->at < 512)
            for (auto it = c.kept.begin(); it != c.kept.end(); ++it)
              if (it->n > out->n) out = it;
          c.bytes -= out->n;
          drop.splice(drop.end(), c.kept, out);
        }
      } catch (const std::bad_alloc &) {   // no room for its entry: not kept
      }
    }
    if (p) free_(p);
    for (const Kept &k : drop) free_(k.p);
  }

  // Frees all of the current context's (ctx); returns their bytes.
  size_t give_up(uint64_t ctx) {
    Context c;
    {
      std::lock_guard<std::mutex> g(mu_);
      const auto of = of_.find(ctx);
      if (of == of_.end()) return 0;
      c.kept.swap(of->second.kept);
      c.bytes = of->second.bytes;
      of->second.bytes = 0;
    }
    for (const Kept &k : c.kept) free_(k.p);
    return c.bytes;
  }

 private:
  struct Kept {
    void *p;
    size_t n;
    uint64_t at;   // the context's `gives` when it was given
  };
  struct Context {
    std::list<Kept> kept;   // most recently given first
    size_t bytes = 0;
    uint64_t gives = 0;
  };
  const Free free_;
  std::mutex mu_;
  std::map<uint64_t, Context> of_;
};

}  // namespace ptb
