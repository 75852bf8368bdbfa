/*
 * lpg_devmem.h — the device memory of one handle.
 *
 * Buffers above kItemBytes are allocations of their own.  Small ones are
 * parts of slabs of kSlabBytes: one allocation for many, and for uploads one
 * copy.  The two are kept in lists of their own: give_back() looks at the
 * allocations made one by one only, so a part of a slab (which may have the
 * slab's own address) is never freed by itself, and stays until clear().
 *
 * Plain C++ over two functions, so that it runs without a device.
 */
#ifndef LPG_DEVMEM_H
#define LPG_DEVMEM_H

#include <stddef.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <utility>
#include <vector>

class DevMem {
 public:
  static constexpr size_t kSlabBytes = 1 << 20, kItemBytes = 1 << 17;
  typedef int (*Alloc)(void** p, size_t bytes); /* 0: done */
  typedef void (*Release)(void* p);

  /* bytes [sent, used) of an upload slab are not on the device yet */
  struct Slab {
    uint8_t* dev = nullptr;
    std::vector<uint8_t> host; /* upload slabs: the bytes to copy */
    size_t used = 0, sent = 0;
  };

  DevMem(Alloc alloc, Release release) : alloc_(alloc), release_(release) {}
  DevMem(const DevMem&) = delete;
  DevMem& operator=(const DevMem&) = delete;

  static size_t pad(size_t n) { return (n + 255) & ~(size_t)255; }

  /* An allocation of its own; the allocator's code on failure. */
  int own(void** p, size_t bytes) {
    const int rc = alloc_(p, bytes);
    if (rc == 0) own_.push_back(*p);
    return rc;
  }

  /* A part of a slab, or an allocation of its own above kItemBytes. */
  int part(void** p, size_t bytes) {
    if (bytes > kItemBytes) return own(p, bytes);
    if (!plain_.dev || plain_.used + bytes > kSlabBytes) {
      Slab s;
      const int rc = slab(&s);
      if (rc) return rc;
      plain_ = std::move(s);
    }
    *p = plain_.dev + plain_.used;
    plain_.used += pad(bytes);
    return 0;
  }

  /* A part of an upload slab with src's bytes (at most kItemBytes), which
   * arrive when the caller copies the slab's unsent bytes. */
  int upload(void** p, const void* src, size_t bytes) {
    if (uploads_.empty() || uploads_.back().used + bytes > kSlabBytes) {
      Slab s;
      const int rc = slab(&s);
      if (rc) return rc;
      s.host.resize(kSlabBytes);
      uploads_.push_back(std::move(s));
    }
    Slab& s = uploads_.back();
    *p = s.dev + s.used;
    if (bytes) memcpy(s.host.data() + s.used, src, bytes);
    s.used = std::min(kSlabBytes, s.used + pad(std::max<size_t>(bytes, 1)));
    return 0;
  }
  std::vector<Slab>& uploads() { return uploads_; }

  /* Frees an allocation of its own; does nothing for a part of a slab. */
  void give_back(void* p) {
    const auto it = std::find(own_.begin(), own_.end(), p);
    if (!p || it == own_.end()) return;
    own_.erase(it);
    release_(p);
  }

  /* Frees everything. */
  void clear() {
    for (void* p : own_) release_(p);
    for (void* p : slabs_) release_(p);
    own_.clear();
    slabs_.clear();
    uploads_.clear();
    plain_ = Slab();
  }

 private:
  int slab(Slab* s) {
    void* p = nullptr;
    const int rc = alloc_(&p, kSlabBytes);
    if (rc) return rc;
    slabs_.push_back(p);
    s->dev = (uint8_t*)p;
    return 0;
  }

  Alloc alloc_;
  Release release_;
  std::vector<void*> own_, slabs_;
  Slab plain_;
  std::vector<Slab> uploads_;
};

#endif /* LPG_DEVMEM_H */
