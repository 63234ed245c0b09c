// Host side of the target uploads: the arrays of a batch (hundreds of
// resolution matrices, 0.2 MB each) gathered into one pinned buffer.
//
// One core copies at about 6 GB/s into pinned memory -- 11 to 14 ms for 100
// DESI targets, half of fitz's time for them -- while the memory of the machine
// takes several times that, so arrays of 4 MB and more are split into equal
// byte ranges over up to kMaxThreads threads that live for the call (the
// callers come here for batches of 16 MB and more).
#include <algorithm>
#include <cstdint>
#include <cstring>
#include <exception>
#include <thread>

#include "../../include/redrock_b200.h"

namespace {

constexpr int kMaxThreads = 16;
constexpr int64_t kBytesPerThread = 2 << 20;

// bytes [lo, hi) of the concatenation of src[0..n)
void copy_range(const void* const* src, const int64_t* bytes, int64_t n, char* dst, int64_t lo,
                int64_t hi) {
  int64_t at = 0;
  for (int64_t i = 0; i < n && at < hi; at += bytes[i], ++i) {
    const int64_t a = std::max(lo, at), b = std::min(hi, at + bytes[i]);
    if (a < b) std::memcpy(dst + a, static_cast<const char*>(src[i]) + (a - at), (size_t)(b - a));
  }
}

}  // namespace

extern "C" int rr_host_gather(const void* const* src, const int64_t* bytes, int64_t n, void* dst,
                              int64_t dst_bytes) {
  if (n < 0 || dst_bytes < 0 || (n > 0 && (!src || !bytes))) return RR_EINVAL;
  int64_t total = 0;
  for (int64_t i = 0; i < n; ++i) {
    if (bytes[i] < 0 || (bytes[i] > 0 && !src[i]) || bytes[i] > dst_bytes - total) return RR_EINVAL;
    total += bytes[i];
  }
  if (total == 0) return RR_OK;
  if (!dst) return RR_EINVAL;
  char* out = static_cast<char*>(dst);
  const int64_t cores = (int64_t)std::thread::hardware_concurrency();
  const int64_t k = std::max<int64_t>(
      1, std::min<int64_t>({total / kBytesPerThread, cores, (int64_t)kMaxThreads}));
  std::thread th[kMaxThreads];
  const int64_t per = (total / k + 63) & ~(int64_t)63;
  int started = 0;
  // the last range, and those whose thread the system refuses or has no memory
  // for, are this thread's own: nothing may leave a C entry, least of all past
  // threads that still run
  int64_t rest = 0;
  try {
    for (; started + 1 < k && rest + per < total; ++started, rest += per)
      th[started] = std::thread(copy_range, src, bytes, n, out, rest, rest + per);
  } catch (const std::exception&) {
  }
  copy_range(src, bytes, n, out, rest, total);
  for (int i = 0; i < started; ++i) th[i].join();
  return RR_OK;
}
