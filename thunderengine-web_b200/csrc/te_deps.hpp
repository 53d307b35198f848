// Dependencies between the kernels of a captured step.
//
// A step captured on one stream is a chain: every kernel waits for the one before it, although
// many do not need it (the faces of a variable in x, y and z; the halo fills of different
// fields; a variable's flux while another variable's halos are filled).  StepDeps sets
// the capture's dependencies before each launch from the memory ranges the launch reads
// and writes, so that the graph holds only the orders the data needs: a reader waits for
// the last writer of every word it reads, a writer for the last writer and for the readers
// since.  The results are those of the chain, word for word: every pair of launches that
// touch a common word, one of them writing, keeps its order.
//
// What bounded the chain: a small grid's step is one kernel latency after another (about
// 1.6 us a launch at 12 x 10 x 8, 333 launches).  One B200, per step, chain -> this: exact
// 12x10x8 505 -> 280 us, exact 128x128x64 1977 -> 1584 us, fused 37x29x13 381 -> 295 us, fused
// 256x256x80 5.40 -> 5.35 ms, recorded full physics (718 launches) 3.84 -> 3.11 ms.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <map>
#include <utility>
#include <vector>

namespace te {

// Device bytes [lo, hi) a launch reads, or (write) may read and write, or (add) only adds to
// with atomics: additions keep no order among themselves.
struct Access {
  uintptr_t lo = 0, hi = 0;
  bool write = false, add = false;
};

inline Access access_words(const void* p, uint64_t words, bool write) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(p);
  return Access{a, a + words * 4, write, false};
}

class StepDeps {
 public:
  explicit StepDeps(cudaStream_t s) : s_(s) {}

  // Runs `launch`, which enqueues work that touches `acc` on the capturing stream, after the
  // launches it depends on and no others.
  template <class F>
  cudaError_t run(const std::vector<Access>& acc, F launch) {
    std::vector<int> after;
    std::vector<int> ids;
    for (const Access& a : acc) {
      if (a.hi <= a.lo) continue;
      const int id = range_id(a.lo, a.hi);
      ids.push_back(id);
      for (int q : ranges_[id].overlap) {
        const Range& r = ranges_[q];
        if (r.writer >= 0) after.push_back(r.writer);
        if (a.write || a.add) after.insert(after.end(), r.readers.begin(), r.readers.end());
        if (!a.add) after.insert(after.end(), r.adders.begin(), r.adders.end());
      }
    }
    const int me = (int)tail_.size();
    std::sort(after.begin(), after.end(), [](int x, int y) { return x > y; });
    after.erase(std::unique(after.begin(), after.end()), after.end());
    // a launch that an already chosen one waits for is waited for through it
    std::vector<uint64_t> reach((me + 64) / 64, 0);
    std::vector<cudaGraphNode_t> nodes;
    for (int d : after) {
      if (reach[d / 64] >> (d % 64) & 1u) continue;
      reach[d / 64] |= 1ull << (d % 64);
      for (size_t w = 0; w < reach_[d].size(); w++) reach[w] |= reach_[d][w];
      nodes.insert(nodes.end(), tail_[d].begin(), tail_[d].end());
    }
    cudaError_t e = set(nodes);
    if (e != cudaSuccess) return e;
    launch();
    cudaStreamCaptureStatus st;
    const cudaGraphNode_t* dep = nullptr;
    size_t n = 0;
    unsigned long long id = 0;
    e = cudaStreamGetCaptureInfo(s_, &st, &id, nullptr, &dep, &n);
    if (e != cudaSuccess) return e;
    if (st != cudaStreamCaptureStatusActive) return cudaErrorStreamCaptureInvalidated;
    tail_.emplace_back(dep, dep + n);  // a launch of nothing passes on what it waited for
    reach_.push_back(std::move(reach));
    size_t q = 0;
    for (const Access& a : acc) {
      if (a.hi <= a.lo) continue;
      Range& r = ranges_[ids[q++]];
      if (a.write) {
        r.writer = me;
        r.readers.clear();
        r.adders.clear();
      } else if (a.add) {
        r.adders.push_back(me);
      } else if (r.readers.empty() || r.readers.back() != me) {
        r.readers.push_back(me);
      }
    }
    return cudaSuccess;
  }

  // Joins every launch: the stream's next work would wait for all of them.
  cudaError_t finish() {
    std::vector<uint64_t> reach((tail_.size() + 63) / 64 + 1, 0);
    std::vector<cudaGraphNode_t> nodes;
    for (int d = (int)tail_.size() - 1; d >= 0; d--) {
      if (reach[d / 64] >> (d % 64) & 1u) continue;
      for (size_t w = 0; w < reach_[d].size(); w++) reach[w] |= reach_[d][w];
      nodes.insert(nodes.end(), tail_[d].begin(), tail_[d].end());
    }
    return set(nodes);
  }

 private:
  struct Range {
    uintptr_t lo, hi;
    int writer = -1;           // the last launch that wrote (part of) it
    std::vector<int> readers;  // launches that read it since
    std::vector<int> adders;   // launches that added to it since
    std::vector<int> overlap;  // the known ranges that share a byte with it, itself included
  };

  int range_id(uintptr_t lo, uintptr_t hi) {
    auto it = id_.find({lo, hi});
    if (it != id_.end()) return it->second;
    const int me = (int)ranges_.size();
    Range r;
    r.lo = lo;
    r.hi = hi;
    for (int q = 0; q < me; q++)
      if (ranges_[q].lo < hi && lo < ranges_[q].hi) {
        r.overlap.push_back(q);
        ranges_[q].overlap.push_back(me);
      }
    r.overlap.push_back(me);
    ranges_.push_back(std::move(r));
    id_[{lo, hi}] = me;
    return me;
  }

  cudaError_t set(std::vector<cudaGraphNode_t>& nodes) {
    std::sort(nodes.begin(), nodes.end());
    nodes.erase(std::unique(nodes.begin(), nodes.end()), nodes.end());
    return cudaStreamUpdateCaptureDependencies(s_, nodes.empty() ? nullptr : nodes.data(), nodes.size(),
                                               cudaStreamSetCaptureDependencies);
  }

  cudaStream_t s_;
  std::vector<Range> ranges_;
  std::map<std::pair<uintptr_t, uintptr_t>, int> id_;
  std::vector<std::vector<cudaGraphNode_t>> tail_;  // per launch: the capture's dependencies after it
  std::vector<std::vector<uint64_t>> reach_;        // per launch: the launches before it, as bits
};

}  // namespace te
