#pragma once
// The node pairs that a decision of the dual walk opens a pair (a, b) into, and
// the rule by which they go into the next frontier.  Plain C++ too, so that the
// rule is checked on the host.
#include <stdint.h>

#ifdef __CUDACC__
#define JB_WALK_FN __host__ __device__ __forceinline__
#else
#define JB_WALK_FN inline
#endif

enum : int { kNone = 0, kSelf = 1, kFar = 2, kNear = 3, kSplitA = 4, kSplitB = 5 };

// Pairs that walk_children writes: (A, A) has both children with themselves and
// with one another, in both orders in the directed walk.
template <bool DIRECTED>
JB_WALK_FN unsigned walk_child_count(int decision) {
  return decision == kSelf ? (DIRECTED ? 4 : 3) : (decision >= kSplitA ? 2 : 0);
}

// Writes them to next[at], next[at + 1], ..., each under its own bound: a step
// reads every place below min(pairs appended, cap), so one that is left out
// because its neighbour lies past the end would be read as it was before.
template <bool DIRECTED, typename Pair>
JB_WALK_FN void walk_children(int decision, int a, int b, const int* left, const int* right, Pair* next, int64_t at,
                              int64_t cap) {
  auto put = [&](int k, int x, int y) {
    if (at + k < cap) next[at + k] = Pair{x, y};
  };
  if (decision == kSelf) {
    const int l = left[a], r = right[a];
    put(0, l, l);
    put(1, r, r);
    put(2, l, r);
    if (DIRECTED) put(3, r, l);
  } else if (decision == kSplitA) {
    put(0, left[a], b);
    put(1, right[a], b);
  } else if (decision == kSplitB) {
    put(0, a, left[b]);
    put(1, a, right[b]);
  }
}
