// Time blocks of the batched schedules: how T steps of a grid are split into
// launches (or work items) of several fused steps each. Host code only.
#pragma once
#include <vector>

namespace gbs {

// Blocks of T steps: blocks of degree bs plus single steps, with as many
// blocks as T has parity (launch k reads plane k%2).
inline std::vector<int> batch_blocks(int T, int bs) {
  std::vector<int> out;
  if (T <= 0) return out;
  int n = T / bs, r = T - n * bs;
  if (((n + r) - T) % 2 != 0) {  // only possible for even bs
    if (n > 0) {
      --n;
      r += bs;
    }
  }
  for (int i = 0; i < n; ++i) out.push_back(bs);
  for (int i = 0; i < r; ++i) out.push_back(1);
  return out;
}

// Blocks of T steps for the layered schedule: what is left over by full
// blocks of bs steps first, so that the grids of a stencil soon run at the
// same degree, then the full blocks; as many blocks as T has parity, for
// which the rest, or a full block, is split in two. For odd T the last block
// has the steps that batch_blocks gives it at the persistent schedule's
// degree: the plane without the result keeps the state before it, from which
// a run of odd T that is repeated starts, under every schedule.
inline std::vector<int> layered_blocks(int T, int bs, int persistent_bs) {
  std::vector<int> out;
  if (T <= 0 || bs < 1) return out;
  const int last = T % 2 ? batch_blocks(T, persistent_bs).back() : 0;
  T -= last;  // an even rest
  int full = T / bs;
  const int rest = T - full * bs;
  auto halves = [&](int x) {
    out.push_back((x + 1) / 2);
    out.push_back(x / 2);
  };
  if (T == 0) {
  } else if ((full + (rest > 0) - T) % 2 == 0) {
    if (rest > 0) out.push_back(rest);
  } else if (rest >= 2) {
    halves(rest);
  } else {  // a full block goes, and one or three blocks take its steps
    --full;
    halves(bs);
    if (rest > 0) out.push_back(rest);
  }
  out.insert(out.end(), full, bs);
  if (last > 0) out.push_back(last);
  return out;
}

}  // namespace gbs
