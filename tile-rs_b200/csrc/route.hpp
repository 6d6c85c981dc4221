// Which kernel a problem runs on, where that depends on its size: host arithmetic only, so that the rules can be looked at
// without a GPU (tests/test_routes.py).  The figures beside a rule are device times in microseconds as graph replays, the
// other side first.
#pragma once

#include <algorithm>
#include <cstdint>

namespace tsm100 {
namespace route {

constexpr int64_t div_up(int64_t a, int64_t b) { return (a + b - 1) / b; }

// 16-bit attention with heads of 32 or 64: the tcgen05 kernel (64-wide form, 256 query rows and 128 keys at a time) or the
// warp-level one (64 query rows).  Up to 64 keys a tcgen05 tile is mostly padding, and its start alone is longer than the
// warp-level kernel's whole work: causal, 2048 heads of 64 keys x 64 61 warp-level, 97 tcgen05, 1 head 6.7 / 7.7; from 65 keys on it
// leads (98.4 / 97.3, 1 head 9.6 / 7.7).  Heads of 32 fill half of its width: there it leads from 129 keys on when it has query
// blocks for all SMs (256 heads of 160 19.1 / 17.7), from 449 on when there are fewer (8 heads of 300 10.0 / 11.8, of 400 13.1 / 13.8, of
// 512 15.6 / 14.1); 2048 heads of 64 keys x 32 31 / 96.
inline bool attention_narrow_on_tcgen05(int32_t head_dim, int64_t seq_kv, int64_t query_blocks, int sms) {
  if (head_dim == 64) return seq_kv > 64;
  return seq_kv > (query_blocks > sms ? 128 : 448);
}

}  // namespace route
}  // namespace tsm100
