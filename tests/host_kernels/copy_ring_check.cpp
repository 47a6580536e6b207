// The copying thread of the shared-memory ring (csrc/copy_ring.cuh) against a
// model of its barriers: readers that release a slot behind every block, that
// stop after some blocks, and copies that never land.
#include <cstdio>
#include <set>
#include <vector>

#include "cuda_runtime.h"

namespace c3d {

struct Bar { int id; };              // full: 0 .. RING-1, empty: 100 ..
constexpr int RING = 8;
using Slot = int;                    // a slot is its number

struct Model {
  int readers = 0;                   // blocks the readers release
  int lost = -1;                     // this block's copy never lands
  std::vector<int> issued;           // blocks in order
  std::set<int> flight;              // copies that nobody has seen land
  int armed[RING] = {};              // arrivals expected per slot
  bool misuse = false, overwritten = false;
};
static Model M;
static const int* g_src[1000];
static int g_blocks[1000];

inline bool mbar_wait(Bar* b, unsigned parity, long long) {
  if (b->id >= 100) {                // a slot's `empty`: use u of it has been read
    const int slot = b->id - 100, g = (int)M.issued.size() - RING;   // the block before the next one there
    if (g < 0 || g % RING != slot || parity != (unsigned)(g / RING & 1)) { M.misuse = true; return false; }
    if (g >= M.readers || g == M.lost) return false;
    M.flight.erase(g);
    return true;
  }
  int g = -1;                        // the last block issued to the slot
  for (int k : M.issued) if (k % RING == b->id) g = k;
  if (g < 0 || parity != (unsigned)(g / RING & 1)) { M.misuse = true; return false; }
  if (g == M.lost) return false;
  M.flight.erase(g);
  return true;
}
inline void mbar_arrive_expect_tx(Bar* b, unsigned) { M.armed[b->id]++; }
inline void bulk_load(Slot s, const int* src, unsigned, Bar* b) {
  const int g = *src;
  if (s != b->id || g % RING != s || g != (int)M.issued.size()) M.misuse = true;
  if (M.flight.count(g - RING)) M.overwritten = true;
  M.issued.push_back(g);
  M.flight.insert(g);
}

}  // namespace c3d

#include "../../channel3d_parallel_b200/csrc/copy_ring.cuh"

int main() {
  using namespace c3d;
  Slot ring[RING];
  Bar full[RING], empty[RING];
  for (int k = 0; k < RING; ++k) { ring[k] = k; full[k].id = k; empty[k].id = 100 + k; }
  for (int k = 0; k < 1000; ++k) { g_blocks[k] = k; g_src[k] = g_blocks + k; }
  auto src = [](int g) { return g_src[g]; };
  int bad = 0, runs = 0;
  for (int total : {0, 1, 7, 8, 9, 16, 17, 145})
    for (int readers : {0, 1, 5, 8, 20, 1000})
      for (int lost : {-1, 0, 6, total - 1}) {
        if (lost >= total) continue;
        M = Model{};
        M.readers = readers;
        M.lost = lost;
        const bool ok = copy_ring<RING>(total, ring, full, empty, 64, 1, src);
        const int could = lost < 0 ? readers : (lost < readers ? lost : readers);   // releases that can come
        const int want = total < could + RING ? total : could + RING;
        const bool fine = want == total && lost < 0;
        std::set<int> left = M.flight;
        if (lost >= 0) left.erase(lost);             // waited for as well, but it never comes
        if (ok != fine || (int)M.issued.size() != want || !left.empty() || M.misuse || M.overwritten) {
          std::printf("total %d readers %d lost %d: ok %d issued %d of %d in flight %d\n", total, readers, lost,
                      (int)ok, (int)M.issued.size(), want, (int)left.size());
          ++bad;
        }
        ++runs;
      }
  std::printf("%d runs, %d mismatches\n", runs, bad);
  return bad != 0;
}
