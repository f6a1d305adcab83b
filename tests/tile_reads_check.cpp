// Check of tiles_read_mutually (vt_common.h), compiled and run by
// tests/test_one_way_meshes.py on the CPU: tables of neighbours whose tiles do
// and do not read each other mutually, whatever the elements' own links.
#include <cstdio>
#include <numeric>
#include <vector>

#include "vt_common.h"

namespace {

int failures = 0;

void expect(const char* name, bool want, const std::vector<int32_t>& nb, int per_tile) {
  const int K = static_cast<int>(nb.size() / 3), ntiles = (K + per_tile - 1) / per_tile;
  std::vector<int> column(K);
  std::iota(column.begin(), column.end(), 0);
  const bool got = vt::tiles_read_mutually(K, nb.data(), column.data(), per_tile, ntiles);
  std::printf("%s %s\n", got == want ? "OK" : "WRONG", name);
  failures += got != want;
}

}  // namespace

int main() {
  // 6 elements in a ring, in tiles of two
  std::vector<int32_t> ring;
  for (int e = 0; e < 6; ++e) ring.insert(ring.end(), {(e + 1) % 6, (e + 5) % 6, e});
  expect("ring", true, ring, 2);
  expect("one tile", true, ring, 64);
  // 6 elements that read the next one only: mutual in tiles of three, not of two
  std::vector<int32_t> next;
  for (int e = 0; e < 6; ++e) next.insert(next.end(), {(e + 1) % 6, (e + 1) % 6, e});
  expect("one way round, three tiles", false, next, 2);
  expect("one way round, two tiles", true, next, 3);
  // two separate rings; element 1 of the first reads the second
  std::vector<int32_t> two;
  for (int e = 0; e < 8; ++e) two.insert(two.end(), {e / 4 * 4 + (e + 1) % 4, e / 4 * 4 + (e + 3) % 4, e});
  expect("two rings", true, two, 2);
  two[3 * 1 + 2] = 6;
  expect("two rings, one link", false, two, 2);
  two[3 * 7 + 2] = 0;  // and another element of that tile reads back
  expect("two rings, a link either way", true, two, 2);
  return failures != 0;
}
