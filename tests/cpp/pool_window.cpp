// Numbers the entries of 32 lists through, a window of each at a time, as a warp of the point
// locator does; prints whether every window's numbers stay within an int and whether the
// windows cover the lists.
#include <climits>
#include <cstdio>
#include <cstdlib>

#include "place_list.cuh"

int main(int argc, char** argv) {
  int left[32];
  long long want = 0, got = 0;
  for (int l = 0; l < 32; ++l) want += left[l] = std::atoi(argv[1 + l % (argc - 1)]);
  bool fits = true;
  for (bool any = true; any;) {
    long long upto = 0;
    any = false;
    for (int l = 0; l < 32; ++l) {
      const int part = otm::pool_part(left[l]);
      upto += part;
      left[l] -= part;
      any |= left[l] > 0;
    }
    fits &= upto <= INT_MAX;
    got += upto;
  }
  std::printf("%d %d\n", fits ? 1 : 0, got == want ? 1 : 0);
}
