// Asks for places of a short list with its counter near the limits of 31 and 32 bits and at the
// most a call can reach. Prints the number of answers that are places of the list.
#include <cstdio>
#include <initializer_list>

#include "place_list.cuh"

int main() {
  const int room = 65536;
  int places = 0;
  for (unsigned long long start : {0ull, 1ull << 31, 1ull << 32, 3ull << 31, 1ull << 62}) {
    otm::PlaceCount counter = (otm::PlaceCount)(start ? start - 1000 : 0);
    for (int k = 0; k < 100000; ++k) places += otm::take_place(room, [&] { return counter++; }) != room;
  }
  std::printf("%d\n", places);
}
