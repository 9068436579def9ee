// Rules that keep counts and places in range. Plain C++, so that they also compile for the host.
#pragma once

#include <climits>

#ifdef __CUDACC__
#define OTM_PLACES __host__ __device__ __forceinline__
#else
#define OTM_PLACES inline
#endif

namespace otm {

// Places in a list of limited room, handed out by one counter that goes on counting when the list
// is full. 64 bits: as many as the rasterizer can ask for (2^31 faces times 2^32 pixels) do not wrap it. A mesh
// of 256^2 quads with random corners asks 5.7e9 times when it is drawn at 1024^2, and a 32-bit counter
// that has wrapped hands out places before the list.
using PlaceCount = unsigned long long;

// A place of the list, or `room` when it is full. next() adds one to the counter and returns the
// number of places asked for before.
template <class Next>
OTM_PLACES int take_place(int room, Next next) {
  const PlaceCount i = next();
  return i < (PlaceCount)room ? (int)i : room;
}

// A warp that pools the lists of its 32 lanes numbers their entries through: it takes this much of
// what is left of each list at a time, so that the numbers stay within an int. (A bin of a mesh that
// has collapsed into few of them lists up to all n^2 faces, 2^26 at 8192^2.)
constexpr int POOL_WINDOW = INT_MAX / 32;
OTM_PLACES int pool_part(int left) { return left < POOL_WINDOW ? left : POOL_WINDOW; }

}  // namespace otm
