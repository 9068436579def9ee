// Places in a list of limited room, handed out by one counter that goes on counting when the list
// is full. Plain C++ beside the operation on the counter, so that it also compiles for the host.
#pragma once

#ifdef __CUDACC__
#define OTM_PLACES __host__ __device__ __forceinline__
#else
#define OTM_PLACES inline
#endif

namespace otm {

// 64 bits: as many as the rasterizer can ask for (2^31 faces times 2^32 pixels) do not wrap it. A mesh
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

}  // namespace otm
