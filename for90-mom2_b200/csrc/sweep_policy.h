// Which contexts of one sweep factorise on a single stream (host code only).
#pragma once

namespace mom {

// Contexts of one sweep on one device from which on each factorises on one
// stream.  The device serves eight queues of launches: a second branch per
// context makes contexts wait for one another.  Sweeps of up to 3,840 unknowns,
// with and without the branch: 4 contexts 172 and 192 ms, 8 contexts 149 and 149
// (four particles) and 103 and 90 (two), 12 contexts 147 and 138, 16 contexts 144
// and 127.
constexpr int kCrowd = 8;

// crowded[i]: context i shares its device (device[i], negative: no context) with
// others to kCrowd or more in all.
inline void crowded_contexts(int n, const int *device, bool *crowded) {
  for (int i = 0; i < n; i++) {
    int same = 0;
    for (int k = 0; k < n; k++) same += device[i] >= 0 && device[k] == device[i];
    crowded[i] = same >= kCrowd;
  }
}

}  // namespace mom
