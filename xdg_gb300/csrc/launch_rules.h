// launch_rules.h -- waits of the particle loops by batch size, where the
// tuning keys are at their defaults; other values of a key are taken as they
// are.  Host code without CUDA, so that it can be checked as such.
#pragma once

#include <algorithm>
#include <cstdint>

namespace xdgcu {

constexpr int32_t kFlushWait = 4;           // trace_flush_wait
constexpr int32_t kTransportEventWait = 4;  // transport_event_wait

// a particle for every lane of 16 warps on each of `sms` SMs
inline int64_t full_batch(int sms) { return (int64_t)sms * 16 * 32; }

// SurfArgs::flush_wait of the surface particle loop.  Where every lane has a
// particle, the others' work covers a longer wait for fuller drains.  With
// event_wait 20 a wait for 12 lanes leaves two lanes searching at the least,
// and beyond that sum of 32 lanes nothing is left (1e6 particles of the
// nested spheres, ms with 8 / 12 / 16 lanes: 73.9 / 70.4 / 72.2, 3e6 191 / 183 /
// 185, 200,000 29.2 / 28.2 / 28.2; event_wait 24 with 12: 85.7).
inline int32_t particle_flush_wait(int32_t key, int32_t event_wait, bool mixed, int64_t n, int sms) {
  if (key != kFlushWait || !mixed || n < full_batch(sms)) return key;
  return std::max(key, std::min(12, 32 - event_wait));
}

// TransportArgs::event_wait.  Waiting for fuller batches of collisions pays
// once every lane has a particle; before that the lanes that wait are what
// the launch waits for (ms with 1 / 2 / 4 lanes, mixed: 20,000 particles 11.5 /
// 12.1 / 12.2, 200,000 25.7 / 23.8 / 23.6; FP64: 14.8 / 15.6 / 15.8 and 34.0 / 32.2 /
// 32.6), and, mixed, fuller ones where a lane runs many particles (ms with 4 /
// 8 lanes: 600,000 particles 38.8 / 38.6, 1e6 53.6 / 51.7, 3e6 128.8 / 118.0; FP64
// 600,000 52.4 / 53.6).
inline int32_t transport_event_wait(int32_t key, bool mixed, int64_t n, int sms) {
  if (key != kTransportEventWait) return key;
  if (n < full_batch(sms)) return 1;
  return mixed && n >= 8 * full_batch(sms) ? 8 : key;
}

}  // namespace xdgcu
