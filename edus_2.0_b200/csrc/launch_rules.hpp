// Which launch serves a call, by sizes alone (host code, no CUDA headers).
#pragma once
#include <cstddef>

namespace edus {

// Threads of a plane CTA in the device-buffer right-hand side.  With more planes
// than SMs, 256, so that two CTAs (128 registers a thread) share an SM and the planes run
// in one wave where they would take two: 196 planes of 48 x 48 with HSEX 50 -> 32 us.
// A plane too large for two CTAs an SM has it to itself either way and keeps 512:
// 169 plane pairs of 65 x 56, the whole call 147 us against 161 with 256.
// (cta_reserved: what the system takes of an SM's shared memory for each CTA.)
inline int rhs_plane_threads(int planes, int sms, size_t plane_smem, size_t sm_smem, size_t cta_reserved) {
    return planes > sms && 2 * (plane_smem + cta_reserved) <= sm_smem ? 256 : 512;
}

// Estimated microseconds of a stage in launches, for problems where nothing but
// latency counts: the launches and ten passes over the solves' states (`elements`)
// at about 2 TB/s.  Two launches take 9 us at the least.  Where planes are spread over
// many CTAs there are four: measured 17 to 19 us replayed from a CUDA graph (RK4, long
// calls) and 24 to 27 launched, with HSEX 25 to 27 and 33 to 35; Adams-Bashforth has
// no graphs.  The choice must not depend on a call's length, or a split call would
// round differently, so RK4 counts near its replayed time.
inline double staged_stage_us(bool spread, bool hsex, bool rk, double elements) {
    const double launches = !spread ? 9.0 : (hsex ? 26.0 : 20.0) + (rk ? 0.0 : 4.0);
    return launches + 160.0 * elements / 2.0e6;
}

// State (all solves) from which the TMA-fed commutator serves without HSEX.  Below,
// the launch that writes H0 + E.xi costs as much as the tiles it relieves: RK4 from
// 12 MB gains 6 to 26% over 12 to 24 bands.  Adams-Bashforth writes H every step
// instead of twice in four stages, and 16 bands fill the direct-load kernel's 8 x 8
// tiles: 28 x 28, four solves (12.2 MB) 82 -> 87 us a step, and even or faster from
// 14 MB (64 x 64, 16 MB: 105 -> 98; 15 bands, 63 x 60, 13 MB: 87 -> 81).
inline size_t ws_ipa_bytes(int nb, bool adams) { return (size_t)(adams && nb == 16 ? 14 : 12) << 20; }

// Observables: a thread per k point (few bands) or a CTA per k point.  A thread
// does nb^3 dependent products whatever the grid, a CTA spreads them: with
// velocities and populations, a call of 4 bands takes 50 us against 49 (24 x 24) and
// 52 against 68 (120 x 120), of 5 bands 62 against 49 and 64 against 75, of 8 bands
// 86 against 47 and 96 against 99.  Up to four bands the thread never loses by more
// than the two calls' spread; from five on the CTA is what is never slower than
// the form before both (an atomic a value from every k point).
constexpr int kObsThreadBands = 4;
inline bool obs_by_thread(int nb) { return nb <= kObsThreadBands; }

}  // namespace edus
