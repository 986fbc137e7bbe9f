// How the single-GPU reductions cut their vectors: the argument block of the kernels, and the host's side of it.
//
// Plain C++, so that the self-test (tools/planner_selftest.cpp) replays every access of every thread for what these
// functions make of a vector, and finds each inside it.
#pragma once
#include <stddef.h>
#include <stdint.h>

#include "../api/ft_types.h"

namespace ftk {

// What a call does about its neighbours on the stream: its first `ahead` CTAs fetch their sources before the kernel in front
// has ended, and those from `ask` on ask for the one behind.  Why, and why these sizes: pdl.cuh.  `moved`: the call's bytes;
// `fetched`: bytes of sources per CTA; `ctas`: of 128 threads each.
struct Seam {
  uint32_t ahead, ask;
};
constexpr uint32_t kNoCta = ~0u;
inline Seam seam_of(unsigned long long moved, unsigned fetched, unsigned long long ctas) {
  if (moved < (50u << 20)) return {0, kNoCta};
  const unsigned asking = moved < (100u << 20) ? 148 * 16 : 148 * 20;
  return {(12u << 20) / fetched, ctas > asking ? (uint32_t)(ctas - asking) : 0};
}

// One launch covers a whole vector: the body in 32- or 16-byte vectors, and the elements in front of and behind it
// (the edges) one by one in a CTA of their own (the last one; in calls that fetch ahead by the first CTA, beside its part of
// the body), so that neither a ragged length nor a slice that starts off a vector boundary costs a second launch or takes
// the rest of the vector off the vector loads.
struct NwayArgs {
  const void* src[FT_MAX_FANIN];  // start of the body in every source
  void* dst;
  unsigned long long nvec;    // body length, in the kernel's vectors
  unsigned long long nbody;   // ... and in scalar units (see ScalarOp)
  int n;
  uint16_t head, edge;        // scalar units in front of the body; in front of and behind it together
  uint8_t shift[FT_MAX_FANIN];  // shifted kernels: bytes by which source k's body lies behind a 16-byte (realign: 32-byte) boundary
  Seam seam;                  // set at the launch
  float scale;                // scaled kernels
  uint32_t fill[3];           // to a size that is cheap to launch with (pdl.cuh)
};

// CTAs of a launch that covers the body once, `per_cta` vectors each; and with the one for the edges.
inline unsigned long long body_ctas(const NwayArgs& a, unsigned per_cta) { return (a.nvec + per_cta - 1) / per_cta; }
inline unsigned long long nway_grid(const NwayArgs& a, unsigned per_cta) { return body_ctas(a, per_cta) + (a.edge && !a.seam.ahead); }
constexpr unsigned kWideThreads = 128;                  // wide and scaled kernels: a vector each
constexpr unsigned kRealignThreads = 128, kRealignPerCta = kRealignThreads / 32 * 31;   // a warp stores 31 of the 32 it sums
inline bool shift_long(const NwayArgs& a) { return a.nvec >= (3u << 20) / 16; }   // shifted kernel: 64 threads, two vectors each; else 128, one

// Cut the vector for the 32-byte kernel: possible when every pointer has the same offset from a 32-byte boundary
// (a slice of a flat buffer reduced into the same slice of another, or whole tensors).
inline bool layout_wide(const NwayArgs& in, size_t bytes, size_t unit, NwayArgs* out) {
  uintptr_t differ = 0;
  for (int k = 0; k < in.n; ++k) differ |= (uintptr_t)in.src[k] ^ (uintptr_t)in.dst;
  if (differ & 31) return false;
  // The body starts on a 128-byte line where that is possible, or each 1 KiB request of a warp touches nine lines
  // instead of eight: bf16 x2 of 4 M one element off, in L2, took 3.2 us from the next 32 bytes and 2.9 from the next line.
  const size_t to = (differ & 127) == 0 && bytes >= 4096 ? 128 : 32;
  const size_t head = (to - ((uintptr_t)in.dst & (to - 1))) & (to - 1);
  if (bytes < head + 32) return false;
  *out = in;
  out->nvec = (bytes - head) / 32;
  out->nbody = out->nvec * 32 / unit;
  out->head = (uint16_t)(head / unit);
  out->edge = (uint16_t)((bytes - out->nvec * 32) / unit);
  for (int k = 0; k < in.n; ++k) out->src[k] = (const unsigned char*)in.src[k] + head;
  out->dst = (unsigned char*)in.dst + head;
  return true;
}
// Cut it for the realigning kernel: the sources agree modulo 32, the result lies elsewhere.  The body is what the
// result's whole 32-byte units between the first and the last whole unit of the sources hold.
inline bool layout_realign(const NwayArgs& in, size_t bytes, size_t unit, NwayArgs* out) {
  const uintptr_t phase = (uintptr_t)in.src[0] & 31;
  for (int k = 1; k < in.n; ++k)
    if (((uintptr_t)in.src[k] & 31) != phase) return false;
  const size_t first = (32 - phase) & 31;   // bytes in front of the sources' first whole unit
  const size_t shift = (32 - (((uintptr_t)in.dst + first) & 31)) & 31, head = first + shift;
  if (shift == 0 || bytes < first + 64) return false;
  *out = in;
  out->nvec = (bytes - first) / 32 - 1;
  out->nbody = out->nvec * 32 / unit;
  out->head = (uint16_t)(head / unit);
  out->edge = (uint16_t)((bytes - out->nvec * 32) / unit);
  out->shift[0] = (uint8_t)shift;
  for (int k = 0; k < in.n; ++k) out->src[k] = (const unsigned char*)in.src[k] + head;
  out->dst = (unsigned char*)in.dst + head;
  return true;
}
// Cut it on the result's 16-byte boundaries for the shifted kernel.  A source that lies s bytes behind such a
// boundary is read from s bytes before the body to 16 - s bytes behind it; the body is kept small enough for these
// to be the vector's own bytes.  A vector too short for that is all edges.
inline void layout_shift(const NwayArgs& in, size_t bytes, size_t unit, NwayArgs* out) {
  *out = in;
  size_t head = (16 - ((uintptr_t)in.dst & 15)) & 15, widest = 0;
  for (int k = 0; k < in.n; ++k) {
    out->shift[k] = (uint8_t)(((uintptr_t)in.src[k] + head) & 15);
    if (out->shift[k] > widest) widest = out->shift[k];
  }
  if (widest > head) head += 16;
  unsigned long long nvec = bytes > head ? (bytes - head) / 16 : 0;
  for (int k = 0; k < in.n; ++k)
    if (out->shift[k]) {
      const unsigned long long whole = (bytes > head ? bytes - head + out->shift[k] : 0) / 16;
      const unsigned long long fits = whole ? whole - 1 : 0;
      if (fits < nvec) nvec = fits;
    }
  if (!nvec) {   // no body, and with it no vector behind the body for the kernel to look at
    head = 0;
    for (int k = 0; k < in.n; ++k) out->shift[k] = 0;
  }
  out->nvec = nvec;
  out->nbody = nvec * 16 / unit;
  out->head = (uint16_t)(head / unit);
  out->edge = (uint16_t)((bytes - nvec * 16) / unit);
  for (int k = 0; k < in.n; ++k) out->src[k] = (const unsigned char*)in.src[k] + head;
  out->dst = (unsigned char*)in.dst + head;
}

// First element from which every source lies on a boundary of `sa` bytes and the output on one of `da`, or -1.
inline int common_head(const NwayArgs& a, size_t is, size_t os, size_t sa, size_t da) {
  for (size_t h = 0; h < sa / is; ++h) {
    bool ok = ((uintptr_t)a.dst + h * os) % da == 0;
    for (int k = 0; ok && k < a.n; ++k) ok = ((uintptr_t)a.src[k] + h * is) % sa == 0;
    if (ok) return (int)h;
  }
  return -1;
}

// Cut it for the scaled kernel: units of 32 bytes of every source, E elements, from an element that lies on a boundary in
// all of them and in the result.  `wide`: boundaries for 256-bit accesses, else for 128-bit ones.  False: no such element.
inline bool layout_scaled(const NwayArgs& in, unsigned long long len, bool in_bf16, bool out_bf16, NwayArgs* out, bool* wide) {
  const unsigned E = in_bf16 ? 16 : 8;
  const size_t is = in_bf16 ? 2 : 4, os = out_bf16 ? 2 : 4, da = in_bf16 || !out_bf16 ? 32 : 16;
  int head = len >= 4096 / is ? common_head(in, is, os, 128, da) : -1;   // whole lines: see layout_wide
  if (head < 0) head = common_head(in, is, os, 32, da);
  *wide = head >= 0;
  if (head < 0) head = common_head(in, is, os, 16, 16);
  if (head < 0) return false;
  *out = in;
  out->nvec = len >= head + E ? (len - head) / E : 0;   // shorter: all edges
  out->nbody = out->nvec * E;
  out->head = (uint16_t)(out->nvec ? head : 0);
  out->edge = (uint16_t)(len - out->nbody);
  for (int k = 0; k < in.n; ++k) out->src[k] = (const unsigned char*)in.src[k] + out->head * is;
  out->dst = (unsigned char*)in.dst + out->head * os;
  return true;
}

}  // namespace ftk
