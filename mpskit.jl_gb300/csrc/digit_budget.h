// When an FP64 operator may keep the digits of its constants.
//
// They are a convenience: without them the constants are cut again in every application.  They
// take 1.75 times the constants (3.5 times a complex right operand), so they must not be what
// makes a solve run out of memory that fitted without them.
#pragma once

#include <cstdint>

namespace gb {

// Sets of at most this (of 280 GB) are kept without asking: a query of the free memory takes 9 us,
// an application of an operator of this size 15 to 60.
constexpr uint64_t DIGITS_SMALL = 64ull << 20;

// Vectors of the operator that its solves may still allocate: a basis at the largest dimension they
// accept (64 + 2), the restart's copies (39), the matvec's result, x in digits (up to 10) and a few
// of the caller's own.
constexpr uint64_t DIGITS_VECTORS = 128;

// `bytes` of digits against the free memory of the device and the unused part of the stream-ordered
// pool, which the digits are taken from first.  `need`: what the operator's solves may still
// allocate.  Beyond that they leave as much as they take, for operators built later.
inline bool digits_affordable(uint64_t bytes, uint64_t need, uint64_t free_bytes,
                              uint64_t pool_unused) {
  if (bytes <= DIGITS_SMALL) return true;
  const uint64_t fresh = bytes > pool_unused ? bytes - pool_unused : 0;
  if (fresh > free_bytes) return false;
  const uint64_t left = free_bytes - fresh;
  return left >= need && left - need >= bytes;
}

}  // namespace gb
