// Words of the messages between the CTAs of the complex128 panel (zpanel.cu).
//
// Every 64-bit word of a message carries the tag of its column, so that a reader
// that sees the tag has the data.  The tag is 21 bits wide: column + 1, no two
// columns of a factorisation share one.  With a shorter one that comes round
// again, what a CTA left in its slot when it last had a row could pass for
// the current column's: a CTA may be absent for some panels and come back
// (beyond 32 rows a CTA the grid shrinks with the panel and grows when the rows
// per CTA drop).
// A complex128 number is 128 of the 129 bits that three words leave, a candidate
// 86 of two words' (64 of its size, 22 of its position): nothing is rounded.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define MGT_HD __host__ __device__ __forceinline__
#else
#define MGT_HD inline
#endif

namespace mgt {
namespace zp {

constexpr int kTagShift = 43;
constexpr int kMaxColumns = (1 << 21) - 2;     // tags 1 .. 2^21 - 1 (zero: a cleared slot)
constexpr int kNoPos = (1 << 22) - 1;          // position of a CTA without a candidate
constexpr uint64_t kWordData = (1ull << kTagShift) - 1;

MGT_HD uint64_t column_tag(int column) { return (uint64_t)(uint32_t)(column + 1) << kTagShift; }
MGT_HD bool has_tag(uint64_t tag, uint64_t w) { return ((w ^ tag) >> kTagShift) == 0; }

// the bits x, y of a number's parts
MGT_HD void pack_number(uint64_t tag, uint64_t x, uint64_t y, uint64_t* w) {
  w[0] = tag | (x >> 21);
  w[1] = tag | ((x & 0x1FFFFFull) << 22) | (y >> 42);
  w[2] = tag | (y & 0x3FFFFFFFFFFull);
}
MGT_HD void unpack_number(const uint64_t* w, uint64_t* x, uint64_t* y) {
  *x = ((w[0] & kWordData) << 21) | ((w[1] & kWordData) >> 22);
  *y = ((w[1] & 0x3FFFFFull) << 42) | (w[2] & 0x3FFFFFFFFFFull);
}

// a candidate: its size as an ordered integer, its position in the panel (< kNoPos)
MGT_HD void pack_key(uint64_t tag, uint64_t key, int pos, uint64_t* w) {
  w[0] = tag | (key >> 21);
  w[1] = tag | ((key & 0x1FFFFFull) << 22) | (uint64_t)(uint32_t)pos;
}
MGT_HD void unpack_key(uint64_t w0, uint64_t w1, uint64_t* key, int* pos) {
  *key = ((w0 & kWordData) << 21) | ((w1 & kWordData) >> 22);
  *pos = (int)(w1 & 0x3FFFFFull);
}

}  // namespace zp
}  // namespace mgt
