// Numbers, slots and ready words of the enumeration's queue of handed-off
// records, shared by the kernel, the host code and host tests.
//
// The queue is a ring: record number t lies in slot t mod kQueueSlots, use
// t / kQueueSlots of that slot.  Its ready word says free for that use, then
// published until its ticket holder has read it, then free for the next use.  A
// holder that leaves before its record is reserved marks the word: the record,
// if it is written, is nobody's in this pass.
// Numbers wrap from 2^32 - 1 to 0, and uses with them: the slot count divides
// 2^32.
#pragma once
#include <stdint.h>

namespace fsig {

constexpr uint32_t kQueueSlots = 1u << 20;

__host__ __device__ __forceinline__ uint32_t queue_slot(uint32_t number) { return number % kQueueSlots; }
// the slot's ready word while it is free for record `number`, and from its publication on
__host__ __device__ __forceinline__ uint32_t ready_free(uint32_t number) { return 2 * (number / kQueueSlots); }
__host__ __device__ __forceinline__ uint32_t ready_published(uint32_t number) { return ready_free(number) + 1; }
// once it is read: free for the slot's next record
__host__ __device__ __forceinline__ uint32_t ready_next(uint32_t number) { return ready_free(number + kQueueSlots); }
// Records of one hand-off, at most: 32 pieces of a range and a buffer's entries.
constexpr uint32_t kHandOff = 32 + 128;
// The record of a warp that left is not read in the pass, so its slot must not
// come round: once one has left, records are reserved only up to the tail of
// that moment plus this.  Every warp may reserve one hand-off beyond (a warp
// checks the limit, then adds), and hold one ticket beyond the records: a full
// ring in all.  (Half a ring as the limit, right for hand-offs of up to 64
// records, was not for 160: 4,864 warps reserve 778,240.)
__host__ __device__ constexpr uint32_t queue_room(uint32_t warps) { return kQueueSlots - warps * (kHandOff + 1); }
// Warps of one launch, at most; a GB300 holds 4,864.
constexpr uint32_t kQueueWarps = kQueueSlots / 8 * 7 / (kHandOff + 1);

// added to the free word by a holder that left; publishing sets the low bit only
constexpr uint32_t kHolderLeft = 0x80000000u;
__host__ __device__ __forceinline__ bool ready_writable(uint32_t word, uint32_t number) {
  return (word & ~kHolderLeft) == ready_free(number);
}

// whether number a comes after number b (they are less than 2^31 apart)
__host__ __device__ __forceinline__ bool queue_after(uint32_t a, uint32_t b) { return int32_t(a - b) > 0; }

}  // namespace fsig
