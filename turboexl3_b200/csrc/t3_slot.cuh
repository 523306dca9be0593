// A sorted row-slot's bank and its expert's number inside that bank in one word, as the prefill chain hands them from the routing
// to the prepares.
#pragma once

#include "t3_lane.cuh"

namespace t3 {

// `bits` of the word are the expert's: 24 beside a bank's number (a layer of several banks has 2^24 experts at most, which its entry
// point checks), 31 where there is one bank (its experts are an int).
struct SlotId {
    uint32_t bits;
    static T3_HD uint32_t bits_for(uint32_t banks) { return banks > 1u ? 24u : 31u; }
    T3_HD uint32_t pack(uint32_t bank, uint32_t expert) const { return (bank << bits) | expert; }
    T3_HD uint32_t bank(uint32_t id) const { return id >> bits; }
    T3_HD uint32_t expert(uint32_t id) const { return id & ((1u << bits) - 1u); }
};

}  // namespace t3
