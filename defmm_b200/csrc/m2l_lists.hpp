// Compaction of the M2L lists (m2l_lists.cu).
#pragma once

#include <cstdint>
#include <string>
#include <vector>

#include "device_slab.hpp"

namespace dfb {

// From the CSR of the M2L lists on the device (ptr: nT + 1, src: nent source
// slots): the target slots with a list in tlist (their list pointers, still
// into src, in cptr with one past the last), the source slots that occur in
// slist, both in slot order, and src rewritten to positions in slist.
// atT / atS: slot numbers (<= nT / <= nS), replaced by how many listed slots
// lie before each.  Room: nT + 1, nT and nS entries; scratch is what slab has
// free, or given back.  0, -4 or -5 (out of device memory) with err set.
int device_m2l_lists(const int64_t* ptr, int32_t* src, int64_t nent, int64_t nT, int64_t nS,
                     std::vector<int64_t>& atT, std::vector<int64_t>& atS, int64_t* cptr, int32_t* tlist,
                     int32_t* slist, DeviceSlab& slab, std::string& err);

}  // namespace dfb
