// Register passes of the search: compiled sides, table j (split across
// translation units so that they compile in parallel).
#define VG_PASS_TYPES_ONLY
#include "vesper_regpass.cuh"

namespace vg {

const RegEntry *find_reg_j(int d, int kind) {
    static const RegEntry table[] = {
        RegSide<27, 3, false, kVec | kVal | kPlain | kProb>::entry(),   // 81
        RegSide<12, 7, false, kVec | kVal | kPlain | kProb>::entry(),   // 84
        RegSide<8, 11, false, kVec | kVal | kPlain | kProb>::entry(),   // 88
    };
    return find_in(table, (int)(sizeof(table) / sizeof(table[0])), d, kind);
}

}  // namespace vg
