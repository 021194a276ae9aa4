// Register passes of the search: compiled sides, table l (split across
// translation units so that they compile in parallel).
#define VG_PASS_TYPES_ONLY
#include "vesper_regpass.cuh"

namespace vg {

const RegEntry *find_reg_l(int d, int kind) {
    static const RegEntry table[] = {
        RegSide<14, 7, false, kVec | kVal | kPlain | kProb>::entry(),   // 98
        RegSide<9, 11, false, kVec | kVal | kPlain | kProb>::entry(),   // 99
        RegSide<20, 5, false, kVec | kVal | kPlain | kProb>::entry(),   // 100
    };
    return find_in(table, (int)(sizeof(table) / sizeof(table[0])), d, kind);
}

}  // namespace vg
