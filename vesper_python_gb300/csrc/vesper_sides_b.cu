// Register passes of the search: compiled sides, table b (split across
// translation units so that they compile in parallel).
#define VG_PASS_TYPES_ONLY
#include "vesper_regpass.cuh"

namespace vg {

const RegEntry *find_reg_b(int d, int kind) {
    static const RegEntry table[] = {
        RegSide<3, 11, false, kVal | kPlain | kProb>::entry(),   // 33
        RegSide<5, 7, false, kVal | kPlain | kProb>::entry(),   // 35
        RegSide<12, 3, false, kVec | kVal | kPlain | kProb>::entry(),   // 36
        RegSide<3, 13, false, kVec | kVal | kPlain | kProb>::entry(),   // 39
    };
    return find_in(table, (int)(sizeof(table) / sizeof(table[0])), d, kind);
}

}  // namespace vg
