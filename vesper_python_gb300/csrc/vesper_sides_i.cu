// Register passes of the search: compiled sides, table i (split across
// translation units so that they compile in parallel).
#define VG_PASS_TYPES_ONLY
#include "vesper_regpass.cuh"

namespace vg {

const RegEntry *find_reg_i(int d, int kind) {
    static const RegEntry table[] = {
        RegSide<7, 11, false, kVec | kVal | kPlain | kProb>::entry(),   // 77
        RegSide<6, 13, false, kVec | kVal | kPlain | kProb>::entry(),   // 78
        RegSide<16, 5, false, kVec | kVal | kPlain | kProb>::entry(),   // 80
    };
    return find_in(table, (int)(sizeof(table) / sizeof(table[0])), d, kind);
}

}  // namespace vg
