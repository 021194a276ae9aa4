// Register passes of the search: compiled sides, table c (split across
// translation units so that they compile in parallel).
#define VG_PASS_TYPES_ONLY
#include "vesper_regpass.cuh"

namespace vg {

const RegEntry *find_reg_c(int d, int kind) {
    static const RegEntry table[] = {
        RegSide<8, 5, false, kVec | kVal | kPlain | kProb>::entry(),   // 40
        RegSide<6, 7, false, kVal | kPlain | kProb>::entry(),   // 42
        RegSide<4, 11, false, kVal | kPlain | kProb>::entry(),   // 44
        RegSide<9, 5, false, kVec | kVal | kPlain | kProb>::entry(),   // 45
    };
    return find_in(table, (int)(sizeof(table) / sizeof(table[0])), d, kind);
}

}  // namespace vg
