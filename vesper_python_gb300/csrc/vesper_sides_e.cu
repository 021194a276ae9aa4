// Register passes of the search: compiled sides, table e (split across
// translation units so that they compile in parallel).
#define VG_PASS_TYPES_ONLY
#include "vesper_regpass.cuh"

namespace vg {

const RegEntry *find_reg_e(int d, int kind) {
    static const RegEntry table[] = {
        RegSide<4, 13, false, kVec | kVal | kPlain | kProb>::entry(),   // 52
        RegSide<18, 3, false, kVec | kVal | kPlain | kProb>::entry(),   // 54
        RegSide<5, 11, false, kVec | kVal | kPlain | kProb>::entry(),   // 55
    };
    return find_in(table, (int)(sizeof(table) / sizeof(table[0])), d, kind);
}

}  // namespace vg
