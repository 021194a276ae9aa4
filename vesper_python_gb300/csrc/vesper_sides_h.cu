// Register passes of the search: compiled sides, table h (split across
// translation units so that they compile in parallel).
#define VG_PASS_TYPES_ONLY
#include "vesper_regpass.cuh"

namespace vg {

const RegEntry *find_reg_h(int d, int kind) {
    static const RegEntry table[] = {
        RegSide<10, 7, false, kVec | kVal | kPlain | kProb>::entry(),   // 70
        RegSide<24, 3, false, kVec | kVal | kPlain | kProb>::entry(),   // 72
        RegSide<15, 5, false, kProb>::entry(),   // 75
    };
    return find_in(table, (int)(sizeof(table) / sizeof(table[0])), d, kind);
}

}  // namespace vg
