// Register passes of the search: compiled sides, table d (split across
// translation units so that they compile in parallel).
#define VG_PASS_TYPES_ONLY
#include "vesper_regpass.cuh"

namespace vg {

const RegEntry *find_reg_d(int d, int kind) {
    static const RegEntry table[] = {
        RegSide<16, 3, false, kVec | kVal | kPlain | kProb>::entry(),   // 48
        RegSide<7, 7, false, kVec | kVal | kPlain | kProb>::entry(),   // 49
        RegSide<10, 5, false, kVec | kVal | kPlain | kProb>::entry(),   // 50
    };
    return find_in(table, (int)(sizeof(table) / sizeof(table[0])), d, kind);
}

}  // namespace vg
