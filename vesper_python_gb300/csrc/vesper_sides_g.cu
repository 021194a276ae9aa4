// Register passes of the search: compiled sides, table g (split across
// translation units so that they compile in parallel).
#define VG_PASS_TYPES_ONLY
#include "vesper_regpass.cuh"

namespace vg {

const RegEntry *find_reg_g(int d, int kind) {
    static const RegEntry table[] = {
        RegSide<16, 4, false, kVec | kVal | kPlain>::entry(),   // 64
        RegSide<5, 13, false, kVec | kVal | kPlain | kProb>::entry(),   // 65
        RegSide<6, 11, false, kVec | kVal | kPlain | kProb>::entry(),   // 66
    };
    return find_in(table, (int)(sizeof(table) / sizeof(table[0])), d, kind);
}

}  // namespace vg
