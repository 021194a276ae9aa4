// Register passes of the search: compiled sides, table a (split across
// translation units so that they compile in parallel).
#define VG_PASS_TYPES_ONLY
#include "vesper_regpass.cuh"

namespace vg {

const RegEntry *find_reg_a(int d, int kind) {
    static const RegEntry table[] = {
        RegSide<5, 5, false, kVec | kVal | kPlain | kProb>::entry(),   // 25
        RegSide<2, 13, false, kVec | kVal | kPlain | kProb>::entry(),   // 26
        RegSide<9, 3, false, kVal | kPlain | kProb>::entry(),   // 27
        RegSide<4, 7, false, kVal | kPlain | kProb>::entry(),   // 28
        RegSide<6, 5, false, kVal | kPlain>::entry(),   // 30
        RegSide<8, 4, false, kVal | kPlain>::entry(),   // 32
    };
    return find_in(table, (int)(sizeof(table) / sizeof(table[0])), d, kind);
}

}  // namespace vg
