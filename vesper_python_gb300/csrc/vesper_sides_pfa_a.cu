// Register passes of the search: compiled sides, table pfa_a (split across
// translation units so that they compile in parallel).
#define VG_PASS_TYPES_ONLY
#include "vesper_regpass.cuh"

namespace vg {

const RegEntry *find_reg_pfa_a(int d, int kind) {
    static const RegEntry table[] = {
        RegSide<13, 1, true, kVec>::entry(),   // 13
        RegSide<9, 3, true, kVec>::entry(),   // 27
        RegSide<7, 4, true, kVec>::entry(),   // 28
        RegSide<10, 3, true, kVec | kProb>::entry(),   // 30
        RegSide<8, 4, true, kVec | kProb>::entry(),   // 32
        RegSide<11, 3, true, kVec>::entry(),   // 33
        RegSide<7, 5, true, kVec>::entry(),   // 35
    };
    return find_in(table, (int)(sizeof(table) / sizeof(table[0])), d, kind);
}

}  // namespace vg
