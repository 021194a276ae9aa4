// Register passes of the search: compiled sides, table pfa_b (split across
// translation units so that they compile in parallel).
#define VG_PASS_TYPES_ONLY
#include "vesper_regpass.cuh"

namespace vg {

const RegEntry *find_reg_pfa_b(int d, int kind) {
    static const RegEntry table[] = {
        RegSide<7, 6, true, kVec>::entry(),   // 42
        RegSide<11, 4, true, kVec>::entry(),   // 44
        RegSide<8, 8, true, kProb>::entry(),   // 64
        RegSide<15, 5, true, kVec | kVal | kPlain>::entry(),   // 75
    };
    return find_in(table, (int)(sizeof(table) / sizeof(table[0])), d, kind);
}

}  // namespace vg
