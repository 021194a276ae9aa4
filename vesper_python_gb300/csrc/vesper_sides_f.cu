// Register passes of the search: compiled sides, table f (split across
// translation units so that they compile in parallel).
#define VG_PASS_TYPES_ONLY
#include "vesper_regpass.cuh"

namespace vg {

const RegEntry *find_reg_f(int d, int kind) {
    static const RegEntry table[] = {
        RegSide<8, 7, false, kVec | kVal | kPlain | kProb>::entry(),   // 56
        RegSide<12, 5, false, kVec | kVal | kPlain | kProb>::entry(),   // 60
        RegSide<9, 7, false, kVec | kVal | kPlain | kProb>::entry(),   // 63
    };
    return find_in(table, (int)(sizeof(table) / sizeof(table[0])), d, kind);
}

}  // namespace vg
