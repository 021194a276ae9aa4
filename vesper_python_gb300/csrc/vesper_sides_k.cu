// Register passes of the search: compiled sides, table k (split across
// translation units so that they compile in parallel).
#define VG_PASS_TYPES_ONLY
#include "vesper_regpass.cuh"

namespace vg {

const RegEntry *find_reg_k(int d, int kind) {
    static const RegEntry table[] = {
        RegSide<18, 5, false, kVec | kVal | kPlain | kProb>::entry(),   // 90
        RegSide<7, 13, false, kVec | kVal | kPlain | kProb>::entry(),   // 91
        RegSide<32, 3, false, kVec | kVal | kPlain | kProb>::entry(),   // 96
    };
    return find_in(table, (int)(sizeof(table) / sizeof(table[0])), d, kind);
}

}  // namespace vg
