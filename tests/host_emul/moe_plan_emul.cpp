// Host build of the SwitchGLU's choice between its two ways for few tokens (ponyexl3_b200/csrc/exl3_moe_plan.h).
#include "../../ponyexl3_b200/csrc/exl3_moe_plan.h"

extern "C" int emul_by_expert(int64_t pairs, int64_t experts, int64_t d, int64_t h, int k) { return exl3::moe_by_expert(pairs, experts, d, h, k); }
extern "C" int emul_most_tiles(int64_t hit, int64_t slots, int64_t cols, int sets) { return exl3::moe_most_tiles(hit, slots, cols, sets); }
