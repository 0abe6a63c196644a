#include "step_roles.cuh"

namespace islbm {
const RoleTable &roles_fp16() {
    static const RoleTable t = role_table<__half>();
    return t;
}
}  // namespace islbm
