#include "step_roles.cuh"

namespace islbm {
const RoleTable &roles_fp32() {
    static const RoleTable t = role_table<float>();
    return t;
}
}  // namespace islbm
