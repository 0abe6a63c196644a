#include "step_roles.cuh"

namespace islbm {
const RoleTable &roles_bf16() {
    static const RoleTable t = role_table<__nv_bfloat16>();
    return t;
}
}  // namespace islbm
