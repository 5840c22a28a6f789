// lbx_roles.h — registers of the two-role fluid kernels (k_cg_lean2, k_cg_lean2_multi).
//
// A CTA is launched with kLaunchRegs registers per thread; its phase half then
// shrinks to kPhaseRegs and its collision half grows to kCollideRegs.  Growing
// waits, without a limit, until the CTA's own launch allocation has that many
// free, so the two shares must fit in what the launch really allocated, which
// the compiler decides (the launch bounds only cap it).
#pragma once

namespace lbx {

constexpr int kLaunchRegs = 128, kPhaseRegs = 56, kCollideRegs = 200;

// numRegs: registers per thread the kernel is launched with.  The halves have
// the same number of threads; neither share may lie on the wrong side of it.
constexpr bool role_regs_fit(int numRegs) {
  return kPhaseRegs + kCollideRegs <= 2 * numRegs && kPhaseRegs <= numRegs && numRegs <= kCollideRegs;
}
static_assert(role_regs_fit(kLaunchRegs), "the roles share out the launch allocation");
static_assert(kPhaseRegs % 8 == 0 && kCollideRegs % 8 == 0, "register shares are multiples of 8");

}  // namespace lbx
