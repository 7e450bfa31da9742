// The coarse levels of a V-cycle in one kernel (mg_tail.cu).
#pragma once

#include <memory>

#include "pmg_internal.hpp"

struct pmg_mg;

namespace pmg {
struct TailPlan; // the coarse levels' index maps as the kernel keeps them
// the plan of a hierarchy's coarse levels, null where the kernel does not apply
std::shared_ptr<TailPlan> mg_tail_plan(const pmg_mg &mg);
// the finest level the kernel takes now, -1: none (a level's tensor-core switch, a Chebyshev degree
// beyond the kernel's tables)
int mg_tail_top(const pmg_mg &mg);
// the V-cycle from level `top` down, from mg.def[top] into mg.sol[top] (every smoother estimated)
void mg_tail(pmg_mg &mg, int top, cudaStream_t s);
} // namespace pmg
