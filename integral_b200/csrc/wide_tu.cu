// The wide kernels (wide.cuh) of one bra pair class: compiled with -DPCB=<n>,
// it instantiates every ket class pck <= PCB that has one (wide_class) and
// adds their registration and its module constants to the registry at load
// time.
#include <utility>

#include "launch.hpp"
#include "wide.cuh"

#ifndef PCB
#error "compile with -DPCB=<bra pair class>"
#endif

namespace igpu {
namespace {

template <int K>
void register_one(WideEntry* tab, int npc) {
  constexpr int LA = pc_la(PCB), LB = pc_lb(PCB), LC = pc_la(K), LD = pc_lb(K);
  WideEntry e;
  if constexpr (wide_class<LA, LB, LC, LD, double>()) {
    e.k64 = wide_kernel<LA, LB, LC, LD, double>;
    e.tab64 = wide_tab_doubles<LA, LB, LC, LD, double>();
  }
  if constexpr (wide_class<LA, LB, LC, LD, float>()) {
    e.k32 = wide_kernel<LA, LB, LC, LD, float>;
    e.tab32 = wide_tab_doubles<LA, LB, LC, LD, float>();
  }
  tab[PCB * npc + K] = e;
}

template <int... I>
void register_all(WideEntry* tab, int npc, std::integer_sequence<int, I...>) {
  (register_one<I>(tab, npc), ...);
}

void register_unit(WideEntry* tab, int npc) { register_all(tab, npc, std::make_integer_sequence<int, PCB + 1>{}); }

cudaError_t upload_unit(const ConstData& c) { return upload_module_constants(c); }

const int g_added = add_wide_unit(register_unit, upload_unit);

}  // namespace
}  // namespace igpu
