// Launch-table entries of the class-templated kernels.  Each k_<kind>_c<B>.cu
// translation unit instantiates the kernels of one kind for bra pair class B
// and every ket pair class, so the classes compile in parallel.  Entries are
// null where the generic runtime-class kernels take over (total angular
// momentum above kTemplatedMaxL) or where a kernel is never used (J/K with the
// ket class above the bra class).
#pragma once
#include "fock_kernels.cuh"

namespace lgb {

// the pair classes of s, p and d shells with total angular momentum up to
// kTemplatedMaxL; classes with an f shell run on the cooperative kernels
constexpr int kTemplatedPairClasses = 6;
template <int B, int K, int MAXL = kTemplatedMaxL>
constexpr bool templated_class() {
  return B < kTemplatedPairClasses && K < kTemplatedPairClasses && pc_L(B) + pc_L(K) <= MAXL;
}
// FP32 and double-float kernels stop at kTemplatedMaxL4
template <typename R>
constexpr int max_l() {
  return std::is_same<R, double>::value ? kTemplatedMaxL : kTemplatedMaxL4;
}

template <typename R, int B, int K>
constexpr JKFn jk_entry() {
  if constexpr (templated_class<B, K, max_l<R>()>() && B >= K) return &jk_tasks_kernel<R, pc_la(B), pc_lb(B), pc_la(K), pc_lb(K)>;
  else return nullptr;
}
template <int B, int K>
constexpr JKFn jkr_entry() {
  if constexpr (templated_class<B, K, kTemplatedMaxL4>() && B >= K) return &jk32_row_kernel<pc_la(B), pc_lb(B), pc_la(K), pc_lb(K)>;
  else return nullptr;
}
template <typename R, int B, int K>
constexpr CPFn cp_entry() {
  if constexpr (templated_class<B, K, max_l<R>()>()) return &cp_tasks_kernel<R, pc_la(B), pc_lb(B), pc_la(K), pc_lb(K)>;
  else return nullptr;
}
template <int B, int K>
constexpr ITFn it_entry() {
  if constexpr (templated_class<B, K, kTemplatedMaxL4>()) return &it_kernel<pc_la(B), pc_lb(B), pc_la(K), pc_lb(K)>;
  else return nullptr;
}

template <int B, int K>
constexpr MXFn mx_entry() {
  if constexpr (templated_class<B, K>()) return &mp2x_kernel<double, pc_la(B), pc_lb(B), pc_la(K), pc_lb(K)>;
  else return nullptr;
}

template <int B, int K>
constexpr MXFn mxd_entry() {
  if constexpr (templated_class<B, K, kTemplatedMaxL4>() && QClass<pc_la(B), pc_lb(B), pc_la(K), pc_lb(K)>::NINT <= 27)
    return &mp2x_kernel<dd32, pc_la(B), pc_lb(B), pc_la(K), pc_lb(K)>;
  else return nullptr;
}
template <int B, int K>
constexpr G12Fn g12_entry() {
  if constexpr (templated_class<B, K, kTemplatedMaxL4>()) return &g12_kernel<pc_la(B), pc_lb(B), pc_la(K), pc_lb(K)>;
  else return nullptr;
}

static_assert(kNumPairClasses == 10, "launch-table rows list every pair class");
#define LGB_ROW(F, ...)                                                                                   \
  { F<__VA_ARGS__, 0>(), F<__VA_ARGS__, 1>(), F<__VA_ARGS__, 2>(), F<__VA_ARGS__, 3>(), F<__VA_ARGS__, 4>(), \
    F<__VA_ARGS__, 5>(), F<__VA_ARGS__, 6>(), F<__VA_ARGS__, 7>(), F<__VA_ARGS__, 8>(), F<__VA_ARGS__, 9>() }

#define LGB_JK_TABLES(B)                                   \
  extern const JKFn kJK64_##B[kNumPairClasses];                          \
  extern const JKFn kJK32_##B[kNumPairClasses];                          \
  extern const JKFn kJKR_##B[kNumPairClasses];                           \
  const JKFn kJK64_##B[kNumPairClasses] = LGB_ROW(jk_entry, double, B); \
  const JKFn kJK32_##B[kNumPairClasses] = LGB_ROW(jk_entry, float, B);  \
  const JKFn kJKR_##B[kNumPairClasses] = LGB_ROW(jkr_entry, B);

// Classes with double-float J/K kernels: those where they clearly beat FP64.  ns per
// quartet on the whole GPU, FP64 / double-float (12 waters with d shells, 480
// functions): (ss|ss) .121/.064, (ps|ss) .253/.109, (ps|ps) .429/.216, (pp|ss)
// .479/.193, (pp|ps) .954/.580, (ds|ss) .400/.177, (ds|ps) .740/.500, (dp|ss)
// .847/.567.  Above 27 integrals the code (some 27,000 instructions for (pp|pp))
// outgrows the instruction cache and 5 to 18 % are left, at two launches a class
// instead of one and less of a quartet's precision: (pp|pp) 2.64/2.38, (ds|pp)
// 1.86/1.52, (dp|ps) 1.78/1.57, (ds|ds) 1.87/1.78; (dd|ss) loses, 1.85/2.05.
template <int B, int K>
constexpr JKFn jkd_entry() {
  if constexpr (templated_class<B, K, kTemplatedMaxL4>() && B >= K &&
                QClass<pc_la(B), pc_lb(B), pc_la(K), pc_lb(K)>::NINT <= 27)
    return &jk_tasks_kernel<dd32, pc_la(B), pc_lb(B), pc_la(K), pc_lb(K)>;
  else return nullptr;
}

#define LGB_JKD_TABLE(B)                                   \
  extern const JKFn kJKD_##B[kNumPairClasses];                           \
  const JKFn kJKD_##B[kNumPairClasses] = LGB_ROW(jkd_entry, B);

#define LGB_CP_TABLES(B)                                   \
  extern const CPFn kCP64_##B[kNumPairClasses];                          \
  extern const CPFn kCP32_##B[kNumPairClasses];                          \
  const CPFn kCP64_##B[kNumPairClasses] = LGB_ROW(cp_entry, double, B); \
  const CPFn kCP32_##B[kNumPairClasses] = LGB_ROW(cp_entry, float, B);

#define LGB_IT_TABLE(B)                      \
  extern const ITFn kIT_##B[kNumPairClasses];              \
  extern const MXFn kMX_##B[kNumPairClasses];              \
  const ITFn kIT_##B[kNumPairClasses] = LGB_ROW(it_entry, B); \
  const MXFn kMX_##B[kNumPairClasses] = LGB_ROW(mx_entry, B);

#define LGB_MXD_TABLE(B)                     \
  extern const MXFn kMXD_##B[kNumPairClasses];             \
  const MXFn kMXD_##B[kNumPairClasses] = LGB_ROW(mxd_entry, B);

#define LGB_G12_TABLE(B)                     \
  extern const G12Fn kG12_##B[kNumPairClasses];            \
  const G12Fn kG12_##B[kNumPairClasses] = LGB_ROW(g12_entry, B);

}  // namespace lgb
