// team_inst.cu -- the team kernels of one force-field kind (TEAM_PART: the
// TKIND, TK_TS64 for both Tersoff kinds).  Compiled once per kind, side by
// side: together they are most of the library's compile time.
#include "team.cuh"

namespace gg {

template <int KIND, int MINB, bool RES>
static const void* fn_k(int K) {
  switch (K) {
    case 1: return (const void*)k_team<KIND, 1, MINB, RES>;
    case 2: return (const void*)k_team<KIND, 2, MINB, RES>;
    case 4: return (const void*)k_team<KIND, 4, MINB, RES>;
    case 8: return (const void*)k_team<KIND, 8, MINB, RES>;
    case 16: return (const void*)k_team<KIND, 16, MINB, RES>;
    default: return (const void*)k_team<KIND, 32, MINB, RES>;
  }
}

// blocks per SM asked for: two in FP64 (128 registers), three in mixed precision
#if TEAM_PART == 5
const void* team_fn_ts(bool mixed, int K) {
  if (!mixed) return (const void*)k_team<TK_TS64, 4, 2, false>;
  return K == 2 ? (const void*)k_team<TK_TS32, 2, 3, false> : (const void*)k_team<TK_TS32, 4, 3, false>;
}
#else
#define TEAM_NAME2(n) team_fn_##n
#define TEAM_NAME(n) TEAM_NAME2(n)
const void* TEAM_NAME(TEAM_PART)(int K, bool res) {
  constexpr int MINB = team_mixed(TEAM_PART) ? 3 : 2;
  return res ? fn_k<TEAM_PART, MINB, true>(K) : fn_k<TEAM_PART, MINB, false>(K);
}
#endif

}  // namespace gg
