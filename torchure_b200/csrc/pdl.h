// Programmatic dependent launch, host side: who turns the overlap on (the kernels' side is in common.cuh).
#pragma once

namespace tb {

// A launch sequence that gains from it turns the overlap on for the launches its own thread makes (PdlScope).
inline thread_local bool t_pdl_scope = false;
struct PdlScope {
  bool before;
  explicit PdlScope(bool on) : before(t_pdl_scope) { t_pdl_scope = before || on; }
  ~PdlScope() { t_pdl_scope = before; }
  PdlScope(const PdlScope&) = delete;
  PdlScope& operator=(const PdlScope&) = delete;
};

}  // namespace tb
