#include "pdl.h"

namespace lb {

namespace {
thread_local bool t_pdl = false;
}

bool pdl_enabled() { return t_pdl; }
PdlScope::PdlScope(bool on) : saved(t_pdl) { t_pdl = on; }
PdlScope::~PdlScope() { t_pdl = saved; }

}  // namespace lb
