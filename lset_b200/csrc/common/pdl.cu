#include "pdl.h"

namespace lb {

namespace {
thread_local bool t_pdl = false;
}

bool pdl_enabled() { return t_pdl; }
bool pdl_enabled(long long bytes) { return t_pdl && bytes < kPdlMaxBytes; }
PdlScope::PdlScope(bool on) : saved(t_pdl) { t_pdl = on; }
PdlScope::~PdlScope() { t_pdl = saved; }

}  // namespace lb
