// pt_persist_checked.cu — the persistent kernel built a second time with index
// checks (PT_DEBUG_CHECKS); see pt_wavefront_checked.cu.
#define PT_DEBUG_CHECKS 1
#define PTK_WF(name) name##_checked
#include "pt_persist.cu"
