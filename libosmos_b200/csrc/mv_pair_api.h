// what mv.cu asks of the paired F32-activation matvec (mv_pair.cu)
#pragma once
#include <cstdint>

#include "mv_staged_api.h"

namespace osmos {
namespace mvp {

using mvs::Request;

// 1: queued on the stream; 0: not a shape or a type this kernel takes (nothing queued: use another kernel); -1: the
// launch was refused
int try_launch(uint32_t type, const Request& r, void* stream);
// the current device's status word, read and cleared (synchronizes): bit 0 a copy never landed, bit 1 a grouped
// entry's matrix started on an odd byte (its rows were not written; MXFP4's are)
uint32_t read_status();

}  // namespace mvp
}  // namespace osmos
