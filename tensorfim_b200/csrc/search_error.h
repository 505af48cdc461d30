// What the resident search's kernels record in ResStatus::error, and the status that a caller gets.
#pragma once
#include <cstdint>

#include "tfim.h"

namespace tfim {

constexpr int32_t kErrRow = 1;         // a counted row below the threshold
constexpr int32_t kErrProjected = 2;   // a projected family of another size than its support
constexpr int32_t kErrWait = 3;        // a wait of the device loop's grid barrier expired

inline int search_error_status(int32_t error) {
    return error == 0 ? TFIM_OK : error == kErrWait ? TFIM_E_TIMEOUT : TFIM_E_STATE;
}

}  // namespace tfim
