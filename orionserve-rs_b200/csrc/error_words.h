// When the host looks into the error words of bounded waits one by one, after a step.
#pragma once

#include <cstdint>

namespace orion {

// The functions that poll the words also switch the phase traces on and print them, so that a build with traces (ORION_TRACE) polls after every step.
#ifdef ORION_TRACE
constexpr bool kPollEveryStep = true;
#else
constexpr bool kPollEveryStep = false;
#endif

// came: the OR of all words came with the step (`all`); a step that brings none has to ask.
inline bool poll_after_step(bool came, uint32_t all) { return kPollEveryStep || !came || all != 0; }

}  // namespace orion
