// The product of many rows (linear_many.cu) as the others of the library see it.
#pragma once

namespace l3ci {

// The device word where its waits that ran out are recorded (of the current device); null without a device.
int* linear_many_wait_status();

}  // namespace l3ci
