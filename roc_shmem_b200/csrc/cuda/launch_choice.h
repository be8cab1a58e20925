// launch_choice.h — which of two forms of a launch runs.  Plain C++.
#pragma once

namespace bshmem {

// The preferred form where it fits and the device accepts it, the general one otherwise: a form that is only the faster one does not
// turn a call away that the other can serve.
template <class Status, class Preferred, class General>
Status launch_preferred(bool fits, Status success, Preferred preferred, General general) {
  if (fits && preferred() == success) return success;
  return general();
}

}  // namespace bshmem
