// The library's settings in the process environment, found in one pass: getenv walks the whole of it for every name, and a
// plan asks for eleven (what os.environ sets reaches it).
#pragma once
#include <unistd.h>

#include <cstring>

namespace tdb {

// f(name, its length, value) for every variable whose name begins with TRIDIST_.
template <typename F>
void each_setting(F f) {
  for (char** e = environ; e != nullptr && *e != nullptr; ++e) {
    // (two characters in front of the call: repeated launches look through the environment too)
    if ((*e)[0] != 'T' || (*e)[1] != 'R' || std::strncmp(*e, "TRIDIST_", 8) != 0) continue;
    const char* eq = std::strchr(*e, '=');
    if (eq != nullptr) f(*e, static_cast<size_t>(eq - *e), eq + 1);
  }
}

}  // namespace tdb
