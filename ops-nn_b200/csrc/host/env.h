// The library's tuning and test switches (OPSNN_* environment variables).
#pragma once

#include <cstdlib>
#include <cstring>

extern char** environ;

namespace opsnn {

// Whether any OPSNN_* variable is set: 0 not looked for yet, 1 none, 2 some.
inline thread_local int tl_env_state = 0;

inline int env_state()
{
    if (tl_env_state != 0) return tl_env_state;
    for (char** e = environ; e != nullptr && *e != nullptr; ++e)
        if ((*e)[0] == 'O' && std::strncmp(*e, "OPSNN_", 6) == 0) return 2;
    return 1;
}

// One entry point's call: the environment is walked once at its start, not once for each of the ten to fifteen switches that the
// call's plan and launch ask for (a process has dozens of variables and getenv compares its way through them all).
struct EnvScope {
    int outer = tl_env_state;
    EnvScope() { tl_env_state = env_state(); }
    ~EnvScope() { tl_env_state = outer; }
    EnvScope(const EnvScope&) = delete;
    EnvScope& operator=(const EnvScope&) = delete;
};

// getenv for OPSNN_* names.
inline const char* env(const char* name) { return env_state() == 1 ? nullptr : std::getenv(name); }

}  // namespace opsnn
