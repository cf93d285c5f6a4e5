// fake_kernels.cu -- what the tests on the stand-in runtime (fake_cudart.cpp)
// need of the kernels' effects: the look launch of a cooperative sweep lists
// every window, the launch after it empties the list, and the Courant read-back
// writes its two words, each only into memory that is there.
#include <string>

#include "hb_kernels.cuh"

bool pinned_word(const void* p, size_t n);

void act_out(const std::string& name, void** args, std::string& faults) {
    const bool look = name.find("steady_") != std::string::npos;
    if (look || name.find("coop_") != std::string::npos) {
        const hb::SweepArgs& a = *(const hb::SweepArgs*)args[0];
        if (!look) {
            a.todo_count[0] = a.todo_count[1] = a.todo_count[2] = 0u;
            return;
        }
        // The narrow windows: rows of 124 outputs, or 60 of each of 4 columns (of a
        // grid that is not square).
        const bool x = a.n == a.nxt && a.nlines == a.ny;
        const int out = hb::coop_outputs(x ? 1 : 2, 4);
        a.todo_count[0] += (unsigned)((x ? a.ny : (a.nx + 5) / 4) * ((a.n - 2 + out - 1) / out));
        if (a.todo_count[0] > hb::coop_list_size(a.nx, a.ny)) faults += "list beyond its room;";
    } else if (name.find("courant_read") != std::string::npos) {
        unsigned long long* host = *(unsigned long long**)args[1];
        if (pinned_word(host, 16)) host[0] = host[1] = 0x4000000000000000ull;  // 2.0
        else faults += "maxima written to memory that is gone;";
    }
}
