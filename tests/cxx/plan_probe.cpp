// plan_probe.cpp -- the host-side job plan seen from a test: what
// kernel_state.hpp builds for a configuration, without a device.
#include "../../openpstd_gb300/csrc/kernel_state.hpp"

using namespace pstd;

extern "C" {

// The four-strip records of a scene in serving slot `slot`, as the serving
// loop places them, copy jobs included: (kind, scene, transform length) each.
// Returns their number, -1 on an error.
int probe_served_records(const pstd_config* cfg, int slot, int* out, int cap) {
    try {
        Kernel k;
        k.build_scenes(cfg, 1);
        std::vector<DevDomain> doms = k.layout_fields().doms;
        for (DevDomain& d : doms) d.scene = slot;
        std::vector<int> lengths;
        for (const StripRun& r : k.scenes[0].runs) {
            const int L = Kernel::run_length(k.scenes[0], r);
            if (std::find(lengths.begin(), lengths.end(), L) == lengths.end()) lengths.push_back(L);
        }
        std::vector<DevJob> jobs;
        for (int L : lengths) {
            const auto js = k.make_jobs(L, serve_variant(L), false);
            jobs.insert(jobs.end(), js.begin(), js.end());
        }
        const auto copies = k.make_jobs(-1, serve_variant(lengths.front()), true);
        jobs.insert(jobs.end(), copies.begin(), copies.end());
        int n = 0;
        for (const QJob& q : Kernel::quad_jobs_of(jobs, doms)) {
            const int v[3] = {q.kind, q.scene, q.L};
            if (n < cap) std::memcpy(out + 3 * n, v, sizeof v);
            n++;
        }
        return n;
    } catch (...) {
        return -1;
    }
}

}  // extern "C"
