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

// What a scene's plan may run, one line each: "bucket L wmin wmax", then the
// variant it starts from ("first"), with every PSTD_VARIANT index ("forced i")
// and those the autotuner may time ("tune"); tensor maps present, staging
// limit of sm_103a.  PSTD_PLAN and PSTD_DFT are followed.  Returns 0, or the
// error code with its message in buf.
int probe_plan(const pstd_config* cfg, char* buf, int cap) {
    std::string s;
    int code = 0;
    Kernel k;
    static unsigned char map;
    k.smem_optin = 232448;
    k.dmaps.p = &map;   // (never read)
    try {
        k.build_scenes(cfg, 1);
        std::map<int, int> lengths;
        for (const StripRun& r : k.scenes[0].runs) lengths[Kernel::run_length(k.scenes[0], r)]++;
        for (auto& kv : lengths) {
            Bucket b = k.bucket_of(kv.first);
            s += "bucket " + std::to_string(b.L) + " " + std::to_string(b.wmin) + " " + std::to_string(b.wmax) + "\n";
            k.choose_variant(b, -1);
            s += std::string("first ") + b.var->name + "\n";
            const StageVariant* vs;
            const int nv = stage_variants(b.L, &vs);
            for (int i = 0; i < nv; i++) {
                k.choose_variant(b, i);
                s += "forced " + std::to_string(i) + " " + b.var->name + "\n";
                if (k.may_tune(vs[i], b)) s += std::string("tune ") + vs[i].name + "\n";
            }
        }
    } catch (SceneError& e) {
        code = e.code;
        s = e.what();
    }
    k.dmaps.p = nullptr;
    std::strncpy(buf, s.c_str(), (size_t)cap - 1);
    buf[cap - 1] = 0;
    return code;
}

// the plan cache's key of a scene (its length; the text in buf)
int probe_signature(const pstd_config* cfg, char* buf, int cap) {
    try {
        Kernel k;
        k.build_scenes(cfg, 1);
        const std::string s = k.plan_signature();
        std::strncpy(buf, s.c_str(), (size_t)cap - 1);
        buf[cap - 1] = 0;
        return (int)s.size();
    } catch (...) {
        return -1;
    }
}

// 1: the plan that `from` would cache (every length on variant `index`) is
// accepted for `to`, 0: it is not
int probe_plan_applies(const pstd_config* from, const pstd_config* to, int index) {
    Kernel a, b;
    a.build_scenes(from, 1);
    b.build_scenes(to, 1);
    b.smem_optin = 232448;
    PlanChoice pc;
    auto lengths = [](Kernel& k) {
        std::map<int, int> m;
        for (const StripRun& r : k.scenes[0].runs) m[Kernel::run_length(k.scenes[0], r)]++;
        return m;
    };
    for (auto& kv : lengths(a)) {
        const StageVariant* vs;
        stage_variants(kv.first, &vs);
        pc.vars.push_back({kv.first, &vs[index]});
    }
    for (auto& kv : lengths(b)) b.buckets.push_back(b.bucket_of(kv.first));
    return b.plan_applies(pc);
}

}  // extern "C"
