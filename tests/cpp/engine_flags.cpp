// Scenes that reach (or must not reach) the incremental sort's overflow, run through the engine interface, which reports the
// substeps' flags, and checkpoints, which it takes. Prints "name value" pairs for the Python test. Each run is compared with one that sorts in full (ZR_SORT=full):
// the two give the same particle order, so they differ by the order of grid sums alone.
#include "../../ziran2020_gb300/csrc/engine.h"

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>

using namespace zr;

constexpr uint32_t SORT_OVERFLOW = 1u << 7; // FLAG_SORT: a bucket of the incremental sort had no room for its movers

struct Rng { // seeded, the same on every machine
    uint64_t s;
    double operator()()
    {
        s = s * 6364136223846793005ull + 1442695040888963407ull;
        return (double)(s >> 11) * (1.0 / 9007199254740992.0);
    }
};

// nx x ny x nz cells of a stiffness so low that the body moves freely, 8 particles a cell at random places
static SceneDesc box(int nx, int ny, int nz, int cells, int first, double speed_cells)
{
    SceneDesc d;
    d.dx = 1.0 / cells;
    d.dt = 1e-4;
    d.domain_cells = cells + 4;
    d.materials.push_back({});
    d.materials[0].E = 1.0;
    Rng u{ 12345 };
    for (int i = 0; i < nx; i++)
        for (int j = 0; j < ny; j++)
            for (int k = 0; k < nz; k++)
                for (int q = 0; q < 8; q++) {
                    d.x.push_back((first + i + u()) * d.dx);
                    d.x.push_back((first + j + u()) * d.dx);
                    d.x.push_back((first + k + u()) * d.dx);
                    for (int c = 0; c < 3; c++) d.v.push_back(speed_cells * d.dx / d.dt);
                }
    d.n = (int64_t)d.x.size() / 3;
    d.m.assign(d.n, 1000 * d.dx * d.dx * d.dx / 8);
    d.V0.assign(d.n, d.dx * d.dx * d.dx / 8);
    return d;
}

static void must(int rc, EngineBase& e)
{
    if (!rc) return;
    std::fprintf(stderr, "error %d: %s\n", rc, e.last_error().c_str());
    std::exit(1);
}

static std::unique_ptr<EngineBase> engine(int precision, const SceneDesc& d, bool full_sort)
{
    if (full_sort) setenv("ZR_SORT", "full", 1); // read when the engine is made
    auto e = precision == 8 ? make_engine_f64() : make_engine_f32();
    unsetenv("ZR_SORT");
    e->set_autotune(0);
    must(e->load({ &d }), *e);
    return e;
}

// largest difference of two states: positions and F as they are, velocities in units of the speed, C of the speed over dx
static double difference(const std::vector<double>& a, const std::vector<double>& b, const SceneDesc& d)
{
    double speed = 0, m = 0;
    for (double v : d.v) speed = std::max(speed, std::fabs(v));
    for (size_t i = 0; i < a.size(); i++) {
        const int f = (int)(i % 25);
        const double unit = f < 3 ? 1.0 : (f < 6 ? speed : (f < 15 ? speed / d.dx : 1.0));
        m = std::isfinite(a[i]) && std::isfinite(b[i]) ? std::max(m, std::fabs(a[i] - b[i]) / unit) : 1e30;
    }
    return m;
}

// A written state in which a few percent of the particles moved, all into one place: more than a bucket holds, in all far
// fewer than a quarter.
static void concentrated(SceneDesc& d, std::vector<double>& state)
{
    const int64_t part = 3000;
    for (int64_t p = 0; p < part; p++) // the first layers, beside the box's far end
        for (int c = 0; c < 3; c++) state[25 * p + c] = d.x[3 * p + c] + (c == 0 ? 20 * d.dx : 0.0);
}

int main(int argc, char** argv)
{
    const std::string mode = argc > 1 ? argv[1] : "";
    const int precision = argc > 2 ? std::atoi(argv[2]) : 8;
    if (mode == "written") {
        SceneDesc d = box(16, 16, 16, 64, 8, 0.005);
        std::vector<double> out[2];
        uint32_t flags = 0;
        for (int full = 0; full < 2; full++) {
            auto e = engine(precision, d, full != 0);
            StepReport r;
            must(e->step(4, &r), *e);
            out[full].resize(25 * d.n);
            must(e->get_state(0, out[full].data(), 0), *e);
            concentrated(d, out[full]);
            must(e->set_state(0, out[full].data(), 0), *e);
            StepReport r2;
            must(e->step(3, &r2), *e);
            must(e->get_state(0, out[full].data(), 0), *e);
            if (!full) flags = r2.flags;
        }
        std::printf("particles %lld overflow %d difference %.3e\n", (long long)d.n, (flags & SORT_OVERFLOW) != 0, difference(out[0], out[1], d));
        return 0;
    }
    if (mode == "fast") { // 58% of the particles change cell in every substep: each incremental sort overflows
        const int n = argc > 3 ? std::atoi(argv[3]) : 40;
        SceneDesc d = box(44, 44, 44, 128, 8, 0.25);
        std::vector<double> out[2];
        StepReport r[2];
        for (int full = 0; full < 2; full++) {
            auto e = engine(precision, d, full != 0);
            must(e->step(n, &r[full]), *e);
            out[full].resize(25 * d.n);
            must(e->get_state(0, out[full].data(), 0), *e);
        }
        std::printf("particles %lld overflow %d launched %d done %d difference %.3e ms %.3f full_ms %.3f\n", (long long)d.n,
            (r[0].flags & SORT_OVERFLOW) != 0, r[0].launched, r[0].steps_done, difference(out[0], out[1], d), r[0].device_ms, r[1].device_ms);
        return 0;
    }
    if (mode == "tiles") { // the first n particles of a box that moves 0.04 cells along each axis per substep: no sort overflows
        const int64_t n = std::atoll(argv[3]);
        int side = 1;
        while ((int64_t)side * side * side * 8 < n) side++;
        SceneDesc d = box(side, side, side, 256, 8, 0.04);
        d.n = n;
        d.x.resize(3 * n);
        d.v.resize(3 * n);
        d.m.resize(n);
        d.V0.resize(n);
        std::vector<double> out[2];
        StepReport r[2];
        for (int full = 0; full < 2; full++) {
            auto e = engine(precision, d, full != 0);
            must(e->step(5, &r[full]), *e);
            out[full].resize(25 * d.n);
            must(e->get_state(0, out[full].data(), 0), *e);
        }
        std::printf("particles %lld overflow %d difference %.3e groups %u full_groups %u blocks %u full_blocks %u\n", (long long)d.n,
            (r[0].flags & SORT_OVERFLOW) != 0, difference(out[0], out[1], d), r[0].n_groups, r[1].n_groups, r[0].n_blocks, r[1].n_blocks);
        return 0;
    }
    if (mode == "restore") { // a checkpoint of a written state, before its damage drives were formed: a run, the checkpoint, the run again
        SceneDesc d = box(8, 8, 8, 64, 20, 0.0);
        d.implicit_damage = 1;
        auto& m = d.materials[0];
        m.model = 1;
        m.E = 5e4;
        m.nu = 0.25;
        m.damage = 1;
        m.alpha = -1;
        m.l0 = 0.5 * d.dx;
        m.eta = 0.1;
        m.residual = 0.01;
        d.sigma_c.assign(d.n, 100.0);
        d.F.resize(9 * d.n);
        for (int64_t p = 0; p < d.n; p++)
            for (int c = 0; c < 9; c++) d.F[9 * p + c] = c == 0 ? 1.05 : (c % 4 ? 0.0 : 1.0);
        auto e = engine(precision, d, false);
        std::vector<double> first(25 * d.n), again(25 * d.n);
        StepReport r;
        must(e->checkpoint_save(), *e);
        must(e->step(4, &r), *e);
        must(e->get_state(0, first.data(), 0), *e);
        must(e->checkpoint_restore(), *e);
        must(e->step(4, &r), *e);
        must(e->get_state(0, again.data(), 0), *e);
        double damage = 0, m2 = 0;
        for (int64_t p = 0; p < d.n; p++) {
            damage = std::max(damage, first[25 * p + 24]);
            m2 = std::max(m2, std::fabs(first[25 * p + 24] - again[25 * p + 24]));
        }
        std::printf("particles %lld damage %.6f difference %.3e\n", (long long)d.n, damage, m2);
        return 0;
    }
    if (mode == "stream") { // pipelined one-substep jobs, some of whose states would overflow a bucket of the job before
        SceneDesc d = box(16, 16, 16, 64, 8, 0.005);
        auto e = engine(precision, d, false);
        std::vector<double> plain(25 * d.n);
        must(e->get_state(0, plain.data(), 0), *e);
        std::vector<double> moved = plain;
        concentrated(d, moved);
        const std::vector<double>* jobs[] = { &plain, &plain, &moved, &plain, &moved, &moved, &plain };
        constexpr int J = 7;
        std::vector<double> out[J], want[J];
        const void* in[J];
        void* to[J];
        for (int j = 0; j < J; j++) {
            out[j].resize(25 * d.n);
            in[j] = jobs[j]->data();
            to[j] = out[j].data();
        }
        must(e->stream_steps(0, J, in, to, 0), *e);
        auto f = engine(precision, d, true);
        double m = 0;
        for (int j = 0; j < J; j++) {
            want[j].resize(25 * d.n);
            StepReport r;
            must(f->set_state(0, in[j], 0), *f);
            must(f->step(1, &r), *f);
            must(f->get_state(0, want[j].data(), 0), *f);
            m = std::max(m, difference(out[j], want[j], d));
        }
        std::printf("particles %lld reruns %lld difference %.3e\n", (long long)d.n, (long long)e->stream_reruns(), m);
        return 0;
    }
    return 2;
}
