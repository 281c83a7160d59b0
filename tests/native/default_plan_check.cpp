// Host-side check of the plans that callers get without options (plan_check.cpp asks for its chunk
// counts): chunks long enough for the register solve up to the row counts it ends at, and 64 of them for
// refined builders. The device solve's steps, emulated with the tables the kernels receive, have to
// reproduce the direct banded solve, for A and A^T. No CUDA call is made.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <string>
#include <vector>

#include "../../ddc_b200/csrc/ddcb_internal.hpp"

int main()
{
    int failures = 0, cases = 0;
    std::mt19937_64 rng(777);
    std::uniform_real_distribution<double> U(-1.0, 1.0);
    int const bcs[][2] = {{0, 0}, {1, 1}, {3, 3}, {1, 3}, {2, 2}};
    for (int d = 1; d <= 5; ++d)
        for (int mesh = 0; mesh < 3; ++mesh)
            for (auto const& bc : bcs)
                for (int nc : {11, 16, 17, 18, 19, 33, 35, 36, 52, 64, 101, 289, 513, 1024, 1291, 1722, 2177, 2300}) {
                    if (nc > 600 && mesh == 2) continue;
                    bool const per = bc[0] == 0;
                    ddcb::Basis b;
                    if (mesh == 0) {
                        ddcb::make_uniform_basis(b, d, per, 0.0, 1.0, nc);
                    } else {
                        std::vector<double> br(nc + 1);
                        for (int i = 0; i <= nc; ++i) {
                            double const t = double(i) / nc;
                            br[i] = mesh == 1 ? t + (i > 0 && i < nc ? 0.3 * U(rng) / nc : 0.0) : t * t * t * t + 1e-3 * t;
                        }
                        ddcb::make_non_uniform_basis(b, d, per, br.data(), nc + 1);
                    }
                    auto pts = ddcb::greville_points(b, bc[0], bc[1]);
                    for (int refined = 0; refined < 2; ++refined) {
                        ddcb_builder_options opt {refined ? DDCB_FP32_REFINE : DDCB_FP64, 0, 0, 0, 0.0};
                        ddcb::Builder* bl = nullptr;
                        try {
                            bl = ddcb::create_builder_host(b, pts.data(), long(pts.size()), bc[0], bc[1], &opt);
                        } catch (std::exception const& e) {
                            std::printf("FAIL create d=%d mesh=%d bc=%d,%d nc=%d: %s\n", d, mesh, bc[0], bc[1], nc, e.what());
                            ++failures;
                            continue;
                        }
                        for (int tr = 0; tr < 2; ++tr) {
                            std::vector<double> rhs(bl->n);
                            for (auto& v : rhs) v = U(rng);
                            double const err = ddcb::emulate_device_solve(*bl, rhs.data(), tr != 0);
                            ++cases;
                            if (!(err <= 1e-12)) {
                                ++failures;
                                std::printf("FAIL d=%d mesh=%d bc=%d,%d nc=%d refined=%d tr=%d err=%.3e %s\n", d, mesh, bc[0], bc[1], nc,
                                            refined, tr, err, bl->structure.c_str());
                            }
                        }
                        if (refined && nc >= 513) { // some 64 chunks a line, as many as whole rows allow; more on long lines
                            size_t const at = bl->structure.find("chunks=");
                            int const chunks = at == std::string::npos ? 0 : std::atoi(bl->structure.c_str() + at + 7);
                            ++cases;
                            if (chunks < 48 || chunks > 128) {
                                ++failures;
                                std::printf("FAIL d=%d mesh=%d nc=%d refined: %s\n", d, mesh, nc, bl->structure.c_str());
                            }
                        }
                        ddcb::destroy_builder(bl);
                    }
                }
    std::printf("default_plan_check: %d cases, %d failures\n", cases, failures);
    return failures ? 1 : 0;
}
