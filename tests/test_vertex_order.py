"""The vertex order of a patch size, found from the layout in patches of another
size (csrc/layout.cpp vertex_order), is that size's own layout's: triangulations
0-3, uneven cloths, patches that cut the mesh often and seldom (CPU)."""
import importlib
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include <cstdio>
#include "pdg_solver.h"
using namespace pdg;

int main()
{
    std::vector<ClothSetup> all;
    int wrong = 0, lone = 0;
    auto check = [&](const std::vector<ClothSetup>& cl) {
        for (int own : {16, 24, 100, 192, 512}) {
            HostLayout a;
            std::string err;
            if (!build_layout(cl, own, a, err)) { std::printf("%s\n", err.c_str()); ++wrong; continue; }
            lone += (int)a.hinges.size();
            for (int size : {16, 128, 256, 512}) {
                HostLayout b;
                std::vector<int> order;
                if (!build_layout(cl, size, b, err)) { std::printf("%s\n", err.c_str()); ++wrong; continue; }
                vertex_order(cl, a, size, order);
                if (order != b.perm_global) { std::printf("patches of %d from %d differ\n", size, own); ++wrong; }
            }
        }
    };
    const int dims[][3] = {{2, 2, 0}, {5, 5, 1}, {33, 41, 2}, {30, 27, 3}, {70, 64, 1}, {3, 200, 0}};
    for (const auto& d : dims) {
        ClothSetup c;
        auto m = std::make_shared<MeshData>();
        generate_grid(d[0], d[1], 1.f, d[2], m->rest, m->tris);
        m->N = (int)m->rest.size() / 3;
        m->T = (int)m->tris.size() / 3;
        precompute_rest_state(*m);
        auto t = std::make_shared<Topology>();
        build_topology(*m, *t);
        c.cons.k_stretch.assign(m->T, 1e3f);
        build_bend(*m, *t, 1e-2f, c.cons);
        if (d[0] == 33 && c.cons.bend_k.size() > 40) {   // hinges of pairs that are no edge's: lone ones
            for (int e = 3; e < 40; e += 7) std::swap(c.cons.quads[4 * e + 1], c.cons.quads[4 * e + 2]);
        }
        c.cfg = pdg_config{};
        c.cfg.dt = 1.f / 60.f;
        c.cfg.max_iterations = 3;
        c.mesh = m;
        c.topo = t;
        check({c});
        all.push_back(c);
    }
    check(all);
    std::printf("%d lone hinges\n", lone);
    return wrong ? 1 : (lone > 0 ? 0 : 2);
}
"""


def test_order_from_another_patch_size(tmp_path):
    build = importlib.import_module("build")
    lib = build.build()
    src = tmp_path / "order.cpp"
    src.write_text(SOURCE)
    exe = str(tmp_path / "order")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", os.path.join(ROOT, "cloth-cuda_gb300", "csrc"), "-I",
                    os.path.join(build.cuda_home(), "include"), str(src), lib, "-Wl,-rpath," + os.path.dirname(lib), "-o", exe],
                   check=True)
    p = subprocess.run([exe], stdout=subprocess.PIPE, text=True, timeout=300)
    assert p.returncode == 0, p.stdout
