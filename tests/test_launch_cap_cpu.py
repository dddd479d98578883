"""The cap on resident blocks (dyc_set_configure) holds for the split, grouping
and replay kernels of a set batch: launch shapes recorded without a GPU."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "databases_gpu_gb300")
SMS, SMEM = 152, 228 << 10
GROUP = 43520  # bytes of the grouping's GroupSmem<true>; it has more beside them


def test_set_kernels_stay_within_the_launch_cap(tmp_path):
    from databases_gpu_gb300 import build
    lib = build.build()
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc())))
    libdir = os.path.join(cuda, "lib64")
    exe = str(tmp_path / "launch_cap")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", os.path.join(ROOT, "include"),
                    "-I", os.path.join(PKG, "csrc"), "-I", os.path.join(cuda, "include"),
                    os.path.join(ROOT, "tests", "cpp", "launch_cap_test.cpp"), lib, "-L", libdir, "-lcudart",
                    "-Wl,-rpath," + PKG + ":" + libdir, "-o", exe], check=True)
    out = subprocess.run([exe], check=True, stdout=subprocess.PIPE, text=True).stdout.split("\n")
    rows = [r.split() for r in out if r]
    assert len(rows) == 9 * 3 * 2 * 5
    for cap, n, what, grid, smem in rows:
        cap, n, grid, smem = int(cap), int(n), int(grid), int(smem)
        if what == "group":
            assert grid == -(-n // 1024)
            assert smem == 0 if cap == 0 else (cap + 1) * (GROUP + smem) > SMEM
        else:
            assert grid <= (cap * SMS if cap else grid)
    loops = [int(r[3]) for r in rows if r[0] == "0" and r[1] == str(1 << 24) and r[2] == "loop"]
    assert max(loops) > 8 * SMS  # uncapped launches of that size do go past the largest cap here
