"""A cooperative launch that is refused falls back to the launch chain; a failed one is an error.  The launch is a fake that
returns the status, so this runs without a GPU."""
import subprocess
import textwrap
from pathlib import Path

from conftest import ROOT
from ffai_b200.build import nvcc_path

PROGRAM = textwrap.dedent(r"""
    #include <cstdio>
    #include "coop_launch.hpp"
    using namespace ffai;

    int main() {
        struct { bool fits, opt_in; cudaError_t launch; CoopLaunch want; int launches, clears; } t[] = {
            {true, true, cudaSuccess, CoopLaunch::ran, 1, 0},
            {false, true, cudaErrorUnknown, CoopLaunch::chain, 0, 0},                       // an error of somebody else's is not looked at
            {true, false, cudaErrorUnknown, CoopLaunch::chain, 0, 1},                       // no room for the shared memory
            {true, true, cudaErrorCooperativeLaunchTooLarge, CoopLaunch::chain, 1, 1},      // a part of the SMs
            {true, true, cudaErrorLaunchOutOfResources, CoopLaunch::chain, 1, 1},
            {true, true, cudaErrorNotSupported, CoopLaunch::chain, 1, 1},
            {true, true, cudaErrorLaunchFailure, CoopLaunch::failed, 1, 1},
        };
        int bad = 0;
        for (auto& c : t) {
            int launches = 0, clears = 0;
            cudaError_t status = cudaErrorUnknown;
            const CoopLaunch got = try_cooperative(c.fits, [&] { return c.opt_in; }, [&] { ++launches; return c.launch; }, [&] { ++clears; }, &status);
            bad += got != c.want || launches != c.launches || clears != c.clears;
            bad += got == CoopLaunch::failed && status != c.launch;
        }
        std::printf("bad=%d\n", bad);
        return bad;
    }
""")


def test_refused_cooperative_launch_takes_the_chain(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    cuda = Path(nvcc_path()).resolve().parent.parent / "include"
    subprocess.run(["g++", "-std=c++17", "-Wall", "-I", str(ROOT / "ffai_b200" / "csrc"), "-I", str(cuda), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
