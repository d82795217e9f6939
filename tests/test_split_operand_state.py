"""When the split form of h_a and loa counts as current (exs_ctx::x_valid), on the host alone.

exs_set_scf_inputs that keeps the muffin-tin integrals forms the operands again unless they are marked
current, so the mark may follow only a launch that succeeded.  The library's own header is compiled with
launches that return a chosen status.
"""
import subprocess

import pytest

from exciting_b200 import build

SOURCE = r"""
#include <cstdio>
#include "exs_internal.cuh"

static cudaError_t status;
exs::DevParams exs_ctx::params() const { return exs::DevParams{}; }
exs::OzAtomArgs exs_ctx::oz_atom_args() const { return exs::OzAtomArgs{}; }
namespace exs {
cudaError_t launch_oz_x(const DevParams &, const OzAtomArgs &, const OzScheme &, cudaStream_t) { return status; }
cudaError_t launch_ring_x(const DevParams &, const OzAtomArgs &, const OzRing &, cudaStream_t) { return status; }
}

int main()
{
    for (int mod = 0; mod < 2; mod++)
        for (int before = 0; before < 2; before++)
            for (cudaError_t s : {cudaSuccess, cudaErrorInvalidConfiguration}) {
                exs_ctx c;
                c.oz_sch.mod = mod;
                c.x_valid = before != 0;
                status = s;
                const cudaError_t e = exs::launch_x(&c, nullptr);
                std::printf("%d %d %d\n", (int)s, (int)e, (int)c.x_valid);
            }
    return 0;
}
"""


@pytest.fixture(scope="module")
def lines(tmp_path_factory):
    d = tmp_path_factory.mktemp("xstate")
    (d / "state.cu").write_text(SOURCE)
    flags = [f for f in build.FLAGS if f not in ("-shared", "-lineinfo", "-O3")]
    subprocess.run([build.nvcc(), *build.ARCH, *flags, "-I", build.CSRC, "-o", str(d / "state"), str(d / "state.cu")],
                   check=True)
    out = subprocess.run([str(d / "state")], check=True, capture_output=True, text=True).stdout
    return [tuple(int(x) for x in line.split()) for line in out.splitlines()]


def test_current_only_after_a_launch_that_succeeded(lines):
    assert len(lines) == 8
    for status, returned, valid in lines:
        assert returned == status
        assert valid == (status == 0)
