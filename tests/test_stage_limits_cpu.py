"""The staging loop's own limits hold at compile time: slots that leave a
group no room for a chunk of candidates, with which its rounds would never
end, do not compile."""
import os
import subprocess

import pytest

from fluidgrid_gb300 import build

SOURCE = """
#include "fg_stage.cuh"
__global__ void k(const float4 *p, const uint32_t *s, const uint32_t *e, const FgScene *S)
{
    __shared__ uint32_t idx[FG_STAGE_WINDOW];
    const fg::StageGrid G(S);
    const fg::StageSig sig = fg::fg_stage_sig(p[threadIdx.x], G);
    fg::fg_stage_rounds<%d, %d>(sig, 0u, 1u, 0.f, 0.f, 0.f, G, p, s, e, idx, [](uint32_t, uint32_t, float4) {},
                               [](uint32_t, uint32_t, uint32_t) {});
}
"""


def compiles(tmp_path, cap, groups):
    src = tmp_path / "k.cu"
    src.write_text(SOURCE % (cap, groups))
    r = subprocess.run([build.nvcc(), *build.ARCH, "-std=c++17", "-I", build.CSRC, "-c", str(src), "-o", os.devnull],
                       capture_output=True, text=True)
    assert r.returncode == 0 or "would never end" in r.stdout + r.stderr, r.stdout + r.stderr
    return r.returncode == 0


@pytest.mark.parametrize("cap,groups,ok", [(384, 9, True), (192, 1, True), (288, 9, True), (280, 9, False),
                                           (384, 13, False), (388, 9, False)])
def test_slots_hold_a_chunk_a_group(tmp_path, cap, groups, ok):
    try:
        build.nvcc()
    except RuntimeError:
        pytest.skip("no nvcc")
    assert compiles(tmp_path, cap, groups) == ok
