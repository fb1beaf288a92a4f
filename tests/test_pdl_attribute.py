"""Kernels launched with the programmatic attribute by hand (cudaLaunchKernelEx
instead of BN_LAUNCH_PDL) begin with the wait for the previous kernel too."""
import glob
import os
import re

from test_pdl_sources import CSRC, _kernel_body_start


def test_kernels_with_the_attribute_wait_first():
    launched = set()
    for f in glob.glob(os.path.join(CSRC, "*.cu")):
        src = open(f).read()
        for m in re.finditer(r"cudaLaunchAttributeProgrammaticStreamSerialization;", src):
            # the launch that this configuration is for: the next one in the source
            call = re.search(r"cudaLaunchKernelEx\(\s*&\w+,\s*([A-Za-z_][A-Za-z0-9_]*)",
                             src[m.end():])
            assert call, f
            launched.add((f, call.group(1)))
    assert any(name == "k_tail" for _, name in launched)
    for f, name in sorted(launched):
        body = _kernel_body_start(open(f).read(), name)
        assert body is not None, name
        assert body.lstrip().startswith("BN_PDL_ENTRY();"), name
