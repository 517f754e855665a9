"""Every kernel of the library runs on a non-blocking stream, which waits for no other stream: a plain
cudaMemcpy to the device may return while its copy is still under way on the legacy stream, so
what a kernel reads has to go up on the kernel's own stream."""
import glob
import os
import re

import pytest

from conftest import PKG


@pytest.mark.parametrize("name", sorted(os.path.basename(p) for p in glob.glob(os.path.join(PKG, "csrc", "*.cu"))))
def test_uploads_are_on_the_kernels_stream(name):
    src = open(os.path.join(PKG, "csrc", name)).read()
    assert not re.findall(r"\bcudaMemcpy\([^;]*cudaMemcpyHostToDevice", src)
