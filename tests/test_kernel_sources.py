"""Properties of the kernel sources that no result shows, checked by reading them."""
import glob
import os
import re

from tests.conftest import ROOT


def test_named_barriers_follow_a_reconvergence():
    """bar.sync and bar.arrive need the whole warp together; the stage kernels reach them from
    divergent branches, so every function that issues one reconverges its warp just before."""
    seen = 0
    for path in glob.glob(os.path.join(ROOT, "ch_swe_b200", "csrc", "*.cu*")):
        src = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"asm[^;]*?\"bar(rier)?\.(sync|arrive)", src):
            assert re.search(r"__syncwarp\(\);\s*$", src[:m.start()]), (os.path.basename(path), src[m.start():m.start() + 60])
            seen += 1
    assert seen >= 2


def test_no_transfer_to_the_device_on_the_default_stream():
    """Contexts work on streams that do not wait for the default stream: what a copy or a clear
    there leaves in device memory has no order against their kernels."""
    for path in glob.glob(os.path.join(ROOT, "ch_swe_b200", "csrc", "*.cu*")):
        src = re.sub(r"//[^\n]*", "", open(path).read())
        assert not re.search(r"cudaMemset\(|cudaMemcpy\([^;]*(HostToDevice|DeviceToDevice)", src), os.path.basename(path)
    src = open(os.path.join(ROOT, "ch_swe_b200", "csrc", "swe_api.cu")).read()
    body = src[src.index("static cudaError_t upload_link_tables()"):]
    body = body[:body.index("\n}")]
    assert body.rindex("cudaStreamSynchronize(cudaStreamLegacy)") > body.rindex("upload_tables(")
