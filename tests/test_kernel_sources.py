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


def functions(src):
    """The bodies of the functions at file scope: from a line "{" to the next line "}"."""
    return re.findall(r"^[^\s#/}][^;{}]*\)\n\{\n.*?^\}", src, flags=re.M | re.S)


def test_calls_that_return_results_report_a_failed_tile_load():
    """A kernel whose bounded wait for its tile loads gives up sets the context's error word and
    finishes: what was computed since is incomplete, and no call hands it out as good.  (The
    wait cannot be made to run out on purpose, so this reads the source: a function that copies
    to the host waits through results_ready, which looks at the word, and after the copies.)"""
    src = re.sub(r"//[^\n]*", "", open(os.path.join(ROOT, "ch_swe_b200", "csrc", "swe_api.cu")).read())
    bodies = [f for f in functions(src) if "DeviceToHost" in f]
    assert len(bodies) >= 7
    for f in bodies:
        last = [m.start() for m in re.finditer("DeviceToHost", f)]
        ready = [m.start() for m in re.finditer(r"results_ready\(c\)", f)]
        assert ready and max(ready) > max(last), f.splitlines()[0]
        assert "cudaStreamSynchronize(c->stream)" not in f[min(last):], f.splitlines()[0]
    ready = next(f for f in functions(src) if re.match(r"static int results_ready\(", f))
    assert "cudaStreamSynchronize(c->stream)" in ready and "derr" in ready
