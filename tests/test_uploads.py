"""Host memory reaches the device on the stream of the object that reads it.  A plain
cudaMemcpy or cudaMemset goes through the default stream, which the objects'
non-blocking streams do not wait for, and may return before its last part has arrived:
a kernel behind it could read what was there before (a batch's table of pointers among
it).  Only code that works on the default stream throughout may use them."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "binarytpm_gb300" / "csrc"
DEFAULT_STREAM_ONLY = {"atpm_vfapi.cpp"}  # its kernels run on the default stream


def test_no_upload_through_the_default_stream():
    for p in sorted(CSRC.glob("*.c*")):
        if p.name in DEFAULT_STREAM_ONLY:
            continue
        text = re.sub(r"//[^\n]*", "", p.read_text())
        for m in re.finditer(r"cudaMemcpy(2D)?\([^;]*cudaMemcpyHostToDevice[^;]*;[^;]*;|cudaMemset\([^;]*;[^;]*;", text):
            # followed at once by a wait for the default stream, or by a launch on it
            assert re.search(r"cudaStreamSynchronize\(0\)|launch_wait_selftest\([^;]*nullptr\)", m.group()), \
                f"{p.name}: {m.group()[:100]}"
