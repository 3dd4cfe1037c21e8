"""The evaluators launch on non-blocking streams, which do not wait for the
legacy stream: a memory fill without a stream has no order with their kernels."""
import re

import pytest

from graphgolf_b200 import build


@pytest.mark.parametrize("name", ["apsp_core.cu", "apsp_batch.cu", "sa_device.cu"])
def test_fills_name_their_stream(name):
    text = (build.CSRC / name).read_text()
    assert "cudaStreamNonBlocking" in text
    assert not re.findall(r"cudaMemset(?:2D)?\s*\(", text)


def test_timed_forward_waits_for_its_upload():
    """The features are cast on the legacy stream, the forwards run on another."""
    text = (build.CSRC / "mlp.cu").read_text()
    body = text[text.index("int ggb_mlp_time_forward("):]
    upload, stream = body.index("upload_x("), body.index("cudaStreamCreateWithFlags")
    assert upload < body.index("cudaStreamSynchronize(nullptr)") < stream
