"""CPU: how a training step deals its pairs over the blocks depends on k, d and the
number of pairs, not on the device: the dealing decides the last bits of the gradients,
and a trained projection is the same wherever it was trained."""
import os
import re

from conftest import ROOT


def test_the_steps_ask_the_device_nothing():
    src = open(os.path.join(ROOT, "tensor_bf_main_gb300", "csrc", "k_learn.cu")).read()
    src = re.sub(r"//[^\n]*", "", src)
    for name in ("StepKernel step_kernel(", "int launch_step(", "unsigned wide_clusters("):
        body = src[src.index(name):]
        body = body[: body.index("\n}")]
        assert not re.search(r"cudaOccupancy|cudaDeviceGet|sms", body), name
    train = src[src.index("int train_projection_dev("):]
    train = train[: train.index("\n}")]
    assert "cudaOccupancy" not in train
    # the device's size shapes the sampling of the pairs only (a pair is a hash of its number)
    used = [line.strip() for line in train.splitlines() if re.search(r"\bsms\b", line)]
    assert [u for u in used if not u.startswith(("int sms", "EJ_CUDA(cudaDeviceGetAttribute"))] == [
        u for u in used if u.startswith("sample_grid =")], used
    assert re.search(r"const unsigned grid = sk\.grid \? sk\.grid\s*:", train)
