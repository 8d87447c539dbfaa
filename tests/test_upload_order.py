"""Uploads and clears of device memory by the native library: what a caller's
stream reads next is in place before it can be read.

A copy from pageable host memory, or a cudaMemset, on the default stream may
still be under way when its call returns, and the callers' (non-blocking)
streams do not wait for that stream; nor does it wait for kernels queued on
theirs that still read what is overwritten."""

import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gpu-ocean_b200", "csrc")


def _function(source, name):
    """Text of the function `name` of a source file: from its definition to the
    closing brace in the first column (or the indentation of its first line)."""
    text = open(os.path.join(CSRC, source)).read()
    m = re.search(r"^[\w:<>&* \t\"]*\b%s\([^;{]*\{$" % name, text, re.M)
    assert m, name
    return text[m.start():text.index("\n}\n", m.end())]


def test_model_error_descriptors_are_uploaded_on_the_callers_stream():
    body = _function("batch.cu", "grf_prepare")
    assert "cudaMemcpy(" not in body
    copy, wait = body.index("cudaMemcpyAsync(b->d_grf"), body.index("cudaStreamSynchronize(s)")
    assert re.search(r"cudaMemcpyAsync\(b->d_grf[^;]*, s\)", body) and copy < wait


# functions that fill device memory through the default stream, and the last
# such call of each: it is followed by a wait for that stream
WAITED = [("ocean_noise.cu", "go_noise_batch_create", "cudaMemcpy(b->d_members"),
          ("api.cu", "go_domain_create", "cudaMemset(d->d_status"),
          ("api.cu", "go_domain_set_coriolis", "cudaMemcpy(d->d_frows"),
          ("api.cu", "go_domain_status", "cudaMemset(d->d_status"),
          ("drifters.cu", "go_wind_texture_create", "cudaMemcpy2DToArray("),
          ("open_boundaries.cu", "go_bc_texture_create", "cudaMemcpy2DToArray("),
          ("batch.cu", "batch_commit", "batch_lay_out("),     # calls all that fills the batch's lists
          ("adjoint.cu", "adjoint_batch_commit", "cudaMemcpy(b->d_folds")]


def test_every_upload_is_listed():
    """No other function uses the default stream to fill device memory."""
    layouts = ("batch_commit_pair", "batch_commit_tile", "batch_lay_out", "tile_batch_consts")   # within batch_commit
    known = {w[1] for w in WAITED} | set(layouts)
    for source in sorted(os.listdir(CSRC)):
        text = open(os.path.join(CSRC, source)).read()
        for m in re.finditer(r"\b(cudaMemcpy|cudaMemset|cudaMemcpy2D|cudaMemcpyToSymbol|cudaMemcpy2DToArray)\(([^;]*);", text):
            if "DeviceToHost" in m.group(2) or "//" in text[text.rindex("\n", 0, m.start()):m.start()]:
                continue
            head = re.findall(r"^[\w:<>&*\" ]+?(\w+)\([^;{]*\{$", text[:m.start()], re.M)
            assert head[-1] in known, (source, head[-1])


@pytest.mark.parametrize("source,name,last", WAITED, ids=[w[1] for w in WAITED])
def test_uploads_on_the_default_stream_are_waited_for(source, name, last):
    body = _function(source, name)
    assert "cudaStreamSynchronize(cudaStreamLegacy)" in body[body.rindex(last):]


@pytest.mark.gpu
def test_model_error_with_another_correlation_length_waits_for_the_filter_before():
    """Two perturbations of different correlation lengths queued behind work on
    the batch's stream: each filter reads its own descriptors, so the states
    are those of the same perturbations one at a time."""
    import numpy as np
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    from SWESimulators import BatchedEnsemble, CDKLM16, Common
    ctx = Common.CUDAContext()

    def ensemble():
        sims = []
        for nx, ny in ((130, 96), (64, 200), (96, 33)):
            zero = np.zeros((ny + 4, nx + 4), np.float32)
            H = np.full((ny + 5, nx + 5), 50.0, np.float32)
            sims.append(CDKLM16.CDKLM16(ctx, zero, zero, zero, H, nx, ny, 1000.0, 1000.0, 1.0, 9.81, 1.2e-4, 0.0, 0.0))
        return BatchedEnsemble.BatchedCDKLM16(sims)
    got, want = ensemble(), ensemble()
    got.model_error(1, corr_cells=4.0)               # the batch's lists and the scratch are laid out
    torch.cuda.synchronize()
    with torch.cuda.stream(got.stream):
        torch.cuda._sleep(40_000_000)                # some 20 ms at the SM clock
    for event, corr in ((2, 15.0), (3, 4.0), (4, 15.0)):
        got.model_error(event, corr_cells=corr)
    for event, corr in ((1, 4.0), (2, 15.0), (3, 4.0), (4, 15.0)):
        want.model_error(event, corr_cells=corr)
        torch.cuda.synchronize()
    torch.cuda.synchronize()
    for a, b in zip(got.sims, want.sims):
        assert np.array_equal(a.download()[0], b.download()[0])
