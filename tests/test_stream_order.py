"""Device memory is filled on streams that order it with the kernels: a
cudaMemset on the default stream, or a cudaMemcpy from pageable host memory,
may still be on its way when the call returns, and the batches' non-blocking
streams do not wait for the default one.  Copies to the host return with their
data and may stay."""
import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "gpu_elmm_b200", "csrc")


def _calls(text, name):
    """The argument texts of the calls of one function."""
    for m in re.finditer(r"\b" + name + r"\(", text):
        depth, q = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[q], 0)
            q += 1
        yield text[m.end():q - 1]


def test_no_fill_or_upload_on_the_default_stream():
    found = []
    for f in sorted(os.listdir(CSRC)):
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read())
        found += [(f, a) for a in _calls(text, "cudaMemset")]
        found += [(f, a) for a in _calls(text, "cudaMemcpy") if "cudaMemcpyDeviceToHost" not in a]
        for name, nargs in (("cudaMemsetAsync", 4), ("cudaMemcpyAsync", 5)):  # with their stream argument
            for a in _calls(text, name):
                depth, commas = 0, 0
                for c in a:
                    depth += {"(": 1, "[": 1, ")": -1, "]": -1}.get(c, 0)
                    commas += c == "," and depth == 0
                if commas + 1 != nargs:
                    found.append((f, a))
    assert not found, found


def test_every_chain_runs_at_the_highest_priority():
    """The streams that steps run on (a batch's and the serving loop's) come
    from chain_stream, which takes the highest priority."""
    found = {}
    for f in sorted(os.listdir(CSRC)):
        text = open(os.path.join(CSRC, f)).read()
        for name in ("cudaStreamCreate", "cudaStreamCreateWithFlags", "cudaStreamCreateWithPriority", "chain_stream"):
            for a in _calls(text, name):
                found.setdefault(a.split(",")[0].strip(), []).append((f, name))
    assert found["&stream"] == [("elmm_api.cu", "chain_stream"), ("elmm_server.inl", "chain_stream")], found
