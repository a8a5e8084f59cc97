"""The training kernels are launched so that one may be resident while the
previous one still writes what it will read.  That must not change the weights
(against a process whose launches are serialised, ragged batches included), and
no buffer that changes under a resident kernel may be declared constant."""
from __future__ import annotations

import os
import re
import subprocess
import sys

import pytest

from conftest import ROOT

SOURCE = os.path.join(ROOT, "kokkos-particletransport_gb300", "csrc", "kpt_surrogate.cu")
TRAIN = """
import hashlib, importlib, sys
sys.path.insert(0, {root!r})
kpt = importlib.import_module("kokkos-particletransport_gb300")
with kpt.Context(0) as ctx:
    settings = kpt.default_settings(focused=1, closure=kpt.CLOSURE_SURROGATE)
    for hidden, batch, steps in ((64, 8192, 400), (32, 4096, 300), (64, 1001, 300), (32, 257, 300),
                                 (64, 33, 200)):
        net = ctx.train_surrogate(settings, samples=20000, steps=steps, batch=batch,
                                  hidden_width=hidden)
        print(hidden, batch, hashlib.sha256(net.parameters()[0].tobytes()).hexdigest())
        net.close()
"""


def test_handed_on_buffers_are_not_declared_constant():
    with open(SOURCE) as f:
        text = f.read()
    overlapped = []
    for m in re.finditer(r"__global__(?P<head>[^{;]*)\{", text):
        body = text[m.end():text.index("\n}\n", m.end())]
        if "previous_done()" not in body:
            continue
        name, params = re.search(r"(\w+)\(([^()]*)\)\s*$", m["head"]).groups()
        overlapped.append(name)
        declared = re.findall(r"__restrict__\s+(\w+)", params)
        assert set(declared) <= {"x", "t"}, (name, declared)  # the training set is constant
    assert len(overlapped) == 3, overlapped


@pytest.mark.gpu
def test_overlapped_launches_train_the_same_weights():
    outs = []
    for blocking in ("0", "1"):
        done = subprocess.run([sys.executable, "-c", TRAIN.format(root=ROOT)], text=True,
                              capture_output=True, timeout=300,
                              env=dict(os.environ, CUDA_LAUNCH_BLOCKING=blocking))
        assert done.returncode == 0, done.stderr[-2000:]
        outs.append(done.stdout)
    assert outs[0] and outs[0] == outs[1]
