"""Small tables on the device (ops.device_table, ops.drift_tables): shared by threads, streams and
CUDA graphs."""

from __future__ import annotations

import sys
import threading

import numpy as np
import pytest
import torch

import jfli_b200 as jf
from jfli_b200 import ops


def test_threads_share_the_tables():
    """More tables than are kept, met again by several threads: every call returns its own."""
    wrong, interval = [], sys.getswitchinterval()

    def loop(seed):
        rng = np.random.default_rng(seed)
        try:
            for _ in range(1500):
                v = float(rng.integers(0, 90))
                if ops.device_table(np.full(3, v), "cpu")[0] != v:
                    wrong.append(v)
        except Exception as exc:
            wrong.append(exc)

    sys.setswitchinterval(1e-6)
    try:
        threads = [threading.Thread(target=loop, args=(i,)) for i in range(8)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    finally:
        sys.setswitchinterval(interval)
    assert not wrong


@pytest.mark.gpu
def test_another_stream_reads_the_table_after_its_copy():
    values = np.random.default_rng(1).uniform(size=3000)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(a):
        torch.cuda._sleep(20_000_000)  # the copy stands behind about 10 ms of work
        t = ops.device_table(values)
    with torch.cuda.stream(b):
        u = ops.device_table(values)
        got = u.clone()
    b.synchronize()
    assert u is t
    np.testing.assert_array_equal(got.cpu().numpy(), values.astype(np.float32))


@pytest.mark.gpu
def test_a_graph_reads_the_table_of_the_warm_up():
    values = np.random.default_rng(2).uniform(size=50)
    warm = ops.device_table(values)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        t = ops.device_table(values)
        out = 2.0 * t
    assert t is warm
    for i in range(2 * ops._TABLES_MOST):  # the graph still reads it
        ops.device_table(np.full(50, float(i)))
    g.replay()
    np.testing.assert_array_equal(out.cpu().numpy(), 2.0 * values.astype(np.float32))


@pytest.mark.gpu
def test_a_table_first_met_in_a_capture_belongs_to_that_capture():
    values = np.random.default_rng(3).uniform(size=50)
    g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(g, stream=s):
        out = 2.0 * ops.device_table(values)
    with torch.cuda.stream(s):  # nothing has been replayed: the captured copy has not run
        t = ops.device_table(values)
    s.synchronize()
    np.testing.assert_array_equal(t.cpu().numpy(), values.astype(np.float32))
    g.replay()
    np.testing.assert_array_equal(out.cpu().numpy(), 2.0 * values.astype(np.float32))


@pytest.mark.gpu
def test_drift_tables_serve_any_stream():
    want = ops._drift_tables_host(jf.Planck18(), 4096)
    torch.cuda._sleep(20_000_000)
    tables = ops.drift_tables(jf.Planck18())
    with torch.cuda.stream(torch.cuda.Stream()):
        got = [t.clone() for t in tables]
        torch.cuda.current_stream().synchronize()
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g.cpu().numpy(), w)


@pytest.mark.gpu
def test_bin_edges_may_be_a_device_tensor():
    from jfli_b200.pm.adjoint import PowerSpectrum

    m = torch.randn(16, 16, 16, device="cuda", requires_grad=True)
    ke = np.linspace(0.05, 0.3, 6)
    pk = PowerSpectrum.apply(m, torch.as_tensor(ke, device="cuda"), (300.0,) * 3)
    torch.testing.assert_close(pk, PowerSpectrum.apply(m, ke, (300.0,) * 3))
