"""Calls that put work on a context's second stream join it to the first on every way out.  An error in between (the record buffer is
exhausted, a runtime call fails) returns a status, and the next call may use the arena again, so nothing may still be running that
the context's stream has not been made to wait for.  Shown on the CPU, against a runtime that only keeps the order of the
operations (tests/cabi/fake_cudart.c)."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INCLUDE = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")

DRIVER = r"""
import ctypes as C
import sys
import numpy as np
import zklm_compile_b200 as zk
from tests.util import rand_layer
from zklm_compile_b200 import _lib, attention, pcs, qwen, tables
from oracle import pyoracle as O

fake = C.CDLL(None)
fake.fake_calls.restype = fake.fake_waits.restype = fake.fake_unordered.restype = fake.fake_graph_flags.restype = C.c_long
fake.fake_unordered.argtypes = [C.c_void_p]
fake.fake_fail_at.argtypes = [C.c_long]
ctx = zk.Context(0)
ctx_stream = _lib.lib().zkb_ctx_stream
ctx_stream.restype, ctx_stream.argtypes = C.c_void_p, [C.c_void_p]
main = ctx_stream(ctx.h)

def poly(n):
    return np.arange(n, dtype=np.uint32)

def batch(sizes):
    b = pcs.BasefoldBatch(ctx, [poly(n) for n in sizes], [max(1, (n - 1).bit_length()) for n in sizes])
    return lambda tr: b.prove(tr)

def basefold(n):
    log_n = (n - 1).bit_length()
    return lambda tr: pcs.basefold_commit_and_prove(ctx, tr, poly(n), poly(log_n))

def basefold_verify(n):
    log_n = (n - 1).bit_length()
    blob = pcs.basefold_commit_and_prove(ctx, zk.Transcript(ctx, b"p"), poly(n), poly(log_n))
    return lambda tr: pcs.basefold_verify_opening(ctx, tr, blob, poly(log_n), 0)

def batch_verify(sizes):
    blob = batch(sizes)(zk.Transcript(ctx, b"p"))
    return lambda tr: pcs.basefold_batch_verify_opening(ctx, tr, blob)

T = tables.build_exp_table(100)

def attention_prove(H=2, S=5, D=8):
    Q, V = np.ones(H * S * D, np.uint32), poly(H * S * D)
    return lambda tr: attention.prove_row_attention(Q, Q, V, H, S, D, T, tr)

def attention_verify(H=2, S=5, D=8):
    Q, V = np.ones(H * S * D, np.uint32), poly(H * S * D)
    blob, status = O.prove_row_attention(O.Transcript(b"p"), Q, Q, V, H, S, D, T)     # a proof of zeros would be turned away before any launch
    assert status == 0
    return lambda tr: attention.verify_row_attention(blob, Q, V, H, S, D, tr)

KEEP = []

def layer(binding, graph=False, d_model=24, d_ff=40, d_head=8):
    silu, sigmoid = ctx.upload(tables.build_silu_table(1000)), ctx.upload(tables.build_sigmoid_table(1000))
    cfg, weights, x = rand_layer(1, d_model=d_model, d_ff=d_ff, heads=2, kv=1, d_head=d_head)
    L = qwen.QwenLayer(ctx, cfg, weights, silu, sigmoid)
    L.set_binding(binding)
    L.use_graph(graph)
    L.forward(x)
    KEEP.append(L)                           # freeing one waits for the device
    return lambda tr: L.prove(0, bytes(32))

def in_order(what):
    left = fake.fake_unordered(main)
    assert left == 0, "%s: %d operations of the second stream are not joined" % (what, left)
    assert ctx_stream(ctx.h) == main, "%s: the context's stream was not given back" % what

if sys.argv[1] == "exhausted":
    # a large polynomial and 1100 that join it with 48 paths each: more words than the record buffer holds
    prove = batch([1 << 14] + [1 << 10] * 1100)
    tr = zk.Transcript(ctx, b"t")            # kept: freeing one waits for the whole device
    try:
        prove(tr)
        raise SystemExit("accepted")
    except zk.ZkbError as e:
        assert "proof record buffer exhausted" in str(e), e
    in_order("record buffer exhausted")
    ok = batch([1 << 14, 1 << 10])
    ok(tr)
    in_order("the call behind it")
elif sys.argv[1] == "graph":
    prove = layer(2, True)
    for i in range(3):                       # launch by launch, captured, replayed
        prove(None)
        in_order("proof %d" % i)
        assert KEEP[0].graph_state() == (1, 2, 2)[i], (i, KEEP[0].graph_state())
    use_node_priority = 8
    assert fake.fake_graph_flags() & use_node_priority, "a replay runs every kernel at the priority of the stream it is launched into"
elif sys.argv[1] == "waits":
    tr = zk.Transcript(ctx, b"t")
    for make in (attention_prove, attention_verify):
        waits = []
        for shape in ((2, 5, 8), (1, 32, 32), (11, 8, 21), (2, 32, 8), (3, 23, 17)):      # 130, 2048, 2552, 2560, 2760 words
            call = make(*shape)
            call(tr)
            before = fake.fake_waits()
            call(tr)
            waits.append(fake.fake_waits() - before)
        assert waits == [waits[0]] * 3 + [waits[0] + 1] * 2, waits
elif sys.argv[1] == "arena":
    # Matrices of 2^22 coefficients, every one bound by an opening: 42 bytes a coefficient are in use at most (codeword and tree 20, those of
    # the folds 20, values 2), and the first proof asks for them in pieces of 64 MB and more.
    for in_order_option in (0, 1):
        ctx = zk.Context(0)
        KEEP.append(ctx)
        ctx.set_option(ctx.OPT_BASEFOLD_IN_ORDER, in_order_option)
        prove = layer(2, False, d_model=1024, d_ff=4096, d_head=128)
        for _ in range(3):
            prove(None)
        assert ctx.scratch_bytes <= 64 << 22, ctx.scratch_bytes
else:
    call = eval(sys.argv[1])
    tr = zk.Transcript(ctx, b"t")
    call(tr)
    in_order("no failure")
    fake.fake_fail_at(-1)
    call(tr)
    n = fake.fake_calls()
    refused = 0
    for i in range(n):
        fake.fake_fail_at(i)
        try:
            call(tr)
        except zk.ZkbError:
            refused += 1
        fake.fake_fail_at(-1)
        in_order("runtime call %d of %d fails" % (i, n))
        call(tr)
        in_order("the call behind it")
    assert refused > n // 2, (refused, n)
    print(n, refused)
import os
sys.stdout.flush()
os._exit(0)                                  # nothing is freed: that waits for streams of contexts that are gone
"""


@pytest.fixture(scope="module")
def runtime(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("fake") / "libfake_cudart.so")
    subprocess.run(["gcc", "-std=gnu11", "-O1", "-Wall", "-Werror", "-shared", "-fPIC", "-I", CUDA_INCLUDE,
                    os.path.join(ROOT, "tests", "cabi", "fake_cudart.c"), "-o", out], check=True)
    return out


def run(runtime, what):
    env = dict(os.environ, LD_PRELOAD=runtime, PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", DRIVER, what], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


def test_batch_that_exhausts_the_record_buffer(runtime):
    run(runtime, "exhausted")


def test_replays_of_a_layer_proof_keep_the_priorities_of_their_streams(runtime):
    run(runtime, "graph")


def test_commitments_ahead_take_no_more_memory_than_between_the_openings(runtime):
    run(runtime, "arena")


def test_short_streams_of_row_attention_do_not_make_the_host_wait(runtime):
    run(runtime, "waits")


@pytest.mark.parametrize("call", ["basefold(5000)", "batch([1 << 14, 1 << 13, 1 << 13, 300, 7])", "basefold_verify(300)", "batch_verify([300, 70])",
                                  "attention_prove()", "attention_verify()", "attention_prove(2, 32, 32)", "attention_verify(2, 32, 32)", "layer(1)", "layer(2)"])
def test_any_failing_runtime_call(runtime, call):
    run(runtime, call)
