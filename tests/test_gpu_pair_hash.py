"""GPU parity of the compressions that two warps share: every split of a tail's warps into hash, helper and workers (the lines at which
the helper starts lie at 128 or 512 elements a warp), byte-aligned and ragged streams, against the CPU oracle, bit-exact."""
import numpy as np
import pytest

import zklm_compile_b200 as zk
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu
P = (1 << 31) - 1
PROVE = {"product": zk.prove_product, "product_ef_full": zk.prove_product_ef_full, "triple": zk.prove_triple, "product_ef": zk.prove_product_ef}


@pytest.fixture(scope="module")
def ctx():
    c = zk.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("option,kind,threads", [("OPT_PIPE_THREADS", k, t) for k in ("product", "product_ef_full") for t in (96, 128, 160, 224, 256, 512)] +
                         [("OPT_SINGLE_CTA_THREADS", k, t) for k in ("triple", "product_ef") for t in (64, 96, 1024)])
def test_tails_match_oracle(ctx, option, kind, threads):
    rng = np.random.default_rng(threads)
    ctx.set_option(getattr(ctx, option), threads)
    try:
        for nv in (1, 2, 8, 10, 12):
            label = b"pair"[: nv % 5]                  # the four alignments of the stream
            tabs = [rng.integers(0, P, (1 << nv, 4) if kind.endswith("full") else 1 << nv, dtype=np.int64).astype(np.uint32)
                    for _ in range(3 if kind == "triple" else 2)]
            t, o = zk.Transcript(ctx, label), O.Transcript(label)
            proof, *finals = PROVE[kind](*tabs, nv, t)
            ref = O.prove(kind, o, tabs, nv)
            assert proof.round_polys.reshape(nv, -1).tolist() == ref[0].reshape(nv, -1).tolist()
            assert proof.challenges.reshape(nv, -1).tolist() == ref[1].reshape(nv, -1).tolist()
            assert t.squeeze_ef().tolist() == o.squeeze_ef().tolist()
    finally:
        ctx.set_option(getattr(ctx, option), 0)


@pytest.mark.parametrize("heads,seq,d", [(1, 31, 2), (2, 16, 16), (3, 21, 17), (11, 8, 21), (2, 32, 8), (3, 23, 17)])
def test_attention_transcript_at_the_host_absorb_line(ctx, heads, seq, d):
    """Streams of 1023, 1024, 2394, 2552, 2560 and 2760 words: the caller's transcript absorbs them on the device below 2560 words, on the host
    from there on."""
    from zklm_compile_b200 import attention, tables
    rng = np.random.default_rng(seq)
    q, k = (np.mod(rng.integers(-1, 2, heads * seq * d), P).astype(np.uint32) for _ in range(2))
    v = rng.integers(0, P, heads * seq * d, dtype=np.int64).astype(np.uint32)
    table = tables.build_exp_table(100)
    for label in (b"", b"abc"):                        # an aligned stream and a ragged one
        t, o = zk.Transcript(ctx, label), O.Transcript(label)
        proof = attention.prove_row_attention(q, k, v, heads, seq, d, table, t)
        ref, status = O.prove_row_attention(o, q, k, v, heads, seq, d, table)
        assert status == 0 and bytes(proof) == bytes(ref)
        t2 = zk.Transcript(ctx, label)
        assert attention.verify_row_attention(proof, k, v, heads, seq, d, t2)
        assert t.squeeze_ef().tolist() == o.squeeze_ef().tolist() == t2.squeeze_ef().tolist()


def test_op_list_whose_attention_streams_the_host_absorbs(ctx):
    """Two attention ops of 2560 and 2760 words, behind and in front of other ops of the same transcript; a second proof on the same list."""
    from zklm_compile_b200 import oplist, tables
    rng = np.random.default_rng(9)
    table = tables.build_exp_table(100)
    small = lambda n: np.mod(rng.integers(-1, 2, n), P).astype(np.uint32)
    shapes = [(2, 32, 8), (3, 23, 17)]
    x = small(int(np.prod(shapes[0])))
    g, o = oplist.OpList(ctx, len(x)), O.OpList()
    for i, (h, s, d) in enumerate(shapes):
        n = h * s * d
        if i:
            q = small(n)
            g.set_input("in", q); o.set_input("in", q)
        k, v = small(n), rng.integers(0, P, n, dtype=np.int64).astype(np.uint32)
        g.attention("attn%d" % i, h, s, d, ctx.upload(table), k, v); o.attention("attn%d" % i, h, s, d, table, k, v)
        w = rng.integers(0, P, (5 + i, n), dtype=np.int64).astype(np.uint32)
        g.linear("out%d" % i, w, None, 5 + i, n); o.linear("out%d" % i, w, None, 5 + i, n)
    want = o.prove(x)
    assert g.prove(x) == want and g.prove(x) == want
