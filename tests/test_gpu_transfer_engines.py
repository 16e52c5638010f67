"""The copy-hardware transfer engines against the register engine and the PyTorch oracle, at the sizes where their hand-out of pages can
go wrong: fewer pages than CTAs, chunks that do not divide the page count, one head, eight heads over four destinations."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,layers,heads,n_dst,ppc,ctas", [(1, 1, 8, 1, 8, None), (3, 5, 8, 4, 7, None), (2, 3, 1, 1, 5, 4), (40, 36, 8, 2, 8, None),
                                                         (9, 2, 6, 3, 1, 300)])
@pytest.mark.parametrize("form", ["bf16", "fp8", "keep"])
def test_copy_engines_move_the_bytes_of_the_register_engine(form, n, layers, heads, n_dst, ppc, ctas):
    import skygdr_b200.ops as ops

    torch.manual_seed(n * 31 + heads)
    if form == "keep":
        n_dst = 1
    hd = heads // n_dst
    g = ops.KVGeometry(layers=layers, kv_heads=heads)
    src = ops.PagedKVPool(g, n + 2, "nhd")
    src.data.normal_()
    src.data[0] = 0                                   # zero groups have a scale of their own
    sb, db = torch.randperm(n + 2, device="cuda")[:n].int(), torch.randperm(n + 1, device="cuda")[:n].int()
    got = {}
    for method in ("auto", "simt"):
        if form == "keep":
            bufs = [torch.zeros((n + 1, *src.data.shape[1:]), dtype=torch.bfloat16, device="cuda")]
            rem = [ops.RemotePool(bufs[0].data_ptr(), src.strides, heads, num_blocks=n + 1)]
        else:
            dt = torch.uint8 if form == "fp8" else torch.bfloat16
            bufs = [torch.zeros((n + 1, layers, 2, hd, 16, 128), dtype=dt, device="cuda") for _ in range(n_dst)]
            sc = [torch.zeros((n + 1, layers, 2, hd, 16, 4), dtype=torch.uint8, device="cuda") for _ in range(n_dst)] if form == "fp8" else []
            rem = [ops.RemotePool(b.data_ptr(), b.stride()[:3], hd, sc[i].data_ptr() if sc else 0, 0, n + 1) for i, b in enumerate(bufs)]
            bufs = bufs + sc
        flow = ops.KvTransferFlow("cuda", page=ops.CreditPage(unlimited=True), pages_per_chunk=ppc, ctas=ctas, method=method)
        for _ in range(2):                            # the second launch finds the working block as the first one left it
            flow.transfer(src, rem, sb, db, fp8=form == "fp8", keep_layout=form == "keep")
            st = flow.result()
            assert st["status"] == 0 and st["bytes_done"] == ops.link_bytes(g, n, fp8=form == "fp8") and st["cursor"] == 2**64 - 1
            assert st["chunks_done"] == -(-n * layers * 2 // ppc)
        assert flow.page.read()["completed_bytes"] == flow.consumed == 2 * st["bytes_done"]
        got[method] = bufs
    assert all(torch.equal(a, b) for a, b in zip(got["auto"], got["simt"]))
    if form == "bf16":
        for i, b in enumerate(got["auto"]):
            assert torch.equal(b[db.long()], ops.reference_transfer(src, sb, slice(i * hd, (i + 1) * hd)))


def test_a_refused_flow_stops_and_a_stopped_one_leaves_a_cursor():
    import skygdr_b200.ops as ops

    g = ops.KVGeometry(layers=4)
    n = 64
    src, dst = ops.PagedKVPool(g, n, "nhd"), ops.PagedKVPool(g, n, "hnd")
    src.data.normal_()
    ids = torch.arange(n, device="cuda").int()
    total = ops.link_bytes(g, n)
    page = ops.CreditPage(unlimited=False)
    flow = ops.KvTransferFlow("cuda", page=page, max_wait_ms=1.0)
    page.grant(total // 3)
    flow.transfer(src, [ops.RemotePool.of(dst)], ids, ids)
    st = flow.result()
    assert st["status_name"] == "YIELD_CREDIT" and st["bytes_done"] <= total // 3
    page.grant(total, stop=True)
    flow.resume(st)
    st2 = flow.result()
    assert st2["status_name"] == "STOPPED" and st2["bytes_done"] == 0 and st2["cursor"] == st["cursor"]
    page.grant(2 * total)
    flow.resume(st2)
    assert flow.result()["status"] == 0
    assert torch.equal(dst.data, ops.reference_transfer(src, ids))
