"""The kernels that compute in 32 bits, on the CUDA cores or on the tensor cores in parts, at the sizes where their tiles,
slabs and dispatch end, against 64-bit restatements."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _ops():
    from vipera_rs_b200.kernels import ops

    return ops


def _rel(got, want):
    return float((got.double() - want).norm() / want.norm())


# rows at the borders of the tiles (8, 32, 64, 128), columns that end inside one, inner sizes of a part of a chunk,
# of fewer than eight slabs, of slabs that end early, of rows that do not start on 16 bytes
@pytest.mark.parametrize("m", [1, 2, 3, 8, 9, 33, 64, 65, 129])
@pytest.mark.parametrize("n,k", [(64, 32), (257, 16), (33, 4), (70, 5), (96, 100), (130, 770), (200, 771), (1536, 808), (9600, 520)])
@pytest.mark.parametrize("types", ["f32", "bf16", "mixed"])
def test_product_tiles_and_slabs(m, n, k, types):
    ops = _ops()
    torch.manual_seed(m * 31 + n + k)
    a = torch.randn(m, k, device=DEV).to(torch.bfloat16 if types == "bf16" else torch.float32)
    w = torch.randn(n, k, device=DEV).to(torch.float32 if types == "f32" else torch.bfloat16)
    if types == "mixed":
        a = a.to(torch.float32)
    bias = torch.randn(n, device=DEV)
    out = torch.full((m, n), float("nan"), device=DEV)
    ops.gemm_simt(a, w, epilogue=ops.EPI_STORE, bias=bias, out=out)
    # the error of a chain of k roundings of random sign, 2^-24 each, is some sqrt(k) 2^-24 of the sum at most
    assert _rel(out, a.double() @ w.double().T + bias.double()) < 2.0 ** -24 * (k ** 0.5 + 4)
    # a row's result does not depend on the rows beside it, within its class (up to eight rows, up to 64, more)
    beside = 1 if m <= 8 else 9 if m <= 64 else 65
    last = torch.empty(beside, n, device=DEV)
    ops.gemm_simt(a[-beside:].contiguous(), w, epilogue=ops.EPI_STORE, bias=bias, out=last)
    assert torch.equal(last[-1], out[-1])


# inner sizes short enough to lie in shared memory whole (up to 320, and the next), rows that are and are not whole pieces,
# all endings and types of the output
@pytest.mark.parametrize("k", [1, 63, 128, 130, 256, 319, 320, 321])
@pytest.mark.parametrize("m,n", [(1, 32), (9, 160), (31, 96), (33, 128), (100, 288)])
@pytest.mark.parametrize("epilogue", [0, 1, 2])
@pytest.mark.parametrize("types", ["f32", "bf16", "mixed"])
def test_short_products(m, n, k, epilogue, types):
    ops = _ops()
    torch.manual_seed(m + n + k)
    a = (torch.randn(m, k, device=DEV) * k ** -0.5).to(torch.bfloat16 if types == "bf16" else torch.float32)
    w, bias = torch.randn(n, k, device=DEV).to(torch.float32 if types == "f32" else torch.bfloat16), torch.randn(n, device=DEV)
    y = a.double() @ w.double().T + bias.double()
    if epilogue == 2:
        gate, up = y.view(m, n // 32, 2, 16)[:, :, 0], y.view(m, n // 32, 2, 16)[:, :, 1]
        y = (up * gate * torch.sigmoid(gate)).reshape(m, n // 2)
    out = torch.randn(m, y.shape[1], device=DEV)
    want = y + out.double() if epilogue == 1 else y
    ops.gemm_simt(a, w, epilogue=epilogue, bias=bias, **({"resid": out} if epilogue == 1 else {"out": out}))
    # k roundings of random sign, 2^-24 each, and those of the ending
    assert _rel(out, want) < 2.0 ** -24 * (k ** 0.5 + 8)
    if epilogue == 0:
        narrow = torch.empty(m, n, device=DEV, dtype=torch.bfloat16)
        ops.gemm_simt(a, w, epilogue=epilogue, bias=bias, out=narrow)
        assert torch.equal(narrow, out.bfloat16())
        # a row's result does not depend on the rows beside it (from nine rows on)
        if m > 17:
            last = torch.empty(9, n, device=DEV)
            ops.gemm_simt(a[-9:].contiguous(), w, epilogue=epilogue, bias=bias, out=last)
            assert torch.equal(last, out[-9:]) or (types == "f32" and k > 128 and m > 64)


# the tensor-core form of many rows: tiles that end inside, one block and clusters of two and four that share K (one
# share may be empty), all endings, numbers of very different sizes, and numbers that have no parts
@pytest.mark.parametrize("m,n,k", [(65, 32, 4), (128, 128, 64), (129, 160, 68), (200, 96, 700), (300, 1152, 896), (1024, 896, 4864), (70, 5024, 300)])
@pytest.mark.parametrize("epilogue", [0, 1, 2])
def test_product_in_parts(m, n, k, epilogue):
    ops = _ops()
    torch.manual_seed(m + n + k)
    a = torch.randn(m, k, device=DEV) * torch.exp(4 * torch.randn(m, 1, device=DEV))
    w, bias = torch.randn(n, k, device=DEV), torch.randn(n, device=DEV)
    y = a.double() @ w.double().T + bias.double()
    if epilogue == 2:
        a = a / a.norm(dim=1, keepdim=True)
        y = a.double() @ w.double().T + bias.double()
        gate, up = y.view(m, n // 32, 2, 16)[:, :, 0], y.view(m, n // 32, 2, 16)[:, :, 1]
        y = (up * gate * torch.sigmoid(gate)).reshape(m, n // 2)
    out = torch.randn(m, y.shape[1], device=DEV)
    want = y + out.double() if epilogue == 1 else y
    ops.gemm_simt(a, w, epilogue=epilogue, bias=bias, **({"resid": out} if epilogue == 1 else {"out": out}))
    torch.cuda.synchronize()
    ops.check_kernel_status(a.device)
    # no worse than a chain of k roundings of 2^-24, row by row
    error = (out.double() - want).norm(dim=1) / want.norm(dim=1)
    assert float(error.max()) < 2.0 ** -24 * (k ** 0.5 + 6)


# Numbers whose parts are as large as they get and of one sign: what the left-out products of parts come to does not
# average out.  Cut-off parts of 1 + 2^-7 - 2^-23 would leave out 4.7e-7 of every product; rounded ones leave out 2^-24 at most.
@pytest.mark.parametrize("value", [1 + 2.0 ** -7 - 2.0 ** -23, 1 + 2.0 ** -8 - 2.0 ** -23, 1 + 2.0 ** -8 + 2.0 ** -16 - 2.0 ** -23, 1.99999988079071])
@pytest.mark.parametrize("m,n,k", [(65, 64, 192), (256, 256, 2048)])
def test_product_in_parts_of_one_sign(value, m, n, k):
    ops = _ops()
    a, w = torch.full((m, k), value, device=DEV), torch.full((n, k), value, device=DEV)
    a[1::2] *= -0.5
    out = torch.empty(m, n, device=DEV)
    ops.gemm_simt(a, w, epilogue=ops.EPI_STORE, out=out)
    want = a.double() @ w.double().T
    # 2^-24 of what is left out, 2^-24 a step of the tensor cores' four within 64 values (the leading product's: towards zero),
    # half of 2^-24 a sum of K / 64 in a row
    assert float((out.double() / want - 1).abs().max()) < 2.0 ** -24 * (1 + 4 + 0.5 * k / 64)


# positive numbers: the tensor cores' rounding towards zero does not average out either, and is held against what one chain
# of fused multiply-adds loses
def test_product_in_parts_of_positive_numbers():
    ops = _ops()
    torch.manual_seed(3)
    a, w = torch.rand(300, 4864, device=DEV), torch.rand(256, 4864, device=DEV)
    out, chain = torch.empty(300, 256, device=DEV), torch.zeros(300, 256, device=DEV)
    ops.gemm_simt(a, w, epilogue=ops.EPI_STORE, out=out)
    for k in range(4864):
        torch.addcmul(chain, a[:, k:k + 1], w[:, k].view(1, -1), out=chain)
    want = a.double() @ w.double().T
    assert _rel(out, want) < _rel(chain, want) < 2.0 ** -24 * 4864


# a number above bfloat16's largest, a finite one, has no leading part: its row is computed with multiply-adds
def test_product_in_parts_of_large_numbers():
    ops = _ops()
    torch.manual_seed(4)
    a, w = torch.randn(130, 512, device=DEV), torch.randn(96, 512, device=DEV)
    a[77, 5], a[90, 500] = 3.4028e38, -3.4028e38
    w[:, 5], w[:, 500] = w[:, 5] * 1e-3, w[:, 500] * 1e-3
    out = torch.empty(130, 96, device=DEV)
    ops.gemm_simt(a, w, epilogue=ops.EPI_STORE, out=out)
    want = a.double() @ w.double().T
    assert float(((out.double() - want).norm(dim=1) / want.norm(dim=1)).max()) < 2.0 ** -24 * (512 ** 0.5 + 6)


# a row of more than 64 is summed in one order, whatever the count of rows, its place among them, how many blocks share its
# K (one, two and four), and what splits its numbers (its own block or the kernel ahead)
@pytest.mark.parametrize("n,k", [(9728, 896), (1152, 896), (896, 4864), (256, 2048), (160, 700), (2048, 1540), (6144, 2048)])
def test_a_row_of_many_does_not_depend_on_the_others(n, k):
    ops = _ops()
    torch.manual_seed(n + k)
    a, w = torch.randn(4200, k, device=DEV), torch.randn(n, k, device=DEV)
    whole = torch.empty(4200, n, device=DEV)
    ops.gemm_simt(a, w, epilogue=ops.EPI_STORE, out=whole)
    for m in (65, 130, 257, 500, 700, 1100, 2300):
        out = torch.empty(m, n, device=DEV)
        ops.gemm_simt(a[-m:].contiguous(), w, epilogue=ops.EPI_STORE, out=out)
        assert torch.equal(out, whole[-m:]), m
    ops.check_kernel_status(a.device)


# more rows than the room for the left operand's parts holds are taken in turns: every ending's rows are those of products of
# one turn
@pytest.mark.parametrize("epilogue,dtype", [(0, torch.float32), (0, torch.bfloat16), (1, torch.float32), (2, torch.float32), (2, torch.bfloat16)])
def test_rows_in_turns(epilogue, dtype):
    ops = _ops()
    m, n, k, one = 2400, 160, 14336, 700
    of_tile, room = ops.gemm_simt_room(128, n, k), ops.gemm_simt_room(m, n, k)
    assert room < -(-m // 128) * of_tile // 2 and ops.gemm_simt_room(one, n, k) == -(-one // 128) * of_tile   # three turns, and one
    torch.manual_seed(epilogue)
    a, w, bias = torch.randn(m, k, device=DEV) * k ** -0.5, torch.randn(n, k, device=DEV), torch.randn(n, device=DEV)
    before = torch.randn(m, n // 2 if epilogue == 2 else n, device=DEV).to(dtype)

    def product(rows):
        out = before[rows].clone()
        ops.gemm_simt(a[rows].contiguous(), w, epilogue=epilogue, bias=bias, **({"resid": out} if epilogue == 1 else {"out": out}))
        return out

    whole = product(slice(0, m))
    for first in range(0, m, one):
        rows = slice(min(first, m - one), min(first, m - one) + one)
        assert torch.equal(whole[rows], product(rows)), first
    if epilogue == 0 and dtype == torch.float32:
        assert _rel(whole, a.double() @ w.double().T + bias.double()) < 2.0 ** -24 * (k ** 0.5 + 6)
    ops.check_kernel_status(a.device)


# rows with an infinity or a NaN in the forms that split both operands and that split the left one ahead, one block and
# clusters: what such a row gives is as multiply-adds give it, and the rows beside it do not notice
@pytest.mark.parametrize("m,n,k,ahead", [(140, 130, 256, False), (256, 256, 2048, True), (1024, 896, 1300, True)])
def test_product_in_parts_without_parts(m, n, k, ahead):
    ops = _ops()
    assert (ops._function("gemm_simt", "vipera_gemm_simt_parts", [ops._c_int] * 3)(m, n, k) > 0) == ahead
    torch.manual_seed(m + n + k)
    a, w = torch.randn(m, k, device=DEV), torch.randn(n, k, device=DEV)
    clean, out = torch.empty(m, n, device=DEV), torch.empty(m, n, device=DEV)
    a[0, 7], w[4, 7] = 1.0, 0.0
    ops.gemm_simt(a, w, epilogue=ops.EPI_STORE, out=clean)
    a[3, 7], a[5, 9], a[m - 3, k - 56], a[64, 1], w[n - 1, k - 1] = (float(x) for x in ("inf", "nan", "-inf", "-nan", "inf"))
    a[70, 3], a[70, k - 3] = float("inf"), float("-inf")
    ops.gemm_simt(a, w, epilogue=ops.EPI_STORE, out=out)
    ops.check_kernel_status(a.device)
    want = a.double() @ w.double().T
    assert torch.equal(torch.isnan(out), torch.isnan(want)) and torch.equal(torch.isinf(out), torch.isinf(want))
    fine = torch.isfinite(want)
    assert torch.equal(out[torch.isinf(want)].sign(), want[torch.isinf(want)].float().sign())
    assert torch.equal(out[fine], clean[fine])
    assert int(fine.sum()) == (m - 5) * (n - 1)


def _attention_want(q, keys, values, entry, position, heads, kv_heads, scale, mask, sink, chunk, window, keep_first, gate):
    out = torch.zeros(len(q), heads, values[0].shape[-1], dtype=torch.float64)
    for t in range(len(q)):
        e, p = int(entry[t]), int(position[t])
        j = torch.arange(p + 1)
        first = p // chunk * chunk if chunk else (max(0, p - window + 1) if window else 0)
        seen = (j >= first) | ((j < keep_first) if window else (j < 0))
        for h in range(heads):
            k, v = keys[e][: p + 1, h // (heads // kv_heads)][seen], values[e][: p + 1, h // (heads // kv_heads)][seen]
            score = (k.double() @ q[t, h].double()) * scale
            if sink is not None:
                score = torch.cat([score, sink[h:h + 1].double()])
            out[t, h] = torch.softmax(score, 0)[: len(k)] @ v.double()
    return out * torch.sigmoid(gate.double()).view(len(q), heads, 1)


# counts of tokens at the borders of two forms (64) and of a tile (64 rows, several requests in one), head sizes of
# every instance, rows that are not whole 16-byte pieces, every mask, narrow (a warp per token and head takes most of those) and
# wide; a value nobody may see yet is infinite
@pytest.mark.parametrize("counts,firsts", [([1], [0]), ([1, 1, 1], [5, 130, 700]), ([7, 40, 1, 30, 7], [100, 3, 64, 0, 33]), ([64], [3]), ([65], [0]), ([1, 70, 130, 1], [90, 0, 65, 200]),
                                          ([1, 1, 70, 1, 1, 1], [0, 3, 40, 200, 7, 64])])
@pytest.mark.parametrize("d,dv,heads,kv_heads", [(64, 64, 7, 1), (128, 96, 4, 2), (80, 256, 12, 1), (30, 18, 2, 2)])
@pytest.mark.parametrize("mask", ["all", "window", "chunk", "wide window", "wide chunk"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_attention_forms(counts, firsts, d, dv, heads, kv_heads, mask, dtype):
    ops = _ops()
    torch.manual_seed(sum(counts) + d + dv)
    page, entries = 16, len(counts)
    longest = max(c + f for c, f in zip(counts, firsts))
    width = -(-longest // page)
    table = torch.randperm(entries * width).view(entries, width).to(torch.int32)
    k_pool = torch.full((entries * width, page, kv_heads, d), float("nan")).to(dtype)
    v_pool = torch.full((entries * width, page, kv_heads, dv), float("nan")).to(dtype)
    keys, values = [], []
    for e, (c, f) in enumerate(zip(counts, firsts)):
        k, v = torch.randn(c + f, kv_heads, d).to(dtype), torch.randn(c + f, kv_heads, dv).to(dtype)
        if c > 1:
            v[-1] = float("inf")
        at = torch.arange(c + f)
        k_pool[table[e].long()[at // page], at % page], v_pool[table[e].long()[at // page], at % page] = k, v
        keys.append(k)
        values.append(v)
    entry = torch.cat([torch.full((c,), e, dtype=torch.int32) for e, c in enumerate(counts)])
    position = torch.cat([torch.arange(f, f + c, dtype=torch.int32) for c, f in zip(counts, firsts)])
    tokens, scale = sum(counts), d ** -0.5
    q = torch.randn(tokens, heads, d).to(dtype)
    sink, gate = torch.randn(heads), torch.randn(tokens, heads)
    options = {"all": dict(window=0, keep_first=0, chunk=0), "window": dict(window=50, keep_first=3, chunk=0),
               "chunk": dict(window=0, keep_first=0, chunk=48), "wide window": dict(window=600, keep_first=7, chunk=0),
               "wide chunk": dict(window=0, keep_first=0, chunk=520)}[mask]
    learned = sink if "chunk" not in mask else None
    want = _attention_want(q, keys, values, entry, position, heads, kv_heads, scale, mask, learned, gate=gate, **options)
    out = torch.full((tokens, heads * dv), float("nan"), device=DEV, dtype=dtype)
    ops.attention(q.view(tokens, -1).to(DEV), out, k_pool.to(DEV), v_pool.to(DEV), token_seq=entry.to(DEV), positions=position.to(DEV),
                  block_table=table.to(DEV), num_heads=heads, num_kv_heads=kv_heads, head_dim=d, scale=scale, value_dim=dv,
                  sink_values=None if learned is None else learned.to(DEV), gate=gate.to(DEV), gate_per_head=True, **options)
    got = out.double().cpu().view(tokens, heads, dv)
    last = torch.zeros(tokens, dtype=torch.bool)
    for e, c in enumerate(counts):
        last |= (entry == e) & (position == firsts[e] + c - 1) & (c > 1)
    assert torch.isinf(got[last]).all() and torch.isfinite(got[~last]).all()
    # 32-bit: a few roundings of 2^-24 per term, bfloat16: the output's own rounding
    if (~last).any():
        assert _rel(got[~last], want[~last]) < (2e-6 if dtype == torch.float32 else 4e-3)
