"""tcgen05 GEMM numerics against a plain fp32 PyTorch reference of the same operation."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rand(m, k, seed, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(m, k, generator=g, device="cuda") * scale).to(torch.bfloat16)


@pytest.mark.parametrize("m,n,k,bn", [(128, 256, 64, 0), (256, 512, 512, 256), (384, 448, 1024, 224), (1024, 1024, 4096, 0),
                                       (200, 264, 72, 128), (128, 3584, 8192, 0), (4096, 7168, 1024, 0),
                                       (2560, 2048, 512, 0)])   # the last two leave a small final wave on 74 CTA pairs
def test_gemm_matches_fp32_reference(m, n, k, bn):
    from purlin_b200.ops.gemm import gemm
    a, w = _rand(m, k, 1), _rand(n, k, 2, 0.05)
    out = gemm(a, w, bn=bn)
    torch.cuda.synchronize()
    ref = a.float() @ w.float().t()
    err = (out.float() - ref).abs().max().item()
    tol = 2e-2 * ref.abs().max().item() + 1e-3      # bf16 output rounding dominates
    assert err <= tol, f"max abs error {err} > {tol}"
    # a stricter check on a sample of entries in relative terms
    rel = ((out.float() - ref).abs() / (ref.abs() + 1.0)).max().item()
    assert rel < 2e-2


def test_gemm_exact_on_small_integers():
    # integer operands and K small enough that every partial sum is exact in fp32 and the result in bf16
    from purlin_b200.ops.gemm import gemm
    g = torch.Generator(device="cuda").manual_seed(0)
    a = torch.randint(-2, 3, (512, 256), generator=g, device="cuda").to(torch.bfloat16)
    w = torch.randint(-1, 2, (768, 256), generator=g, device="cuda").to(torch.bfloat16)
    out = gemm(a, w)
    ref = (a.float() @ w.float().t())
    assert torch.equal(out.float(), ref.to(torch.bfloat16).float())


def test_partial_last_wave_is_exact_on_small_integers():
    # 10 x 8 tiles on 74 CTA pairs: a full wave and a last wave of six tiles
    from purlin_b200.ops.gemm import gemm
    g = torch.Generator(device="cuda").manual_seed(1)
    a = torch.randint(-2, 3, (2560, 256), generator=g, device="cuda").to(torch.bfloat16)
    w = torch.randint(-1, 2, (2048, 256), generator=g, device="cuda").to(torch.bfloat16)
    out = gemm(a, w)
    ref = (a.float() @ w.float().t())
    assert torch.equal(out.float(), ref.to(torch.bfloat16).float())


@pytest.mark.parametrize("m,i,k", [(256, 512, 256), (1024, 3584, 2048), (2560, 1024, 512)])
def test_swiglu_epilogue(m, i, k):
    from purlin_b200.ops.gemm import gemm_swiglu, interleave_gate_up
    a, wg, wu = _rand(m, k, 3), _rand(i, k, 4, 0.05), _rand(i, k, 5, 0.05)
    out = gemm_swiglu(a, interleave_gate_up(wg, wu))
    torch.cuda.synchronize()
    g = a.float() @ wg.float().t()
    u = a.float() @ wu.float().t()
    ref = torch.nn.functional.silu(g) * u
    err = (out.float() - ref).abs().max().item()
    assert err <= 2e-2 * ref.abs().max().item() + 1e-3


def test_repeated_calls_are_bitwise_stable():
    from purlin_b200.ops.gemm import gemm
    a, w = _rand(1024, 2048, 7), _rand(2048, 2048, 8, 0.05)
    first = gemm(a, w).clone()
    for _ in range(5):
        assert torch.equal(gemm(a, w), first)


def test_one_activation_against_more_weights_than_the_map_cache_holds():
    # the tensor map of `a` is found in the cache while the weight's is made: every product has to see its own operands
    from purlin_b200.ops.gemm import gemm
    g = torch.Generator(device="cuda").manual_seed(2)
    a = torch.randint(-2, 3, (256, 128), generator=g, device="cuda").to(torch.bfloat16)
    ws = [torch.randint(-1, 2, (256, 128), generator=g, device="cuda").to(torch.bfloat16) for _ in range(20)]
    outs = [torch.empty(256, 256, device="cuda", dtype=torch.bfloat16) for _ in ws]
    for _ in range(2):
        for w, out in zip(ws, outs):
            gemm(a, w, out)
    for w, out in zip(ws, outs):
        assert torch.equal(out.float(), (a.float() @ w.float().t()).to(torch.bfloat16).float())


def _small_integers(m, n, k, seed):
    # every partial sum is exact in fp32, whatever the order, so the bf16 result is one value
    g = torch.Generator(device="cuda").manual_seed(seed)
    a = torch.randint(-2, 3, (m, k), generator=g, device="cuda").to(torch.bfloat16)
    w = torch.randint(-1, 2, (n, k), generator=g, device="cuda").to(torch.bfloat16)
    return a, w


@pytest.mark.parametrize("m,n,k", [(1, 8, 8), (1, 136, 72), (15, 264, 200), (16, 1024, 64), (17, 128, 520), (33, 640, 1024), (64, 4096, 4096),
                                    (65, 2048, 1096), (96, 384, 2048), (128, 1024, 4096), (129, 4096, 4096), (255, 4104, 4160)])
def test_few_rows_are_exact_on_small_integers(m, n, k):
    # tiles of 128 weight rows with and without a remainder, one to eight k-splits, one column up to a full pass
    from purlin_b200.ops.gemm import gemm
    a, w = _small_integers(m, n, k, 11)
    assert torch.equal(gemm(a, w).float(), (a.float() @ w.float().t()).to(torch.bfloat16).float())


@pytest.mark.parametrize("m,n,k", [(129, 8, 2048), (300, 32, 4096), (4096, 64, 2056), (1000, 256, 2112), (257, 248, 7168)])
def test_few_weight_rows_are_exact_on_small_integers(m, n, k):
    # a router's shape: the tokens are the rows of the tile
    from purlin_b200.ops.gemm import gemm
    a, w = _small_integers(m, n, k, 12)
    assert torch.equal(gemm(a, w).float(), (a.float() @ w.float().t()).to(torch.bfloat16).float())


@pytest.mark.parametrize("m,i,k", [(1, 16, 72), (16, 80, 128), (100, 3584, 512), (300, 528, 200), (777, 1024, 256), (1000, 7168, 64)])
def test_swiglu_at_odd_sizes(m, i, k):
    from purlin_b200.ops.gemm import gemm_swiglu, interleave_gate_up
    a, wg, wu = _rand(m, k, 3), _rand(i, k, 4, 0.05), _rand(i, k, 5, 0.05)
    out = gemm_swiglu(a, interleave_gate_up(wg, wu)).float()
    ref = torch.nn.functional.silu(a.float() @ wg.float().t()) * (a.float() @ wu.float().t())
    # one rounding to bf16 (2^-9 relative) on top of fp32 sums; the absolute term covers cancellation at K <= 512 of unit values
    assert ((out - ref).abs() <= 2 ** -8 * ref.abs() + 1e-4).all()


@pytest.mark.parametrize("m,n,k", [(129, 264, 72), (257, 14336, 72), (513, 8192, 136), (777, 8200, 328), (1000, 14336, 64), (2049, 4104, 72),
                                    (2368, 8192, 64)])
def test_ragged_rows_are_exact_on_small_integers(m, n, k):
    # row counts that are no multiple of a tile: narrow remainder tiles, half tiles in the last wave, more than one wave
    from purlin_b200.ops.gemm import gemm
    a, w = _small_integers(m, n, k, 13)
    assert torch.equal(gemm(a, w).float(), (a.float() @ w.float().t()).to(torch.bfloat16).float())


@pytest.mark.parametrize("likely", [1, 8, 12, 13, 400])
@pytest.mark.parametrize("counts", [[0, 1, 0, 31, 33, 0], [300, 0, 129, 1, 256, 515], [0, 0, 0, 0, 0, 700], [0, 0, 0, 0, 0, 0]])
@pytest.mark.parametrize("swiglu", [False, True])
def test_grouped_gemm(likely, counts, swiglu):
    # `likely` picks the kernel and the columns of a pass; any counts have to come out right, and rows beyond them stay as they were
    from purlin_b200.ops.gemm import grouped_gemm
    n, k, rows = 544, 136, sum(counts) + 37
    a, _ = _small_integers(rows, 8, k, 14)
    w = torch.stack([_small_integers(1, n, k, 20 + e)[1] for e in range(len(counts))])
    out = torch.full((rows, n // 2 if swiglu else n), 7.0, device="cuda", dtype=torch.bfloat16)
    grouped_gemm(a, w, torch.tensor(counts, dtype=torch.int32, device="cuda"), likely, out, swiglu=swiglu)
    first = 0
    for e, c in enumerate(counts):
        ref = a[first:first + c].float() @ w[e].float().t()
        got = out[first:first + c].float()
        if swiglu:
            v = ref.view(c, n // 32, 2, 16)
            ref = (torch.nn.functional.silu(v[:, :, 0]) * v[:, :, 1]).reshape(c, n // 2)
            assert ((got - ref).abs() <= 2 ** -8 * ref.abs() + 1e-6).all()      # one rounding to bf16
        else:
            assert torch.equal(got, ref.to(torch.bfloat16).float())
        first += c
    assert (out[first:] == 7).all()


@pytest.mark.parametrize("m", [512, 1024, 4096])
@pytest.mark.parametrize("n,bn", [(8, 0), (32, 0), (64, 0), (72, 0), (128, 0), (264, 0), (320, 0), (1000, 0), (448, 224), (320, 160), (192, 96), (72, 32)])
@pytest.mark.parametrize("swiglu", [False, True])
def test_tiles_wider_than_the_output_are_exact_on_small_integers(m, n, bn, swiglu):
    # The staging tiles of the epilogue rotate: columns past the output take none, a tile that leaves by plain stores counts like
    # one that leaves by TMA. Several calls with a short k, so that the epilogues follow each other closely.
    from purlin_b200.ops.gemm import gemm, gemm_swiglu
    n = (n + 31) // 32 * 32 if swiglu else n
    a, w = _small_integers(m, n, 72, 15)
    ref = a.float() @ w.float().t()
    if swiglu:
        v = ref.view(m, n // 32, 2, 16)
        ref = (torch.nn.functional.silu(v[:, :, 0]) * v[:, :, 1]).reshape(m, n // 2)
    for _ in range(4):
        out = torch.full(ref.shape, 7.0, device="cuda", dtype=torch.bfloat16)
        (gemm_swiglu if swiglu else gemm)(a, w, out, bn=bn)
        if swiglu:
            assert ((out.float() - ref).abs() <= 2 ** -8 * ref.abs() + 1e-6).all()      # one rounding to bf16
        else:
            assert torch.equal(out.float(), ref.to(torch.bfloat16).float())


@pytest.mark.parametrize("likely", [1, 400])
@pytest.mark.parametrize("counts", [[100, 200, 30, 300], [0, 256, 1, 0], [300, 5, 5, 5], [10, -7, 20, -1], [2 ** 31 - 1] * 4, [255] + [2 ** 31 - 1] * 45, [1] * 300])
def test_grouped_gemm_counts_never_lead_past_the_rows(likely, counts):
    # counts that add up to more than the 256 rows, and past 2^31: groups are cut at the last row, later ones are empty
    from purlin_b200.ops.gemm import grouped_gemm
    rows, n, k = 256, 40, 72
    a, w = _small_integers(rows, len(counts) * n, k, 16)
    guard = torch.full((rows + 64, n), 7.0, device="cuda", dtype=torch.bfloat16)
    grouped_gemm(a, w.view(len(counts), n, k), torch.tensor(counts, dtype=torch.int32, device="cuda"), likely, guard[32:32 + rows])
    ref, first = torch.full((rows, n), 7.0, device="cuda"), 0
    for e, c in enumerate(counts):
        end = min(first + max(c, 0), rows)
        ref[first:end] = a[first:end].float() @ w[e * n:(e + 1) * n].float().t()
        first = end
    assert torch.equal(guard[32:32 + rows].float(), ref)
    assert (guard[:32] == 7).all() and (guard[32 + rows:] == 7).all()


@pytest.mark.parametrize("swiglu", [False, True])
def test_a_wait_that_runs_out_reports_and_leaves_no_half_sums(swiglu):
    # k so long that the wait for the accumulator outlasts its limit in some CTAs of a cluster: their peers must not add what is
    # not a partial tile. A row piece is the product or untouched, the status says which wait it was, the next call is whole.
    from purlin_b200.ops.gemm import grouped_gemm
    rows, n, k = 8, 64, 1 << 21
    a = torch.zeros(rows, k, device="cuda", dtype=torch.bfloat16)
    a[:, ::4096] = 1
    w = torch.full((1, n, k), 0.125, device="cuda", dtype=torch.bfloat16)
    counts = torch.tensor([rows], dtype=torch.int32, device="cuda")
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    width = n // 2 if swiglu else n
    ref = torch.full((rows, width), 64.0 * 64.0 if swiglu else 64.0, device="cuda")      # 512 ones x 0.125; silu(64) = 64 in fp32
    out = torch.full((rows, width), 7.0, device="cuda", dtype=torch.bfloat16)
    grouped_gemm(a, w, counts, rows, out, swiglu=swiglu, status_ptr=status.data_ptr(), timeout_ns=1)
    torch.cuda.synchronize()
    assert status[0].item() == 5 and status[1].item() in (1, 3, 5)
    assert ((out == 7) | (out.float() == ref)).all()
    status.zero_()
    grouped_gemm(a, w, counts, rows, out, swiglu=swiglu, status_ptr=status.data_ptr())
    assert status[0].item() == 0 and torch.equal(out.float(), ref)


@pytest.mark.parametrize("swiglu", [False, True])
def test_a_wait_that_runs_out_in_the_kernel_of_many_rows_an_expert_reports(swiglu):
    # the same on CTA pairs (more than a dozen rows an expert): a row is the product or untouched, and the next call is whole
    from purlin_b200.ops.gemm import grouped_gemm
    rows, n, k = 16, 64, 1 << 21
    a = torch.zeros(rows, k, device="cuda", dtype=torch.bfloat16)
    a[:, ::4096] = 1
    w = torch.full((1, n, k), 0.125, device="cuda", dtype=torch.bfloat16)
    counts = torch.tensor([rows], dtype=torch.int32, device="cuda")
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    width = n // 2 if swiglu else n
    ref = torch.full((rows, width), 64.0 * 64.0 if swiglu else 64.0, device="cuda")      # 512 ones x 0.125; silu(64) = 64 in fp32
    out = torch.full((rows, width), 7.0, device="cuda", dtype=torch.bfloat16)
    grouped_gemm(a, w, counts, rows, out, swiglu=swiglu, status_ptr=status.data_ptr(), timeout_ns=1)
    torch.cuda.synchronize()
    assert status[0].item() == 5 and status[1].item() in (1, 2, 3, 5)
    assert ((out == 7) | (out.float() == ref)).all()
    status.zero_()
    grouped_gemm(a, w, counts, rows, out, swiglu=swiglu, status_ptr=status.data_ptr())
    assert status[0].item() == 0 and torch.equal(out.float(), ref)


def _swiglu_ref(a, w):
    v = (a.float() @ w.float().t()).view(a.shape[0], w.shape[0] // 32, 2, 16)
    return (torch.nn.functional.silu(v[:, :, 0]) * v[:, :, 1]).reshape(a.shape[0], w.shape[0] // 2)


@pytest.mark.parametrize("m,n,k", [(1, 7168, 8192), (33, 1024, 4096), (64, 14336, 2048), (16, 64, 8200), (128, 2080, 1032)])
def test_few_rows_swiglu_with_the_k_range_split(m, n, k):
    # gate and up are summed over a cluster of two to eight CTAs; both sums are exact, so what is left is one rounding to bf16
    from purlin_b200.ops.gemm import gemm_swiglu
    a, w = _small_integers(m, n, k, 17)
    ref = _swiglu_ref(a, w)
    assert ((gemm_swiglu(a, w).float() - ref).abs() <= 2 ** -8 * ref.abs() + 1e-6).all()


@pytest.mark.parametrize("likely,n,k,counts", [
    (1, 64, 4104, [100, 0, 515]), (1, 544, 1032, [33, 1, 0, 64, 200]),                # several passes of a cluster of eight, of four
    (12, 160, 2048, [300, 40, 0, 41]),
    (400, 96, 72, [7] * 33), (400, 64, 136, [0, 65, 1, 300] * 16), (400, 32, 72, [1, 0, 3, 2] * 128),      # 33, 64, 512 groups in the scan
    (5, 32, 72, [1, 0, 3, 2] * 128)])
@pytest.mark.parametrize("swiglu", [False, True])
def test_grouped_gemm_split_over_clusters_and_over_many_groups(likely, n, k, counts, swiglu):
    from purlin_b200.ops.gemm import grouped_gemm
    rows, experts = sum(counts) + 5, len(counts)
    a, w = _small_integers(rows, experts * n, k, 18)
    out = torch.full((rows, n // 2 if swiglu else n), 7.0, device="cuda", dtype=torch.bfloat16)
    grouped_gemm(a, w.view(experts, n, k), torch.tensor(counts, dtype=torch.int32, device="cuda"), likely, out, swiglu=swiglu)
    ref, first = torch.full(out.shape, 7.0, device="cuda"), 0
    for e, c in enumerate(counts):
        ae, we = a[first:first + c], w[e * n:(e + 1) * n]
        if c:
            ref[first:first + c] = _swiglu_ref(ae, we) if swiglu else (ae.float() @ we.float().t()).to(torch.bfloat16).float()
        first += c
    if swiglu:
        assert ((out.float() - ref).abs() <= 2 ** -8 * ref.abs() + 1e-6).all()      # one rounding to bf16
    else:
        assert torch.equal(out.float(), ref)


@pytest.mark.parametrize("m,n,k", [(33, 264, 504), (33, 264, 512), (64, 96, 72), (64, 11168, 1072), (80, 12056, 1320), (192, 5824, 4104), (65, 4096, 1536)])
@pytest.mark.parametrize("swiglu", [False, True])
def test_few_rows_around_the_limits_of_the_split(m, n, k, swiglu):
    # where the few-rows kernel begins to be used and where one more split would not have room on the GPU
    from purlin_b200.ops.gemm import gemm, gemm_swiglu
    n = (n + 31) // 32 * 32
    a, w = _small_integers(m, n, k, 19)
    if swiglu:
        ref = _swiglu_ref(a, w)
        assert ((gemm_swiglu(a, w).float() - ref).abs() <= 2 ** -8 * ref.abs() + 1e-6).all()      # one rounding to bf16
    else:
        assert torch.equal(gemm(a, w).float(), (a.float() @ w.float().t()).to(torch.bfloat16).float())


@pytest.mark.parametrize("m,n,k", [(257, 14336, 768), (513, 8192, 840), (777, 8200, 776), (1000, 14336, 832), (2049, 4104, 768), (2368, 8192, 1032), (1000, 14336, 760)])
@pytest.mark.parametrize("swiglu", [False, True])
def test_ragged_rows_with_a_k_that_hides_the_epilogue(m, n, k, swiglu):
    # the sizes of the ragged kernel's remainders and waves at the shortest k it is used for, and one below
    from purlin_b200.ops.gemm import gemm, gemm_swiglu
    n = (n + 31) // 32 * 32 if swiglu else n
    a, w = _small_integers(m, n, k, 21)
    if swiglu:
        ref = _swiglu_ref(a, w)
        assert ((gemm_swiglu(a, w).float() - ref).abs() <= 2 ** -8 * ref.abs() + 1e-6).all()      # one rounding to bf16
    else:
        assert torch.equal(gemm(a, w).float(), (a.float() @ w.float().t()).to(torch.bfloat16).float())


@pytest.mark.parametrize("m,n,k", [(200, 8192, 4104), (333, 8192, 1096), (384, 7944, 4160), (250, 4096, 4096), (97, 4128, 3080), (512, 4352, 2056), (130, 2304, 5000),
                                    (300, 1312, 1032), (1030, 14336, 520), (2048, 4096, 512), (2240, 5792, 584), (511, 18944, 648)])
@pytest.mark.parametrize("swiglu", [False, True])
def test_tiles_of_one_accumulator_and_k_shared_by_the_pairs_of_a_cluster(m, n, k, swiglu):
    # few tiles: 256 rows of W each, with columns in two halves (a multiple of 128) or not, k over one, two or four pairs, an odd last
    # k-block; many: column tiles of unequal width, a last tile of W without its second half
    from purlin_b200.ops.gemm import gemm, gemm_swiglu
    n = (n + 31) // 32 * 32 if swiglu else n
    a, w = _small_integers(m, n, k, 23)
    if swiglu:
        ref = _swiglu_ref(a, w)
        assert ((gemm_swiglu(a, w).float() - ref).abs() <= 2 ** -8 * ref.abs() + 1e-6).all()      # one rounding to bf16
    else:
        assert torch.equal(gemm(a, w).float(), (a.float() @ w.float().t()).to(torch.bfloat16).float())


@pytest.mark.parametrize("m,n,k", [(33, 8, 520), (128, 32, 7168), (97, 136, 4104), (200, 504, 7176), (129, 2080, 4096), (300, 256, 7168), (257, 200, 2056), (50, 600, 1000),
                                    (255, 1024, 3080)])
@pytest.mark.parametrize("swiglu", [False, True])
def test_few_rows_with_the_columns_of_a_tile_shared(m, n, k, swiglu):
    # few tiles: several CTAs take 32 to 64 columns each of the same weight rows (or, with few weight rows, of the same tokens); odd last groups
    from purlin_b200.ops.gemm import gemm, gemm_swiglu
    n = (n + 31) // 32 * 32 if swiglu else n
    a, w = _small_integers(m, n, k, 37)
    if swiglu:
        ref = _swiglu_ref(a, w)
        assert ((gemm_swiglu(a, w).float() - ref).abs() <= 2 ** -8 * ref.abs() + 1e-6).all()      # one rounding to bf16
    else:
        assert torch.equal(gemm(a, w).float(), (a.float() @ w.float().t()).to(torch.bfloat16).float())


@pytest.mark.parametrize("k", [8, 64, 72, 128, 136, 192, 256, 328])
@pytest.mark.parametrize("counts", [[257, 0, 300, 31], [513, 1030, 64, 65]])
def test_grouped_gemm_with_a_k_shorter_than_the_lead_of_an_accumulator(k, counts):
    from purlin_b200.ops.gemm import grouped_gemm
    n, rows = 776, sum(counts)
    a, _ = _small_integers(rows, 8, k, 29)
    w = torch.stack([_small_integers(8, n, k, 31 + e)[1] for e in range(len(counts))])
    out = torch.zeros(rows, n, dtype=torch.bfloat16, device="cuda")
    grouped_gemm(a, w, torch.tensor(counts, dtype=torch.int32, device="cuda"), 400, out)
    at = 0
    for e, c in enumerate(counts):
        assert torch.equal(out[at:at + c].float(), (a[at:at + c].float() @ w[e].float().t()).to(torch.bfloat16).float())
        at += c


@pytest.mark.parametrize("swiglu", [False, True])
@pytest.mark.parametrize("counts", [[64, 1, 0, 64, 33, 32, 64], [64, 65, 64, 0, 1], [0, 0, 300, 1, 64], [257] + [31] * 40, [640] + [20] * 31, [16] * 70, [0, 0]])
def test_grouped_gemm_of_few_rows_an_expert_and_of_one_that_has_many(counts, swiglu):
    # tiles of 64 columns and a ring of more stages where that is few more tiles (an expert of 300 rows among many), of 256 otherwise
    from purlin_b200.ops.gemm import grouped_gemm
    n, k, rows = 1056, 1096, sum(counts) + 8
    a, _ = _small_integers(rows, 8, k, 41)
    w = torch.stack([_small_integers(8, n, k, 43 + e)[1] for e in range(len(counts))])
    width = n // 2 if swiglu else n
    out = torch.full((rows, width), 7.0, dtype=torch.bfloat16, device="cuda")
    grouped_gemm(a, w, torch.tensor(counts, dtype=torch.int32, device="cuda"), 32, out, swiglu=swiglu)
    at = 0
    for e, c in enumerate(counts):
        if swiglu:
            ref = _swiglu_ref(a[at:at + c], w[e])
            assert ((out[at:at + c].float() - ref).abs() <= 2 ** -8 * ref.abs() + 1e-6).all()      # one rounding to bf16
        else:
            assert torch.equal(out[at:at + c].float(), (a[at:at + c].float() @ w[e].float().t()).to(torch.bfloat16).float())
        at += c
    assert (out[at:] == 7).all()
