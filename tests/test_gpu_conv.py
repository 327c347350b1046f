"""Convolutions that read the grid in place (k_conv_fwd, k_conv_back, k_im2col_t) against the column
matrix and its GEMM: the accumulation order is the same, so the values are equal (needs a B200)."""
import pytest

pytestmark = pytest.mark.gpu

GRIDS = ((1, 1, 2), (3, 5, 7), (2, 16, 64), (6, 33, 130))
CHANNELS = ((64, 64), (64, 128), (128, 128), (128, 64), (64, 8))


def setup(cin, cout, grid):
    import torch
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    from water_flow_simulation_b200 import _native as nat
    Z, Y, X = grid
    g = torch.Generator(device="cuda").manual_seed(cin + cout + X)
    t = dict(x=torch.randn(Z * Y * X, cin, device="cuda", generator=g).to(torch.bfloat16),
             W=(torch.randn(cout, 27 * cin, device="cuda", generator=g) * 0.05).to(torch.bfloat16),
             b=torch.randn(cout, device="cuda", generator=g),
             g=torch.randn(Z * Y * X, cout, device="cuda", generator=g).to(torch.bfloat16),
             err=torch.zeros(1, dtype=torch.int32, device="cuda"))
    return torch, nat, nat.load(), t, torch.cuda.current_stream().cuda_stream


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("cin,cout", CHANNELS)
@pytest.mark.parametrize("epi", (2, 3, 4))
def test_forward_equals_the_column_matrix_product(cin, cout, grid, epi):
    torch, nat, lib, t, st = setup(cin, cout, grid)
    Z, Y, X = grid
    V = Z * Y * X
    dt = torch.float32 if epi == 4 else torch.bfloat16
    got, want = (torch.empty(V, cout, dtype=dt, device="cuda") for _ in range(2))
    nat.check(lib.lbm_conv3_bf16(t["x"].data_ptr(), cin, X, Y, Z, t["W"].data_ptr(), cout, got.data_ptr(), epi,
                                 t["b"].data_ptr(), t["err"].data_ptr(), st), "conv")
    col = torch.empty(V, 27 * cin, dtype=torch.bfloat16, device="cuda")
    nat.check(lib.lbm_nn_im2col(t["x"].data_ptr(), cin, X, Y, Z, col.data_ptr(), st), "im2col")
    nat.check(lib.lbm_gemm_bf16(col.data_ptr(), 27 * cin, t["W"].data_ptr(), 27 * cin, V, cout, 27 * cin,
                                want.data_ptr(), cout, epi, t["b"].data_ptr(), t["err"].data_ptr(), st), "gemm")
    assert int(t["err"].item()) == 0 and torch.equal(got, want)


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("cin,cout", CHANNELS)
def test_backward_equals_the_gathered_product(cin, cout, grid):
    torch, nat, lib, t, st = setup(cin, cout, grid)
    Z, Y, X = grid
    V = Z * Y * X
    Wt = t["W"].t().contiguous()
    got, want = (torch.empty(V, cin, dtype=torch.float32, device="cuda") for _ in range(2))
    nat.check(lib.lbm_conv3_back(t["g"].data_ptr(), cout, X, Y, Z, Wt.data_ptr(), cin, got.data_ptr(),
                                 t["err"].data_ptr(), st), "conv back")
    dcol = torch.empty(V, 27 * cin, dtype=torch.float32, device="cuda")
    nat.check(lib.lbm_gemm_bf16(t["g"].data_ptr(), cout, Wt.data_ptr(), cout, V, 27 * cin, cout, dcol.data_ptr(),
                                27 * cin, 0, None, t["err"].data_ptr(), st), "gemm")
    nat.check(lib.lbm_nn_col2im(dcol.data_ptr(), cin, X, Y, Z, want.data_ptr(), st), "col2im")
    assert int(t["err"].item()) == 0 and torch.equal(got, want)


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("cin", (8, 64, 72, 128))
def test_transposed_column_matrix(cin, grid):
    torch, nat, lib, t, st = setup(cin, 8, grid)
    Z, Y, X = grid
    V = Z * Y * X
    Vp = (V + 7) // 8 * 8
    col = torch.empty(V, 27 * cin, dtype=torch.bfloat16, device="cuda")
    colT = torch.full((27 * cin, Vp), float("nan"), dtype=torch.bfloat16, device="cuda")
    nat.check(lib.lbm_nn_im2col(t["x"].data_ptr(), cin, X, Y, Z, col.data_ptr(), st), "im2col")
    nat.check(lib.lbm_nn_im2col_t(t["x"].data_ptr(), cin, X, Y, Z, Vp, colT.data_ptr(), st), "im2col_t")
    assert torch.equal(colT[:, :V], col.t()) and not bool(colT[:, V:].any())


def test_argument_errors():
    torch, nat, lib, t, st = setup(64, 8, (1, 1, 2))
    p = t["x"].data_ptr()
    e, b = t["err"].data_ptr(), t["b"].data_ptr()
    assert lib.lbm_conv3_bf16(p, 72, 2, 1, 1, p, 8, p, 2, b, e, st) == -1            # channels
    assert lib.lbm_conv3_bf16(p, 64, 2, 1, 1, p, 8, p, 1, b, e, st) == -1            # epilogue
    assert lib.lbm_conv3_bf16(p + 2, 64, 2, 1, 1, p, 8, p, 2, b, e, st) == -1        # alignment
    assert lib.lbm_conv3_back(p, 8, 2, 1, 1, p, 72, p, e, st) == -1
    assert lib.lbm_nn_im2col_t(p, 8, 2, 1, 1, 12, p, st) == -1


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("cout", (8, 40, 64, 72))
@pytest.mark.parametrize("epi", (2, 3, 4))
def test_input_layer_equals_the_column_matrix_product(cout, grid, epi):
    test_forward_equals_the_column_matrix_product(8, cout, grid, epi)


@pytest.mark.parametrize("C", (8, 12, 64))
@pytest.mark.parametrize("grid", ((2, 2, 2), (2, 6, 10), (4, 8, 66)))
def test_pooling_and_upsampling(C, grid):
    """Sums of eight in index order in float32, one rounding to bf16: equal to the same sums in torch."""
    torch, nat, lib, _, st = setup(8, 8, (1, 1, 1))
    Z, Y, X = grid
    g = torch.Generator(device="cuda").manual_seed(C + X)
    full = torch.randn(Z, Y, X, C, device="cuda", generator=g).to(torch.bfloat16)
    half = torch.randn(Z // 2, Y // 2, X // 2, C, device="cuda", generator=g).to(torch.bfloat16)

    def children(a):
        s = torch.zeros_like(half, dtype=torch.float32)
        for d in range(8):
            s = s + a[d >> 2::2, d >> 1 & 1::2, d & 1::2].float()
        return s

    def up(a):
        return a[:, None, :, None, :, None].expand(-1, 2, -1, 2, -1, 2, -1).reshape(Z, Y, X, C)
    out_h, out_f = torch.empty_like(half), torch.empty_like(full)
    nat.check(lib.lbm_nn_pool2(full.data_ptr(), C, X, Y, Z, out_h.data_ptr(), st), "pool2")
    assert torch.equal(out_h, (0.125 * children(full)).to(torch.bfloat16))
    nat.check(lib.lbm_nn_up2_add(half.data_ptr(), full.data_ptr(), C, X, Y, Z, out_f.data_ptr(), st), "up2_add")
    assert torch.equal(out_f, (up(half).float() + full.float()).to(torch.bfloat16))
    ff, hf = full.float(), half.float()
    out_hf = torch.empty_like(hf)
    nat.check(lib.lbm_nn_up2_back(ff.data_ptr(), C, X, Y, Z, out_hf.data_ptr(), st), "up2_back")
    assert torch.equal(out_hf, children(ff))
    for acc in (0, 1):
        out_ff = ff.clone()
        nat.check(lib.lbm_nn_pool2_back(hf.data_ptr(), C, X, Y, Z, out_ff.data_ptr(), acc, st), "pool2_back")
        assert torch.equal(out_ff, 0.125 * up(hf) + (ff if acc else 0))
