"""The prompt GEMM against the verify GEMV in pieces of 32 rows, plane by plane and bit for bit: every cut (column tiles per
range, weight tiles per item) on shapes whose K parts are odd and even numbers of blocks, longer than the rings, whose CTAs
take one and several items, with ragged last tiles, column ranges and rows. Both launchers are internal to the library
(csrc/kernels.h), so they are called by their C++ names. Which cut a call takes is a rule on its sizes (gemm_cut)."""
import ctypes

import pytest
import torch

import hipster_b200 as hb
from hipster_b200 import kernels as K_

CUTS = [(ntc, G) for ntc in (4, 6, 8, 10, 12, 14, 16) for G in (8, 4)]
SHAPES = [(100, 5120), (4999, 5120), (2100, 17408), (34816, 1024), (4096, 768), (40, 256)]


class XQ8F(ctypes.Structure):
    _fields_ = [("q", ctypes.c_void_p), ("sc", ctypes.c_void_p)]


def sym(name, *argtypes):
    f = getattr(hb.lib(), name)
    f.argtypes = argtypes
    return f


CUT = "_ZN2hp15gemm_q4k_q8_cutEPKvRKNS_4XQ8FEPfiiiimPvPiP11CUstream_stbii"
P, I, Z, B = ctypes.c_void_p, ctypes.c_int, ctypes.c_size_t, ctypes.c_bool


def gemm_cut(N, K, R):
    f = sym("_ZN2hp8gemm_cutEiiiPiS0_", I, I, I, P, P)
    ntc, G = I(), I()
    f(N, K, R, ctypes.addressof(ntc), ctypes.addressof(G))
    return ntc.value, G.value


def pack(R, K):
    f = sym("_ZN2hp15gemm_pack_bytesEii", I, I)
    f.restype = Z
    return torch.full((f(R, K),), 0xA5, dtype=torch.uint8, device="cuda")


def run_gemm(wt, xq, N, K, R, ldy, cut, err):
    y = torch.full((hb.lib().hp_gemv_parts(N, K), R, ldy), float("nan"), device="cuda")
    f = sym(CUT, P, P, P, I, I, I, I, Z, P, P, P, B, I, I)
    x, pk = XQ8F(xq.q.data_ptr(), xq.sc.data_ptr()), pack(R, K)
    hb.check(f(wt.data_ptr(), ctypes.addressof(x), y.data_ptr(), N, K, R, ldy, R * ldy, pk.data_ptr(), err.data_ptr(), torch.cuda.current_stream().cuda_stream, True, *cut))
    return y


def run_gemv(wt, xq, N, K, R, ldy, err):
    L = hb.lib()
    y = torch.full((L.hp_gemv_parts(N, K), R, ldy), float("nan"), device="cuda")
    f = sym("_ZN2hp17gemv_q4k_q8_partsEPKvRKNS_4XQ8FEPfiiiimPiP11CUstream_stbbb", P, P, P, I, I, I, I, Z, P, P, B, B, B)
    for r0 in range(0, R, 32):
        x = XQ8F(xq.q.data_ptr() + L.hp_xq8_q_bytes(r0, K), xq.sc.data_ptr() + L.hp_xq8_sc_bytes(r0, K)) if r0 else XQ8F(xq.q.data_ptr(), xq.sc.data_ptr())
        hb.check(f(wt.data_ptr(), ctypes.addressof(x), y.data_ptr() + 4 * r0 * ldy, N, K, min(32, R - r0), ldy, R * ldy, err.data_ptr(),
                   torch.cuda.current_stream().cuda_stream, False, True, False))
    return y


@pytest.fixture(scope="module")
def weights():
    out = {}
    for i, (N, K) in enumerate(SHAPES):
        g = torch.Generator(device="cuda").manual_seed(i)
        blk = torch.randint(0, 256, (N * (K // 256), 144), dtype=torch.uint8, device="cuda", generator=g)
        blk[:, :4] = torch.randn((blk.shape[0], 2), device="cuda", generator=g).mul_(0.01).abs_().half().view(torch.uint8)
        out[N, K] = K_.repack_tiled(blk.reshape(-1), N, K, 0)
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("ntc,G", CUTS)
def test_every_cut_gives_the_bits_of_the_gemv(weights, ntc, G):
    for N, K in SHAPES:
        for R in {8 * ntc - 3, 8 * ntc + 1, 16 * ntc + 5} if N < 30000 else {8 * ntc + 8}:
            ldy = N + 5
            x = torch.randn((R, K), device="cuda", generator=torch.Generator(device="cuda").manual_seed(R))
            xq = K_.quantize_x_q8(x); err = torch.zeros(1, dtype=torch.int32, device="cuda")
            got, want = run_gemm(weights[N, K], xq, N, K, R, ldy, (ntc, G), err), run_gemv(weights[N, K], xq, N, K, R, ldy, err)
            assert err.item() == 0
            assert not torch.isnan(want[:, :, :N]).any()
            assert torch.equal(got.view(torch.int32), want.view(torch.int32)), (N, K, R)   # and nothing beyond column N


# rows whose last column ranges are two tiles narrower: one of three, both of the two behind the first, and with more rows left empty than that
@pytest.mark.gpu
@pytest.mark.parametrize("ntc,G", CUTS)
def test_narrow_ranges_give_the_bits_of_the_gemv(weights, ntc, G):
    for N, K in SHAPES:
        for R in (24 * ntc - 16, 24 * ntc - 35, 16 * ntc + 1) if N < 30000 else (24 * ntc - 32,):
            xq = K_.quantize_x_q8(torch.randn((R, K), device="cuda", generator=torch.Generator(device="cuda").manual_seed(R)))
            err = torch.zeros(1, dtype=torch.int32, device="cuda")
            got, want = run_gemm(weights[N, K], xq, N, K, R, N, (ntc, G), err), run_gemv(weights[N, K], xq, N, K, R, N, err)
            assert err.item() == 0
            assert torch.equal(got.view(torch.int32), want.view(torch.int32)), (N, K, R)


# The GEMM takes each sub-block's integer dot from an fp32 accumulator of the tensor core: the dots that need most of its bits (16: nibbles of
# 15 against 127, odd ones beside them), one-signed sums and large ones that cancel to a residue. Scales of 1 and no minimum, so that every sum is a
# whole number below 2^24 and the result exact.
@pytest.mark.gpu
@pytest.mark.parametrize("ntc,G", CUTS)
def test_dots_of_full_width_are_exact(ntc, G):
    N, K, R = 400, 768, 8 * ntc + 5
    g = torch.Generator(device="cuda").manual_seed(ntc)
    ri = lambda hi, *shape: torch.randint(0, hi, shape, device="cuda", generator=g)
    full, part = torch.full((N, K // 32, 32), 15, device="cuda"), torch.tensor([0, 1, 14, 15], device="cuda")[ri(4, N, K // 32, 32)]
    one = full.clone(); one.scatter_(2, ri(32, N, K // 32, 1), 14)
    q = torch.where(ri(2, N, K // 32, 1) == 0, full, torch.where(ri(2, N, K // 32, 1) == 0, one, part))
    sign = 1 - 2 * ri(2, R, K // 32, 1)
    flat, near, far = torch.full((R, K // 32, 32), 127, device="cuda"), 119 + ri(3, R, K // 32, 32), torch.tensor([127, 126, 121, 1, 0, -1, -120, -127], device="cuda")[ri(8, R, K // 32, 32)]
    cancel = flat.clone(); cancel[..., ::2] = -127; cancel.scatter_(2, 1 + 2 * ri(16, R, K // 32, 1), 126)
    kind = ri(4, R, K // 32, 1)
    x = sign * torch.where(kind == 0, flat, torch.where(kind == 1, near, torch.where(kind == 2, far, cancel)))
    x[..., 31] = 127 * sign[..., 0]                              # a largest value of 127: the quantised row is the row itself
    blk = torch.zeros((N, K // 256, 144), dtype=torch.uint8, device="cuda")
    blk[..., 1] = 0x3C                                            # d = 1
    blk[..., 4:8] = 1; blk[..., 12:16] = 1                        # scales of 1, minima of 0
    qs = q.reshape(N, K // 256, 4, 2, 32)
    blk[..., 16:] = (qs[..., 0, :] | qs[..., 1, :] << 4).reshape(N, K // 256, 128).to(torch.uint8)
    wt = K_.repack_tiled(blk.reshape(-1), N, K, 0)
    xq = K_.quantize_x_q8(x.reshape(R, K).float()); err = torch.zeros(1, dtype=torch.int32, device="cuda")
    got, gemv = run_gemm(wt, xq, N, K, R, N, (ntc, G), err), run_gemv(wt, xq, N, K, R, N, err)
    want = x.reshape(R, K).double() @ q.reshape(N, K).double().T
    assert err.item() == 0 and (want.abs() < 2 ** 24).all() and (q * 127).sum(-1).max() == 60960
    assert torch.equal(gemv.double().sum(0), want) and torch.equal(got.view(torch.int32), gemv.view(torch.int32))


# rows from the smallest to the largest of fp32, scales of the weights from subnormal ones up: products of the scales that are subnormal, and dots
# of few nibbles beside products that leave no factor of 512 to the largest number
@pytest.mark.gpu
@pytest.mark.parametrize("N,K", [(400, 768), (2100, 17408)])
@pytest.mark.parametrize("ntc,G", CUTS)
def test_rows_at_the_ends_of_the_range_give_the_bits_of_the_gemv(ntc, G, N, K):
    R = 8 * ntc + 5
    g = torch.Generator(device="cuda").manual_seed(ntc)
    blk = torch.randint(0, 256, (N, K // 256, 144), dtype=torch.uint8, device="cuda", generator=g)
    blk[N // 2:, :, 16:] *= (torch.rand((N - N // 2, K // 256, 128), device="cuda", generator=g) < 1 / 64).to(torch.uint8)
    d = torch.randn((N, K // 256, 2), device="cuda", generator=g).mul_(0.01).abs_()
    d[::3] *= 2.0 ** -12                                          # subnormal f16
    d[N // 2:, :, 1] = 0
    blk[..., :4] = d.half().view(torch.uint8)
    wt = K_.repack_tiled(blk.reshape(-1), N, K, 0)
    e = torch.linspace(-140, 125, R, device="cuda").round().double()
    x = (torch.randn((R, K), device="cuda", generator=g).clamp_(-3.9, 3.9).double() * 2.0 ** e[:, None]).float()
    xq = K_.quantize_x_q8(x); err = torch.zeros(1, dtype=torch.int32, device="cuda")
    got, want = run_gemm(wt, xq, N, K, R, N, (ntc, G), err), run_gemv(wt, xq, N, K, R, N, err)
    assert err.item() == 0 and torch.isfinite(want).float().mean() > 0.95
    same = (got.view(torch.int32) == want.view(torch.int32)) | (torch.isnan(got) & torch.isnan(want))
    assert same.all(), e[(~same).nonzero()[:, 1].unique()].tolist()


# the tile-major form of the GEMV on both sides of its row limits (4 rows; three column tiles whose activations leave room for one-block
# stages only: 20 blocks), against the row-major one
@pytest.mark.gpu
@pytest.mark.parametrize("R", [1, 4, 5, 8, 16, 17, 24, 25, 32])
@pytest.mark.parametrize("N,K", [(100, 5120), (16480, 5120), (4096, 768), (2100, 17408)])
def test_tile_major_gemv_gives_the_bits_of_the_row_major_one(N, K, R):
    g = torch.Generator(device="cuda").manual_seed(R)
    blk = torch.randint(0, 256, (N * (K // 256), 144), dtype=torch.uint8, device="cuda", generator=g)
    blk[:, :4] = torch.randn((blk.shape[0], 2), device="cuda", generator=g).mul_(0.01).abs_().half().view(torch.uint8)
    xq = K_.quantize_x_q8(torch.randn((R, K), device="cuda", generator=g)); err = torch.zeros(1, dtype=torch.int32, device="cuda")
    planes = run_gemv(K_.repack_tiled(blk.reshape(-1), N, K, 0), xq, N, K, R, N, err)
    got = planes[0].clone()
    for p in planes[1:]:
        got += p
    assert err.item() == 0
    assert torch.equal(got.view(torch.int32), K_.gemv_q4k_q8(blk, xq, N, K).view(torch.int32))


# rows 25 to 32 of a large matrix run as two launches in both layouts: against one launch per column tile, in one K part and in two, an
# even and an odd number of blocks per part; three tiles stay in one
@pytest.mark.gpu
@pytest.mark.parametrize("R", [24, 25, 32])
@pytest.mark.parametrize("N,K,parts", [(16480, 5120, 1), (8192, 10240, 2), (16480, 5888, 1)])
def test_two_launches_give_the_bits_of_single_column_tiles(N, K, parts, R):
    assert hb.lib().hp_gemv_parts(N, K) == parts
    g = torch.Generator(device="cuda").manual_seed(R)
    blk = torch.randint(0, 256, (N * (K // 256), 144), dtype=torch.uint8, device="cuda", generator=g)
    blk[:, :4] = torch.randn((blk.shape[0], 2), device="cuda", generator=g).mul_(0.01).abs_().half().view(torch.uint8)
    x = torch.randn((R, K), device="cuda", generator=g); xq = K_.quantize_x_q8(x); err = torch.zeros(1, dtype=torch.int32, device="cuda")
    tiled = K_.repack_tiled(blk.reshape(-1), N, K, 0)
    planes, rows = run_gemv(tiled, xq, N, K, R, N, err), K_.gemv_q4k_q8(blk, xq, N, K)
    for r0 in range(0, R, 8):
        r1 = min(R, r0 + 8); x8 = K_.quantize_x_q8(x[r0:r1].contiguous())
        assert torch.equal(planes[:, r0:r1].view(torch.int32), run_gemv(tiled, x8, N, K, r1 - r0, N, err).view(torch.int32))
        assert torch.equal(rows[r0:r1].view(torch.int32), K_.gemv_q4k_q8(blk, x8, N, K).view(torch.int32))
    assert err.item() == 0


@pytest.mark.parametrize("ntc,G", [(5, 8), (0, 8), (18, 8), (2, 8), (-4, 8), (8, 2), (8, 16), (8, 0)])
def test_cuts_that_do_not_exist_are_refused(ntc, G):
    f = sym(CUT, P, P, P, I, I, I, I, Z, P, P, P, B, I, I)       # refused on the host, before any pointer is used
    x = XQ8F(4096, 4096)
    assert f(4096, ctypes.addressof(x), 4096, 40, 256, 8, 40, 320, 4096, 4096, None, False, ntc, G) == 1
    assert b"no cut" in hb.lib().hp_last_error()


def test_the_rule_takes_tested_cuts_only_and_all_widths_occur():
    seen = set()
    for E, F, heads, kv in ((5120, 17408, 24, 4), (2048, 0, 24, 2), (512, 1024, 4, 2)):
        lins = [(16480 if E > 512 else 1544, E), (heads * 512 + kv * 512, E), (E, heads * 256), (E, 2 * E)] + ([(2 * F, E), (E, F)] if F else [])
        for N, K in lins:
            seen |= {gemm_cut(N, K, R) for R in range(33, 513)}
    assert seen <= set(CUTS)
    assert {c[0] for c in seen} == {4, 6, 8, 10, 12, 14, 16}
