"""Each kernel alone against a plain float32/float64 PyTorch statement of the same operation,
at sizes other than the engine's tiny configurations (widths and vocabularies that are no power
of two, head sizes in steps of 16, odd numbers of heads and groups)."""

import math
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

from mini_rsglang_b200 import BackendError, InvalidRequest, kernels
from mini_rsglang_b200.parts.position import RotaryPosition
from mini_rsglang_b200.sampling import Sampler, SamplingParams, uniform_from_counter
import plain_qwen3 as P

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
DTYPES = [torch.float32, torch.bfloat16]


def close(got, want, dtype, what=""):
    got, want = got.double().cpu(), want.double().cpu()
    if dtype is torch.float32:
        tol = 2e-5 * max(1.0, want.abs().max().item())
    else:
        tol = 2 ** -7 * max(1.0, want.abs().max().item())     # one bfloat16 rounding of the result, with room
    err = (got - want).abs().max().item()
    assert err <= tol, f"{what}: max error {err:.3e} > {tol:.3e}"


@pytest.mark.parametrize("dtype", DTYPES)
def test_embed(dtype):
    table = torch.randn(301, 72, device=DEV).to(dtype)
    ids = torch.tensor([0, 300, 5, 5, 17], dtype=torch.int32, device=DEV)
    out = torch.empty(5, 72, device=DEV)
    kernels.embed(table, ids, out)
    assert torch.equal(out, table.float()[ids.long()])


def test_patch_tokens_fills_ids_from_what_another_step_sampled():
    """ids[rows[i]] = sampled[index[i]]; a value that is no token (the sampler's mark of a bad row, or beyond the
    vocabulary) becomes token 0; the other ids stay."""
    ids = torch.arange(100, 140, dtype=torch.int32, device=DEV)
    rows = torch.tensor([3, 0, 39, 17, 20], dtype=torch.int32, device=DEV)
    index = torch.tensor([2, 2, 0, 4, 1], dtype=torch.int32, device=DEV)
    sampled = torch.tensor([7, -1, 299, 5, 300], dtype=torch.int32, device=DEV)
    kernels.patch_tokens(ids, rows, index, sampled, 300)
    want = list(range(100, 140))
    want[3], want[0], want[39], want[17], want[20] = 299, 299, 7, 0, 0
    assert ids.tolist() == want
    big_rows = torch.randperm(5000, device=DEV)[:3000].to(torch.int32)
    big_index = torch.randint(0, 64, (3000,), device=DEV, dtype=torch.int32)
    big_sampled = torch.randint(0, 1000, (64,), device=DEV, dtype=torch.int32)
    big = torch.full((5000,), -5, dtype=torch.int32, device=DEV)
    kernels.patch_tokens(big, big_rows, big_index, big_sampled, 1000)
    expect = torch.full((5000,), -5, dtype=torch.int32, device=DEV)
    expect[big_rows.long()] = big_sampled[big_index.long()]
    assert torch.equal(big, expect)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("width", [72, 75, 1000, 4096, 5120, 16384, 16388])
def test_add_rmsnorm(dtype, width):
    rows = 7
    residual = torch.randn(rows, width, device=DEV)
    delta = torch.randn(rows, width, device=DEV).to(dtype)
    weight = 1 + 0.1 * torch.randn(width, device=DEV)
    eps = 1e-5
    total = residual.double() + delta.double()
    want = total * torch.rsqrt(total.pow(2).mean(-1, keepdim=True) + eps) * weight.double()
    work = residual.clone()
    out = torch.empty(rows, width, device=DEV, dtype=dtype)
    kernels.add_rmsnorm(work, delta, weight, eps, out)
    close(out, want, dtype, "add_rmsnorm")
    close(work, total, torch.float32, "residual written back")
    # picked rows, nothing written back, a row asked for twice
    pick = torch.tensor([6, 0, 6], dtype=torch.int32, device=DEV)
    work = residual.clone()
    out = torch.empty(3, width, device=DEV, dtype=dtype)
    kernels.add_rmsnorm(work, delta, weight, eps, out, rows=pick, write_back=False)
    close(out, want[pick.long()], dtype, "picked rows")
    assert torch.equal(work, residual)
    # no delta
    out = torch.empty(rows, width, device=DEV, dtype=dtype)
    kernels.add_rmsnorm(residual.clone(), None, weight, eps, out)
    x = residual.double()
    close(out, x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * weight.double(), dtype, "no delta")
    # plain norm of activations
    x = torch.randn(rows, width, device=DEV).to(dtype)
    out = torch.empty_like(x)
    kernels.rmsnorm(x, weight, eps, out)
    xd = x.double()
    close(out, xd * torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + eps) * weight.double(), dtype, "rmsnorm")


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("inter", [136, 75, 12288])
def test_silu_mul(dtype, inter):
    gate_up = torch.randn(5, 2 * inter, device=DEV).to(dtype) * 3
    out = torch.empty(5, inter, device=DEV, dtype=dtype)
    kernels.silu_mul(gate_up, out)
    g, u = gate_up.double()[:, :inter], gate_up.double()[:, inter:]
    close(out, g / (1 + torch.exp(-g)) * u, dtype, "silu_mul")


@pytest.mark.parametrize("m,n,k", [(1, 7, 5), (33, 100, 72), (64, 64, 16), (130, 301, 257)])
def test_gemm_f32_is_true_float32(m, n, k):
    x = torch.randn(m, k, device=DEV)
    w = torch.randn(n, k, device=DEV)
    out = torch.empty(m, n, device=DEV)
    kernels.gemm_f32(x, w, out)
    want = x.double() @ w.double().T
    close(out, want, torch.float32, "gemm_f32")
    # a product that a tensor-core mode with a shortened mantissa would get wrong by 1e-3
    x = torch.full((1, 8), 1.0 + 2 ** -12, device=DEV)
    w = torch.full((1, 8), 1.0 + 2 ** -12, device=DEV)
    out = torch.empty(1, 1, device=DEV)
    kernels.gemm_f32(x, w, out)
    assert abs(out.item() - 8 * (1 + 2 ** -12) ** 2) < 1e-5
    # a row's result does not depend on the other rows of the batch
    x = torch.randn(70, 72, device=DEV)
    w = torch.randn(50, 72, device=DEV)
    whole, alone = torch.empty(70, 50, device=DEV), torch.empty(1, 50, device=DEV)
    kernels.gemm_f32(x, w, whole)
    kernels.gemm_f32(x[69:70].contiguous(), w, alone)
    assert torch.equal(whole[69:70], alone)


@pytest.mark.parametrize("m", [1, 4, 5, 8, 9, 31, 33, 64, 65, 700, 2100])
@pytest.mark.parametrize("n,k", [(16, 128), (1, 4), (33, 132), (1000, 1020), (257, 1026), (64, 37), (4100, 96)])
def test_gemm_f32_sizes_keep_a_rows_bits(m, n, k):
    """Every kernel that the sizes choose (few rows, three tile shapes, sixteen- and four-byte copies), at whole and ragged
    tiles and stages: within the rounding of a chain of k multiply-adds of the 64-bit product, and every element the same bits
    as the product of its row alone (a chain in ascending order whatever the kernel)."""
    g = torch.Generator(device=DEV).manual_seed(m * 7 + n + k)
    x, w = torch.randn(m, k, device=DEV, generator=g), torch.randn(n, k, device=DEV, generator=g)
    out = torch.full((m, n), float("nan"), device=DEV)
    kernels.gemm_f32(x, w, out)
    want, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    assert ((out.double() - want).abs() <= size * k * 2.0 ** -24).all()
    for row in {0, m // 2, m - 1}:
        alone = torch.empty(1, n, device=DEV)
        kernels.gemm_f32(x[row:row + 1].clone(), w, alone)
        assert torch.equal(out[row:row + 1], alone)
    shifted = torch.empty(m * k + 1, device=DEV)[1:].view(m, k)           # off a 16-byte boundary: four-byte copies
    shifted.copy_(x)
    other = torch.empty_like(out)
    kernels.gemm_f32(shifted, w, other)
    assert torch.equal(out, other)


@pytest.mark.parametrize("m,n,k", [(1, 130, 1024), (17, 127, 3072), (95, 129, 2048), (97, 128, 1000), (260, 300, 4100)])
def test_gemm_f32_keeps_every_bit_of_its_inputs(m, n, k):
    """Both sides of the tiles' edges, short and long ranges of K, one CTA and clusters a tile.  A product of two float32 loses at most
    2^-24 of itself (parts of 2^-8 and 2^-17 twice), 32 are added by the tensor cores, the rest is k / 32 + 4 additions: within 2^-23 of the sum of the products'
    sizes for the first and, a rounding each, (k / 32 + 4) 2^-24 for the others; and closer than a chain of k multiply-adds in
    float32 comes."""
    g = torch.Generator(device=DEV).manual_seed(m + n + k)
    x, w = torch.randn(m, k, device=DEV, generator=g), torch.randn(n, k, device=DEV, generator=g)
    out = torch.empty(m, n, device=DEV)
    kernels.gemm_f32(x, w, out)
    want, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    assert ((out.double() - want).abs() <= size * 2.0 ** -23 + want.abs().max() * (k / 32 + 4) * 2.0 ** -24).all()
    chain = torch.zeros(m, n, device=DEV, dtype=torch.float64)
    for i in range(k):                                       # a multiply-add: exact in 64 bits, then rounded
        chain = (chain + x[:, i, None].double() * w[:, i].double()).float().double()
    assert (out.double() - want).norm() <= (chain - want).norm()


@pytest.mark.parametrize("m", [1, 20, 100])
def test_gemm_f32_of_values_at_the_ends_of_the_range(m):
    """Infinities, NaN, values that bfloat16 rounds to infinity and products far below one: what the sum of the products is."""
    g = torch.Generator(device=DEV).manual_seed(m)
    n, k = 140, 300
    x, w = torch.randn(m, k, device=DEV, generator=g), torch.randn(n, k, device=DEV, generator=g)
    w[3] *= 1e-30                                            # small results, their factors' parts partly below bfloat16's range
    w[5, 7], w[6, 8], w[7, 9] = math.inf, math.nan, 0.0
    x[m // 2, 9], x[m // 2, 11] = math.inf, 3.4e38           # infinity times 0 in column 7
    w[:, 11] *= 1e-3
    w[11] = 0.0
    x[m - 1] *= 1e-9
    out = torch.empty(m, n, device=DEV)
    kernels.gemm_f32(x, w, out)
    want, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    assert torch.equal(out.isnan(), want.isnan())
    infinite = want.float().isinf()
    assert torch.equal(out[infinite], want.float()[infinite])
    finite = want.float().isfinite()
    assert ((out.double() - want).abs() <= size * k * 2.0 ** -24)[finite].all() and out[finite].isfinite().all()
    assert (out[m - 1, 3].double() - want[m - 1, 3]).abs() <= 2.0 ** -23 * size[m - 1, 3] or not want[m - 1, 3].isfinite()


@pytest.mark.parametrize("m,n,k", [(1, 140, 1024), (7, 4096, 300), (20, 140, 3072), (100, 500, 301), (97, 4100, 1024)])
def test_gemm_f32_of_factors_with_bits_under_the_parts_range(m, n, k):
    """Elements below 2^-110, whose last bits bfloat16 has no room for, and subnormal ones, beside factors that bring their products
    back to ordinary numbers or up to 1: one CTA and clusters a tile, whole rows and single elements.  A result is the sum of the products
    to a rounding each of k / 32 + 8 additions; what shares a tile with such rows keeps its bits."""
    g = torch.Generator(device=DEV).manual_seed(m + n)
    x, w = torch.randn(m, k, device=DEV, generator=g), torch.randn(n, k, device=DEV, generator=g)
    plain = torch.empty(m, n, device=DEV)
    kernels.gemm_f32(x, w, plain)
    whole, single = sorted({0, m // 2}), sorted({m // 3, m - 1} - {0, m // 2})
    for row in whole:
        x[row] = torch.ldexp(x[row], torch.tensor(-120 if row == 0 else -136, device=DEV))       # from 2^-126 on down: subnormal
    for row in single:
        x[row, k // 2] = 1.2345678e-38
    w[3] = torch.ldexp(w[3], torch.tensor(70, device=DEV))
    w[5] = torch.ldexp(w[5], torch.tensor(120, device=DEV))
    w[7] = 0.0
    w[7, k // 2] = 1e30                                      # 1.2e-38 times 1e30 alone
    w[n - 1] = torch.ldexp(w[n - 1], torch.tensor(-125, device=DEV))
    out = torch.empty(m, n, device=DEV)
    kernels.gemm_f32(x, w, out)
    torch.cuda.synchronize()
    kernels.check_device_errors()
    want, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    assert ((out.double() - want).abs() <= size * (k / 32 + 8) * 2.0 ** -24 + 2.0 ** -149).all()
    odd = torch.zeros(n, dtype=torch.bool, device=DEV)
    odd[[3, 5, 7, n - 1]] = True
    rows = [r for r in range(m) if r not in whole + single]
    assert torch.equal(out[rows][:, ~odd], plain[rows][:, ~odd])


@pytest.mark.parametrize("exponents", [(-30, -31), (-50, -49), (-50, -52), (-55, -60), (-62, -63), (-109, 3)])
def test_gemm_f32_of_small_results(exponents):
    """Results on both sides of 2^-100, below which they are computed again, down to 2^-125, and factors that just have their parts: the
    error of ordinary ones, a rounding to a subnormal beside it."""
    g = torch.Generator(device=DEV).manual_seed(2)
    for k in (1, 300, 1024):
        x, w = (torch.ldexp(torch.randn(rows, k, device=DEV, generator=g), torch.tensor(e, device=DEV)) for rows, e in zip((70, 300), exponents))
        out = torch.empty(70, 300, device=DEV)
        kernels.gemm_f32(x, w, out)
        want, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
        assert ((out.double() - want).abs() <= size * (2.0 ** -23 + (k / 32 + 4) * 2.0 ** -24) + 2.0 ** -149).all()


@pytest.mark.parametrize("k", [1, 3, 32, 1024])
def test_gemm_f32_of_factors_whose_parts_are_largest(k):
    """Factors just below 1 + 2^-8, whose second part is 2^-8 and whose third would be 2^-16 if the second were cut off: a product loses at most
    2^-24 of itself and is rounded once, few of them are added by few roundings; on average they come within half of that."""
    g = torch.Generator(device=DEV).manual_seed(k)
    x, w = (1 + 2.0 ** -8 - torch.randint(1, 200, (rows, k), generator=g, device=DEV) * 2.0 ** -23 for rows in (64, 256))
    out = torch.empty(64, 256, device=DEV)
    kernels.gemm_f32(x, w, out)
    want = x.double() @ w.double().T
    error = (out.double() - want).abs() / want
    assert error.max() <= 2.0 ** -24 + (1 + k / 32 + 4 * (k > 1)) * 2.0 ** -24 and error.mean() <= 2.0 ** -24 * (1 + (k > 32))


def plain_qk(qkv, positions, q_w, k_w, eps, theta, nq, nkv, d):
    """q and k after head norm and rotation, v untouched, from the plain implementation's parts."""
    ar = P.Arith(None)
    T = qkv.shape[0]
    x = qkv.double().cpu().view(T, nq + 2 * nkv, d)
    q, k, v = x[:, :nq], x[:, nq:nq + nkv], x[:, nq + nkv:]
    if q_w is not None:
        q = P.rms_norm(ar, q, q_w.cpu(), eps)
        k = P.rms_norm(ar, k, k_w.cpu(), eps)
    if theta is not None:
        q = P.rope(ar, q, positions.cpu(), theta)
        k = P.rope(ar, k, positions.cpu(), theta)
    return q, k, v


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("nq,nkv,d,page", [(3, 3, 48, 8), (8, 2, 128, 16), (5, 1, 16, 4), (2, 1, 256, 32), (32, 8, 128, 16),
                                           (7, 7, 64, 8), (20, 1, 64, 16)])
def test_qk_norm_rope_store(dtype, nq, nkv, d, page):
    T, pages, eps, theta = 9, 12, 1e-5, 50000.0
    qkv = torch.randn(T, (nq + 2 * nkv) * d, device=DEV).to(dtype)
    positions = torch.tensor([0, 1, 2, 40, 41, 1000, 7, 8, 9], dtype=torch.int32, device=DEV)
    perm = torch.randperm(pages * page)[:T].to(torch.int32).to(DEV)       # scattered, distinct slots
    q_w, k_w = 1 + 0.1 * torch.randn(d, device=DEV), 1 + 0.1 * torch.randn(d, device=DEV)
    inv_freq = RotaryPosition.inverse_frequencies(d, theta).to(DEV)
    assert torch.equal(inv_freq.cpu().double(), P.rope_inverse_frequencies(d, theta))
    q_out = torch.empty(T, nq * d, device=DEV, dtype=dtype)
    kc = torch.zeros(pages, nkv, page, d, device=DEV, dtype=dtype)
    vc = torch.zeros_like(kc)
    kernels.qk_norm_rope_store(qkv, q_out, kc, vc, positions, perm, q_w, k_w, eps, inv_freq, nq, nkv, d, page)
    q, k, v = plain_qk(qkv, positions, q_w, k_w, eps, theta, nq, nkv, d)
    close(q_out.view(T, nq, d), q, dtype, "q")
    slot = perm.long().cpu()
    got_k = kc.cpu()[slot // page, :, slot % page]
    got_v = vc.cpu()[slot // page, :, slot % page]
    close(got_k, k, dtype, "k in the cache")
    assert torch.equal(got_v.double(), v)
    assert kc.count_nonzero().item() <= T * nkv * d                     # nothing else was written
    # no norms, no rotation, no cache: q passes through
    q_only = torch.empty_like(q_out)
    kernels.qk_norm_rope_store(qkv, q_only, None, None, positions, None, None, None, 0.0, None, nq, nkv, d, page)
    assert torch.equal(q_only.view(T, nq, d), qkv.view(T, nq + 2 * nkv, d)[:, :nq])
    with pytest.raises(BackendError, match="refused"):
        kernels.qk_norm_rope_store(torch.zeros(1, 3 * 258, device=DEV), torch.zeros(1, 258, device=DEV), None, None,
                                   positions[:1], None, None, None, 0.0, None, 1, 1, 258, page)


def test_rotation_table_and_many_tokens():
    """The step's table of cosines and sines equals float32 cos and sin of position * frequency, and the kernel that
    reads it gives the same bits with a table handed in as with one it makes itself; 5,000 tokens with 11 heads (the
    warps go around the grid more than once, the last four heads of a token are three), some tokens without a slot."""
    nq, nkv, d, page, eps, theta, tokens = 5, 3, 128, 16, 1e-6, 1e6, 5000
    g = torch.Generator().manual_seed(5)
    positions = torch.randint(0, 40000, (tokens,), generator=g, dtype=torch.int32).to(DEV)
    inv_freq = RotaryPosition.inverse_frequencies(d, theta).to(DEV)
    table = kernels.rotation_table(positions, inv_freq)
    angles = positions.float()[:, None] * inv_freq[None, :]                    # float32 products, as in the kernel
    close(table[..., 0], torch.cos(angles.double()), torch.float32, "cosines")
    close(table[..., 1], torch.sin(angles.double()), torch.float32, "sines")
    qkv = torch.randn(tokens, (nq + 2 * nkv) * d, generator=g).to(torch.bfloat16).to(DEV)
    q_w, k_w = (1 + 0.1 * torch.randn(d, generator=g)).to(DEV), (1 + 0.1 * torch.randn(d, generator=g)).to(DEV)
    pages = tokens // page + 2
    slots = torch.randperm(pages * page, generator=g)[:tokens].to(torch.int32)
    slots[::7] = -1
    outs = []
    for rotations in (None, table):
        q_out = torch.empty(tokens, nq * d, device=DEV, dtype=torch.bfloat16)
        kc = torch.zeros(pages, nkv, page, d, device=DEV, dtype=torch.bfloat16)
        vc = torch.zeros_like(kc)
        kernels.qk_norm_rope_store(qkv, q_out, kc, vc, positions, slots.to(DEV), q_w, k_w, eps, inv_freq, nq, nkv, d, page,
                                   rotations=rotations)
        outs.append((q_out, kc, vc))
    assert all(torch.equal(a, b) for a, b in zip(*outs))
    q, k, v = plain_qk(qkv, positions, q_w, k_w, eps, theta, nq, nkv, d)
    q_out, kc, vc = outs[0]
    close(q_out.view(tokens, nq, d), q, torch.bfloat16, "q")
    keep = (slots >= 0).nonzero().flatten()
    slot = slots[keep].long()
    close(kc.cpu()[slot // page, :, slot % page], k[keep], torch.bfloat16, "k in the cache")
    assert torch.equal(vc.cpu()[slot // page, :, slot % page].double(), v[keep].double())
    assert kc.count_nonzero().item() <= keep.numel() * nkv * d and vc.count_nonzero().item() <= keep.numel() * nkv * d


class PagedCase:
    """Requests with scattered pages; builds the kernel's inputs and the plain answer."""

    def __init__(self, dtype, nq, nkv, d, page, spans, seed=0, window=0):
        # spans: for every request (context already in the cache, new tokens in this step)
        g = torch.Generator().manual_seed(seed)
        self.nq, self.nkv, self.d, self.page, self.window, self.dtype = nq, nkv, d, page, window, dtype
        total_pages = sum(-(-(c + n) // page) for c, n in spans) + 3
        order = torch.randperm(total_pages, generator=g).tolist()
        self.kc = torch.zeros(total_pages, nkv, page, d, dtype=dtype)
        self.vc = torch.zeros_like(self.kc)
        width = max(-(-(c + n) // page) for c, n in spans)
        self.table = torch.full((len(spans), width), -1, dtype=torch.int32)
        q_rows, pos, seq, self.want, self.q_start = [], [], [], [], [0]
        self.ks, self.vs = [], []
        for i, (c, n) in enumerate(spans):
            L = c + n
            k = torch.randn(L, nkv, d, generator=g).to(dtype)
            v = torch.randn(L, nkv, d, generator=g).to(dtype)
            q = torch.randn(n, nq, d, generator=g).to(dtype)
            self.ks.append(k), self.vs.append(v)
            for lp in range(-(-L // page)):
                page_id = order.pop()
                self.table[i, lp] = page_id
                rows = slice(lp * page, min(L, (lp + 1) * page))
                self.kc[page_id, :, :rows.stop - rows.start] = k[rows].transpose(0, 1)
                self.vc[page_id, :, :rows.stop - rows.start] = v[rows].transpose(0, 1)
            q_rows.append(q)
            pos += list(range(c, L))
            seq += [i] * n
            self.q_start.append(self.q_start[-1] + n)
        self.q = torch.cat(q_rows)
        self.positions = torch.tensor(pos, dtype=torch.int32)
        self.seq = torch.tensor(seq, dtype=torch.int32)
        self.spans = spans

    def plain(self):
        ar = P.Arith(None)
        out = []
        for i, (c, n) in enumerate(self.spans):
            L = c + n
            full_q = torch.zeros(L, self.nq, self.d, dtype=torch.float64)
            full_q[c:] = self.q[self.q_start[i]:self.q_start[i + 1]].double()
            o = P.causal_attention(ar, full_q, self.ks[i].double(), self.vs[i].double(), self.window)
            out.append(o[c:])
        return torch.cat(out).reshape(-1, self.nq * self.d)

    def dev(self, t):
        return t.to(DEV)

    def run_simt(self):
        out = torch.empty(self.q.shape[0], self.nq * self.d, device=DEV, dtype=self.dtype)
        kernels.attention_simt(self.dev(self.q.reshape(-1, self.nq * self.d)), self.dev(self.kc), self.dev(self.vc),
                               self.dev(self.positions), self.dev(self.seq), self.dev(self.table), out, self.nq,
                               self.nkv, self.d, self.window)
        return out

    def run_mma(self, mode, splits=1):
        group = self.nq // self.nkv
        per_tile = {"rows": 64}.get(mode, 16) // group
        if mode in ("tc", "tc_shares", "tc_pairs"):          # two tiles of 128 rows, each a whole number of tokens
            per_tile = 2 * (128 // group)
        tiles = []
        for i in range(len(self.spans)):
            first, n = self.q_start[i], self.q_start[i + 1] - self.q_start[i]
            if mode == "tc_pairs":               # the first tile of a request with its last, the second with the last but one, ...
                one = 128 // group
                count = -(-n // one)
                for a in range(count // 2):
                    b = count - 1 - a
                    tiles.append((i, first + a * one, one + min(one, n - b * one), ((b - a - 1) * one) << 16))
                if count % 2:
                    tiles.append((i, first + (count // 2) * one, min(one, n - (count // 2) * one), 0))
                continue
            for s in range(0, n, per_tile):
                if mode == "tc_shares":          # `splits` entries that walk one share of the keys each
                    tiles += [(i, first + s, min(per_tile, n - s), share | splits << 8) for share in range(splits)]
                else:
                    tiles.append((i, first + s, min(per_tile, n - s), 0))
        tiles = torch.tensor(tiles, dtype=torch.int32, device=DEV)
        out = torch.zeros(self.q.shape[0], self.nq * self.d, device=DEV, dtype=self.dtype)
        args = (self.dev(self.q.reshape(-1, self.nq * self.d)), self.dev(self.kc), self.dev(self.vc),
                self.dev(self.positions), self.dev(self.table), tiles, out, self.nq, self.nkv, self.d, self.window)
        if mode == "keys":
            kernels.attention_mma_keys(*args, splits=splits)
        elif mode in ("tc", "tc_shares", "tc_pairs"):
            kernels.attention_prefill_tc(*args, shares=mode == "tc_shares")
            torch.cuda.synchronize()
            kernels.check_device_errors()
        elif mode == "tma":
            kernels.attention_decode_tma(*args, splits=splits)
            torch.cuda.synchronize()
            kernels.check_device_errors()
        else:
            kernels.attention_mma_rows(*args)
        return out


SHAPES = [(3, 3, 48, 8), (8, 2, 128, 16), (6, 1, 32, 4), (4, 2, 16, 16), (2, 1, 256, 32), (5, 5, 80, 16), (12, 2, 64, 64)]
SPANS = [(0, 1), (0, 70), (130, 3), (257, 1), (63, 66), (1, 2), (300, 1)]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("nq,nkv,d,page", SHAPES)
def test_attention_simt(dtype, nq, nkv, d, page):
    case = PagedCase(dtype, nq, nkv, d, page, SPANS, seed=nq * d)
    close(case.run_simt(), case.plain(), dtype, "attention_simt")


@pytest.mark.parametrize("m", [65535 * 32, 65535 * 32 + 1, 65535 * 64])
def test_gemm_f32_takes_as_many_rows_as_its_highest_tiles_cover(m):
    """Few columns choose low tiles, whose grid ends at 2,097,120 rows; more rows go to the high ones (4,194,240, as before them)."""
    x = torch.arange(m, device=DEV, dtype=torch.float32).view(m, 1) * torch.tensor([[1.0, 0.5, 0.0, 0.25]], device=DEV)
    w = torch.tensor([[1.0, 0.0, 0.0, 0.0], [0.0, 0.0, 0.0, 2.0]], device=DEV)
    out = torch.full((m, 2), float("nan"), device=DEV)
    kernels.gemm_f32(x, w, out)
    assert torch.equal(out[:, 0], x[:, 0]) and torch.equal(out[:, 1], 0.5 * x[:, 0])


@pytest.mark.parametrize("nq,nkv,d,page,window", [(4, 2, 128, 16, 0), (16, 8, 128, 16, 0), (5, 1, 64, 8, 0), (12, 1, 96, 4, 0), (64, 1, 36, 16, 0),
                                                  (3, 3, 256, 32, 0), (4, 2, 128, 16, 700), (2, 1, 20, 4, 37)])
def test_attention_f32_gives_a_row_the_same_bits_in_every_cut(monkeypatch, nq, nkv, d, page, window):
    """Tiles of rows that begin and end anywhere, single tokens, contexts on both sides of a chunk's and a block's end; a row's
    bits are the same as a single token, inside a prompt, beside other requests, with a chunk's keys in blocks of their own or
    in one walk; a value behind a row's last key does not reach it, not even one that is no number."""
    spans = [(0, 1), (511, 2), (0, 130), (1030, 1), (480, 77), (1535, 1), (96, 1), (31, 33)]
    case = PagedCase(torch.float32, nq, nkv, d, page, spans, seed=d + window, window=window)
    got = case.run_simt()
    close(got, case.plain(), torch.float32, "attention_f32")
    monkeypatch.setattr(kernels, "ATTENTION_F32_PARTS_BYTES", 0)
    assert torch.equal(got, case.run_simt())
    monkeypatch.undo()
    q, table = case.dev(case.q.reshape(-1, nq * d)), case.dev(case.table)
    for row in (0, 2, 3, 130, 133, 134, 150, 210, 211, 212, 213, 230, q.shape[0] - 1):
        seq, position = int(case.seq[row]), int(case.positions[row])
        kc, vc = case.kc.clone(), case.vc.clone()
        length = spans[seq][0] + spans[seq][1]
        for p in range(position + 1, length):                      # what the request's later tokens left behind this one
            kc[case.table[seq, p // page], :, p % page] = float("inf")
            vc[case.table[seq, p // page], :, p % page] = float("nan")
        first = max(0, row - (position - spans[seq][0]))             # the request's rows up to this one, in one step
        for rows in (slice(row, row + 1), slice(first, row + 1), slice(first, case.q_start[seq + 1])):
            out = torch.empty(rows.stop - rows.start, nq * d, device=DEV)
            kernels.attention_simt(q[rows].clone(), case.dev(kc), case.dev(vc), case.dev(case.positions)[rows].clone(), case.dev(case.seq)[rows].clone(),
                                   table, out, nq, nkv, d, window, longest=length)
            assert torch.equal(out[row - rows.start], got[row]), (row, rows)


@pytest.mark.parametrize("window", [0, 900])
def test_attention_f32_joins_chunks_the_same_way_every_time(monkeypatch, window):
    """Heads of 128, walks over up to 16 chunks: at a chunk's end the two threads of a row exchange their sums through memory that also
    carries the blocks' maxima.  Tiles that begin with an even and an odd block, run after run: the bits of chunks in blocks of their own."""
    case = PagedCase(torch.float32, 8, 2, 128, 16, [(0, 1100), (2900, 75), (4000, 1), (190, 700)], seed=window, window=window)
    want = case.run_simt()
    monkeypatch.setattr(kernels, "ATTENTION_F32_PARTS_BYTES", 0)
    for _ in range(20):
        assert torch.equal(case.run_simt(), want)


@pytest.mark.parametrize("nq,nkv,d,page,window", [(2, 1, 128, 16, 0), (8, 1, 64, 4, 0), (3, 3, 256, 1, 0), (6, 2, 40, 16, 90), (1, 1, 128, 64, 33)])
def test_attention_f32_single_tokens_at_the_edges_of_steps(monkeypatch, nq, nkv, d, page, window):
    """One to eight rows a tile: contexts around a block of 32 keys, a step of 64 and a chunk of 256, windows that begin inside
    them; chunks in blocks of their own and in one walk give the same bits, and those of the rows inside a prompt."""
    spans = [(p, 1) for p in (0, 30, 31, 32, 62, 63, 64, 95, 96, 254, 255, 256, 287, 320, 511, 512, 700)]
    case = PagedCase(torch.float32, nq, nkv, d, page, spans, seed=d + window, window=window)
    got = case.run_simt()
    close(got, case.plain(), torch.float32, "attention_f32")
    monkeypatch.setattr(kernels, "ATTENTION_F32_PARTS_BYTES", 0)
    assert torch.equal(got, case.run_simt())


@pytest.mark.parametrize("window", [1, 5, 64, 100])
def test_attention_window_edges(window):
    for dtype in DTYPES:
        case = PagedCase(dtype, 4, 2, 32, 8, [(0, 130), (120, 1), (99, 2), (3, 4)], seed=window, window=window)
        close(case.run_simt(), case.plain(), dtype, f"simt window {window}")
    case = PagedCase(torch.bfloat16, 4, 2, 32, 8, [(0, 130), (120, 1), (99, 2), (3, 4)], seed=window, window=window)
    close(case.run_mma("rows"), case.plain(), torch.bfloat16, f"mma rows window {window}")
    close(case.run_mma("keys", 1), case.plain(), torch.bfloat16, f"mma keys window {window}")
    close(case.run_mma("keys", 3), case.plain(), torch.bfloat16, f"mma keys split window {window}")


@pytest.mark.parametrize("nq,nkv,d,page", SHAPES)
def test_attention_mma_rows_mode(nq, nkv, d, page):
    case = PagedCase(torch.bfloat16, nq, nkv, d, page, SPANS, seed=nq + d)
    close(case.run_mma("rows"), case.plain(), torch.bfloat16, "attention_mma rows")


@pytest.mark.parametrize("splits", [1, 2, 5, 16])
@pytest.mark.parametrize("nq,nkv,d,page", SHAPES)
def test_attention_mma_keys_mode(nq, nkv, d, page, splits):
    case = PagedCase(torch.bfloat16, nq, nkv, d, page, SPANS, seed=nq + d + splits)
    close(case.run_mma("keys", splits), case.plain(), torch.bfloat16, f"attention_mma keys, {splits} splits")


TMA_SHAPES = [(8, 2, 128, 16), (2, 1, 256, 32), (12, 2, 64, 64), (4, 4, 64, 8), (16, 1, 128, 128), (3, 1, 192, 16)]


@pytest.mark.parametrize("splits", [1, 2, 5, 16])
@pytest.mark.parametrize("nq,nkv,d,page", TMA_SHAPES)
def test_attention_decode_tma(nq, nkv, d, page, splits):
    """Head sizes 64 to 256, pages of 8 to 128 rows (a copy of a whole page, and of 64 rows of a
    longer one), groups of 1 to 16 query heads."""
    assert kernels.attention_decode_tma_supported(d, nq // nkv, page)
    case = PagedCase(torch.bfloat16, nq, nkv, d, page, SPANS, seed=nq + d + splits)
    close(case.run_mma("tma", splits), case.plain(), torch.bfloat16, f"attention_decode_tma, {splits} splits")


TC_SHAPES = [(8, 2, 128, 16), (12, 3, 64, 8), (4, 4, 64, 64), (16, 1, 128, 128), (2, 1, 128, 32), (32, 1, 64, 16),
             (10, 2, 128, 16), (3, 1, 64, 8), (14, 2, 128, 32), (48, 1, 64, 16)]      # groups of 5, 3, 7, 48: rows of a tile stay empty
TC_SPANS = [(0, 1), (0, 70), (130, 3), (257, 1), (63, 66), (1, 2), (300, 200), (0, 513), (1000, 37)]


@pytest.mark.parametrize("nq,nkv,d,page", TC_SHAPES)
def test_attention_prefill_tc(nq, nkv, d, page):
    """Head sizes 64 and 128, groups of 1 to 48 query heads (among them groups that do not divide a tile's 128
    rows), pages of 8 to 128 rows; portions of 1 to 513 tokens on contexts up to 1,037: several tiles a request,
    several blocks of keys a tile, blocks that need no mask, the diagonal, and tiles that are not full."""
    assert kernels.attention_prefill_tc_supported(d, nq // nkv, page)
    case = PagedCase(torch.bfloat16, nq, nkv, d, page, TC_SPANS, seed=nq + d)
    close(case.run_mma("tc"), case.plain(), torch.bfloat16, "attention_prefill_tc")


@pytest.mark.parametrize("shares", [2, 3, 7])
@pytest.mark.parametrize("nq,nkv,d,page", [(8, 2, 128, 16), (4, 4, 64, 8), (4, 1, 128, 32), (10, 2, 128, 16)])
def test_attention_prefill_tc_shares_of_the_keys(nq, nkv, d, page, shares):
    """Entries that walk one share of their key blocks each, merged by the second kernel: portions deep in a long
    context, a fresh prompt whose first entries have fewer blocks than shares (empty shares), a tile without
    a block in the last share, a ragged last entry."""
    case = PagedCase(torch.bfloat16, nq, nkv, d, page, [(1000, 70), (0, 300), (130, 3 + 2 * (128 // (nq // nkv))), (2000, 40)], seed=shares)
    close(case.run_mma("tc_shares", shares), case.plain(), torch.bfloat16, f"{shares} shares of the keys")


@pytest.mark.parametrize("nq,nkv,d,page", [(8, 2, 128, 16), (4, 4, 64, 8), (10, 2, 128, 16), (2, 1, 128, 32), (16, 8, 128, 16)])
def test_attention_prefill_tc_tiles_that_are_no_neighbours(nq, nkv, d, page):
    """Entries whose two tiles lie apart in their request (the first tile with the last, and so on inwards): a tile
    that is done after one block beside one that walks a dozen, a last tile that is not full, an odd count whose
    middle tile stands alone, requests of one and two tiles, and cached tokens before the portion."""
    one = 128 // (nq // nkv)
    case = PagedCase(torch.bfloat16, nq, nkv, d, page, [(0, 12 * one), (0, 7 * one + 3), (300, 5 * one - 1), (0, one), (64, 2 * one), (0, 3)], seed=nq)
    close(case.run_mma("tc_pairs"), case.plain(), torch.bfloat16, "tiles that are no neighbours")
    assert torch.equal(case.run_mma("tc_pairs"), case.run_mma("tc"))          # a row's walk is the same whoever shares its CTA


def test_attention_prefill_tc_rescales_when_the_maximum_grows():
    """Keys whose scores rise block after block by far more than 2^8: the accumulator in tensor
    memory is rescaled again and again; then keys that fall: it is not."""
    nq, nkv, d, page = 4, 2, 64, 16
    for rising in (True, False):
        case = PagedCase(torch.bfloat16, nq, nkv, d, page, [(0, 600)], seed=3)
        case.q.mul_(0.05)
        case.q[:, :, 5] = 4.0
        ramp = torch.arange(600, dtype=torch.float32) / 600 * 24 - 12          # scores from -6 to +6 (in natural units)
        case.ks[0].mul_(0.05)
        case.ks[0][:, :, 5] = (ramp if rising else -ramp).to(torch.bfloat16)[:, None] * (d ** 0.5) / 4.0 / 2
        for lp in range(-(-600 // page)):
            rows = slice(lp * page, min(600, (lp + 1) * page))
            case.kc[case.table[0, lp], :, :rows.stop - rows.start] = case.ks[0][rows].transpose(0, 1)
        close(case.run_mma("tc"), case.plain(), torch.bfloat16, f"prefill_tc, scores {'rising' if rising else 'falling'}")


@pytest.mark.parametrize("window", [1, 5, 64, 100, 300])
def test_attention_prefill_tc_window_edges(window):
    case = PagedCase(torch.bfloat16, 4, 2, 64, 8, [(0, 330), (120, 40), (99, 2), (3, 4)], seed=window, window=window)
    close(case.run_mma("tc"), case.plain(), torch.bfloat16, f"prefill_tc window {window}")


@pytest.mark.parametrize("window", [1, 5, 64, 100])
def test_attention_decode_tma_window_edges(window):
    case = PagedCase(torch.bfloat16, 4, 2, 64, 8, [(0, 130), (120, 1), (99, 2), (3, 4)], seed=window, window=window)
    close(case.run_mma("tma", 1), case.plain(), torch.bfloat16, f"tma window {window}")
    close(case.run_mma("tma", 3), case.plain(), torch.bfloat16, f"tma split window {window}")
    # pages that the window has passed are gone from the table: the kernel must not need them
    table = case.table.clone()
    for i, (c, n) in enumerate(case.spans):
        passed = max(0, c - window + 1) // case.page
        case.table[i, :passed] = -1
    close(case.run_mma("tma", 2), case.plain(), torch.bfloat16, f"tma window {window}, passed pages given back")
    case.table = table


@pytest.mark.parametrize("runner", ["simt32", "simt16", "rows", "keys1", "keys7", "tma1", "tma7", "tc"])
def test_one_far_key_among_hundreds(runner):
    """One key far back scores far above the rest: the output must be that key's value row, so a
    kernel that skips, repeats or misplaces a block of keys cannot pass."""
    dtype = torch.float32 if runner == "simt32" else torch.bfloat16
    nq, nkv, d, page = 4, 2, 64, 16
    for far in (0, 15, 16, 63, 64, 200, 511, 689):
        case = PagedCase(dtype, nq, nkv, d, page, [(700, 1), (690, 12)], seed=far)
        for i in range(2):
            case.ks[i].mul_(0.01)
            case.ks[i][far] = 0
            case.ks[i][far, :, 3] = 16.0
        case.q.mul_(0.01)
        case.q[:, :, 3] = 16.0
        # rebuild the cache pages from the edited keys
        for i, (c, n) in enumerate(case.spans):
            L = c + n
            for lp in range(-(-L // page)):
                rows = slice(lp * page, min(L, (lp + 1) * page))
                case.kc[case.table[i, lp], :, :rows.stop - rows.start] = case.ks[i][rows].transpose(0, 1)
        got = {"simt32": case.run_simt, "simt16": case.run_simt, "rows": lambda: case.run_mma("rows"),
               "keys1": lambda: case.run_mma("keys", 1), "keys7": lambda: case.run_mma("keys", 7),
               "tma1": lambda: case.run_mma("tma", 1), "tma7": lambda: case.run_mma("tma", 7),
               "tc": lambda: case.run_mma("tc")}[runner]()
        want_rows = torch.cat([case.vs[0][far].reshape(1, -1).repeat(1, 1)] +
                              [case.vs[1][far].reshape(1, -1)] * 12).double()
        want = want_rows.view(13, nkv, 1, d).expand(13, nkv, nq // nkv, d).reshape(13, nq * d)
        close(got, want, dtype, f"{runner}, far key at {far}")
        close(got, case.plain(), dtype, f"{runner} vs plain, far key at {far}")


@pytest.mark.parametrize("runner", ["simt16", "tma1", "tma16", "tma7", "tma15", "tma32", "tc"])
def test_one_far_key_among_tens_of_thousands(runner):
    """The same at a context of 40,000 tokens with heads of 128 (block tables of 2,500 pages, scattered): a decoded
    token and a portion of a prompt find one key at the start, in the middle and near the end.  The shares of the
    keys as one cluster (16) and as counts that are no cluster and meet through memory (7, 15, 32: what the plan
    takes for few requests with long contexts)."""
    dtype = torch.bfloat16
    nq, nkv, d, page = 8, 2, 128, 16
    case = PagedCase(dtype, nq, nkv, d, page, [(39990, 1), (39000, 70)], seed=9)
    case.q.mul_(0.01)
    case.q[:, :, 5] = 16.0
    keys_as_drawn = [k.clone() for k in case.ks]
    for far in (0, 17, 20000, 38999):
        for i, (c, n) in enumerate(case.spans):
            case.ks[i] = keys_as_drawn[i] * 0.01
            case.ks[i][far] = 0
            case.ks[i][far, :, 5] = 16.0
            for lp in range(-(-(c + n) // page)):
                rows = slice(lp * page, min(c + n, (lp + 1) * page))
                case.kc[case.table[i, lp], :, :rows.stop - rows.start] = case.ks[i][rows].transpose(0, 1)
        if runner.startswith("tma"):
            got = case.run_mma("tma", int(runner[3:]))
        else:
            got = {"simt16": case.run_simt, "tc": lambda: case.run_mma("tc")}[runner]()
        want_rows = torch.cat([case.vs[0][far].reshape(1, -1)] + [case.vs[1][far].reshape(1, -1)] * 70).double()
        want = want_rows.view(71, nkv, 1, d).expand(71, nkv, nq // nkv, d).reshape(71, nq * d)
        close(got, want, dtype, f"{runner}, far key at {far} of 40,000")


def test_attention_refuses_what_it_cannot_do():
    case = PagedCase(torch.bfloat16, 4, 2, 32, 8, [(0, 4)])
    with pytest.raises(InvalidRequest):
        kernels.attention_simt(case.dev(case.q.reshape(-1, 128)).float(), case.dev(case.kc), case.dev(case.vc),
                               case.dev(case.positions), case.dev(case.seq), case.dev(case.table),
                               torch.empty(4, 128, device=DEV), 4, 2, 32)
    assert not kernels.attention_mma_supported(24, 1) and not kernels.attention_mma_supported(128, 128)
    assert kernels.attention_mma_supported(112, 7)
    assert not kernels.attention_decode_tma_supported(48, 1, 16) and not kernels.attention_decode_tma_supported(128, 4, 4)


# --------------------------------------------------------------------------------- tcgen05 product
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("m,n,k", [(1, 7, 8), (8, 128, 64), (16, 300, 72), (17, 1000, 1000), (64, 4096, 4096),
                                   (100, 257, 136), (128, 6144, 520), (3, 24576, 4096)])
def test_gemm_tc(m, n, k, out_dtype):
    """Rows up to 128 (every padded size), widths and depths that are no multiples of the tiles,
    one and several ranges of K."""
    g = torch.Generator().manual_seed(m + n + k)
    x = torch.randn(m, k, generator=g).to(torch.bfloat16)
    w = (torch.randn(n, k, generator=g) / k ** 0.5).to(torch.bfloat16)
    assert kernels.gemm_tc_supported(x.to(DEV), w.to(DEV))
    out = torch.full((m, n), float("nan"), dtype=out_dtype, device=DEV)
    kernels.gemm_tc(x.to(DEV), w.to(DEV), out)
    torch.cuda.synchronize()
    kernels.check_device_errors()
    close(out, x.double() @ w.double().T, out_dtype, f"gemm_tc {m}x{n}x{k}")


@pytest.mark.parametrize("m,inner,k", [(1, 64, 72), (8, 128, 64), (19, 3072, 1024), (32, 192, 4096), (100, 12288, 520)])
def test_gemm_tc_gated(m, inner, k):
    """silu(x . gate^T) * (x . up^T) out of one product over weights in blocks of 64 gate and 64 up rows;
    the same result as the product followed by the kernel that does it alone."""
    g = torch.Generator().manual_seed(m + inner)
    x = torch.randn(m, k, generator=g).to(torch.bfloat16)
    gate = (torch.randn(inner, k, generator=g) / k ** 0.5 * 2).to(torch.bfloat16)
    up = (torch.randn(inner, k, generator=g) / k ** 0.5 * 2).to(torch.bfloat16)
    mixed = torch.stack([gate.view(-1, 64, k), up.view(-1, 64, k)], dim=1).reshape(2 * inner, k).contiguous()
    out = torch.full((m, inner), float("nan"), dtype=torch.bfloat16, device=DEV)
    kernels.gemm_tc(x.to(DEV), mixed.to(DEV), out, gated=True)
    torch.cuda.synchronize()
    kernels.check_device_errors()
    gd, ud = x.double() @ gate.double().T, x.double() @ up.double().T
    want = gd / (1 + torch.exp(-gd)) * ud
    close(out, want, torch.bfloat16, f"gated gemm_tc {m}x{inner}x{k}")
    both = torch.cat([gd.unsqueeze(0), ud.unsqueeze(0)])      # the kernel alone on the blocked layout
    blocked = torch.stack([gd.view(m, -1, 64), ud.view(m, -1, 64)], dim=2).reshape(m, 2 * inner).to(torch.bfloat16).to(DEV)
    alone = torch.empty((m, inner), dtype=torch.bfloat16, device=DEV)
    kernels.silu_mul(blocked, alone, 64)
    close(alone, want, torch.bfloat16, "silu_mul on blocks of 64")
    del both


@pytest.mark.parametrize("t,inner,k", [(1, 64, 72), (128, 128, 64), (200, 192, 136), (513, 3072, 1024), (2048, 12288, 4096), (300, 64, 520)])
def test_gemm_gated_rows(t, inner, k):
    """The gated product for many rows (tiles of 128 tokens x 256 weight rows): token counts and widths that end inside
    a tile, a weight matrix of one and a half tiles, a depth that ends inside a block of 64."""
    g = torch.Generator().manual_seed(t + inner)
    x = torch.randn(t, k, generator=g).to(torch.bfloat16)
    gate = (torch.randn(inner, k, generator=g) / k ** 0.5 * 2).to(torch.bfloat16)
    up = (torch.randn(inner, k, generator=g) / k ** 0.5 * 2).to(torch.bfloat16)
    mixed = torch.stack([gate.view(-1, 64, k), up.view(-1, 64, k)], dim=1).reshape(2 * inner, k).contiguous()
    assert kernels.gemm_gated_rows_supported(x.to(DEV), mixed.to(DEV))
    out = torch.full((t, inner), float("nan"), dtype=torch.bfloat16, device=DEV)
    kernels.gemm_gated_rows(x.to(DEV), mixed.to(DEV), out)
    torch.cuda.synchronize()
    kernels.check_device_errors()
    gd, ud = x.double() @ gate.double().T, x.double() @ up.double().T
    close(out, gd / (1 + torch.exp(-gd)) * ud, torch.bfloat16, f"gated rows {t}x{inner}x{k}")
    assert not kernels.gemm_gated_rows_supported(x.to(DEV), mixed.to(DEV)[:64])          # half a block of gate rows


@pytest.mark.parametrize("gate", ["silu", "gelu_tanh"])
def test_gated_products_give_an_activation_the_same_bits_for_few_and_many_rows(gate):
    """Rows with a single 1 make every sum a weight itself, 8 million pairs of a gate and an up value over all gates that count and
    some whose exponential overflows: the products for many rows (dense and of one expert) divide as the product for few rows does."""
    g = torch.Generator().manual_seed(5)
    rows, inner = 1024, 8192
    scale = torch.cat([torch.full((inner - 1024,), 1.0), torch.full((1024,), 30.0)])
    gates = (torch.randn(inner, rows, generator=g) * scale[:, None]).bfloat16()
    ups = torch.randn(inner, rows, generator=g).bfloat16()
    mixed = torch.stack([gates.view(-1, 64, rows), ups.view(-1, 64, rows)], dim=1).reshape(2 * inner, rows).to(DEV).contiguous()
    x = torch.eye(rows, dtype=torch.bfloat16, device=DEV)
    few = torch.empty(rows, inner, dtype=torch.bfloat16, device=DEV)
    for first in range(0, rows, 128):
        kernels.gemm_tc(x[first:first + 128], mixed, few[first:first + 128], gated=True, gate=gate)
    z = gates.double().t()
    want = z * ups.double().t() * (torch.sigmoid(z) if gate == "silu" else 0.5 * (1 + torch.tanh(math.sqrt(2 / math.pi) * (z + 0.044715 * z ** 3))))
    close(few, want, torch.bfloat16, "gated gemm_tc")
    many = torch.empty(rows, inner, dtype=torch.bfloat16, device=DEV)
    kernels.gemm_gated_rows(x, mixed, many, gate)
    assert torch.equal(many, few)
    if gate == "silu":
        listed = torch.arange(rows, dtype=torch.int32, device=DEV)
        tile_expert = torch.tensor([0] * (rows // 128) + [rows // 128], dtype=torch.int32, device=DEV)
        many.zero_()
        kernels.moe_product_tc(x, listed, tile_expert, mixed.view(1, 2 * inner, rows), many, gated=True)
        assert torch.equal(many, few)


@pytest.mark.parametrize("m,nq,nkv,k,page", [(1, 2, 1, 64, 8), (8, 32, 8, 4096, 16), (19, 3, 3, 520, 4), (32, 8, 2, 1024, 32)])
def test_gemm_tc_qkv_heads(m, nq, nkv, k, page):
    """The fused q/k/v projection with head norms, rotation and cache write in its epilogue, against the
    plain functions; and against the product followed by the kernel that does the rest alone."""
    d, eps, theta, pages = 128, 1e-6, 1e6, 9
    g = torch.Generator().manual_seed(m + nq + k)
    x = torch.randn(m, k, generator=g).to(torch.bfloat16)
    w = (torch.randn((nq + 2 * nkv) * d, k, generator=g) / k ** 0.5).to(torch.bfloat16)
    q_w, k_w = 1 + 0.1 * torch.randn(d, generator=g), 1 + 0.1 * torch.randn(d, generator=g)
    positions = torch.randint(0, 3000, (m,), generator=g, dtype=torch.int32)
    slots = torch.randperm(pages * page, generator=g)[:m].to(torch.int32)
    slots[m // 2] = -1 if m > 1 else slots[0]                 # a row that writes nothing
    inv_freq = RotaryPosition.inverse_frequencies(d, theta)
    q_out = torch.full((m, nq * d), float("nan"), dtype=torch.bfloat16, device=DEV)
    kc = torch.zeros(pages, nkv, page, d, dtype=torch.bfloat16, device=DEV)
    vc = torch.zeros_like(kc)
    kernels.gemm_tc_qkv_heads(x.to(DEV), w.to(DEV), q_out, kc, vc, positions.to(DEV), slots.to(DEV), q_w.to(DEV), k_w.to(DEV),
                              eps, inv_freq.to(DEV), nq, nkv)
    torch.cuda.synchronize()
    kernels.check_device_errors()
    qkv = (x.double() @ w.double().T).float()                  # the plain functions on the unrounded product
    q, kk, v = plain_qk(qkv.to(DEV), positions.to(DEV), q_w.to(DEV), k_w.to(DEV), eps, theta, nq, nkv, d)
    close(q_out.view(m, nq, d), q, torch.bfloat16, "q")
    keep = (slots >= 0).nonzero().flatten()
    slot = slots[keep].long()
    close(kc.cpu()[slot // page, :, slot % page], kk[keep], torch.bfloat16, "k in the cache")
    close(vc.cpu()[slot // page, :, slot % page], v[keep], torch.bfloat16, "v in the cache")
    assert kc.count_nonzero().item() <= keep.numel() * nkv * d and vc.count_nonzero().item() <= keep.numel() * nkv * d
    # q only: nothing is written without slots
    kc.zero_()
    kernels.gemm_tc_qkv_heads(x.to(DEV), w.to(DEV), q_out, None, None, positions.to(DEV), None, q_w.to(DEV), k_w.to(DEV), eps,
                              inv_freq.to(DEV), nq, nkv)
    close(q_out.view(m, nq, d), q, torch.bfloat16, "q without a cache")
    assert kc.count_nonzero().item() == 0


@pytest.mark.parametrize("m,n,k", [(1, 128, 64), (8, 4096, 4096), (5, 136, 192), (8, 1000, 12288), (19, 520, 1024), (32, 256, 320)])
def test_gemm_tc_adds_to_the_stream_and_prepares_the_next_norm(m, n, k):
    """The product whose epilogue adds to the residual stream: stream += bfloat16(x . w^T), out = stream * the next
    norm's weights, and parts of the rows' sums of squares that add up to the rows' sums of squares."""
    g = torch.Generator().manual_seed(m * n + k)
    x = torch.randn(m, k, generator=g).to(torch.bfloat16)
    w = (torch.randn(n, k, generator=g) / k ** 0.5).to(torch.bfloat16)
    stream = 3 * torch.randn(m, n, generator=g)
    next_w = 1 + 0.2 * torch.randn(n, generator=g)
    on_device = stream.clone().to(DEV)
    out = torch.full((m, n), float("nan"), dtype=torch.bfloat16, device=DEV)
    sums = kernels.gemm_tc(x.to(DEV), w.to(DEV), out, residual=(on_device, next_w.to(DEV)))
    torch.cuda.synchronize()
    kernels.check_device_errors()
    product = (x.double() @ w.double().T)
    want_stream = stream.double() + product
    error = (on_device.cpu().double() - want_stream).abs()              # one bfloat16 rounding of the product, one float32 sum
    assert (error <= 2.0 ** -8 * product.abs() + 1e-5).all(), f"stream: {error.max().item():.3e}"
    close(out, want_stream * next_w.double(), torch.bfloat16, "stream times the next norm's weights")
    assert sums.shape[0] == (n + 127) // 128
    got = sums[:, :m].sum(0).cpu().double()
    exact = (on_device.cpu().double() ** 2).sum(1)                      # of the stream that the kernel wrote
    assert ((got - exact).abs() / exact).max().item() < 1e-5, "sums of squares"


@pytest.mark.parametrize("m", [1, 8, 16, 30])
def test_gemm_tc_more_ranges_for_the_tiles_of_the_last_round(m):
    """A plan of two counts of ranges (the first tiles 2, the tiles behind them 4 or 3), as the library plans a last
    round of units that would fill the GPU partly: plain, gated and adding to the stream, all equal to the same
    product with one count; and the plans of the shapes it was made for."""
    lib = kernels.gemm_tc_library()
    assert lib.mrs_gemm_tc_splits(24576, 4096, 148) == 2 | 3 << 8 | 148 << 16           # gate/up of the 8B shape: 44 tiles in the last round
    assert lib.mrs_gemm_tc_splits(151936, 4096, 148) == 1 | 16 << 8 | 1184 << 16        # the head: 3 tiles
    assert lib.mrs_gemm_tc_splits(4096, 4096, 148) == 4 and lib.mrs_gemm_tc_splits(6144, 4096, 148) == 3
    n, k = 20 * 128 + 72, 1024
    g = torch.Generator().manual_seed(m)
    x = torch.randn(m, k, generator=g).to(torch.bfloat16).to(DEV)
    w = (torch.randn(n, k, generator=g) / k ** 0.5).to(torch.bfloat16).to(DEV)
    want = x.double().cpu() @ w.double().cpu().T
    for plan in (2 | 4 << 8 | 12 << 16, 1 | 3 << 8 | 20 << 16, 3 | 2 << 8 | 1 << 16):
        out = torch.full((m, n), float("nan"), dtype=torch.float32, device=DEV)
        kernels.gemm_tc(x, w, out, splits=plan)
        close(out, want, torch.float32, f"plan {plan:#x}")
        stream = (3 * torch.randn(m, n, generator=g)).to(DEV)
        before = stream.clone()
        folded = torch.full((m, n), float("nan"), dtype=torch.bfloat16, device=DEV)
        sums = kernels.gemm_tc(x, w, folded, splits=plan, residual=(stream, torch.ones(n, device=DEV)))
        error = (stream.double().cpu() - before.double().cpu() - want).abs()
        assert (error <= 2.0 ** -8 * want.abs() + 1e-5).all(), f"stream with plan {plan:#x}: {error.max().item():.3e}"
        exact = (stream.double() ** 2).sum(1).cpu()
        assert ((sums[:, :m].sum(0).cpu().double() - exact).abs() / exact).max().item() < 1e-5
    inner = 20 * 64
    mixed = (torch.randn(2 * inner, k, generator=g) / k ** 0.5 * 2).to(torch.bfloat16).to(DEV)
    outs = []
    for plan in (2 | 4 << 8 | 12 << 16, 2):
        out = torch.full((m, inner), float("nan"), dtype=torch.bfloat16, device=DEV)
        kernels.gemm_tc(x, mixed, out, gated=True, splits=plan)
        outs.append(out)
    both = x.double().cpu() @ mixed.double().cpu().T
    gd, ud = both.view(m, -1, 2, 64)[:, :, 0].reshape(m, inner), both.view(m, -1, 2, 64)[:, :, 1].reshape(m, inner)
    close(outs[0], gd / (1 + torch.exp(-gd)) * ud, torch.bfloat16, "gated with two counts of ranges")
    assert torch.equal(outs[0][:, :12 * 64], outs[1][:, :12 * 64])      # the tiles with 2 ranges: the same bits either way
    torch.cuda.synchronize()
    kernels.check_device_errors()


@pytest.mark.parametrize("m,n,k,out_dtype", [(1, 256, 136, torch.float32), (8, 151936 // 8, 4096, torch.float32),
                                            (7, 520, 1024, torch.bfloat16), (40, 384, 512, torch.bfloat16)])
def test_gemm_tc_finishes_a_norm(m, n, k, out_dtype):
    """A product over rows that were multiplied by a norm's weights but not divided by their root mean square,
    with the rows' sums of squares in parts: equal to the product over the normalised rows."""
    eps = 1e-5
    g = torch.Generator().manual_seed(m + n + k)
    stream = 5 * torch.randn(m, k, generator=g) * (1 + torch.arange(m).float()[:, None])      # rows of very different size
    norm_w = 1 + 0.2 * torch.randn(k, generator=g)
    w = (torch.randn(n, k, generator=g) / k ** 0.5).to(torch.bfloat16)
    scaled = (stream * norm_w).to(torch.bfloat16)
    parts = 3
    stride = 48
    sums = torch.zeros(parts, stride)
    cut = [0, k // 3, k // 2, k]
    for p in range(parts):
        sums[p, :m] = (stream[:, cut[p]:cut[p + 1]] ** 2).sum(1)
    out = torch.full((m, n), float("nan"), dtype=out_dtype, device=DEV)
    kernels.gemm_tc(scaled.to(DEV), w.to(DEV), out, row_sums=(sums.to(DEV), k, eps))
    torch.cuda.synchronize()
    kernels.check_device_errors()
    factor = torch.rsqrt((stream.double() ** 2).mean(1, keepdim=True) + eps)
    normed = stream.double() * factor * norm_w.double()
    close(out, normed @ w.double().T, torch.bfloat16, "product over the normalised rows")     # x was rounded to bfloat16


@pytest.mark.parametrize("m", [1, 8])
def test_gemm_tc_gated_and_heads_finish_a_norm(m):
    """The same through the gated epilogue and through the q/k/v epilogue (whose head norms are not invariant
    under the factor, because of their eps)."""
    eps, k, inner, nq, nkv, d, page, pages, theta = 1e-6, 1024, 384, 4, 2, 128, 16, 4, 1e4
    g = torch.Generator().manual_seed(m)
    stream = 0.01 * torch.randn(m, k, generator=g)                         # small rows: the factor is large
    norm_w = 1 + 0.2 * torch.randn(k, generator=g)
    scaled = (stream * norm_w).to(torch.bfloat16)
    sums = torch.zeros(2, 16)
    sums[0, :m] = (stream[:, :600] ** 2).sum(1)
    sums[1, :m] = (stream[:, 600:] ** 2).sum(1)
    factor = torch.rsqrt((stream.double() ** 2).mean(1, keepdim=True) + eps)
    normed = scaled.double() * factor                                       # the rounding that the kernel sees
    gate = (torch.randn(inner, k, generator=g) / k ** 0.5 * 2).to(torch.bfloat16)
    up = (torch.randn(inner, k, generator=g) / k ** 0.5 * 2).to(torch.bfloat16)
    mixed = torch.stack([gate.view(-1, 64, k), up.view(-1, 64, k)], dim=1).reshape(2 * inner, k).contiguous()
    act = torch.full((m, inner), float("nan"), dtype=torch.bfloat16, device=DEV)
    kernels.gemm_tc(scaled.to(DEV), mixed.to(DEV), act, gated=True, row_sums=(sums.to(DEV), k, eps))
    gd, ud = normed @ gate.double().T, normed @ up.double().T
    close(act, gd / (1 + torch.exp(-gd)) * ud, torch.bfloat16, "gated")
    w = (torch.randn((nq + 2 * nkv) * d, k, generator=g) / k ** 0.5 * 0.02).to(torch.bfloat16)     # head norms feel their eps
    q_w, k_w = 1 + 0.1 * torch.randn(d, generator=g), 1 + 0.1 * torch.randn(d, generator=g)
    positions = torch.randint(0, 3000, (m,), generator=g, dtype=torch.int32)
    slots = torch.randperm(pages * page, generator=g)[:m].to(torch.int32)
    inv_freq = RotaryPosition.inverse_frequencies(d, theta)
    q_out = torch.full((m, nq * d), float("nan"), dtype=torch.bfloat16, device=DEV)
    kc = torch.zeros(pages, nkv, page, d, dtype=torch.bfloat16, device=DEV)
    vc = torch.zeros_like(kc)
    kernels.gemm_tc_qkv_heads(scaled.to(DEV), w.to(DEV), q_out, kc, vc, positions.to(DEV), slots.to(DEV), q_w.to(DEV), k_w.to(DEV),
                              1e-3, inv_freq.to(DEV), nq, nkv, row_sums=(sums.to(DEV), k, eps))
    torch.cuda.synchronize()
    kernels.check_device_errors()
    qkv = (normed @ w.double().T).float()
    q, kk, v = plain_qk(qkv.to(DEV), positions.to(DEV), q_w.to(DEV), k_w.to(DEV), 1e-3, theta, nq, nkv, d)
    close(q_out.view(m, nq, d), q, torch.bfloat16, "q")
    slot = slots.long()
    close(kc.cpu()[slot // page, :, slot % page], kk, torch.bfloat16, "k in the cache")
    close(vc.cpu()[slot // page, :, slot % page], v, torch.bfloat16, "v in the cache")


@pytest.mark.parametrize("m", [1, 7, 16, 20, 64, 100])
@pytest.mark.parametrize("n,k,splits", [(1024, 2048, 8), (1024, 3072, 12), (4096, 1024, 4), (6144, 4096, 3), (4096, 4096, 4), (300, 1032, 2),
                                        (128, 8192, 16), (384, 8192, 5), (24576, 4096, 2)])
def test_gemm_tc_ranges_merged_in_a_cluster(m, n, k, splits, monkeypatch):
    """Where every range has a CTA of its own the ranges of a tile meet in a cluster's shared memory: the same bits as
    with fewer CTAs, whose partial sums go through global memory (both add the ranges in their order), in every epilogue."""
    torch.manual_seed(31)
    x = torch.randn(m, k, dtype=torch.bfloat16, device=DEV)
    w = torch.randn(n, k, dtype=torch.bfloat16, device=DEV) / k ** 0.5
    lib = kernels.gemm_tc_library()
    assert lib.mrs_gemm_tc_splits(6144, 1024, 148) == 2 and lib.mrs_gemm_tc_splits(1024, 3072, 148) == 8     # by N, K and SMs alone
    state = kernels._gemm_device_state(x.device)
    mpad = 16 if m <= 16 else (32 if m <= 32 else (64 if m <= 64 else 128))
    if (n, k, splits) in ((1024, 2048, 8), (300, 1032, 2)) and m <= 20:      # few tiles, sums that find room: clusters for certain
        assert lib.mrs_gemm_tc_in_cluster(m, n, k, splits, mpad, state["sms"])
    assert not lib.mrs_gemm_tc_in_cluster(m, n, k, splits, mpad, 5)
    results = []
    for sms in (state["sms"], 5):
        monkeypatch.setitem(state, "sms", sms)
        stream = torch.linspace(-2, 2, m * n, device=DEV).view(m, n).contiguous()
        plain, folded = torch.empty(m, n, device=DEV), torch.empty(m, n, dtype=torch.bfloat16, device=DEV)
        for _ in range(3):                       # back to back: a launch begins under the one before it
            kernels.gemm_tc(x, w, plain, splits=splits)
        rounded = torch.empty(m, n, dtype=torch.bfloat16, device=DEV)
        kernels.gemm_tc(x, w, rounded, splits=splits)
        assert torch.equal(rounded, plain.bfloat16())
        out = [plain, rounded]
        if n % 128 == 0:
            gated = torch.empty(m, n // 2, dtype=torch.bfloat16, device=DEV)
            kernels.gemm_tc(x, w, gated, gated=True, splits=splits)
            out.append(gated)
        if m <= 32:
            sums = kernels.gemm_tc(x, w, folded, splits=splits, residual=(stream, torch.ones(n, device=DEV)))
            out += [folded, stream, sums[:, :m]]
        results.append(out)
    for a, b in zip(*results):
        assert torch.equal(a, b)
    close(results[0][0], x.double() @ w.double().T, torch.float32, f"gemm_tc {m}x{n}x{k} in {splits} ranges")


FIRST_PRODUCTS = """
import torch
from mini_rsglang_b200 import kernels
lib, sms = kernels.gemm_tc_library(), kernels.sm_count(torch.device("cuda", 0))
g = torch.Generator(device="cuda").manual_seed(4)
for n, k in ((4096, 4096), (1024, 3072), (3072, 2048), (4096, 4096)):      # 4, 8 and 4 ranges: each new count is asked about in between
    x, w = torch.randn(16, k, device="cuda", generator=g).bfloat16(), (torch.randn(n, k, device="cuda", generator=g) / k ** 0.5).bfloat16()
    assert lib.mrs_gemm_tc_splits(n, k, sms) > 1
    for m in (1, 16):
        out = torch.empty(m, n, device="cuda", dtype=torch.bfloat16)
        kernels.gemm_tc(x[:m].contiguous(), w, out)
        want = x[:m].double() @ w.double().T
        assert ((out.double() - want).abs() <= want.abs() * 2.0 ** -8 + 1e-4).all(), (n, k, m)
"""


def test_gemm_tc_plain_bfloat16_product_as_a_process_first():
    """Asking how many clusters the GPU holds leaves the limits of shared memory as the launches set them: bfloat16 products of full
    rings and clusters are taken as a process's first ones, and after another count of ranges was asked about."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    done = subprocess.run([sys.executable, "-c", FIRST_PRODUCTS], cwd=root, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]


def test_gemm_tc_rows_do_not_depend_on_the_batch():
    """The same row alone, among 8 and among 100 others: equal bit for bit, twice in a row (the
    counters of the ranges of K are left ready for the next launch)."""
    g = torch.Generator().manual_seed(5)
    n, k = 4096, 4096
    x = torch.randn(100, k, generator=g).to(torch.bfloat16).to(DEV)
    w = (torch.randn(n, k, generator=g) / 64).to(torch.bfloat16).to(DEV)
    outs = []
    for m in (1, 8, 100, 1):
        out = torch.empty((m, n), dtype=torch.float32, device=DEV)
        kernels.gemm_tc(x[:m].contiguous(), w, out)
        outs.append(out[0].clone())
    torch.cuda.synchronize()
    kernels.check_device_errors()
    for other in outs[1:]:
        assert torch.equal(outs[0], other)
    assert not kernels.gemm_tc_supported(x[:, :100].contiguous(), w[:, :100].contiguous())      # rows of 200 bytes
    assert not kernels.gemm_tc_supported(torch.zeros(129, 64, dtype=torch.bfloat16, device=DEV), w[:, :64].contiguous())


# --------------------------------------------------------------------------------- sampling
def test_argmax_takes_the_smaller_id_on_a_tie():
    logits = torch.randn(6, 1000, device=DEV)
    logits[0, 17] = logits[0, 900] = 50.0
    logits[1, 999] = 60.0
    logits[2, 0] = 60.0
    logits[3] = 0.0
    out = torch.empty(6, dtype=torch.int32, device=DEV)
    kernels.argmax(logits, out)
    want = [17, 999, 0, 0] + [int(logits[i].argmax()) for i in (4, 5)]
    assert out.tolist() == want


@pytest.mark.parametrize("tokens,top,routed,tile", [(1, 1, 1, 32), (5, 3, 33, 32), (2047, 4, 32, 128), (2048, 4, 200, 128), (2049, 4, 7, 128), (7001, 6, 64, 128)])
def test_expert_lists_hold_every_pair_once(tokens, top, routed, tile):
    """On both sides of the choices that one block's threads keep in registers, experts beyond a warp's, choices without weights
    (numbers from `routed` on): every pair of a routed expert once, in tiles of its expert, the others nowhere."""
    g = torch.Generator().manual_seed(tokens)
    chosen = torch.randint(0, routed + 2, (tokens, top), generator=g, dtype=torch.int32)
    capacity = kernels.moe_capacity(tokens * top, routed, tile)
    rows = torch.full((capacity,), 77, dtype=torch.int32, device=DEV)
    experts = torch.full((capacity // tile + 1,), 77, dtype=torch.int32, device=DEV)
    kernels.moe_align(chosen.to(DEV), routed, tile, rows, experts)
    rows, experts, flat = rows.cpu(), experts.cpu(), chosen.flatten()
    assert sorted(rows[rows >= 0].tolist()) == (flat < routed).nonzero().flatten().tolist()
    used = sum(-(-int((flat == e).sum()) // tile) for e in range(routed))
    assert int(experts[-1]) == used and (experts[used:-1] == -1).all() and (rows[used * tile:] == -1).all()
    for i in range(used):
        listed = rows[i * tile:(i + 1) * tile]
        assert (flat[listed[listed >= 0].long()] == experts[i]).all() and (listed >= 0).any()
    assert experts[:used].tolist() == sorted(experts[:used].tolist())


@pytest.mark.parametrize("vocab", [16384, 70001, 151936])
def test_argmax_of_long_rows_shared_by_a_cluster(vocab):
    """Rows long enough to be shared by the blocks of a cluster: ties across shares, the last id,
    a share's edge."""
    logits = torch.randn(5, vocab, device=DEV)
    share = -(-vocab // (8 if vocab >= 65536 else 4))
    logits[0, 5] = logits[0, vocab - 1] = 40.0          # a tie between the first and the last share
    logits[1, vocab - 1] = 41.0
    logits[2, share - 1] = logits[2, share] = 42.0      # a tie across a share's edge
    logits[3, share] = 43.0
    out = torch.empty(5, dtype=torch.int32, device=DEV)
    kernels.argmax(logits, out)
    assert out.tolist() == [5, vocab - 1, share - 1, share, int(logits[4].argmax())]


def plain_draw(logits, params: SamplingParams, index: int) -> int:
    """The kernel's draw restated: the reference's support, then the inverse CDF in id order."""
    ids, weights = P.nucleus_support(logits.double().cpu(), params.temperature, params.top_k, params.top_p)
    pairs = sorted(zip(ids, weights))
    u = uniform_from_counter(params.seed, index) * sum(w for _, w in pairs)
    run = 0.0
    for i, w in pairs:
        run += w
        if run > u:
            return i
    return pairs[-1][0]


@pytest.mark.parametrize("vocab", [3, 301, 5000])
def test_sampler_support_and_repeatability(vocab):
    sampler = Sampler(torch.device(DEV))
    g = torch.Generator().manual_seed(vocab)
    logits = (torch.randn(1, vocab, generator=g) * 2).to(DEV)
    settings = [SamplingParams(temperature=1.0, seed=42), SamplingParams(temperature=0.7, top_k=2, top_p=0.9, seed=42),
                SamplingParams(temperature=1.3, top_p=0.5, seed=7), SamplingParams(temperature=0.5, top_k=min(50, vocab), seed=9),
                SamplingParams(temperature=2.0, top_k=vocab + 5, top_p=0.999, seed=11)]
    for params in settings:
        support, _ = P.nucleus_support(logits[0].cpu(), params.temperature, params.top_k, params.top_p)
        draws = 200
        rows = logits.expand(draws, vocab).contiguous()
        got = sampler.sample(rows, [params] * draws, list(range(draws)))
        assert got == sampler.sample(rows, [params] * draws, list(range(draws)))      # same seed, same draws
        assert set(got) <= set(support), f"drew outside the support with {params}"
        want = [plain_draw(logits[0], params, i) for i in range(draws)]
        agree = sum(a == b for a, b in zip(got, want))
        assert agree >= draws - 2, f"{draws - agree} of {draws} draws differ from the plain draw with {params}"
    tiny = SamplingParams(temperature=1.0, top_k=2, top_p=0.01, seed=1)
    assert set(sampler.sample(logits.expand(20, vocab).contiguous(), [tiny] * 20, list(range(20)))) == {int(logits[0].argmax())}


@pytest.mark.parametrize("vocab", [1, 32, 1025, 8191, 8192, 32768, 65535, 65536, 151936, 196640, 327680, 327681])
def test_sampler_rows_that_several_ctas_share(vocab):
    """One row a cluster of 1, 4 or 8 CTAs, in shared memory or (from 327,681 logits on) read from memory; rows that start off a
    16-byte boundary; equal logits across the shares' edges, of which a cut by count or by weight keeps the first ids; every row
    against the draw restated in float64.  A draw may differ only where u falls within 1e-5 of the weight of its token's interval (float32
    sums of at most 327,681 weights in 1,024 runs), which at most one row in twenty does; the same call again gives the same tokens."""
    sampler = Sampler(torch.device(DEV))
    g = torch.Generator().manual_seed(vocab)
    settings = [SamplingParams(temperature=0.8, top_p=0.95, seed=1), SamplingParams(temperature=0.7, top_k=50, top_p=0.9, seed=2),
                SamplingParams(temperature=1.0, seed=3), SamplingParams(temperature=0.6, top_k=20, seed=4), SamplingParams(temperature=0.0),
                SamplingParams(temperature=5.0, top_p=0.6, seed=5), SamplingParams(temperature=1.0, top_k=max(1, vocab - 1), top_p=0.7, seed=6)]
    params = [settings[i % len(settings)] for i in range(21)]
    logits = torch.randn(21, vocab, generator=g) * 2
    logits[7:14] = (logits[7:14] * 2).round() / 2          # a few dozen values: long runs of equals at every cut
    logits[14:] = logits[14:].clamp(max=1.5)
    got = sampler.sample(logits.to(DEV), params, list(range(21)))
    wrong = sum(not drawn(row, p, i, token, 1e-5) for row, p, i, token in zip(logits.double(), params, range(21), got))
    assert wrong <= 1, wrong
    assert sampler.sample(logits.to(DEV), params, list(range(21))) == got          # whole numbers and fixed orders: the same bits


@pytest.mark.parametrize("vocab", [4000, 20000, 70000])
@pytest.mark.parametrize("bunch", [1, 1000, 1023, 1024, 1025, 3000])
def test_sampler_candidates_up_to_their_limit(vocab, bunch):
    """Thresholds inside a bunch of `bunch` logits that lie within a 64th of a logarithm (half of them equal): as many candidates as
    are sorted at once, and more; temperatures that put every logit into one bin, or nearly all behind the last."""
    g = torch.Generator().manual_seed(vocab + bunch)
    row = torch.randn(vocab, generator=g) * 2 - 9.0
    at = torch.randperm(vocab, generator=g)
    row[at[:20]] = 8.0 - 0.1 * torch.arange(20)
    row[at[20:20 + bunch]] = 4.0001 + 0.01 * torch.rand(bunch, generator=g)
    row[at[20:20 + bunch // 2]] = 4.005
    settings = [SamplingParams(temperature=1.0, top_k=20 + k, seed=k) for k in {1, bunch // 3, bunch - 1, bunch} if k > 0]
    settings += [SamplingParams(temperature=1.0, top_k=min(20 + bunch, 1000), top_p=p, seed=3) for p in (0.5, 0.97, 0.999)]
    settings += [SamplingParams(temperature=1.0, top_p=p, seed=5) for p in (0.4, 0.93, 0.999)]
    settings += [SamplingParams(temperature=t, top_k=k, top_p=0.9, seed=7) for t in (1e-3, 300.0) for k in (None, 3, 40)]
    params = [p for p in settings for _ in range(3)]
    got = Sampler(torch.device(DEV)).sample(row.expand(len(params), vocab).contiguous().to(DEV), params, list(range(len(params))))
    wrong = sum(not drawn(row.double(), p, i, token, 1e-5) for i, (p, token) in enumerate(zip(params, got)))
    assert wrong <= 1, wrong


def test_sampler_launches_that_are_outstanding():
    """Launches behind one another, with more rows each and on streams of their own, before any is read; a sampler that goes while its
    last launch is under way."""
    logits = torch.randn(400, 9000, device=DEV) * 2
    sampler, held = Sampler(torch.device(DEV)), []
    params = [SamplingParams(temperature=1.0, top_k=1 + i % 40, seed=i) for i in range(400)]
    torch.cuda.synchronize()
    for n in (3, 100, 400):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            held.append((n, sampler.launch(logits[:n].contiguous(), params[:n], list(range(n)))))
    got = [sampler.read(chosen) for _, chosen in held]
    last = sampler.launch(logits, params, list(range(400)))
    del sampler
    want = Sampler(torch.device(DEV)).sample(logits, params, list(range(400)))
    assert all(tokens == want[:n] and chosen.tokens.tolist() == tokens for (n, chosen), tokens in zip(held, got))
    assert last.host.tolist() == want


@pytest.mark.parametrize("greedy", [False, True])
def test_sampler_launches_in_a_graph(greedy):
    """More launches recorded in one graph than a sampler has buffers in turn, behind and before ordinary ones; every replay chooses from
    the logits that are there then."""
    params = [SamplingParams(temperature=0.0 if greedy else 0.9, top_k=None if greedy else 30, seed=i) for i in range(7)]
    logits, sampler = torch.randn(7, 5000, device=DEV), Sampler(torch.device(DEV))
    for _ in range(4):
        sampler.sample(logits, params, [0] * 7)
    graph, held = torch.cuda.CUDAGraph(), []
    with torch.cuda.graph(graph):
        for n in range(5):
            held.append(sampler.launch(logits, params, [n] * 7))
    for _ in range(2):
        logits.normal_()
        graph.replay()
        torch.cuda.synchronize()
        for n, chosen in enumerate(held):
            want = sampler.sample(logits, params, [n] * 7)
            assert chosen.tokens.tolist() == want and chosen.host.tolist() == want


def drawn(row, p, index, token, tolerance) -> bool:
    """Whether `token` is the draw restated in float64: the support by a stable sort, then the inverse CDF in id order.  A token that is
    not has to be one that float32 sums may give instead: u within `tolerance` of the kept weight of that token's own interval, and the
    token kept, or the next one at the edge of the support (which one it is hangs on a float32 product: 2^-23 of the weight)."""
    if p.is_greedy():
        assert token == int(row.argmax())
        return True
    order = torch.sort(row, descending=True, stable=True).indices[:p.top_k]
    weight = torch.exp((row[order] - row[order[0]]) / p.temperature)
    total = weight.sum()
    keep = len(order) if p.top_p >= 1.0 else int((torch.cumsum(weight, 0) < p.top_p * total * (1 - 1e-12)).sum()) + 1
    more = 0 if p.top_p >= 1.0 else 1 + int(total * 2.0 ** -23 / weight[min(keep, len(order)) - 1])
    kept = torch.sort(order[:keep]).values
    running = torch.cumsum(torch.exp((row[kept] - row.max()) / p.temperature), 0)
    u = uniform_from_counter(p.seed, index)
    place = int(torch.searchsorted(running, u * running[-1], right=True))
    if token == int(kept[min(place, len(kept) - 1)]):
        return True
    kept = torch.sort(order[:keep + more]).values
    at = int(torch.searchsorted(kept, torch.tensor(token)))
    assert at < len(kept) and int(kept[at]) == token, f"{token} is not kept by {p}"
    running = torch.cumsum(torch.exp((row[kept] - row.max()) / p.temperature), 0) / running[-1]
    before = running[at - 1] if at else 0.0
    assert before - tolerance <= u <= running[at] + tolerance, f"u {u} lies off {token}'s interval, {before} to {running[at]}, with {p}"
    return False


@pytest.mark.parametrize("vocab", [151936, 262144, 1000003])
@pytest.mark.parametrize("ragged", [False, True])
def test_sampler_counts_a_long_tail_of_small_weights(vocab, ragged):
    """One large logit (the last id) and a long tail whose weights are a 2^-35 to 2^-31 of it and together 2.75e-5: the cut by weight at
    1 - 2^-16 keeps the tail's first 1.22e-5 (of equal weights the first ids), so that draws with a small u are tokens of the tail, each
    the one that u names to 2^-23 (the cut's weight is a float32 product; a tail that ends a little earlier or later moves the others)."""
    g = torch.Generator().manual_seed(vocab)
    tail = torch.full((vocab,), 2.75e-5 / vocab, dtype=torch.float64)
    if ragged:
        tail *= torch.rand(vocab, generator=g, dtype=torch.float64) * 1.2 + 0.4
    tail[-1] = 1.0
    logits = torch.log(tail).float()
    p = SamplingParams(temperature=1.0, top_p=1.0 - 2.0 ** -16, seed=77)
    index = torch.arange(1 << 21)
    u = uniforms(p.seed, index)
    small = index[(u > 1e-6) & (u < 1.1e-5)][:8].tolist()
    assert len(small) == 8 and u[small[0]] == uniform_from_counter(p.seed, small[0])
    got = Sampler(torch.device(DEV)).sample(logits.expand(8, vocab).contiguous().to(DEV), [p] * 8, small)
    for i, token in zip(small, got):
        assert token != vocab - 1
        drawn(logits.double(), p, i, token, 2.0 ** -23)
    assert Sampler(torch.device(DEV)).sample(logits[None].to(DEV), [SamplingParams(temperature=1e-42)], [0]) == [vocab - 1]


def uniforms(seed, index):
    """`uniform_from_counter` of many draw indices."""
    with np.errstate(over="ignore"):
        z = np.uint64(seed) + np.uint64(0x9E3779B97F4A7C15) * (index.numpy().astype(np.uint64) + np.uint64(1))
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return torch.from_numpy(((z ^ (z >> np.uint64(31))) >> np.uint64(40)).astype(np.float64)) / 16777216.0


def test_sampler_distribution_ties_and_bad_rows():
    sampler = Sampler(torch.device(DEV))
    logits = torch.tensor([[0.0, 2.0, 1.0, -1.0, 0.5]], device=DEV)
    params = SamplingParams(temperature=0.7, seed=3)
    draws = 4000
    got = sampler.sample(logits.expand(draws, 5).contiguous(), [params] * draws, list(range(draws)))
    probs = torch.softmax(logits[0].double().cpu() / 0.7, 0)
    counts = torch.bincount(torch.tensor(got), minlength=5).double()
    chi2 = ((counts - draws * probs) ** 2 / (draws * probs)).sum().item()
    assert chi2 < 25.0, f"chi-square {chi2:.1f} over 4 degrees of freedom"
    # all logits equal, top_k 3: the three smallest ids, as the reference's sort by (value, id) keeps them
    flat = torch.zeros(300, 40, device=DEV)
    got = sampler.sample(flat, [SamplingParams(temperature=1.0, top_k=3, seed=5)] * 300, list(range(300)))
    assert set(got) == {0, 1, 2}
    got = sampler.sample(flat, [SamplingParams(temperature=1.0, top_p=0.1, seed=5)] * 300, list(range(300)))
    assert set(got) == {0, 1, 2, 3}
    # greedy rows beside sampled rows
    mixed = sampler.sample(logits.expand(3, 5).contiguous(),
                           [SamplingParams(), SamplingParams(temperature=0.9, top_k=1), params], [0, 0, 0])
    assert mixed[0] == 1 and mixed[1] == 1
    bad = logits.clone()
    bad[0, 2] = float("nan")
    with pytest.raises(BackendError, match="nonfinite"):
        sampler.sample(bad, [params], [0])
    bad[0, 2] = float("inf")
    with pytest.raises(BackendError, match="nonfinite"):
        sampler.sample(bad, [params], [0])


@pytest.mark.parametrize("per_expert", [1, 8, 9, 16, 17, 40])
@pytest.mark.parametrize("experts,width,inner,block", [(3, 72, 40, 0), (2, 136, 64, 64), (4, 1032, 200, 0), (2, 4104, 128, 64), (1, 2048, 1032, 0)])
def test_experts_for_few_rows(per_expert, experts, width, inner, block):
    """The tensor-core product for few rows an expert over whole and filled-up tiles of 8, 16 and 32 rows, K split among 1, 2, 4
    and 8 warps with a ragged end, columns beyond the last group, an expert without rows: silu(gate) * up and the down product
    within bfloat16 rounding of the 64-bit result; ungated experts that read gathered rows likewise; a row's bits do not
    depend on the other rows of its tile."""
    g = torch.Generator(device=DEV).manual_seed(per_expert * 31 + width)
    top = 2 if experts > 1 else 1
    tokens = max(1, per_expert * experts // top)
    h = torch.randn(tokens, width, device=DEV, generator=g).bfloat16()
    gate, up = ((torch.randn(experts, inner, width, device=DEV, generator=g) * width ** -0.5).bfloat16() for _ in range(2))
    down = (torch.randn(experts, width, inner, device=DEV, generator=g) * inner ** -0.5).bfloat16()
    chosen = torch.stack([torch.randperm(experts, generator=g, device=DEV)[:top] for _ in range(tokens)]).int()
    if experts > 3:
        chosen = chosen % 3                                   # an expert without rows (and tokens that choose one twice)
    if block:
        laid = torch.stack([gate.view(experts, -1, block, width), up.view(experts, -1, block, width)], dim=2).reshape(experts, 2 * inner, width)
    else:
        laid = torch.cat([gate, up], dim=1)
    y = torch.full((tokens * top, width), 77.0, device=DEV).bfloat16()
    kernels.moe_experts(h, chosen, laid.contiguous(), down, y, experts, kernel="few", block=block)
    plain = torch.full_like(y, 77.0)
    kernels.moe_plain_experts(h, chosen, None, up, down, plain, experts, "relu", kernel="few")
    pairs = chosen.view(-1).long()
    x = h.repeat_interleave(top, dim=0).double()
    z = torch.einsum("pw,piw->pi", x, gate.double()[pairs]).bfloat16().double()
    u = torch.einsum("pw,piw->pi", x, up.double()[pairs])
    act = (z * torch.sigmoid(z) * u.bfloat16().double()).bfloat16().double()
    # three bfloat16 roundings on the way (gate, up, their product) and one at the end, each 2^-9 of its value
    for got, inner_rows in ((y, act), (plain, torch.relu(u).bfloat16().double())):
        want = torch.einsum("pi,pwi->pw", inner_rows, down.double()[pairs])
        size = torch.einsum("pi,pwi->pw", inner_rows.abs(), down.double()[pairs].abs())
        assert ((got.double() - want).abs() <= want.abs() * 2.0 ** -8 + size * 2.0 ** -7).all()
    alone = torch.empty((top, width), device=DEV).bfloat16()
    last = tokens - 1
    kernels.moe_experts(h[last:].clone(), chosen[last:].clone(), laid.contiguous(), down, alone, experts, kernel="few", block=block)
    assert torch.equal(alone, y[last * top:])


@pytest.mark.parametrize("heads,latent,rotated,page,window", [(16, 256, 32, 16, 1024), (16, 256, 32, 16, 0), (32, 256, 32, 8, 100), (5, 192, 64, 64, 0),
                                                              (3, 128, 0, 128, 70), (64, 64, 32, 32, 0), (1, 256, 0, 16, 65), (128, 64, 64, 16, 64)])
def test_attention_latent_tc(heads, latent, rotated, page, window):
    """The tcgen05 latent attention over tiles of 128 rows: whole and ragged tiles, heads that do not divide 128, portions behind
    contexts on both sides of a block's and a page's end, rings gone round several times, windows that begin inside a block with
    the pages before them given back, gates and sinks; entries without tokens are left out."""
    spans = [(0, 1), (0, 130), (63, 2), (64, 65), (500, 40), (1100, 9), (2047, 1)]
    row, per_tile = latent + rotated, 128 // heads
    g = torch.Generator(device=DEV).manual_seed(heads + latent + page)
    pages = [-(-(c + n) // page) for c, n in spans]
    cache = torch.randn(sum(pages) + 3, 1, page, row, device=DEV, generator=g).bfloat16()
    order = torch.randperm(cache.shape[0], generator=g, device=DEV).int().tolist()
    table = torch.full((len(spans), max(pages)), -1, dtype=torch.int32)
    tiles, positions, first = [], [], 0
    for i, (c, n) in enumerate(spans):
        taken = [order.pop() for _ in range(pages[i])]
        gone = max(0, c - window + 1) // page if window else 0
        table[i, :pages[i]] = torch.tensor([-1] * gone + taken[gone:], dtype=torch.int32)
        tiles += [(i, first + s, min(per_tile, n - s), 0) for s in range(0, n, per_tile)] + [(0, 0, 0, 0)]
        positions += range(c, c + n)
        first += n
    q = torch.randn(first, heads * row, device=DEV, generator=g).bfloat16()
    gate, sinks = torch.rand(first, heads, device=DEV, generator=g), torch.randn(heads, device=DEV, generator=g) * 3
    scale = 1.7 * row ** -0.5
    i32 = lambda x: torch.as_tensor(x, dtype=torch.int32).to(DEV)      # noqa: E731
    for use_gate, use_sinks in ((True, True), (False, False)):
        out = torch.full((first, heads * latent), 77.0, device=DEV).bfloat16()
        kernels.attention_latent_tc(q, cache, i32(positions), i32(table), i32(tiles), out, heads, latent, rotated, scale, window=window,
                                    gate=gate if use_gate else None, sink_logits=sinks if use_sinks else None)
        kernels.check_device_errors(certain=True)
        at = 0
        for i, (c, n) in enumerate(spans):
            slots = torch.arange(c + n, device=DEV)
            keys = cache[table[i].to(DEV).long()[slots // page].clamp(min=0), 0, slots % page].double()
            scores = torch.einsum("thd,kd->thk", q[at:at + n].view(n, heads, row).double(), keys) * scale
            query, key = torch.arange(c, c + n, device=DEV)[:, None], slots[None]
            seen = (key <= query) & ((key > query - window) if window else True)
            scores = scores.masked_fill(~seen[:, None], -float("inf"))
            if use_sinks:
                scores = torch.cat([scores, sinks.double()[None, :, None].expand(n, heads, 1)], dim=2)
            weights = torch.softmax(scores, dim=2)[:, :, :c + n]
            want = torch.einsum("thk,ke->the", weights, keys[:, :latent])
            size = torch.einsum("thk,ke->the", weights, keys[:, :latent].abs())
            if use_gate:
                want, size = want * gate[at:at + n].double()[..., None], size * gate[at:at + n].double()[..., None]
            got = out[at:at + n].view(n, heads, latent).double()
            # a weight and the result rounded to bfloat16 (2^-9 each), the scores' float32 sums far below
            assert ((got - want).abs() <= want.abs() * 2.0 ** -8 + size * 2.0 ** -8 + 1e-6).all(), (i, use_gate)
            at += n


@pytest.mark.parametrize("heads,latent,rotated,page,window", [(16, 256, 32, 16, 0), (16, 256, 32, 16, 100), (32, 256, 32, 8, 1024), (5, 192, 64, 64, 70),
                                                              (3, 128, 0, 128, 0), (64, 64, 32, 32, 33)])
def test_attention_latent_tc_leaves_out_rows_that_no_query_sees(heads, latent, rotated, page, window):
    """Rows behind a portion's last key, before its window, on pages of other requests, on the cache's first page (which no table names
    here) and on pages that were given back are no numbers: the results are those over a clean cache, bit for bit."""
    spans = [(0, 1), (0, 130), (63, 1), (64, 65), (500, 3), (1100, 9)]
    row, per_tile = latent + rotated, 128 // heads
    g = torch.Generator(device=DEV).manual_seed(heads + page)
    i32 = lambda x: torch.as_tensor(x, dtype=torch.int32).to(DEV)      # noqa: E731
    scale = row ** -0.5
    for c, n in spans:
        pages = -(-(c + n) // page)
        clean = torch.randn(2 * pages + 3, 1, page, row, device=DEV, generator=g).bfloat16()
        order = (1 + torch.randperm(clean.shape[0] - 1, generator=g, device=DEV)[:pages]).tolist()
        # one portion of a tile's tokens at a time: which of its rows nobody sees is then the portion's own matter
        for start in {0, (n - 1) // per_tile * per_tile}:
            tokens, first = min(per_tile, n - start), c + start
            seen = max(0, first - window + 1) if window else 0
            q = torch.randn(tokens, heads * row, device=DEV, generator=g).bfloat16()
            dirty = torch.full_like(clean, float("nan"))
            dirty[::2] = float("inf")
            slots = torch.arange(seen, first + tokens, device=DEV)
            pages_of = torch.tensor(order, device=DEV)[slots // page]
            dirty[pages_of, 0, slots % page] = clean[pages_of, 0, slots % page]
            results = []
            for cache, gone in ((clean, 0), (dirty, 0), (dirty, seen // page)):
                out = torch.full((tokens, heads * latent), 77.0, device=DEV).bfloat16()
                kernels.attention_latent_tc(q, cache, i32(list(range(first, first + tokens))), i32([[-1] * gone + order[gone:]]), i32([(0, 0, tokens, 0)]), out,
                                            heads, latent, rotated, scale, window=window)
                kernels.check_device_errors(certain=True)
                results.append(out)
            assert torch.isfinite(results[0].float()).all()
            assert torch.equal(results[0], results[1]) and torch.equal(results[0], results[2]), (c, n, start)


def test_attention_latent_tc_makes_a_caches_maps_once(monkeypatch):
    """The tensor maps of a cache are made at its first call and kept; another cache, and the same memory as pages of another size, get
    their own."""
    heads, latent, rotated = 4, 64, 32
    row = latent + rotated
    lib = kernels.attention_latent_tc_library(latent, rotated)
    make, made = lib.mrs_attention_latent_tc_cache_maps, []
    monkeypatch.setattr(lib, "mrs_attention_latent_tc_cache_maps", lambda *a: made.append(a[:3]) or make(*a))
    monkeypatch.setattr(kernels, "_latent_tc_cache_maps", {})
    g = torch.Generator(device=DEV).manual_seed(8)
    caches = [torch.randn(6, 1, 16, row, device=DEV, generator=g).bfloat16() for _ in range(2)]
    caches.append(caches[0].view(3, 1, 32, row))
    q = torch.randn(9, heads * row, device=DEV, generator=g).bfloat16()
    i32 = lambda x: torch.as_tensor(x, dtype=torch.int32).to(DEV)      # noqa: E731
    for again in range(2):
        for cache in caches:
            out = torch.empty(9, heads * latent, device=DEV).bfloat16()
            kernels.attention_latent_tc(q, cache, i32(list(range(70, 79))), i32([list(range(cache.shape[0]))]), i32([(0, 0, 9, 0)]), out, heads, latent, rotated, 0.1)
            keys = cache.view(-1, row)[:79].double()
            scores = torch.einsum("thd,kd->thk", q.view(9, heads, row).double(), keys) * 0.1
            scores = scores.masked_fill(torch.arange(79, device=DEV)[None, None] > torch.arange(70, 79, device=DEV)[:, None, None], -float("inf"))
            want = torch.softmax(scores, 2) @ keys[:, :latent]
            size = torch.softmax(scores, 2) @ keys[:, :latent].abs()
            assert ((out.view(9, heads, latent).double() - want).abs() <= want.abs() * 2.0 ** -8 + size * 2.0 ** -8 + 1e-6).all()
        assert len(made) == 3


def test_attention_latent_tc_scores_that_are_no_numbers():
    """A query that is no number gives its own (token, head) no number and no other one; rows whose scores are all -inf have no
    weights and give zeros; a score of +inf gives no number, as its softmax does."""
    heads, latent, rotated, page, n = 16, 256, 32, 16, 8
    row = latent + rotated
    g = torch.Generator(device=DEV).manual_seed(3)
    cache = torch.randn(9, 1, page, row, device=DEV, generator=g).bfloat16()
    cache[..., latent:] = cache[..., latent:].abs() + 1               # the last elements tell the sign of an infinite score
    q = torch.randn(n, heads, row, device=DEV, generator=g).bfloat16()
    i32 = lambda x: torch.as_tensor(x, dtype=torch.int32).to(DEV)      # noqa: E731

    def attend(q):
        out = torch.full((n, heads * latent), 77.0, device=DEV).bfloat16()
        kernels.attention_latent_tc(q.reshape(n, -1).contiguous(), cache, i32(list(range(100, 100 + n))), i32([[3, 1, 4, 8, 5, 0, 2]]), i32([(0, 0, n, 0)]), out,
                                    heads, latent, rotated, row ** -0.5)
        kernels.check_device_errors(certain=True)
        return out.view(n, heads, latent)

    clean, odd = attend(q), q.clone()
    odd[2, 3, 7] = float("nan")
    odd[5, 0, row - 1] = -float("inf")
    odd[6, 9, row - 1] = float("inf")
    got = attend(odd)
    assert torch.isnan(got[2, 3]).all() and torch.isnan(got[6, 9]).all() and (got[5, 0] == 0).all()
    for token, head in ((2, 3), (5, 0), (6, 9)):
        got[token, head] = clean[token, head]
    assert torch.equal(got, clean)


def test_attention_f32_keeps_what_is_no_number_in_its_row():
    """A query that is no number gives its own (token, head) no number and no other one, in tiles of rows, single tokens and with the
    keys in chunks."""
    nq, nkv, d, page = 4, 2, 64, 16
    case = PagedCase(torch.float32, nq, nkv, d, page, [(0, 90), (700, 3), (1200, 1)], seed=5)
    clean = case.run_simt().view(-1, nq, d)
    odd = case.q.clone().view(-1, nq, d)
    marks = ((0, 1), (70, 2), (91, 0), (93, 3))
    for token, head in marks:
        odd[token, head, 5] = float("nan")
    case.q = odd.view(case.q.shape)
    got = case.run_simt().view(-1, nq, d)
    for token, head in marks:
        assert torch.isnan(got[token, head]).all()
        got[token, head] = clean[token, head]
    assert torch.equal(got, clean)


@pytest.mark.parametrize("exponent", [-90, -105, -113, -122, -126, 100])
def test_attention_f32_on_tensor_cores_of_small_and_large_values(exponent):
    """Heads of 128: values of one power of two keep every bit, also where the last bfloat16 part would lie under that type's range.  The
    error is that of the values before the scaling, beside half a unit of the smallest float32 a key."""
    spans = [(0, 130), (300, 5)]
    case = PagedCase(torch.float32, 4, 2, 128, 16, spans, seed=12)
    want = case.plain()
    error = (case.run_simt().cpu().double() - want).abs().max().item()
    case.vc = torch.ldexp(case.vc, torch.tensor(exponent))
    got = case.run_simt().cpu().double()
    assert (got - want * 2.0 ** exponent).abs().max().item() <= 2 * error * 2.0 ** exponent + 305 * 2.0 ** -150 * 4


@pytest.mark.parametrize("small,large", [(1.2345678e-38, 2e38), (1.3e-40, 3e38), (1.7e-36, 1e37)])
def test_attention_f32_on_tensor_cores_of_factors_with_bits_under_the_parts_range(small, large):
    """Heads of 128: an element of the queries whose last bits bfloat16 has no room for beside large ones of the keys, and the other way
    round; scores of ordinary size come of it.  Rows and keys without such elements keep their bits."""
    nq, nkv, d = 4, 2, 128
    case = PagedCase(torch.float32, nq, nkv, d, 16, [(0, 150), (290, 4)], seed=21)
    clean = case.run_simt().view(-1, nq, d)
    g = torch.Generator().manual_seed(3)
    q, kept = case.q.view(-1, nq, d), case.q.clone()

    def set_key(request, key, head, column, value):
        case.kc[case.table[request, key // 16], head, key % 16, column] = value
        case.ks[request][key, head, column] = value

    # queries of heads 0 and 1 (key head 0) small in column 5, every third key large there
    q[:, :2, 5] = small * (1 + torch.rand(q.shape[0], 2, generator=g))
    for request, length in ((0, 150), (1, 294)):
        for key in range(0, length, 3):
            set_key(request, key, 0, 5, large * (0.5 + 0.5 * float(torch.rand((), generator=g))) * (-1) ** key)
    got = case.run_simt()
    close(got, case.plain(), torch.float32, "small queries, large keys")
    assert torch.equal(got.view(-1, nq, d)[:, 2:], clean[:, 2:])
    # the other way round: every third key small, the others nothing there
    case.q.copy_(kept)
    q[:, :2, 5] = large * (0.5 + 0.5 * torch.rand(q.shape[0], 2, generator=g))
    for request, length in ((0, 150), (1, 294)):
        for key in range(length):
            set_key(request, key, 0, 5, small * (1 + float(torch.rand((), generator=g))) if key % 3 == 0 else 0.0)
    got = case.run_simt()
    close(got, case.plain(), torch.float32, "large queries, small keys")
    assert torch.equal(got.view(-1, nq, d)[:, 2:], clean[:, 2:])


def test_attention_f32_on_tensor_cores_of_a_small_weight_and_a_large_value():
    """Heads of 128: one key's weight is exp(-86), whose last bits bfloat16 has no room for, and its value brings their product to 1."""
    nq, nkv, d = 4, 2, 128
    case = PagedCase(torch.float32, nq, nkv, d, 16, [(0, 90), (400, 2)], seed=22)
    case.q.zero_()
    case.q.view(-1, nq, d)[:, :, 7] = 10.0
    case.kc[:, :, :, 7] = 0.0
    case.vc[:, :, :, 9] = 0.0
    for request in range(2):
        case.ks[request][:, :, 7] = 0.0
        case.vs[request][:, :, 9] = 0.0
        for key in (3, 70):
            case.kc[case.table[request, key // 16], :, key % 16, 7] = -8.6 * d ** 0.5
            case.ks[request][key, :, 7] = -8.6 * d ** 0.5
            case.vc[case.table[request, key // 16], :, key % 16, 9] = 3e37
            case.vs[request][key, :, 9] = 3e37
    got, want = case.run_simt(), case.plain()
    close(got, want, torch.float32, "small weights")
    got, want = (x.double().cpu().view(-1, nq, d)[:, :, 9] for x in (got, want))
    assert (want[3:] > 1e-3).all() and ((got - want).abs() <= 2e-5 * want.abs()).all()


@pytest.mark.parametrize("whole", [False, True])
@pytest.mark.parametrize("window", [0, 300])
def test_attention_f32_on_tensor_cores_of_values_without_parts(monkeypatch, window, whole):
    """Heads of 128: queries, keys and values that bfloat16 has no parts for (infinite, NaN, beyond its largest number), chunks in
    blocks of their own and in one walk.  What sees such a value has it in that column alone, what does not has the same bits as
    without it; a score of such a key is the score of its elements."""
    if whole:
        monkeypatch.setattr(kernels, "ATTENTION_F32_PARTS_BYTES", 0)
    nq, nkv, d, page = 4, 2, 128, 16
    spans = [(0, 200), (700, 3), (400, 70)]
    case = PagedCase(torch.float32, nq, nkv, d, page, spans, seed=11, window=window)
    clean = case.run_simt().view(-1, nq, d)
    position, seq = case.positions, case.seq

    def sees(request, key):
        return (seq == request) & (position >= key) & ((position < key + window) if window else True)

    # a query that is no number: its own (token, head) alone
    kept = case.q.clone()
    case.q.view(-1, nq, d)[201, 2, 7] = math.nan
    got = case.run_simt().view(-1, nq, d)
    assert got[201, 2].isnan().all()
    got[201, 2] = clean[201, 2]
    assert torch.equal(got, clean)
    case.q = kept
    # values: of request 0 key 150 (head 1), request 1 key 690 (head 0), request 2 keys 410 and 411
    marks = ((0, 150, 1, 9, math.inf), (1, 690, 0, 3, math.nan), (2, 410, 1, 100, -math.inf), (2, 411, 0, 64, 3.4e38))
    kept = case.vc.clone()
    for request, key, head, column, value in marks:
        case.vc[case.table[request, key // page], head, key % page, column] = value
    got = case.run_simt().view(-1, nq, d)
    expected = clean.clone()
    for request, key, head, column, value in marks:
        rows, heads = sees(request, key).nonzero().flatten().tolist(), (2 * head, 2 * head + 1)
        assert rows
        for row in rows:
            for h in heads:
                x = float(got[row, h, column])
                if math.isnan(value):
                    assert math.isnan(x)
                elif math.isinf(value):
                    assert x == value
                else:                                        # a weight times the value: from the row's weights in 64 bits
                    keys = torch.arange(max(0, int(position[row]) + 1 - window) if window else 0, int(position[row]) + 1)
                    score = case.ks[request][keys, head].double() @ case.q.view(-1, nq, d)[row, h].double() * d ** -0.5
                    want = float(torch.softmax(score, 0)[keys.tolist().index(key)]) * value
                    assert abs(x - want) <= 1e-4 * abs(want)
                got[row, h, column] = expected[row, h, column]
    assert torch.equal(got, expected)
    case.vc = kept
    # keys: an element beyond bfloat16's range met by a tiny query, and -inf, whose weight is nothing
    q = case.q.view(-1, nq, d)
    q[:, :, 5] = 1e-38
    for request, key, value in ((0, 60, 3.4e38), (1, 650, -3.4e38), (2, 420, -math.inf)):
        case.kc[case.table[request, key // page], 0, key % page, 5] = value
        case.ks[request][key, 0, 5] = value
    close(case.run_simt(), case.plain(), torch.float32, "attention_f32")
