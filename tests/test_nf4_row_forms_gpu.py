"""Fused NF4 calls of long rows: the row form's instances by the number of warps per row, their loads in place, and
sums in half2 or in 32 bits."""
import pytest

pytestmark = pytest.mark.gpu


def _form(name):
    """Kernel's (rows, loads in place, 32-bit sums)"""
    flags = [part[-1] for part in name.split("EEEv")[0].split("ELb")]  # ..., in place, wide, fused, packets
    return "nf4_gemv_kernel" in name and (flags[-4], flags[-3], flags[-2]) if "mma" not in name else None


# more: 32-input chunks beyond whole slices of 2048; form: half sums, 32-bit sums
@pytest.mark.parametrize("rows,n,norm,act,resident,form", [
    # 32-bit sums: 2 to 8 warps per row, rows that fill them, stop in the last one and leave warps without a row
    (6145, 4096, 0, 0, True, None), (6146, 4096, 0, 1, True, "wide"), (14339, 3520, 1, 0, True, "wide"),
    (3586, 5632, 0, 1, True, "wide"), (5803, 6144, 1, 0, True, "wide"), (2050, 6208, 0, 1, True, "wide"),
    (3371, 8192, 1, 0, True, "wide"), (16390, 8192, 1, 2, True, "wide"), (2290, 8256, 1, 1, True, "wide"),
    (2051, 10304, 1, 0, True, "wide"), (1531, 12352, 1, 0, True, "wide"), (2050, 16384, 0, 1, True, "wide"),
    (6146, 8192, 0, 1, False, "wide"), (16386, 6144, 1, 1, False, "wide"), (4097, 12352, 1, 0, False, "wide"),
    # half2, weights resident: few rows
    (1021, 10240, 1, 0, True, "half"), (1023, 14336, 1, 0, True, "half"), (1022, 16384, 1, 1, True, "half"),
    (514, 12288, 0, 1, True, "half"),
    # and without the early fetch
    (10242, 4096, 1, 1, False, "half"), (8195, 8192, 1, 0, False, "half")])
def test_row_form_instances(hq, dev, rows, n, norm, act, resident, form):
    """Elementwise against fp64.  A half2 sum of four products is rounded four times and met three more times by others of its kind,
    7 * 2^-11 of the products' absolute values; in 32 bits n roundings of 2^-24 bound all.  With norm the
    inputs round to fp16, and so does the result."""
    import torch
    from launches import launched
    g = torch.Generator(device=dev).manual_seed(rows + n)
    x = (torch.randn(n, generator=g, device=dev) * 3).half()
    gamma = (torch.rand(n, generator=g, device=dev) + 0.5).half() if norm else None
    mat = torch.randint(0, 256, (rows, n // 2), generator=g, device=dev, dtype=torch.uint8)
    absmax = (torch.rand((rows, n // 64), generator=g, device=dev) + 0.5) / n ** 0.5
    lut = torch.arange(-8, 8, device=dev).float() / 8  # exact in fp16
    rows_out = rows // 2 if act else rows
    y = []
    ((name, _),) = launched(lambda: y.append(hq.gemv_fused(
        "nf4", x, mat, rows_out, gamma=gamma, eps=1e-5, act=act, absmax=absmax.view(-1), lut16=lut, weights_resident=resident)))
    if form:
        assert _form(name) == ("1", "1" if form == "wide" else "0", "1"), name

    xd = x.double()
    if norm:
        xd = xd * torch.rsqrt((xd * xd).mean() + 1e-5) * gamma.double()
    unit = 2.0**-11 * norm + (n * 2.0**-24 if form == "wide" else 7 * 2.0**-11 + n * 2.0**-24)
    sums, errs = [], []
    for part in range(0, rows, 2048):
        m = mat[part:part + 2048].long()
        w = lut[torch.stack([m >> 4, m & 15], 2)].view(len(m), n).double()
        w = w * absmax[part:part + 2048].double().repeat_interleave(64, 1)
        sums.append(w @ xd)
        errs.append(unit * (w.abs() @ xd.abs()))
    v, dv = torch.cat(sums), torch.cat(errs)
    if act:
        gate, dgate, v, dv = v[1::2], dv[1::2], v[0::2], dv[0::2]
        f = gate * torch.sigmoid(gate) if act == 1 else 0.5 * gate * (1 + torch.tanh(0.7978845608028654 * (gate + 0.044715 * gate**3)))
        df = 1.13 * dgate + 2.0**-20  # |f'| is below 1.13; exp and tanh of the kernel
        v, dv = v * f, dv * (f.abs() + df) + v.abs() * df
    err = (y[0].double() - v).abs()
    assert bool((err <= dv + 2.0**-11 * (v.abs() + dv) + 2.0**-24).all()), float((err / (dv + 2.0**-11 * v.abs())).max())


@pytest.mark.parametrize("rows,n,act", [(6146, 4096, 1), (2048, 9216, 0), (28672, 8192, 1)])
def test_wide_rows_hold_sums_beyond_fp16(hq, dev, rows, n, act):
    """Four products of inputs near fp16's largest value exceed it; the layers' sums in 32 bits do not.
    All terms have one sign: every sum is within n * 2^-24 of itself, the result rounds once to fp16."""
    import torch
    g = torch.Generator(device=dev).manual_seed(rows)
    x = (torch.rand(n, generator=g, device=dev) * 3e4 + 3e4).half()
    mat = torch.randint(0, 64, (rows, n // 2), generator=g, device=dev, dtype=torch.uint8) * 2 % 128 | 0x88  # levels 8 to 15
    absmax = torch.full((rows * n // 64,), 1e-4 / n, device=dev)
    lut = torch.arange(-7, 9, device=dev).float() / 8
    rows_out = rows // 2 if act else rows
    y = hq.gemv_fused("nf4", x, mat, rows_out, gamma=None if act else torch.ones(n, device=dev).half(), act=act,
                      absmax=absmax if act else absmax * 1e4, lut16=lut, weights_resident=True)
    xd = x.double() if act else (x.double() * torch.rsqrt((x.double() ** 2).mean() + 1e-5))
    m = mat[:512].long()
    w = lut[torch.stack([m >> 4, m & 15], 2)].view(512, n).double() * (1e-4 if act else 1.0) / n
    v = w @ xd
    if act:
        v = v[0::2] * v[1::2] * torch.sigmoid(v[1::2])
    tol = 2.0**-11 + (2.2 * n * 2.0**-24 + 2.0**-20 if act else n * 2.0**-24 + 2.0**-11)
    assert bool(((y[:len(v)].double() - v).abs() <= tol * v).all())


@pytest.mark.parametrize("rows,n,norm,act,resident,bs", [
    # 32-bit sums
    (14339, 3520, 1, 0, True, 64), (3586, 5632, 0, 1, True, 64), (2050, 6208, 0, 1, True, 64), (2290, 8256, 1, 1, True, 64),
    (4097, 12352, 1, 0, False, 64),
    # half2: fused, plain, loads behind a branch, rows that begin inside an absmax block, four chunks per lane
    (1021, 10304, 1, 0, True, 64), (333, 4160, 0, 0, True, 64), (333, 4160, 0, 0, False, 64), (333, 1376, 0, 0, True, 128),
    (37, 33792, 0, 0, True, 64)])
def test_infinite_level_beside_idle_lanes(hq, dev, rows, n, norm, act, resident, bs):
    """Level 0 is one that no fp16 number holds, and lanes beyond the row's end hold its code: rows without
    it have the value that a finite level 0 gives, bit for bit; one such code makes its row infinite."""
    import torch
    g = torch.Generator(device=dev).manual_seed(rows + n)
    x = torch.randn(n, generator=g, device=dev).half()
    codes = torch.randint(1, 16, (rows, n), generator=g, device=dev)
    codes[::3, 5] = 0
    mat = (codes[:, 0::2] << 4 | codes[:, 1::2]).to(torch.uint8)
    absmax = (torch.rand(-(-rows * n // bs), generator=g, device=dev) + 0.5) / n ** 0.5
    gamma = (torch.rand(n, generator=g, device=dev) + 0.5).half() if norm else None
    got = []
    for level in (-1.0, -1e30):
        lut = torch.linspace(-1, 1, 16, device=dev)
        lut[0] = level
        got.append(hq.gemv_fused("nf4", x, mat, rows // 2, gamma=gamma, act=act, absmax=absmax, lut16=lut, weights_resident=resident)
                   if act else
                   hq.gemv_fused("nf4", x, mat, rows, gamma=gamma, absmax=absmax, lut16=lut, weights_resident=resident)
                   if norm else hq.gemv_nf4(x, mat, absmax, lut, rows, n, bs, weights_resident=resident))
    hit = (codes == 0).any(1)
    if act:
        hit = hit.view(-1, 2).any(1)
    assert torch.equal(got[1][~hit], got[0][~hit]) and bool(got[0].isfinite().all())
    if not act:
        assert bool((got[1][hit] == (float("-inf") if x[5] > 0 else float("inf"))).all())
