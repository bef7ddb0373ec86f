"""Rows of the plain and fused mat-vecs through the ring of copies and from registers: rows that end inside a
step of 32 chunks, at one and just behind it, from one step to more than the ring holds, an odd row at the end."""
import pytest

pytestmark = pytest.mark.gpu

STEP = {16: 256, 8: 512, 4: 1024}  # inputs of a step


def _layer(bits, rows, n, dev):
    """Integer weights and inputs whose products and sums are exact: weights for the kernels, their values less the
    zero point, inputs."""
    import torch
    g = torch.Generator(device=dev).manual_seed(rows * 3 + n)
    x = torch.randint(-3, 4, (n,), generator=g, device=dev).half()
    if bits == 4:
        b = torch.randint(0, 256, (rows, n // 2), generator=g, device=dev).to(torch.uint8)
        return b, torch.stack([b & 15, b >> 4], dim=2).reshape(rows, n).double() - 7.0, x
    if bits == 8:
        w = torch.randint(-128, 128, (rows, n), generator=g, device=dev)
        return w.to(torch.int8), w.double() + 2.0, x
    w = torch.randint(-9, 10, (rows, n), generator=g, device=dev)
    return w.half(), w.double(), x


def _calls(hq, bits, mat, x, rows):
    zero = {16: 0.0, 8: -2.0, 4: 7.0}[bits]
    fmt = {16: "f16", 8: "int8", 4: "int4"}[bits]
    kw = {} if bits == 16 else dict(scale=1.0, zero_point=zero)
    plain = {16: lambda: hq.gemv_fp16(mat, x), 8: lambda: hq.gemv_int8_quantized(mat, x, 1.0, zero),
             4: lambda: hq.gemv_int4_quantized(mat, x, 1.0, zero)}[bits]
    return plain, lambda: hq.gemv_fused(fmt, x, mat, rows, **kw)


@pytest.mark.parametrize("bits", [16, 8, 4])
@pytest.mark.parametrize("rows,steps,more,ring", [
    (37, 1, 0, 0), (37, 1, -1, 0), (299, 4, 0, 0),             # registers: one to four steps
    (299, 4, 1, None), (37, 9, 0, 1), (301, 12, 1, 1),         # the ring: longer rows (4 bits: from nine steps on)
    (19001, 1, 0, 1), (19001, 1, -1, 1), (19001, 2, 1, 1),     # and two rounds of pairs, across the ends of rows
    (35, 56, 0, 1)])
def test_rows_by_ring_and_registers(hq, dev, bits, rows, steps, more, ring):
    """fp16 of exact sums.  more: chunks of 16 bytes beyond the steps."""
    import torch
    from launches import launched
    n = STEP[bits] * steps + more * (128 // bits)
    mat, w, x = _layer(bits, rows, n, dev)
    want = (w @ x.double()).half()
    for call in _calls(hq, bits, mat, x, rows):
        assert torch.equal(call(), want)
        ((name, _),) = launched(call)
        form = ring if ring is not None else (bits != 4)
        assert ("Lb1EE" if form else "Lb0EE") in name


# the longest inputs beside which two rings fit an SM and the shortest beside which one does; rows just beyond a pair per
# warp, and the fewest of 8 and 16 bits that one CTA per SM takes by ring
@pytest.mark.parametrize("bits,n,per_warp,one", [(4, 24576, 1.0, None), (4, 24608, 1.0, True), (4, 57344, 2.0, True),
                                                 (8, 24592, 1.0, False), (8, 24592, 1.4, True), (16, 25096, 1.0, False),
                                                 (16, 25096, 1.5, True)])
def test_one_ring_per_sm(hq, dev, bits, n, per_warp, one):
    """Where the ring leaves an SM room for one CTA, as many are launched as there are SMs, or two of the register form."""
    import torch
    from launches import launched
    sms = torch.cuda.get_device_properties(dev).multi_processor_count
    rows = 2 * int(per_warp * 16 * sms + 1)
    mat, w, x = _layer(bits, rows, n, dev)
    want = w @ x.double()
    finite = want.abs() < 65504
    for call in _calls(hq, bits, mat, x, rows):
        assert torch.equal(call().double()[finite], want.half().double()[finite])
        ((name, blocks),) = launched(call)
        assert ("Lb1EE" in name) == (one is not False) and blocks == (sms if one else 2 * sms)


@pytest.mark.parametrize("n", [1280, 1800, 2048, 2056, 4096])
def test_fp16_rows_from_registers(hq, dev, n):
    """Layers whose last round of pairs is nearly full: each piece's next loads follow its product, to a row's end inside,
    at and behind a turn of four steps."""
    import torch
    from launches import launched
    sms = torch.cuda.get_device_properties(dev).multi_processor_count
    rows = 2 * int(31 * sms) + 1
    mat, w, x = _layer(16, rows, n, dev)
    call = _calls(hq, 16, mat, x, rows)[1]
    assert torch.equal(call(), (w @ x.double()).half())
    ((name, _),) = launched(call)
    assert "Lb0EE" in name


@pytest.mark.parametrize("bits,n", [(16, 60032), (8, 90112), (4, 115712)])
def test_rows_too_long_for_the_ring(hq, dev, bits, n):
    """Inputs that leave the ring no room come from registers, up to the longest vector that the calls take."""
    import torch
    mat, w, x = _layer(bits, 5, n, dev)
    for call in _calls(hq, bits, mat, x, 5):
        got, want = call().double(), w @ x.double()
        finite = want.abs() < 65504
        assert torch.equal(got[finite], want.half().double()[finite])


@pytest.mark.parametrize("bits", [16, 8, 4])
@pytest.mark.parametrize("steps", [2, 12])
def test_an_infinite_input_stays_in_its_products(hq, dev, bits, steps):
    """The products of other lanes' weights and inputs that an instruction forms beside the wanted ones are
    not read: an infinity meets the weights of its own column alone."""
    import torch
    n = STEP[bits] * steps - 3 * (128 // bits)
    mat, w, x = _layer(bits, 21, n, dev)
    x[n - 5] = float("inf")
    zero = {16: 0.0, 8: -2.0, 4: 7.0}[bits]
    if bits == 16:
        got, column = hq.gemv_fp16(mat, x), w[:, n - 5]
        assert bool((got[column > 0] == float("inf")).all() and (got[column < 0] == float("-inf")).all())
        assert bool(got[column == 0].isnan().all())
    else:  # the sum of the inputs is infinite too
        call = hq.gemv_int8_quantized if bits == 8 else hq.gemv_int4_quantized
        got, column = call(mat, x, 1.0, -1.0), w[:, n - 5] + zero
        assert bool((got[column > 0] == float("inf")).all() and got[column <= 0].isnan().all())
