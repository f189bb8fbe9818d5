"""The original-weights experts in 64 bits, from the stored bytes: dequantized matrices, and the products of quantized
vectors with the bound that FP32 sums of exact products keep, in whatever order they are added."""
import numpy as np

E2M1 = np.array([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0])
E2M1 = np.concatenate([E2M1, -E2M1])


def e4m3(codes):
    codes = np.asarray(codes, dtype=np.int64)
    exponent, fraction = (codes >> 3) & 15, codes & 7
    value = np.where(exponent == 0, np.ldexp(fraction.astype(float), -9), np.ldexp(8.0 + fraction, exponent - 10))
    return np.where(codes & 0x80, -value, value)


def e8m0(codes):
    return np.ldexp(1.0, np.asarray(codes, dtype=np.int64) - 127)


def mx_weights(stored, outputs, inputs):
    """MXFP4 with an E8M0 code per 32 inputs -> [outputs][inputs]"""
    words = stored[:outputs * inputs // 2].view(np.uint32).reshape(outputs // 16, inputs // 64, 8, 4, 4)  # tile load g t step
    codes = np.zeros((outputs // 16, 16, inputs // 64, 64), dtype=np.int64)
    for r in range(4):
        for h in range(2):
            nibble = (words >> np.uint32(4 * r + 16 * h)) & np.uint32(15)
            for t in range(4):
                for step in range(4):
                    codes[:, 8 * (r % 2):8 * (r % 2) + 8, :, 16 * step + 2 * t + 8 * (r // 2) + h] = \
                        nibble[:, :, :, t, step].transpose(0, 2, 1)
    scales = stored[outputs * inputs // 2:].reshape(outputs // 16, inputs // 64, 8, 2, 2)  # tile load g q r
    of_block = scales.transpose(0, 4, 2, 1, 3).reshape(outputs, inputs // 32)
    return E2M1[codes.reshape(outputs, inputs)] * np.repeat(e8m0(of_block), 32, axis=1)


def e4m3_weights(stored, outputs, inputs, block128):
    """E4M3 with an E8M0 code per 32 x 32, or an FP32 scale per 128 x 128 -> [outputs][inputs]"""
    groups = stored[:outputs * inputs].reshape(outputs // 16, inputs // 32, 8, 4, 4, 2, 2)  # tile group g t quarter odd upper
    codes = groups.transpose(0, 6, 2, 1, 4, 3, 5).reshape(outputs, inputs)  # tile upper g | group quarter t odd
    rest = stored[outputs * inputs:]
    if block128:
        scales, size = rest.view(np.float32).reshape(outputs // 128, inputs // 128).astype(float), 128
    else:
        scales, size = e8m0(rest.reshape(outputs // 32, inputs // 32)), 32
    return e4m3(codes) * np.repeat(np.repeat(scales, size, axis=0), size, axis=1)


def from_lane_order(codes):
    """Codes of whole vectors [..., width] in the order activation_quantize_entry stores -> natural order"""
    lines = codes.reshape(codes.shape[:-1] + (codes.shape[-1] // 64, 4, 4, 2, 2))  # load t s h r
    return np.moveaxis(lines, (-4, -3, -2, -1), (-2, -4, -1, -3)).reshape(codes.shape)  # load s r t h


def from_stream_order(codes):
    lines = codes.reshape(codes.shape[:-1] + (codes.shape[-1] // 64, 2, 4, 2, 2, 2))  # load q t h r p
    return np.moveaxis(lines, (-5, -1, -2, -4, -3), (-5, -4, -3, -2, -1)).reshape(codes.shape)  # load q p r t h


def vectors(codes, exponents):
    """natural-order codes and exponents -> values"""
    return e4m3(codes) * np.repeat(e8m0(exponents), 32, axis=-1)


def product(weights, values):
    """Products [vectors][outputs] and how far FP32 sums of the (exact) products of codes may lie from them: every addition,
    at most one for 32 inputs and 32 in a group, and a block's scaling, is off by a step of 2^-23 of the terms' size (the
    tensor cores align and cut, they do not round to nearest)."""
    inputs = weights.shape[1]
    return values @ weights.T, (inputs // 32 + 36) * 2.0 ** -23 * (np.abs(values) @ np.abs(weights).T)


def bfloat16_step(values):
    """The distance of bfloat16 neighbours at these values."""
    _, exponent = np.frexp(np.where(values == 0, 1e-30, values))
    return np.ldexp(1.0, exponent - 8)


def check_outputs(got, weights, values):
    """bfloat16 outputs of exactly these quantized vectors: a rounding to nearest of a sum within the bound"""
    exact, bound = product(weights, values)
    assert (np.abs(got - exact) <= 0.5 * bfloat16_step(np.abs(exact) + bound) + bound).all(), \
        float((np.abs(got - exact) / bfloat16_step(exact)).max())


def bfloat16(values):
    bits = np.ascontiguousarray(values, dtype=np.float32).view(np.uint32).astype(np.uint64)
    return (((bits + 0x7FFF + ((bits >> 16) & 1)) >> 16 << 16) & 0xFFFFFFFF).astype(np.uint32).view(np.float32)


def check_hidden(codes, exponents, gate, up, values, route_weights, limit):
    """Natural-order E4M3 codes and exponents of the hidden vectors. A hidden value whose gate and up sums both lie further
    than the bound from a rounding boundary of bfloat16 has one right answer, up to the last bits of expf and of the
    division (they may move its own bfloat16 rounding by a step); in the others gate or up may be either neighbour."""
    rounded, sure = [], np.ones((values.shape[0], gate.shape[0]), dtype=bool)
    for weights in (gate, up):
        exact, bound = product(weights, values)
        low, high = bfloat16(exact - bound), bfloat16(exact + bound)
        sure &= low == high
        rounded.append(bfloat16(exact))
    g, u = rounded
    bounded_gate = np.minimum(g, np.float32(limit))
    with np.errstate(over="ignore"):  # a gate far below zero: its sigmoid is zero
        gated = (bounded_gate / (np.float32(1.0) + np.exp(-bounded_gate))).astype(np.float32)
    hidden = (gated * np.clip(u, -np.float32(limit), np.float32(limit))).astype(np.float32)
    hidden = bfloat16((hidden * route_weights[:, None].astype(np.float32)).astype(np.float32))
    largest = np.maximum(np.abs(hidden.reshape(hidden.shape[0], -1, 32)).max(axis=2), np.float32(1e-4))
    ratio = (largest * np.float32(1.0 / 448.0)).astype(np.float32).view(np.uint32)
    want = (ratio >> 23) + ((ratio & 0x7FFFFF) != 0)
    # a block's largest value decides its exponent: a neighbour of it may cross a power of two
    assert np.abs(exponents.astype(int) - want.astype(int)).max() <= 1 and np.mean(exponents != want) <= 0.01
    scaled = np.clip(hidden.astype(float) / np.repeat(e8m0(exponents), 32, axis=1), -448.0, 448.0)
    half_step = 0.5 * np.ldexp(1.0, np.frexp(np.maximum(np.abs(scaled), 2.0 ** -6))[1] - 4)
    distance = np.abs(e4m3(codes) - scaled)
    assert sure.mean() > 0.5, sure.mean()
    assert (distance <= half_step + np.abs(scaled) * 2.0 ** -7)[sure].all(), float((distance / half_step)[sure].max())
    assert np.mean((distance > half_step)[sure]) <= 1e-3 and np.mean(distance > half_step) <= 1e-2, \
        (np.mean((distance > half_step)[sure]), np.mean(distance > half_step))
