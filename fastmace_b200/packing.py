"""Packs a MACE model for the device: folds every normalisation constant into the weights, restricts the
species-dependent tensors to the species that are present, lays the per-irrep linears out as plain [K][N] matrices and
turns the symmetric contraction into per-(species, channel) polynomial coefficients.

These are the exact algebraic rewrites the reference applies once at set-up ("species tables", 1/sqrt(fan_in) folded
into W, species skip restricted to present species: ``fastmace/config.py:208-219``,
``fastmace/rewrites/generic/modules.py:584-593,726-737``); nothing here runs per step.
"""

from __future__ import annotations

import ctypes
import functools
import math

import numpy as np
import torch

from . import so3
from ._lib import IMAGE_FIRST_PADDED, IMAGE_ONCHIP, IMAGES, MAX_SPECIES, LayerStruct, ModelStruct
from .codegen import message_slots
from .model import SILU_NORM, MaceSpec, e0_table


def _f64(t: torch.Tensor) -> torch.Tensor:
    return t.detach().to(torch.float64).cpu()


def tf32_round(x: torch.Tensor) -> torch.Tensor:
    """fp32 -> nearest tf32 (10-bit mantissa, ties away from zero, like cvt.rna.tf32.f32), returned as fp32."""
    bits = x.contiguous().view(torch.int32)
    return ((bits + 0x1000) & ~0x1fff).view(torch.float32)


def tensor_core_twin(blocks) -> torch.Tensor:
    """For a list of fp32 [K][N] weight blocks: the concatenation of, per block, the transposed block [N][K] rounded
    to tf32 followed by the tf32-rounded remainder -- the operands of the 3xTF32 tensor-core GEMM. The twin of a
    block that starts at float offset o of the concatenated weights starts at 2 o."""
    out = []
    for block in blocks:
        bt = block.to(torch.float32).t().contiguous()
        hi = tf32_round(bt)
        lo = tf32_round(bt - hi)
        out += [hi.reshape(-1), lo.reshape(-1)]
    return torch.cat(out)


def _swizzled_tile_index() -> torch.Tensor:
    """Float index inside a [128 rows][32 K] operand tile (K-major, 128-byte rows in 1024-byte groups of 8 rows, the
    16-byte chunk index XORed with row mod 8) of element (row, k), flattened row-major."""
    row = torch.arange(128).view(128, 1)
    kk = torch.arange(32).view(1, 32)
    return ((row >> 3) * 256 + (row & 7) * 32 + ((((kk >> 2) & 7) ^ (row & 7)) << 2) + (kk & 3)).reshape(-1)


def tensor_core_image(blocks) -> torch.Tensor:
    """For a list of fp32 [K][N] weight blocks: per block (at twice its float offset, like ``tensor_core_twin``) the
    pieces the warp-specialised GEMM copies into shared memory -- for column tile nt and K chunk kc the [128][32] tile
    of the transposed block as 4,096 tf32 values followed by their 4,096 remainders, both in the swizzled operand
    layout. Blocks with N % 128 != 0 or K % 32 != 0 stay zero."""
    index = _swizzled_tile_index()
    source_of = torch.empty_like(index)
    source_of[index] = torch.arange(len(index))          # where each float of a tile comes from
    out = []
    for block in blocks:
        k, n = block.shape
        image = torch.zeros(2 * k * n, dtype=torch.float32)
        if n % 128 == 0 and k % 32 == 0:
            bt = block.to(torch.float32).t().contiguous()
            hi = tf32_round(bt)
            lo = tf32_round(bt - hi)
            view = image.view(n // 128, k // 32, 2, 4096)
            for part, source in enumerate((hi, lo)):
                tiles = source.view(n // 128, 128, k // 32, 32).transpose(1, 2).reshape(n // 128, k // 32, 4096)
                view[:, :, part] = tiles[:, :, source_of]
        out.append(image)
    return torch.cat(out)


def radial_image(w4: torch.Tensor, channels: int = 128) -> torch.Tensor:
    """The last radial layer [64][paths * channels] (fp32, already scaled) as the radial-weight producer streams it:
    per path p, K half h and part (0 = tf32 remainder, 1 = tf32 value) one 16 KB tile [128 channels][32 features] of the
    transposed block in the K-major operand layout with 128-byte swizzle (8-row groups of 1024 bytes, the 16-byte
    chunk index XORed with row mod 8), at float offset ((p * 2 + h) * 2 + part) * 4096."""
    k, n = w4.shape
    assert k == 64 and channels == 128 and n % channels == 0
    bt = w4.to(torch.float32).t().contiguous()                      # [paths * 128][64]
    hi = tf32_round(bt)
    lo = tf32_round(bt - hi)
    row = torch.arange(128).view(128, 1)
    kk = torch.arange(32).view(1, 32)
    offset = (row >> 3) * 256 + (row & 7) * 32 + ((((kk >> 2) & 7) ^ (row & 7)) << 2) + (kk & 3)   # float index in a tile
    offset = offset.reshape(-1)
    n_paths = n // channels
    image = torch.zeros(n_paths, 2, 2, 4096, dtype=torch.float32)
    for p in range(n_paths):
        for h in range(2):
            for part, source in enumerate((lo, hi)):
                image[p, h, part, offset] = source[p * 128:(p + 1) * 128, h * 32:(h + 1) * 32].reshape(-1)
    return image.reshape(-1)


def mlp_image(w0: torch.Tensor, w1: torch.Tensor, w2: torch.Tensor) -> torch.Tensor:
    """The three hidden layers of a radial MLP ([8][64], [64][64], [64][64], fp32, already scaled) as the operand images
    the tcgen05 edge kernel bulk-copies: a layer [K][64] becomes the tile [64 outputs][K] of its transpose, K-major with
    the 128-byte swizzle in halves of 32 K (2,048 floats each; the first layer fills 8 of the 32 columns of one half),
    tf32 values first, then the tf32 remainders. Float offsets: first layer 0 / 2,048, second 4,096 / 8,192, third
    12,288 / 16,384."""
    assert tuple(w0.shape) == (8, 64) and tuple(w1.shape) == (64, 64) and tuple(w2.shape) == (64, 64)
    row = torch.arange(64).view(64, 1)
    kk = torch.arange(32).view(1, 32)
    index = ((row >> 3) * 256 + (row & 7) * 32 + ((((kk >> 2) & 7) ^ (row & 7)) << 2) + (kk & 3)).reshape(-1)
    image = torch.zeros(20480, dtype=torch.float32)

    def parts(w):
        bt = w.to(torch.float32).t().contiguous()                  # [64 outputs][K]
        hi = tf32_round(bt)
        return hi, tf32_round(bt - hi)

    hi, lo = parts(w0)
    for base, source in ((0, hi), (2048, lo)):
        tile = torch.zeros(64, 32, dtype=torch.float32)
        tile[:, :8] = source
        image[base + index] = tile.reshape(-1)
    for layer, w in enumerate((w1, w2)):
        hi, lo = parts(w)
        for part, source in enumerate((hi, lo)):
            for half in range(2):
                base = 4096 + layer * 8192 + part * 4096 + half * 2048
                image[base + index] = source[:, half * 32:half * 32 + 32].reshape(-1)
    return image


ONCHIP_HEADER = 8                      # floats before the image
ONCHIP_NEAREST = 2.0 ** -9             # distance from the cutoff below which the kernels' scales no longer grow


def onchip_image(w4: torch.Tensor, largest: float, largest_tangent: float, long=(math.inf, math.inf, 0.0, 0.0)) -> torch.Tensor:
    """The last radial layer [64][paths * 128] (fp32, already scaled) as the kernels that evaluate the tensor product
    beside it keep it in tensor memory, fp32 words: a header (scale of the hidden features, scale of their d/dr, inverse of
    the product's scale; powers of two that put the ``largest`` magnitudes half way up the fp16 range; then ``onchip_long``'s
    four numbers, one unused), then per half of the
    channels and pair of paths the values and the remainders of 128 rows (path, channel of the half) of 64 weights as fp16
    pairs, [8][128 rows][4 words] each."""
    k, n = w4.shape
    paths = n // 128
    w = w4.to(torch.float64).t().reshape(paths, 2, 64, k)                       # [path][half][channel][64]
    scale = [onchip_scale(v) for v in (largest, largest_tangent, w.abs().max())]
    rows = (w * scale[2]).transpose(0, 1).reshape(2, paths // 2, 128, k)
    value = rows.to(torch.float16)
    rest = (rows - value.to(torch.float64)).to(torch.float16)
    image = torch.stack([value, rest], dim=2)                                   # [half][pair][part][128][64]
    image = image.reshape(2, paths // 2, 2, 128, 8, 8).transpose(3, 4).contiguous()
    header = torch.tensor([scale[0], scale[1], 1.0 / (scale[0] * scale[2]), *long, 0.0], dtype=torch.float64)
    return torch.cat([header.to(torch.float32), image.reshape(-1).view(torch.float32)])


def onchip_scale(largest: float) -> float:
    return 2.0 ** min(math.floor(math.log2(32768.0 / max(float(largest), 1e-30))), 40)


def table_rows(table: torch.Tensor, per: int):
    """Hidden features and their d/dr from a table, in nine places of every interval: lengths [intervals, 9] and
    [intervals, 9, 64] each, float64."""
    u = torch.linspace(-1, 1, 9, dtype=torch.float64)
    powers = torch.stack([u ** k for k in range(table.shape[1])])
    slopes = torch.stack([2.0 * per * k * u ** max(k - 1, 0) for k in range(table.shape[1])])
    r = (torch.arange(len(table), dtype=torch.float64)[:, None] + 0.5 + 0.5 * u) / per
    return r, *(torch.einsum("nkf,ku->nuf", table.double(), p) for p in (powers, slopes))


def onchip_long(r: torch.Tensor, value: torch.Tensor, slope: torch.Tensor, scale: float, tangent_scale: float, r_cut: float):
    """How the kernels scale the features of long edges (``table_rows``): (length from which on they look at them, cutoff, factor a, factor b).
    Near the cutoff the largest value is at most 4 a (cutoff - r)^4 and the largest d/dr 4 b (cutoff - r)^3 under the scales;
    beyond the length one of these is below 1/4, and rows of which that holds are scaled by the inverse of the law."""
    tops = value.abs().amax(2) * scale, slope.abs().amax(2) * tangent_scale
    least = torch.minimum(*tops)
    least[0, 0] = least[0, 1]
    small = torch.nonzero(least.amin(1) < 1.0)
    first = float(r[int(small[0]), 0]) if len(small) else r_cut
    d = (r_cut - r).clamp_min(ONCHIP_NEAREST)
    inside = (r >= first) & (r <= r_cut)
    law = [0.25 * float((top * inside / d ** k).max()) for top, k in zip(tops, (4, 3))]
    reach = r_cut - max((0.0625 / max(a, 1e-30)) ** (1 / k) for a, k in zip(law, (4, 3)))
    return max(reach, first), r_cut, *law


def onchip_is_accurate(w4: torch.Tensor, image: torch.Tensor, r: torch.Tensor, features: torch.Tensor, tangents: torch.Tensor) -> bool:
    """Does the image (``onchip_image``) of the layer give products with the hidden ``features`` and their d/dr [n, 64] at the
    lengths ``r`` that are off by no more than those of tf32 pairs can be: 2^-23 of every term for the remainder of each operand
    and 2^-22 for the product of remainders that is left out? fp16 pairs have fewer bits where a weight is below 2^-17 of the
    layer's largest, or a feature below 2^-2 under its row's scale."""
    n_out = w4.shape[1]
    weights = w4.to(torch.float64)
    parts = image[ONCHIP_HEADER:].view(torch.float16).double().reshape(2, n_out // 256, 2, 8, 128, 8) * float(image[0]) * float(image[2])
    parts = parts.permute(2, 1, 4, 0, 3, 5).reshape(2, n_out // 256, 2, 64, 2, 64)     # [part][pair][path][channel][half][k]
    parts = parts.transpose(3, 4).reshape(2, n_out, 64).transpose(1, 2)
    d = (float(image[4]) - r).clamp_min(ONCHIP_NEAREST)
    for scale, rows, law in ((image[0], features, d ** 4 * float(image[5])), (image[1], tangents, d ** 3 * float(image[6]))):
        h = rows.to(torch.float32).to(torch.float64)
        up = torch.where((r < float(image[3])) | (law >= 0.0625), torch.ones_like(r),
                         torch.exp2(-torch.floor(torch.log2(law.clamp_min(2.0 ** -126)))))
        power = float(scale) * up[:, None]
        if not bool((h * power).abs().max() < 65504.0):
            return False
        value = (h * power).to(torch.float16).double()
        rest = (h * power - value).to(torch.float16).double()
        off = ((h - (value + rest) / power).abs() @ weights.abs() + h.abs() @ (weights - parts.sum(0)).abs()
               + (rest / power).abs() @ parts[1].abs())
        if not bool((off <= 2.0 ** -21 * (h.abs() @ weights.abs())).all()):
            return False
    return True


RADIAL_DEGREE = 5


def radial_hidden_float64(w0, w1, w2, r: torch.Tensor, r_cut: float, with_tangent: bool = True):
    """Third hidden layer of a radial MLP (scaled fp32 weights [8][64], [64][64], [64][64]) and its d/dr (or None) at
    lengths ``r``, [n, 64] float64 each. The envelope polynomial is continued beyond the cutoff (the caller cuts there)."""
    x = (r / r_cut)[:, None]
    x2 = x * x
    x5 = x2 * x2 * x
    envelope = 1 + x5 * (-21 + 35 * x - 15 * x2)
    k = torch.arange(1, 9, dtype=torch.float64) * (math.pi / r_cut)
    a = r[:, None] * k
    bessel = k * torch.sinc(a / math.pi)                  # sin(k r) / r
    value, tangent = math.sqrt(2 / r_cut) * bessel * envelope, None
    if with_tangent:
        d_envelope = x2 * x2 * (-105 + 210 * x - 105 * x2) / r_cut
        # smooth at r = 0, where the quotient loses its digits to cancellation
        d_bessel = torch.where(a < 0.02, k * k * a * (-1 / 3 + a * a / 30), (k * torch.cos(a) - bessel) / r[:, None])
        tangent = math.sqrt(2 / r_cut) * (d_bessel * envelope + bessel * d_envelope)
    for w in (w0, w1, w2):
        w = w.to(torch.float64)
        z = value @ w
        s = torch.sigmoid(z)
        if with_tangent:
            tangent = SILU_NORM * s * (1 + z * (1 - s)) * (tangent @ w)
        value = SILU_NORM * z * s
    return value, tangent


def _table_is_accurate(table, per: int, function, r_cut: float) -> bool:
    """Is a table off by at most 2e-7 (value) and 4e-7 (d/dr) of the largest magnitude its function takes within the same
    quarter of an Å (counted from the cutoff)? Checked between the nodes and at both ends of every interval, where d/dr is
    worst. The features of a pair that nearly touches are a hundred times those of a bond and ten thousand times those
    near the cutoff: one bound for all lengths would let errors of 1e-5 and more pass where a crystal has its neighbours."""
    n = len(table)
    ends, inner = torch.arange(n + 1, dtype=torch.float64) / per, (torch.arange(n, dtype=torch.float64) + 0.75) / per
    r = torch.cat([ends, inner])
    inside = r < r_cut                                              # nothing is looked up at the cutoff or beyond
    windows = max(int(r_cut / 0.25), 1)                             # the one at zero holds the remainder
    window = ((r_cut - r) / 0.25).long().clamp(0, windows - 1)
    value, tangent = function(r)
    largest = [torch.zeros(windows, dtype=torch.float64).scatter_reduce(0, window, f.abs().amax(1) * inside, "amax")
               for f in (value, tangent)]
    n_c, probes = table.shape[1], ((-1.0, slice(0, n)), (1.0, slice(1, n + 1)), (0.5, slice(n + 1, 2 * n + 1)))
    powers = [[u ** k for k in range(n_c)] for u, _ in probes]
    slopes = [[2.0 * per * k * u ** max(k - 1, 0) for k in range(n_c)] for u, _ in probes]
    got = torch.tensor(powers + slopes, dtype=torch.float64) @ table.double()                       # [n, 6, features]
    for q, (_, at) in enumerate(probes):
        for row, exact, bound, top in ((q, value, 2e-7, largest[0]), (q + 3, tangent, 4e-7, largest[1])):
            error = (got[:, row] - exact[at]).abs().amax(1) * inside[at]
            if not bool((error <= bound * top[window[at]]).all()):
                return False
    return True


def radial_table(w0, w1, w2, r_cut: float):
    """The hidden radial features as piecewise polynomials of the length: (coefficients [intervals, 6, 64] fp32,
    intervals per Å), or None where 512 intervals per Å are not enough.

    The features of an edge depend on its length only, through a smooth function fixed by the weights. Polynomials of
    degree 5 through the Chebyshev nodes of intervals of 1/32 Å reproduce it below fp32 rounding for the benchmark's
    models (5e-8 of the local magnitude in value and d/dr from 1 Å on, 3e-7 in d/dr below, rounding of the coefficients
    included; the 3xTF32 chain of three layers they replace is off by 3e-7 to 1e-6). The interval is halved until the
    table is accurate at every length, so a model with a steeper radial function gets a finer table and one that no table
    serves keeps the MLP kernel."""
    n_c = RADIAL_DEGREE + 1
    w0, w1, w2 = (w.cpu() for w in (w0, w1, w2))
    nodes = torch.cos(math.pi * (torch.arange(n_c, dtype=torch.float64) + 0.5) / n_c)
    fit = torch.linalg.inv(torch.stack([nodes ** k for k in range(n_c)], dim=1))
    for per in (32, 64, 128, 256, 512):
        n = int(math.ceil(r_cut * per))
        middle = (torch.arange(n, dtype=torch.float64)[:, None] + 0.5) / per
        at_nodes = radial_hidden_float64(w0, w1, w2, (middle + nodes / (2 * per)).reshape(-1), r_cut, False)[0]
        table = (fit @ at_nodes.reshape(n, n_c, -1)).to(torch.float32)
        if _table_is_accurate(table, per, lambda r: radial_hidden_float64(w0, w1, w2, r, r_cut), r_cut):
            return table.contiguous(), per
    return None


@functools.lru_cache(maxsize=None)
def _contraction_layout(l_out_max: int, correlation: int, sh_lmax: int):
    """(terms int32 [T, 4], per (l_out, degree) block the polynomial terms ordered by their row of the coefficient table,
    the first of every row and that row)."""
    keys = so3.contraction_keys(l_out_max, correlation, sh_lmax)
    terms = np.full((len(keys), 4), -1, dtype=np.int32)
    for t, (m_out, _, mono) in enumerate(keys):
        terms[t, :len(mono)] = mono
        terms[t, 3] = m_out
    row_of = {key: t for t, key in enumerate(keys)}
    rows = {}
    for big_l in range(l_out_max + 1):
        for nu in range(1, correlation + 1):
            mono, m_out, _, _, _ = so3.contraction_polynomial(nu, big_l, sh_lmax)
            row = np.array([row_of[big_l * big_l + int(m), nu, tuple(int(i) for i in q)] for m, q in zip(m_out, mono)])
            order = np.argsort(row, kind="stable")
            row = row[order]
            first = np.flatnonzero(np.concatenate([[True], row[1:] != row[:-1]]))
            rows[big_l, nu] = order, first, row[first]
    return terms, rows


def contraction_terms(spec: MaceSpec, weights, layer: int, species_z):
    """(terms int32 [T, 4], coef float64 [n_species, T, C]) of one layer's symmetric contraction, sorted by output."""
    terms, rows = _contraction_layout(spec.l_out_max(layer), spec.correlation, spec.sh_lmax)
    coefs = np.zeros((len(terms), len(species_z), spec.channels), dtype=np.float64)
    for (big_l, nu), (order, first, row) in rows.items():
        _, _, weight, coef, _ = so3.contraction_polynomial(nu, big_l, spec.sh_lmax)
        w = _f64(weights[f"l{layer}.sc.{big_l}.{nu}"]).numpy()[[z - 1 for z in species_z]]  # [nz, k, C]
        coefs[row] += np.add.reduceat(coef[order, None, None] * w.transpose(1, 0, 2)[weight[order]], first, axis=0)
    return terms.copy(), coefs.transpose(1, 0, 2)


class PackedModel:
    """Device tensors of a model restricted to ``species_z`` (sorted atomic numbers present) and the ``ModelStruct``
    the C ABI reads. Keeps the tensors alive for as long as the struct is used."""

    def __init__(self, spec: MaceSpec, weights, species_z, device):
        species_z = [int(z) for z in species_z]
        if species_z != sorted(set(species_z)):
            raise ValueError("species_z must be sorted and unique")
        if len(species_z) > MAX_SPECIES:
            raise ValueError(f"at most {MAX_SPECIES} species per structure, got {len(species_z)}")
        if spec.num_interactions != 2 or spec.channels != 128 or spec.correlation != 3:
            raise ValueError("the device path takes 2 interactions, 128 channels, correlation 3")
        self.spec = spec
        self.species_z = species_z
        self.device = torch.device(device)
        self.tensors: dict[str, torch.Tensor] = {}
        c, n_el = spec.channels, spec.num_elements
        idx = [z - 1 for z in species_z]
        w = {k: _f64(v) for k, v in weights.items()}
        struct = ModelStruct()
        struct.n_species = len(species_z)
        struct.channels = c
        struct.hidden_lmax = spec.hidden_lmax
        struct.n_layers = spec.num_interactions
        struct.n_bessel = spec.num_bessel
        struct.cutoff_p = spec.cutoff_p
        struct.radial_width = spec.radial_hidden[-1]
        struct.mlp_hidden = spec.mlp_hidden
        struct.r_cut = spec.r_cut
        struct.scale = spec.scale
        struct.shift = spec.shift
        struct.silu_norm = SILU_NORM
        e0 = e0_table(spec)
        for k, z in enumerate(species_z):
            struct.e0[k] = float(e0[z - 1])
        h0 = w["emb"][idx] / math.sqrt(n_el)                                   # [nz, C]
        for t in range(spec.num_interactions):
            layer = struct.layer[t]
            paths = spec.paths(t)
            slots, blocks = message_slots(paths)
            layer.l_in_max = spec.l_in_max(t)
            layer.l_out_max = spec.l_out_max(t)
            layer.n_paths = len(paths)
            layer.mid_dim = so3.mid_dim(paths)
            layer.skip_lmax = spec.skip_lmax(t)
            layer.is_last = int(t == spec.num_interactions - 1)
            widths = (spec.num_bessel, *spec.radial_hidden, len(paths) * c)
            for i in range(4):
                layer.rad_w[i] = self._put(f"l{t}.rad.{i}", w[f"l{t}.rad.{i}"] / math.sqrt(widths[i]))
            layer.tc[0] = self._twin(f"l{t}.rad.3", [self.tensors[f"l{t}.rad.3"]])
            if t > 0 and c == 128:
                layer.rad_img = self._put(f"l{t}.rad.img", radial_image(self.tensors[f"l{t}.rad.3"].cpu(), c))
            if spec.num_bessel == 8 and tuple(spec.radial_hidden) == (64, 64, 64):
                layer.mlp_img = self._put(f"l{t}.rad.mlp_img",
                                          mlp_image(*(self.tensors[f"l{t}.rad.{i}"].cpu() for i in range(3))))
                if spec.cutoff_p == 5:
                    found = radial_table(*(self.tensors[f"l{t}.rad.{i}"] for i in range(3)), spec.r_cut)
                    if found is not None:
                        layer.rad_tab = self._put(f"l{t}.rad.table", found[0])
                        layer.rad_tab_intervals, layer.rad_tab_per_angstrom = int(found[0].shape[0]), float(found[1])
                        if t > 0 and c == 128 and spec.l_in_max(t) == 1:
                            # behind the producer's image the one of the kernels that keep the layer on the SM
                            table, power = found[0].double(), torch.arange(1, RADIAL_DEGREE + 1, dtype=torch.float64)
                            largest = table.abs().sum(1).max()
                            largest_tangent = (table[:, 1:].abs() * power[None, :, None]).sum(1).max() * 2.0 * found[1]
                            w4 = self.tensors[f"l{t}.rad.3"].cpu()
                            if bool(torch.isfinite(w4).all()) and largest > 0 and largest_tangent > 0:
                                rows = table_rows(*found)
                                long = onchip_long(*rows, onchip_scale(largest), onchip_scale(largest_tangent), spec.r_cut)
                                image = onchip_image(w4, largest, largest_tangent, long)
                                # accurate in the middle of every 16th interval and, where the scales begin to grow, of all?
                                some = (torch.arange(len(rows[0])) % 16 == 0) | (rows[0][:, 0] >= long[0] - 0.1)
                                some &= rows[0][:, 4] < spec.r_cut - ONCHIP_NEAREST
                                if onchip_is_accurate(w4, image, *(q[some, 4] for q in rows)):
                                    layer.rad_img = self._put(f"l{t}.rad.img", torch.cat([radial_image(w4, c), image]))
                                    layer.extra_images |= IMAGES | IMAGE_ONCHIP
            if t == 0:
                x_species = h0 @ (w["l0.up.0"] / math.sqrt(c))
                sc = torch.zeros(len(idx), spec.out_dim(0), c, dtype=torch.float64)
                skip = w["l0.skip.0"]                                           # [C, 89, C]
                for k, e in enumerate(idx):
                    sc[k, 0] = h0[k] @ skip[:, e, :] / math.sqrt(c * n_el)
                layer.x_species = self._put("l0.x_species", x_species)
                layer.sc_species = self._put("l0.sc_species", sc)
                # reassociated first layer: message[i, (l, m), :] = sum_z S[i, (l, m), z, :] @ first_l[z], with
                # S[i, lm, z, k] = sum_{e -> i, species(sender) = z} hidden[e, k] * Y[e, lm]  (exact algebra)
                w4 = (w["l0.rad.3"] / math.sqrt(widths[3])).to(torch.float32).to(torch.float64)
                blocks = []
                for l_out in range(spec.sh_lmax + 1):
                    (p0,) = so3.paths_into(paths, l_out)
                    lin_l = w[f"l0.lin.{p0}"] / math.sqrt(c) / spec.avg_num_neighbors
                    per_z = [(w4[:, p0 * c:(p0 + 1) * c] * x_species[z][None, :]) @ lin_l for z in range(len(idx))]
                    blocks.append(torch.cat(per_z, dim=0).to(torch.float32))           # [nz * 64, C]
                layer.first[0] = self._put("l0.first", torch.cat([b.reshape(-1) for b in blocks]))
                layer.first[1] = self._put("l0.first_t", torch.cat([b.t().contiguous().reshape(-1) for b in blocks]))
                layer.first[2] = self._twin("l0.first", blocks)
                layer.first_img[0] = self._image_of("l0.first")
                layer.first[3] = self._twin("l0.first_t", [b.t().contiguous() for b in blocks])
                if len(idx) % 2:
                    # N = 64 for every species: an odd number of them leaves half a column tile
                    padded = [torch.nn.functional.pad(b.t(), (0, 64)) for b in blocks]
                    layer.first_img[1] = self._put("l0.first_t.img", tensor_core_image(padded))
                    layer.extra_images |= IMAGES | IMAGE_FIRST_PADDED
                else:
                    layer.first_img[1] = self._image_of("l0.first_t")
            else:
                up = torch.stack([w[f"l{t}.up.{l}"] / math.sqrt(c) for l in range(spec.l_in_max(t) + 1)])
                layer.w_up = self._put(f"l{t}.w_up", up)
                layer.w_up_t = self._put(f"l{t}.w_up_t", up.transpose(1, 2))
                layer.tc[1] = self._twin(f"l{t}.w_up", list(self.tensors[f"l{t}.w_up"]))
                layer.tc_img[1] = self._image_of(f"l{t}.w_up")
                layer.tc[2] = self._twin(f"l{t}.w_up_t", list(self.tensors[f"l{t}.w_up_t"]))
                layer.tc_img[2] = self._image_of(f"l{t}.w_up_t")
                skip = torch.stack([w[f"l{t}.skip.{l}"][:, idx, :].permute(1, 0, 2) / math.sqrt(c * n_el)
                                    for l in range(spec.skip_lmax(t) + 1)])     # [L, nz, C, C]
                layer.w_skip = self._put(f"l{t}.w_skip", skip)
                layer.w_skip_t = self._put(f"l{t}.w_skip_t", skip.transpose(2, 3))
                layer.tc[3] = self._twin(f"l{t}.w_skip", list(self.tensors[f"l{t}.w_skip"].reshape(-1, c, c)))
                layer.tc_img[3] = self._image_of(f"l{t}.w_skip")
                layer.tc[4] = self._twin(f"l{t}.w_skip_t", list(self.tensors[f"l{t}.w_skip_t"].reshape(-1, c, c)))
                layer.tc_img[4] = self._image_of(f"l{t}.w_skip_t")
            lin, lin_t, lin_blocks = [], [], []
            for l_out in range(spec.sh_lmax + 1):
                into = so3.paths_into(paths, l_out)
                norm = 1.0 / math.sqrt(len(into) * c) / spec.avg_num_neighbors
                block = torch.cat([w[f"l{t}.lin.{p}"] for p in into], dim=0) * norm   # [n_seg * C, C]
                lin.append(block.reshape(-1))
                lin_t.append(block.t().contiguous().reshape(-1))
                lin_blocks.append(block.to(torch.float32))
            layer.w_lin = self._put(f"l{t}.w_lin", torch.cat(lin))
            layer.w_lin_t = self._put(f"l{t}.w_lin_t", torch.cat(lin_t))
            layer.tc[5] = self._twin(f"l{t}.w_lin", lin_blocks)
            layer.tc_img[5] = self._image_of(f"l{t}.w_lin")
            layer.tc[6] = self._twin(f"l{t}.w_lin_t", [b.t().contiguous() for b in lin_blocks])
            layer.tc_img[6] = self._image_of(f"l{t}.w_lin_t")
            prod = torch.stack([w[f"l{t}.prod.{big_l}"] / math.sqrt(c) for big_l in range(spec.l_out_max(t) + 1)])
            layer.w_prod = self._put(f"l{t}.w_prod", prod)
            layer.w_prod_t = self._put(f"l{t}.w_prod_t", prod.transpose(1, 2))
            layer.tc[7] = self._twin(f"l{t}.w_prod", list(self.tensors[f"l{t}.w_prod"]))
            layer.tc_img[7] = self._image_of(f"l{t}.w_prod")
            layer.tc[8] = self._twin(f"l{t}.w_prod_t", list(self.tensors[f"l{t}.w_prod_t"]))
            layer.tc_img[8] = self._image_of(f"l{t}.w_prod_t")
            terms, coefs = contraction_terms(spec, weights, t, species_z)
            layer.n_sc_terms = len(terms)
            layer.sc_terms = self._put(f"l{t}.sc_terms", torch.from_numpy(terms), dtype=torch.int32)
            layer.sc_coef = self._put(f"l{t}.sc_coef", torch.from_numpy(coefs))
            if t < spec.num_interactions - 1:
                layer.w_readout = self._put(f"l{t}.readout", w[f"l{t}.readout"] / math.sqrt(c))
            else:
                ro = torch.cat([(w[f"l{t}.readout.0"] / math.sqrt(c)).reshape(-1),
                                w[f"l{t}.readout.1"] / math.sqrt(spec.mlp_hidden)])
                layer.w_readout = self._put(f"l{t}.readout", ro)
        self.struct = struct

    def _put(self, name: str, tensor: torch.Tensor, dtype=torch.float32) -> int:
        t = tensor.to(dtype).contiguous().to(self.device)
        self.tensors[name] = t
        return t.data_ptr()

    def _twin(self, name: str, blocks) -> int:
        """Tensor-core twin of fp32 [K][N] blocks that are already on the device (so the split is of the fp32 values
        the SIMT path reads)."""
        host = [b.cpu() for b in blocks]
        twin = tensor_core_twin(host).to(self.device)
        self.tensors[name + ".tc"] = twin
        self.tensors[name + ".img"] = tensor_core_image(host).to(self.device)
        return twin.data_ptr()

    def _image_of(self, name: str) -> int:
        return self.tensors[name + ".img"].data_ptr()

    def species_index(self, numbers) -> torch.Tensor:
        """[N] int32 index of each atom's species among the present ones."""
        table = np.full(128, -1, dtype=np.int32)
        for k, z in enumerate(self.species_z):
            table[z] = k
        index = table[np.asarray(numbers, dtype=np.int64)]
        if (index < 0).any():
            raise ValueError("an atom's species is not among the species the model was packed for")
        return torch.as_tensor(index, dtype=torch.int32, device=self.device)

    def pointer(self):
        return ctypes.byref(self.struct)


__all__ = ["PackedModel", "contraction_terms", "mlp_image", "radial_image", "tensor_core_image", "tensor_core_twin", "tf32_round"]
