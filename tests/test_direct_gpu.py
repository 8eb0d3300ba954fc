"""Direct solver on the GPU against the oracle and the reference's outputs.

Restates the contract of the reference's CUDA direct tests
(tests/solvers/cuda_direct_solver_test.cpp) with this backend swapped in:
FP32 bounds against the compensated reference (worst < 2e-4, RMS < 2e-5),
counters N(N-1), empty/single inputs, the origin-padding known answer. The
FP64 form is held to bit equality with the reference's scalar DirectSolver and
the split precision form to a median per-particle relative error below 1e-7.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import relative_errors

pytestmark = pytest.mark.gpu

# Tolerances (per-particle relative error |a - a_ref| / |a_ref|).
FP32_WORST, FP32_RMS = 2e-4, 2e-5        # cuda_direct_solver_test.cpp:122-151 (FP32 build)
# Split precision: median well below 1e-7; the worst particle is one whose
# net force nearly cancels, where FP32 pair rounding (~1e-7 per term) is
# amplified by sum|t| / |sum t|. Measured worst on this case: 1.25e-6.
SPLIT_WORST, SPLIT_MEDIAN = 2e-6, 1e-7


def _xyzm(d):
    return d["x"], d["y"], d["z"], d["m"]


def test_fp64_is_bit_identical_to_reference(b200, golden_plummer):
    g = golden_plummer
    for eps in (0.01, 0.05):
        s = b200.B200DirectSolver(eps, "fp64")
        a = s.evaluate((g["x"], g["y"], g["z"]), g["m"])
        assert np.array_equal(a, g[f"direct_eps{eps}"])
        assert s.interaction_count().particle_particle == 2048 * 2047


# 31-33: the edges of a chunk of sources; 28,417 and on: one target per thread.
# The scales put squared distances below and above the range of the short
# root and division; without softening the target's own argument is zero. (Below
# that range, |d|^2 < 2^-895, the force's 1 / |d|^3 > 2^1342 overflows, in the
# oracle too: opposite infinities make NaN, and only the potential is finite.)
@pytest.mark.parametrize("n,eps,scale", [(1, 0.01, 1.0), (31, 0.0, 1.0), (32, 0.01, 1.0),
                                         (33, 0.05, 1.0), (257, 0.0, 1e-140),
                                         (257, 0.0, 1e137), (4097, 0.01, 1.0),
                                         (16383, 0.01, 1.0), (16384, 0.01, 1.0),
                                         (16415, 0.0, 1.0), (28416, 0.01, 1.0),
                                         (28417, 0.0, 1.0), (28447, 0.01, 1.0)])
def test_fp64_sums_are_bit_identical_at_every_size(b200, restatement, n, eps, scale):
    from orrery_b200 import initial_conditions as ic
    d = ic.plummer_sphere(n, seed=n)
    x, y, z = (d[k] * scale for k in "xyz")
    exact, _ = restatement.direct(x, y, z, d["m"], eps)
    a = b200.B200DirectSolver(eps, "fp64").evaluate((x, y, z), d["m"])
    assert np.array_equal(a, exact, equal_nan=scale < 1e-100)
    s = b200.DeviceSystem(n, eps, precision="fp64")
    s.set_state(x, y, z, d["vx"], d["vy"], d["vz"], d["m"])
    assert s.energy()[1] == restatement.potential_energy(x, y, z, d["m"], eps)


def _square_roots(a, bits):
    """Every r modulo 2^bits with r^2 = a (a = 1 modulo 8), by Hensel lifting."""
    r = 1
    for b in range(3, bits):
        if (r * r - a) % (1 << (b + 1)):
            r += 1 << (b - 1)
    m = 1 << bits
    return {r % m, -r % m, (r + m // 2) % m, (-r + m // 2) % m}


# Prime factors of 2^106 - j.
_FACTORS = {-5: [3, 7, 140627, 173331457829, 158494480927183],
            -4: [2, 2, 257, 78919881726271091143763623681],
            -3: [13, 6951403, 306673771, 2927433831769543],
            -2: [2, 3, 3, 11, 43, 211, 281, 331, 5419, 86171, 664441, 1564921],
            -1: [5, 15358129, 586477649, 1801439824104653],
            1: [3, 107, 6361, 69431, 20394401, 28059810762433],
            2: [2, 7, 7, 31, 71, 127, 151, 337, 29191, 106681, 122921, 152041],
            3: [2327027, 34864072662073401681969743],
            4: [2, 2, 3, 5, 17, 53, 157, 1613, 2731, 8191, 858001, 308761441],
            5: [19, 29, 147240723075511219048618884109]}


def _hard_arguments():
    """Every x whose square root, or the reciprocal of whose rounded square root,
    lies so near a midpoint of two doubles that a result good to 2^-103 before its
    last rounding could round wrongly (at a few exponents each)."""
    found = []
    # Roots: M^2 - j = x 2^k with M an odd 54-bit integer (a midpoint) and
    # |j| <= 2 M^2 2^-103 < 64; x in [1, 2) and [2, 4) stand for every x.
    for low, k in ((1 << 106, 54), (1 << 107, 55)):
        for j in range(-63, 64, 8):
            for r in _square_roots(j % (1 << k), k):
                for odd in range(r, 1 << 54, 1 << k):
                    square = odd * odd - j
                    if odd >= 1 << 53 and low <= square < 2 * low and square % (1 << k) == 0:
                        found += [np.ldexp(float(square >> k), k - 54 - 52 + 2 * e)
                                  for e in (-420, -120, 0, 17, 350)]
    # Reciprocals: s M = 2^106 - j with s a 53-bit integer, M a 54-bit odd one
    # and |j| <= 2^106 2^-103.8 < 5; all x whose rounded root is s: s^2 rounded
    # and its neighbours.
    for j, primes in _FACTORS.items():
        n = (1 << 106) - j
        divisors = {1}
        for p in primes:
            divisors |= {d * p for d in divisors}
        assert max(divisors) == n
        for s in divisors:
            if 1 << 52 <= s < 1 << 53 and (n // s) % 2 == 1:
                for e in (-440, -53, 0, 1, 300):
                    root = float(np.ldexp(float(s), e - 52))
                    for direction in (0.0, np.inf):
                        x = root ** 2
                        while np.sqrt(x) == root:
                            found.append(float(x))
                            x = np.nextafter(x, direction)
    edges = [np.nextafter(4.0 ** k, 0) for k in (-200, 0, 1, 2, 300)]
    edges += [np.nextafter(x, 0) for x in edges]  # both round to the root 2 - 2^-52
    return found + edges + [2.0 ** k for k in range(-1074, 1024, 53)]


def test_inverse_distance_is_correctly_rounded_where_it_is_hardest(b200):
    # Two unit masses at one point: their potential energy is minus the inverse
    # distance of the squared softening alone.
    import ctypes as C
    lib = b200.load_library()
    zero, one = np.zeros(2), np.ones(2)
    z, m = (a.ctypes.data_as(C.POINTER(C.c_double)) for a in (zero, one))
    arguments = _hard_arguments()
    assert len(arguments) > 400
    for x in arguments:
        params = b200.make_params(b200.SOLVER_DIRECT, "fp64")
        params.softening_squared = x
        system, energy = C.c_void_p(), C.c_double()
        assert lib.ob_system_create(C.byref(params), 2, C.byref(system)) == b200.OK
        assert lib.ob_system_set_state(system, z, z, z, None, None, None, m) == b200.OK
        assert lib.ob_system_energy(system, None, C.byref(energy)) == b200.OK
        lib.ob_system_destroy(system)
        assert energy.value == -(1.0 / np.sqrt(np.float64(x))), x.hex()


def test_fp32_within_reference_bounds(b200, restatement, golden_plummer):
    g = golden_plummer
    x, y, z, m = _xyzm(g)
    exact = restatement.reference_accelerations(x, y, z, m, 0.05)
    a = b200.B200DirectSolver(0.05, "fp32").evaluate((x, y, z), m)
    err = relative_errors(a, exact)
    assert err.max() < FP32_WORST
    assert np.sqrt(np.mean(err ** 2)) < FP32_RMS
    # Against the CPU solver (cuda_direct_solver_test.cpp:154-192): 2x the bound.
    assert relative_errors(a, g["direct_eps0.05"]).max() < 2 * FP32_WORST


def test_split_precision_meets_its_target(b200, golden_plummer):
    g = golden_plummer
    x, y, z, m = _xyzm(g)
    a = b200.B200DirectSolver(0.01, "split").evaluate((x, y, z), m)
    err = relative_errors(a, g["direct_eps0.01"])
    assert err.max() < SPLIT_WORST, err.max()
    assert np.median(err) < SPLIT_MEDIAN, np.median(err)


@pytest.mark.parametrize("precision", ["fp32", "split", "fp64"])
def test_pair_known_answer(b200, precision):
    a = b200.B200DirectSolver(0.0, precision).evaluate(
        (np.array([-1.0, 1.0]), np.zeros(2), np.zeros(2)), np.array([2.0, 3.0]))
    tol = 0.0 if precision == "fp64" else 1e-6
    assert np.allclose(a, [[0.75, 0, 0], [-0.5, 0, 0]], rtol=0, atol=tol)


@pytest.mark.parametrize("precision", ["fp32", "split", "fp64"])
def test_origin_particle_survives_padding(b200, precision):
    # cuda_direct_solver_test.cpp:296-337: unsoftened, a particle at the origin
    # next to zero-mass padding must get exactly (1, 1/4, 0).
    a = b200.B200DirectSolver(0.0, precision).evaluate(
        (np.array([0.0, 1.0, 0.0]), np.array([0.0, 0.0, 2.0]), np.zeros(3)), np.ones(3))
    assert np.all(np.isfinite(a))
    tol = 1e-14 if precision == "fp64" else 1e-6
    assert abs(a[0, 0] - 1.0) < tol and abs(a[0, 1] - 0.25) < tol and abs(a[0, 2]) < tol


@pytest.mark.parametrize("precision", ["fp32", "split", "fp64"])
def test_empty_and_single(b200, precision):
    s = b200.B200DirectSolver(0.1, precision)
    assert s.evaluate((np.zeros(0), np.zeros(0), np.zeros(0)), np.zeros(0)).shape == (0, 3)
    a = s.evaluate((np.ones(1), np.ones(1), np.ones(1)), np.ones(1))
    assert a.tolist() == [[0.0, 0.0, 0.0]]
    c = s.interaction_count()
    assert c.evaluations == 2 and c.particle_particle == 0


@pytest.mark.parametrize("n", [2, 3, 31, 33, 511, 513, 1023, 1025, 4097])
def test_ragged_sizes_against_oracle(b200, restatement, n):
    from orrery_b200 import initial_conditions as ic
    d = ic.plummer_sphere(n, seed=100 + n)
    x, y, z, m = _xyzm(d)
    exact, _ = restatement.direct(x, y, z, m, 0.02)
    for precision, bound in (("fp32", 5e-4), ("split", 2e-6)):
        a = b200.B200DirectSolver(0.02, precision).evaluate((x, y, z), m)
        assert relative_errors(a, exact).max() < bound, (precision, n)
    a = b200.B200DirectSolver(0.02, "fp64").evaluate((x, y, z), m)
    assert np.array_equal(a, exact)


@pytest.mark.parametrize("precision", ["fp32", "split"])
def test_heavy_target_keeps_its_self_term_masked(b200, restatement, precision):
    # With softening the kernels add a target's own entry as f * 0, which is
    # zero only while f = m / eps^3 is finite in FP32. A particle of mass
    # 1e32 at eps 1e-3 (f = 1e41) sends its block back to the masked loop;
    # every acceleration stays finite and on the oracle. It sits far from the
    # cluster so that its pair terms with the others stay in FP32 range.
    from orrery_b200 import initial_conditions as ic
    n = 1500
    d = ic.plummer_sphere(n, seed=77)
    x, y, z, m = (np.array(d[k]) for k in ("x", "y", "z", "m"))
    x[700], y[700], z[700], m[700] = 40.0, 40.0, 40.0, 1e32
    exact, _ = restatement.direct(x, y, z, m, 1e-3)
    a = b200.B200DirectSolver(1e-3, precision).evaluate((x, y, z), m)
    assert np.all(np.isfinite(a))
    bound = 5e-4 if precision == "fp32" else 2e-6
    assert relative_errors(a, exact).max() < bound


@pytest.mark.parametrize("precision", ["fp32", "split"])
def test_every_kernel_shape_computes_the_same_sum(b200, golden_plummer, precision):
    g = golden_plummer
    x, y, z, m = _xyzm(g)
    s = b200.B200DirectSolver(0.05, precision)
    results = []
    for shape in b200.direct_shapes(precision):
        s.set_shape(len(m), shape)
        results.append(s.evaluate((x, y, z), m))
    ref = g["direct_eps0.05"]
    bound = 2 * FP32_WORST if precision == "fp32" else SPLIT_WORST
    for a in results:
        assert relative_errors(a, ref).max() < bound
    # Splitting the sources (across a cluster or into source groups) changes
    # only the order of partial sums; in the split form that moves the
    # Kahan-compensated segments (512 or 512/K sources), which shows most on
    # the particles whose net force nearly cancels (measured 1.5e-7).
    spread = max(relative_errors(a, results[0]).max() for a in results)
    assert spread < (1e-5 if precision == "fp32" else 5e-7)


@pytest.mark.parametrize("precision", ["fp32", "split"])
def test_every_shape_masks_self_and_padding_without_softening(b200, restatement, precision):
    # eps = 0: the target's own entry and the padding must be masked, in every
    # shape (source groups included). A jittered lattice of 1500 particles
    # (ragged against every tile and target block) keeps pairs apart.
    rng = np.random.default_rng(11)
    g = np.stack(np.meshgrid(*(np.arange(12.0),) * 3, indexing="ij"), -1).reshape(-1, 3)[:1500]
    p = g + rng.uniform(-0.2, 0.2, g.shape)
    x, y, z = (np.ascontiguousarray(p[:, k]) for k in range(3))
    m = rng.uniform(0.5, 1.5, len(x))
    exact, _ = restatement.direct(x, y, z, m, 0.0)
    s = b200.B200DirectSolver(0.0, precision)
    bound = 2e-4 if precision == "fp32" else 2e-6
    for shape in b200.direct_shapes(precision):
        s.set_shape(len(m), shape)
        a = s.evaluate((x, y, z), m)
        assert np.all(np.isfinite(a)), shape
        assert relative_errors(a, exact).max() < bound, shape


def test_autotune_picks_a_working_shape(b200, golden_plummer):
    g = golden_plummer
    s = b200.B200DirectSolver(0.05, "fp32")
    shape, ms = s.autotune(len(g["m"]))
    assert shape in b200.direct_shapes("fp32") and ms > 0
    a = s.evaluate((g["x"], g["y"], g["z"]), g["m"])
    assert relative_errors(a, g["direct_eps0.05"]).max() < 2 * FP32_WORST


def test_momentum_is_conserved_at_scale(b200):
    # A size-independent property at the precision form's full size (262,144):
    # sum_i m_i a_i = 0 up to rounding (conservation_test.cpp:135-180).
    from orrery_b200 import initial_conditions as ic
    d = ic.plummer_sphere(262144, seed=20260811)
    x, y, z, m = _xyzm(d)
    for precision, bound in (("fp32", 1e-4), ("split", 1e-7)):
        a = b200.B200DirectSolver(0.01, precision).evaluate((x, y, z), m)
        net = np.abs((a * m[:, None]).sum(axis=0)).max()
        scale = (np.linalg.norm(a, axis=1) * m).sum()
        assert net / scale < bound, (precision, net / scale)


def test_device_pointer_entry_point(b200, golden_plummer):
    torch = pytest.importorskip("torch")
    g = golden_plummer
    dev = torch.device("cuda:0")
    ins = [torch.tensor(g[k], dtype=torch.float64, device=dev) for k in ("x", "y", "z", "m")]
    outs = [torch.empty(len(g["m"]), dtype=torch.float64, device=dev) for _ in range(3)]
    s = b200.B200DirectSolver(0.01, "fp64")
    s.evaluate_device(len(g["m"]), *ins, *outs, stream=torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    a = torch.stack(outs, dim=1).cpu().numpy()
    assert np.array_equal(a, g["direct_eps0.01"])


# Parts of a target tile added through a cluster (the grid fits 2 x 148 CTAs) or
# through memory (it does not), ragged last tiles and pairs; the same sums again
# on the next launch, which starts from the words the first one left.
@pytest.mark.parametrize("precision", ["fp32", "split"])
@pytest.mark.parametrize("n,shape", [(513, None), (2367, (256, 2, 4, 8)), (2369, (256, 2, 8, 8)),
                                     (4097, (256, 4, 8, 8)), (9473, (256, 4, 4, 8)),
                                     (9473, (128, 2, 4, 1)), (10007, None), (12289, None)])
def test_parts_are_added_in_order_wherever_they_meet(b200, restatement, precision, n, shape):
    from orrery_b200 import initial_conditions as ic
    d = ic.plummer_sphere(n, seed=n)
    x, y, z, m = _xyzm(d)
    exact, _ = restatement.direct(x, y, z, m, 0.05)
    s = b200.B200DirectSolver(0.05, precision)
    if shape is not None:
        s.set_shape(n, shape)
    a = s.evaluate((x, y, z), m)
    err = relative_errors(a, exact)
    if precision == "fp32":
        assert err.max() < FP32_WORST and np.sqrt(np.mean(err ** 2)) < FP32_RMS
    else:
        assert np.median(err) < SPLIT_MEDIAN and err.max() < 1e-5
    for _ in range(2):
        assert np.array_equal(s.evaluate((x, y, z), m), a)


def _kernel_ms(s, n, xyz, m):
    times = []
    for _ in range(15):
        s.evaluate(xyz, m)
        times.append(s.timings()["traversal_ms"])
    return np.median(times)


@pytest.mark.parametrize("precision,n", [("split", 1500), ("split", 2500)])
def test_tuning_never_picks_a_slower_shape_than_none(b200, precision, n):
    # The default takes three and five parts here; the best shapes of 1, 2, 4 or 8
    # parts are 37 and 38 % slower. 25 %: these kernels take 17 and 21 us, and events
    # tell times about 2 us apart.
    from orrery_b200 import initial_conditions as ic
    d = ic.plummer_sphere(n, seed=n)
    xyz, m = (d["x"], d["y"], d["z"]), d["m"]
    untuned = _kernel_ms(b200.B200DirectSolver(0.05, precision), n, xyz, m)
    s = b200.B200DirectSolver(0.05, precision)
    shape, _ = s.autotune(n)
    assert _kernel_ms(s, n, xyz, m) < 1.25 * untuned
    # What tuning returns can be set by hand.
    again = b200.B200DirectSolver(0.05, precision)
    again.set_shape(n, shape)
    assert np.array_equal(again.evaluate(xyz, m), s.evaluate(xyz, m))


def test_parts_take_a_bounded_amount_of_memory(b200):
    # Eight parts of a million targets would leave 192 MB of sums in memory; they
    # meet in clusters instead.
    torch = pytest.importorskip("torch")
    n = 1 << 20
    rng = torch.Generator(device="cuda")
    rng.manual_seed(3)
    x = torch.rand(3, n, generator=rng, device="cuda", dtype=torch.float64)
    m = torch.full((n,), 1.0 / n, device="cuda", dtype=torch.float64)
    out = torch.zeros(3, n, device="cuda", dtype=torch.float64)
    s = b200.B200DirectSolver(0.05, "fp32")
    s.set_shape(n, (256, 4, 8, 8))
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    s.evaluate_device(n, x[0], x[1], x[2], m, out[0], out[1], out[2],
                      torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    # 16 bytes of packed sources per particle, and what parts may take.
    assert before - torch.cuda.mem_get_info()[0] < 16 * n + (64 << 20) + (8 << 20)
    some = torch.arange(0, n, 4099, device="cuda")
    for i in some.tolist()[:64]:
        diff = x - x[:, i:i + 1]
        w = m * ((diff * diff).sum(0) + 0.05 ** 2) ** -1.5
        exact = (diff * w).sum(1)
        assert float((out[:, i] - exact).norm() / exact.norm()) < FP32_WORST
