"""The moduli of the off-box 1/mu bound (cabs_plain in common.cuh) are FP64:
within two units of 2^-53 of the exact modulus over the whole FP64 range (one
rounding of the sum of squares, halved by the root, one of the product before
it and one of the root), zero, infinities and NaN included."""
from test_rows_plan_cpu import run_program


def test_modulus_is_fp64(tmp_path):
    run_program(tmp_path, r"""
    const double scales[] = {1e-320, 1e-300, 1e-160, 1e-150, 1e-18, 1e-9, 1, 40, 1e18, 1e19, 1e150, 1e160, 1e300};
    unsigned long long s = 1;
    auto uniform = [&]() {
        s = s * 6364136223846793005ull + 1442695040888963407ull;
        return (double)(s >> 11) / 9007199254740992.0 * 2 - 1;
    };
    for (double a : scales)
        for (double b : scales)
            for (int i = 0; i < 200; i++)
            {
                const double2 v = make_double2(a * uniform(), b * uniform());
                const long double x = v.x, y = v.y, want = sqrtl(x * x + y * y);
                const long double d = fabsl((long double)cabs_plain(v) - want);
                if (d > 2 * 0x1p-53L * want && d > 0x1p-1074L) bad++;
            }
    if (cabs_plain(make_double2(0, 0)) != 0 || !std::isinf(cabs_plain(make_double2(INFINITY, 1)))) bad++;
    if (!std::isnan(cabs_plain(make_double2(NAN, 1)))) bad++;
""")
