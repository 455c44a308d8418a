// Device Bessel/Hankel functions of order 0 and 1 for complex argument.
//
// The reference evaluates H0^(1), H1^(1), J0, J1 with Bessels.jl (real
// argument) or AMOS through SpecialFunctions.jl (complex argument),
// src/utils/special_functions_calls.jl:3-7. AMOS is not restated here; these
// routines are written from the published mathematics:
//
//  * 0 < Re z < 128, |Im z| <= 0.4 (every real argument up to 128, and a
//    contour around a real k up to there): Taylor expansions of J0 and Y0 about
//    the centres c = n + 1/2 of unit panels, J1 and Y1 as their derivatives.
//    The coefficients follow from the values at c by Bessel's equation
//    x y'' + y' + x y = 0. For c < 6, where the logarithm of Y is too close,
//    G0 = Y0 - (2/pi) ln z J0, which is entire, takes the place of Y0; it
//    satisfies x y'' + y' + x y = -(4/pi) J0'.
//  * |z| >= 32, Re z > 0 elsewhere: the asymptotic expansion below with a
//    fixed number of terms (below 1e-17 at the range's lower end).
//  * otherwise (wide strips near the origin, Re z <= 0), |z| < 14.5: Miller's
//    backward recurrence for J_n(z) (Abramowitz & Stegun
//    9.1.27 recurrence run downward from n0 ~ |z| + 26), normalised with the
//    generating-function identity exp(-/+ i z) = J0 + 2 sum_{n>=1} (-/+ i)^n J_n
//    (sign chosen so that no cancellation occurs for Im z != 0), and the
//    Neumann series (A&S 9.1.88 for Y0; its derivative for Y1):
//        Y0 = (2/pi) [ (log(z/2)+gamma) J0 - 2 sum_{k>=1} (-1)^k J_{2k}/k ]
//        Y1 = (2/pi) [ (log(z/2)+gamma) J1 - J0/z - J1
//                      + sum_{m>=1} (-1)^{m+1} (2m+1)/(m(m+1)) J_{2m+1} ]
//    and |z| >= 14.5: Hankel's asymptotic expansion (A&S 9.2.5-9.2.10,
//    DLMF 10.17.1-10.17.4), summed until the terms stop decreasing:
//        J_nu = sqrt(2/(pi z)) (P cos w - Q sin w),
//        Y_nu = sqrt(2/(pi z)) (P sin w + Q cos w),   w = z - nu pi/2 - pi/4,
//        a_k(nu) = a_{k-1}(nu) (4 nu^2 - (2k-1)^2) / (8k).
//
// Accuracy (checked against mpmath in tests/test_gpu_core.py and
// tests/test_gpu_bessel_panels.py): max error relative to max(|J|,|Y|) below
// 2e-14, and a few 1e-16 on the Taylor panels; J0 and J1 to 4e-14 of themselves
// for |z| < 1, Re z > 0 (tests/test_gpu_bessel_small.py).
//
// Cost. This part issues 2 FP64 FMAs per clock and SM, so an evaluation costs
// its FP64 instruction count and nothing else: the recurrence takes about
// n0 = |z| + 26 complex steps with a divide in each (some 2000 instructions),
// the general asymptotic sum some 900; the Taylor panels take 64 FMAs at a
// real and 180 at a complex argument (one 16-byte table load per two
// coefficients, from L1), the fixed asymptotic sum about 250. Measured: 24 real k of a 602-node
// DLP operator 21.9 ms with the recurrence and the general sum, 1.5 ms now
// (with the real-k entry of qbg_assemble.cu).
//
// The FP32 variant used by the mixed form takes z in FP64, reduces Re z modulo
// 2*pi in FP64 (k*r reaches several thousand radians) and evaluates the
// asymptotic series in FP32; callers use it only for |z| >= 12, where the
// FP32-truncated series is accurate to FP32 rounding.
#pragma once
#include "qbg_common.cuh"

namespace qbg {

struct Bessel01d {
  cxd j0, j1, y0, y1;
  __device__ __forceinline__ cxd h0() const { return j0 + cmul_i(y0); }
  __device__ __forceinline__ cxd h1() const { return j1 + cmul_i(y1); }
};

__device__ __forceinline__ cxd cexp_d(cxd z) {
  double e = exp(z.re), s, c;
  sincos(z.im, &s, &c);
  return {e * c, e * s};
}

__device__ __forceinline__ cxd clog_d(cxd z) { return {log(hypot(z.re, z.im)), atan2(z.im, z.re)}; }

__device__ __forceinline__ cxd csqrt_d(cxd z) {
  double m = hypot(z.re, z.im);
  if (m == 0.0) return {0.0, 0.0};
  double t = sqrt(0.5 * (m + fabs(z.re)));
  if (z.re >= 0.0) return {t, 0.5 * z.im / t};
  return {0.5 * fabs(z.im) / t, copysign(t, z.im)};
}

__device__ __noinline__ Bessel01d bessel01_miller(cxd z) {
  const double az = hypot(z.re, z.im);
  const int n0 = 2 * (int)((az + 26.0) * 0.5);
  const cxd iz = cinv(z);
  const bool upper = z.im >= 0.0;  // normalise with exp(-iz) (upper) or exp(+iz)
  cxd fp1(0.0, 0.0), f(1e-30, 0.0);
  cxd snorm(0.0, 0.0), sy0(0.0, 0.0), sy1(0.0, 0.0);
  for (int n = n0; n >= 1; --n) {
    // (-i)^n for upper, (+i)^n for lower, n mod 4
    cxd fn2 = 2.0 * f;
    switch (n & 3) {
      case 0: snorm += fn2; break;
      case 1: snorm += upper ? cxd(fn2.im, -fn2.re) : cxd(-fn2.im, fn2.re); break;
      case 2: snorm -= fn2; break;
      default: snorm += upper ? cxd(-fn2.im, fn2.re) : cxd(fn2.im, -fn2.re); break;
    }
    if ((n & 1) == 0) {
      int k = n >> 1;
      double c = ((k & 1) ? -1.0 : 1.0) / (double)k;
      sy0 += c * f;
    } else {
      int m = (n - 1) >> 1;
      if (m >= 1) {
        double c = ((m & 1) ? 1.0 : -1.0) * (double)(2 * m + 1) / ((double)m * (double)(m + 1));
        sy1 += c * f;
      }
    }
    cxd fm1 = (2.0 * (double)n) * (iz * f) - fp1;
    fp1 = f;
    f = fm1;
    if (fabs(f.re) + fabs(f.im) > 1e200) {
      f = 1e-200 * f; fp1 = 1e-200 * fp1;
      snorm = 1e-200 * snorm; sy0 = 1e-200 * sy0; sy1 = 1e-200 * sy1;
    }
  }
  cxd f0 = f, f1 = fp1;
  cxd e = upper ? cexp_d(cxd(z.im, -z.re)) : cexp_d(cxd(-z.im, z.re));  // exp(-iz) or exp(iz)
  cxd sc = e * cinv(f0 + snorm);
  Bessel01d r;
  r.j0 = f0 * sc;
  r.j1 = f1 * sc;
  sy0 = sy0 * sc;
  sy1 = sy1 * sc;
  const double twopi_inv = 0.63661977236758134308;  // 2/pi
  cxd L = clog_d(0.5 * z) + cxd(0.57721566490153286061, 0.0);
  r.y0 = twopi_inv * (L * r.j0 - 2.0 * sy0);
  r.y1 = twopi_inv * (L * r.j1 - r.j0 * iz - r.j1 + sy1);
  return r;
}

__device__ __noinline__ Bessel01d bessel01_asym(cxd z) {
  const cxd w = cinv(z);
  const double aw = hypot(w.re, w.im);
  cxd wk(1.0, 0.0);
  double rk = 1.0, a0 = 1.0, a1 = 1.0, prev = 1e300;
  cxd P0(0, 0), Q0(0, 0), P1(0, 0), Q1(0, 0);
  for (int k = 0; k < 64; ++k) {
    double t = fmax(fabs(a0), fabs(a1)) * rk;
    if (t > prev) break;
    double sg = ((k >> 1) & 1) ? -1.0 : 1.0;
    if ((k & 1) == 0) { P0 += (sg * a0) * wk; P1 += (sg * a1) * wk; }
    else              { Q0 += (sg * a0) * wk; Q1 += (sg * a1) * wk; }
    if (t < 1e-17) break;
    prev = t;
    wk = wk * w;
    rk *= aw;
    double m = (double)(2 * k + 1);
    double d = 8.0 * (double)(k + 1);
    a0 *= (-m * m) / d;
    a1 *= (4.0 - m * m) / d;
  }
  // sqrt(2/(pi z))
  cxd pref = 0.79788456080286535588 * cinv(csqrt_d(z));
  double s, c;
  sincos(z.re, &s, &c);
  const double r2 = 0.70710678118654752440;
  double ca = (c + s) * r2, sa = (s - c) * r2;  // cos, sin of (Re z - pi/4)
  double ch = cosh(z.im), sh = sinh(z.im);
  cxd cw(ca * ch, -sa * sh), sw(sa * ch, ca * sh);  // cos w0, sin w0 (complex)
  Bessel01d r;
  r.j0 = pref * (P0 * cw - Q0 * sw);
  r.y0 = pref * (P0 * sw + Q0 * cw);
  // nu = 1: w1 = w0 - pi/2, cos w1 = sin w0, sin w1 = -cos w0
  r.j1 = pref * (P1 * sw + Q1 * cw);
  r.y1 = pref * (Q1 * sw - P1 * cw);
  return r;
}

// Taylor panels: coefficients a_m of J0 and b_m of Y0 (G0 for the first
// BP_G panels) about n + 1/2, interleaved (a_m, b_m). 16 coefficients reach
// 2e-17 at a real argument (|d| <= 1/2), 18 at |d| <= 0.64 (|Im z| <= 0.4).
constexpr int BP_PANELS = 128, BP_G = 6, BP_REAL = 16, BP_CPLX = 18;
constexpr double BP_STRIP = 0.4;
struct BesselPanels {
  double c[BP_PANELS][BP_CPLX][2];
};
constexpr BesselPanels bessel_panels() {
  // J0, J0', Y0, Y0' (panels 0 .. BP_G - 1: J0, J0', G0, G0') at n + 1/2
  constexpr double v[BP_PANELS][4] = {
    {0.9384698072408129042, -0.2422684576748738864, -0.03039903521526653506, 0.1696694294369484226},
    {0.5118276717359181287, -0.557936507910099642, 0.2503323287223161474, 0.3391007518566298824},
    {-0.04838377646819799633, -0.497094102464274038, 0.5262940097439155855, 0.1563719943977749274},
    {-0.3801277399872633774, -0.1373775273623271857, 0.4921866176793611911, -0.2314832605700143114},
    {-0.3205425089851214244, 0.231060431923370634, 0.1122225886957397609, -0.4768960691825374736},
    {-0.006843869417819196824, 0.3414382154290433502, -0.332053103312106626, -0.3460044072683648423},
    {0.2600946055816063814, 0.1538413014099718371, -0.1732424349189823357, 0.274091273959275453},
    {0.2663396578803783969, -0.1352484275797055052, 0.1173132861482086308, 0.2591285104861162518},
    {0.04193925184293450355, -0.2731219636740537443, 0.270205105365787476, 0.02616867939853747003},
    {-0.1939287476874223554, -0.161264430757529851, 0.1712106262027238449, -0.2031798993872076682},
    {-0.2366481944623471262, 0.07885001422733148815, -0.0675303724978763968, -0.2337042283572685784},
    {-0.06765394811166522843, 0.2283786206653234746, -0.2252321116911878654, -0.05794254714300082167},
    {0.1468840547004211023, 0.1654838046147597185, -0.1712143068446692873, 0.1538382565375011801},
    {0.2149891658804008153, -0.03804929208600142316, 0.03007700904678558868, 0.2140229303400289095},
    {0.08754486801037622291, -0.1934294635960469601, 0.1903018911878445166, 0.08104209092873875211},
    {-0.1092306509000501685, -0.1672131803517471433, 0.1706449112294346175, -0.1147861425133423274},
    {-0.1963806929368610297, 0.005764213735631226989, 0.0001812324575409665639, -0.1964758377859096562},
    {-0.1031103982286859222, 0.1634199694257549059, -0.1604111925050111691, -0.09857279873421604621},
    {0.07716482142255469901, 0.1666336400100160312, -0.1686563450403231259, 0.08174785849680946133},
    {0.178853827040172893, 0.02087707014809752225, -0.02545174297615446711, 0.1795645668963178899},
    {0.1150969602536747623, -0.1362546881933957366, 0.1334095666575904782, 0.1118790983445097298},
    {-0.04894204372155805655, -0.1638520825458122339, 0.1649452034614838544, -0.0527891089341719058},
    {-0.1615403170277827168, -0.04324203319071220007, 0.04681853166548836007, -0.1626199829760663075},
    {-0.1239282315602744426, 0.1109461433817633214, -0.1082861176947909405, -0.1216532806902694229},
    {0.02369743373406790211, 0.1589784118193280788, -0.1594287177497504292, 0.02695465533188541139},
    {0.1440621575468478617, 0.06204853649148410172, -0.06485976549878349112, 0.1453610587230494007},
    {0.1298776261133854109, -0.087027807537331489, 0.08456313574029273476, 0.1283057277317732306},
    {-0.0009922289050674051631, -0.1521418932046569415, 0.1521348331300461849, -0.003757569928524230523},
    {-0.1262911313804614537, -0.07770135790452337075, 0.07990403933540335667, -0.1277119251195870528},
    {-0.133147858298398214, 0.06430437809919239678, -0.06203938540000603999, -0.1321157350610256782},
    {-0.01938975451776215207, 0.1434943001509709411, -0.143157316174107651, -0.01704614288387645417},
    {0.1082389267114726217, 0.09044569145442246721, -0.09215174743370735848, 0.1097148997052929975},
    {0.13391127720843152, -0.0427308926203796142, 0.04066639974238427627, 0.1333016120800622247},
    {0.03754444002435240925, -0.1332093657305239754, 0.1326343726320787672, 0.03556943827909765261},
    {-0.09000065475310386358, -0.10044494700742566, 0.1017383605043284823, -0.09148425440075688465},
    {-0.1323315638913300117, 0.02234797020881734265, -0.02048248506960172862, -0.1320562445896174181},
    {-0.05350364241761478096, 0.1214808570499770248, -0.1207367526017292894, -0.05185503809193530804},
    {0.07172270511060222932, 0.1078233440192769592, -0.1087698194090656407, 0.07317908043183006528},
    {0.1285756853307894659, -0.003244073765967619493, 0.001574408059198233498, 0.128566073473720829},
    {0.06726809850975385967, -0.1085199464011415798, 0.1076599710263504567, 0.06591091580356654401},
    {-0.05358267563226294688, -0.1126905299405943127, 0.1133433143742016849, -0.05498584250054305299},
    {-0.1228203242138017711, -0.01446811651145212114, 0.0159465087140080311, -0.1230213291605513681},
    {-0.07882797369598458372, 0.09455212681048804615, -0.09361839381924884752, -0.07773218351432074142},
    {0.03577573717522485961, 0.1151562691098231548, -0.1155598027730954364, 0.03710619694257796455},
    {0.115254948926731048, 0.03066741696224856478, -0.03196023731678986897, 0.1156212770078977257},
    {0.08817609315509209525, -0.0798137996530667759, 0.07884019170172604669, 0.08731514187303833871},
    {-0.01850466374724187491, -0.1153392519145761344, 0.1155315297416970131, -0.01974786382982732807},
    {-0.1060827141588935375, -0.04523511047496801568, 0.04634908102989063244, -0.1065764183389329298},
    {-0.09531666074729756956, 0.06454862659555296941, -0.06356270937892591254, -0.09466650646080534805},
    {0.00197209936205727762, 0.1133721962832653914, -0.1133863337029157457, 0.003117399704532848896},
    {0.09551989154970056708, 0.05806287642132068648, -0.05900563494765444832, 0.09610872758567612125},
    {0.1002709976667062313, -0.04900372738955581878, 0.048028051986455218, 0.09980947277179286905},
    {0.01362570130150304338, -0.1094044746740236236, 0.109269765105670081, 0.01258574874828167897},
    {-0.08379426962089218808, -0.0690586353103599608, 0.06983864267499291247, -0.08445056773545347783},
    {-0.1030811910957957214, 0.03342580139117648016, -0.0324788157802863082, -0.1027875811519338843},
    {-0.0281040743011523956, 0.1036030058959336272, -0.1033456448067232601, -0.02717424785929639913},
    {0.07114281838573940958, 0.07815086275690760984, -0.078777312762802779, 0.07184269260714857939},
    {0.1038121944022615596, -0.01805724866618377237, 0.01715395388683610156, 0.1036669638486234815},
    {0.04129431799911825368, -0.09615188039980943483, 0.09579546587020109656, 0.04047712070413161417},
    {-0.05780883147438126812, -0.08529170609526627035, 0.08577443311208485931, -0.05853161440531592229},
    {-0.1025527247809908365, 0.003132364367764196285, -0.002284801030573988336, -0.1025373441680937684},
    {-0.05304735880343627548, 0.0872510341904327735, -0.08681691529469134324, -0.05234332928262824717},
    {0.04403870948258147505, 0.09045911175007760979, -0.09080849418578369681, 0.04476653965650351898},
    {0.09941519189110788463, 0.01112632284945246481, -0.01190870211390043792, 0.09951203607452658054},
    {0.06323677689948930697, -0.07711419701138436716, 0.07662171754000450196, 0.06264474507865848405},
    {-0.030078517787695294, -0.09365809982633242483, 0.09388495904154732382, -0.03079603117769199008},
    {-0.09453482556598131247, -0.02451150147635595499, 0.0252215368212298359, -0.09472712166145709258},
    {-0.07176122579142253673, 0.06596628696291754466, -0.06543295694548396711, -0.07127853188077291904},
    {0.01617043217167417306, 0.09492128159072181043, -0.09503677675156072396, 0.01686452496949748284},
    {0.08806813230646535463, 0.03683425478635325502, -0.03746683642640900334, 0.0883399422923072623},
    {0.07854626293837299522, -0.05404039094017062507, 0.05348200861639030288, 0.07816895176896187544},
    {-0.002549171644835308335, -0.09430869296611806822, 0.0943242128459745484, -0.003208811599964979191},
    {-0.08019078786203466094, -0.04792690915924440181, 0.04847877024626356432, -0.08052701478440719757},
    {-0.08354560162634329071, 0.04157444956890405255, -0.04100518990330663192, -0.08326860021925824531},
    {-0.01056149280236191994, 0.09190700557990992022, -0.0918340586089733683, -0.009945422377788484333},
    {0.07109506027151367851, 0.05764550342032911381, -0.05811503694867779305, 0.07148146980293387989},
    {0.08674179289234569252, -0.02880775162089463414, 0.02824023297263483568, 0.08655907633704204474},
    {0.0229520737645530248, -0.08782817196233676344, 0.08767827597152626549, 0.02238690854661886371},
    {-0.06098685037974146496, -0.06587183692049402504, 0.06625892873726503269, -0.06141010145291483597},
    {-0.0881463486291085164, 0.01597733319087644452, -0.01542267060760413841, -0.08805109743687824382},
    {-0.03443047577005887091, 0.08220756051450883176, -0.08199213367749001257, -0.03392189147860259335},
    {0.05008243266675789669, 0.07251506212887258867, -0.07282093466873044057, 0.05053011233650872478},
    {0.08779932155396742912, -0.003314369368606637372, 0.002782220719043657226, 0.08778407233545474117},
    {0.04482481290320406038, -0.07520163716129763213, 0.07493189163353386221, 0.04437693847134480887},
    {-0.0386049767059406478, -0.07751279607089761446, 0.0777398592446396585, -0.03906563546053194279},
    {-0.0857683635977974619, -0.0089593603944990824, 0.009460750889471284368, -0.08582515399905084324},
    {-0.05398588032729748624, 0.06698525306069462276, -0.06667209276583695679, -0.05360140708995039093},
    {0.02678092773299819843, 0.08083173387597459898, -0.08098344084484668997, 0.02724411229837273214},
    {0.08214729081420695758, 0.02063485824705617962, -0.02109861576733237951, 0.0822677990109578593},
    {0.06178923273698054451, -0.05774860061086658621, 0.05740252454345091345, 0.06146952228022981392},
    {-0.01483632302709028607, -0.08246775684660841818, 0.08254846336255870587, -0.01529260435940001961},
    {-0.07705418965772834194, -0.03151907658644975936, 0.03193964838506537263, -0.07722986827153393614},
    {-0.06813683148442760958, 0.04769390276471575552, -0.04732491507161681852, -0.06788202384741543993},
    {0.002993118670219192021, 0.08244553666521865061, -0.0824603633509734893, 0.003434113363745607904},
    {0.07062910607989263133, 0.04143780744618106164, -0.04181091082195910281, 0.070851310088232277},
    {0.07295823113238305607, -0.03703190297081175037, 0.03664943094756928466, 0.07276735432999537323},
    {0.008534401495985850787, -0.08081764645462531522, 0.08077234390465311209, 0.008116017713204742578},
    {-0.06303136507066916964, -0.05023823784398897979, 0.05056080238871265792, -0.06329147309890235637},
    {-0.07621128541917213724, 0.02597822465914419041, -0.02559104565527778092, -0.07608236669865854136},
    {-0.01954306640744078356, 0.07766319824307693544, -0.07756401519388381423, -0.01915355403677695903},
    {0.05443657381441359099, 0.05779112399693202059, -0.05806122757035574851, 0.05472610209468348646},
    {0.07788236197513819429, -0.01474966990943906933, 0.014365847982673354, 0.07781254079245830669},
    {0.02984404384865724676, -0.07308603479899686184, 0.07293958987747029006, 0.02948860445714870088},
    {-0.04503336636380667816, -0.06399254548236853575, 0.06420934375909300516, -0.04534407460583387266},
    {-0.07798606448359291484, 0.003560526668473968001, -0.003187359664492999815, -0.07797170685743641352},
    {-0.03926579330115592443, 0.06721251164615469326, -0.06702566938117065327, -0.03894858415192149471},
    {0.03501995152919449817, 0.06876520901727358322, -0.06892885876988096265, 0.03534393995666092598},
    {0.07656447019649210816, 0.007381047441090369657, -0.007737069876274584617, 0.07660128384946273503},
    {0.04765669284359344435, -0.06018891220896342183, 0.05996866410121695092, 0.04738085138066732405},
    {-0.02460052843382097681, -0.07205928044346387027, 0.07217085698895086987, -0.02493032528719326424},
    {-0.0736858996534613364, -0.01787649907635600782, 0.01820972621734899649, -0.07376904916629363494},
    {-0.0548872941733784384, 0.0521785453453615455, -0.05193189684609552211, -0.05465497218862840979},
    {0.01398163582702135393, 0.0738527326219682421, -0.07391414207235947182, 0.01431027471094239236},
    {0.06944324396932289983, 0.02774014871131226867, -0.02804578804735432884, 0.06956746504445520285},
    {0.06085216728898875387, -0.0433585798919944614, 0.04309244415277822964, 0.06066457439178817826},
    {-0.003368501734740270243, -0.07415120612009672329, 0.07416509324959213349, -0.003689588288805852056},
    {-0.06395188301033797682, -0.03680219805431982306, 0.03707632316819677519, -0.06411159485752916836},
    {-0.06547130440315789927, 0.03391667518136899222, -0.03363777441208901245, -0.06532876023055100926},
    {-0.007038540656567084811, 0.07298738867497741583, -0.07295704134981223866, -0.00673077316637479349},
    {0.05734723504088439671, 0.04491142308021561909, -0.04515097029169344816, 0.05753664985343693192},
    {0.06869106112012379695, -0.02404746972070039185, 0.02376224493784551462, 0.06859305556551055319},
    {0.01704750683160438055, -0.07041992828887199823, 0.07034917950584023525, 0.01675815327219995771},
    {-0.04978198486899480777, -0.05193750671041130811, 0.05214026082500085164, -0.04999521334933515917},
    {-0.07048462166325228854, 0.01394899229517803465, -0.01366352216273508053, -0.07042988226469908428},
    {-0.02647802341631065623, 0.06653190330644363969, -0.06642503195461615062, -0.02621147402891698638},
    {0.04142304304355081176, 0.05777297222820010904, -0.05793754188436181766, 0.04165419495703250756},
    {0.07085198383213736541, -0.003819060643636823622, 0.003538990009174531754, 0.07083854934709516847},
    {0.03516434225656891892, -0.06142888079880234327, 0.061290512298760913, 0.03492426136694922321},
  };
  BesselPanels t{};
  for (int n = 0; n < BP_PANELS; ++n) {
    const double c = n + 0.5;
    t.c[n][0][0] = v[n][0];
    t.c[n][1][0] = v[n][1];
    t.c[n][0][1] = v[n][2];
    t.c[n][1][1] = v[n][3];
    for (int m = 0; m + 2 < BP_CPLX; ++m) {
      const double p = m + 1.0, den = 1.0 / (c * p * (m + 2.0));
      for (int f = 0; f < 2; ++f) {
        const double low = m > 0 ? t.c[n][m - 1][f] : 0.0;
        const double rhs = (f == 1 && n < BP_G) ? -1.27323954473516268615 * p * t.c[n][m + 1][0] : 0.0;
        t.c[n][m + 2][f] = (rhs - (p * p * t.c[n][m + 1][f] + c * t.c[n][m][f] + low)) * den;
      }
    }
  }
  return t;
}
static __device__ const BesselPanels g_bessel_panels = bessel_panels();

// Coefficients (-1)^{k/2} a_k(nu) of P (even k) and Q (odd k), A&S 9.2.9-9.2.10
struct HankelCoef {
  double p0[9], q0[8], p1[9], q1[8];
};
constexpr HankelCoef hankel_coef() {
  HankelCoef h{};
  double a0 = 1.0, a1 = 1.0;
  for (int k = 0; k < 17; ++k) {
    const double sg = ((k >> 1) & 1) ? -1.0 : 1.0;
    if (k & 1) {
      h.q0[k >> 1] = sg * a0;
      h.q1[k >> 1] = sg * a1;
    } else {
      h.p0[k >> 1] = sg * a0;
      h.p1[k >> 1] = sg * a1;
    }
    const double m = 2.0 * k + 1.0, d = 8.0 * (k + 1.0);
    a0 *= -m * m / d;
    a1 *= (4.0 - m * m) / d;
  }
  return h;
}

// On panel 0 the derivative series leaves J1 an absolute error of a few 1e-16
// (5e-13 of J1 at 1e-3, 5e-8 at 1e-8); below 0.25 the power series
// (z/2) sum (-z^2/4)^m / (m! (m+1)!) keeps it to rounding in six terms (q = -z^2/4).
constexpr double BP_SMALL = 0.25;
template <class T>
__device__ __forceinline__ T j1_small(T z, T q) {
  T s = q * (1.0 / 86400.0) + T(1.0 / 2880.0);
  s = s * q + T(1.0 / 144.0);
  s = s * q + T(1.0 / 12.0);
  s = s * q + T(0.5);
  return 0.5 * (z * (s * q + T(1.0)));
}

// J0, J1, Y0, Y1 at a real x > 0
struct Bessel01r {
  double j0, j1, y0, y1;
};

__device__ __forceinline__ Bessel01r bessel01_real(double x) {
  const double two_over_pi = 0.63661977236758134308;
  Bessel01r r;
  if (x < (double)BP_PANELS) {
    const int n = (int)x;
    const double d = x - ((double)n + 0.5);
    const double2* c = reinterpret_cast<const double2*>(g_bessel_panels.c[n]);
    double2 v = __ldg(c + BP_REAL - 1);
    double a = v.x, b = v.y, ap = 0.0, bp = 0.0;
#pragma unroll
    for (int m = BP_REAL - 2; m >= 0; --m) {
      v = __ldg(c + m);
      ap = m == BP_REAL - 2 ? a : fma(ap, d, a);
      bp = m == BP_REAL - 2 ? b : fma(bp, d, b);
      a = fma(a, d, v.x);
      b = fma(b, d, v.y);
    }
    r.j0 = a;
    r.j1 = -ap;
    if (n < BP_G) {
      if (x < BP_SMALL) r.j1 = j1_small(x, -0.25 * x * x);
      const double l = two_over_pi * log(x);
      r.y0 = fma(l, a, b);
      r.y1 = fma(l, r.j1, -two_over_pi * a / x) - bp;
    } else {
      r.y0 = b;
      r.y1 = -bp;
    }
    return r;
  }
  constexpr HankelCoef h = hankel_coef();
  const double w = 1.0 / x, t = w * w;
  double p0 = h.p0[4], q0 = h.q0[3], p1 = h.p1[4], q1 = h.q1[3];
#pragma unroll
  for (int m = 3; m >= 0; --m) {
    p0 = fma(p0, t, h.p0[m]);
    p1 = fma(p1, t, h.p1[m]);
    if (m < 3) {
      q0 = fma(q0, t, h.q0[m]);
      q1 = fma(q1, t, h.q1[m]);
    }
  }
  q0 *= w;
  q1 *= w;
  double s, c;
  sincos(x, &s, &c);
  const double f = 0.56418958354775628695 * sqrt(w);  // sqrt(1/(pi x))
  const double ca = f * (c + s), sa = f * (s - c);
  r.j0 = p0 * ca - q0 * sa;
  r.y0 = p0 * sa + q0 * ca;
  r.j1 = p1 * sa + q1 * ca;
  r.y1 = q1 * sa - p1 * ca;
  return r;
}

static __device__ __noinline__ Bessel01d bessel01_real_c(double x) {
  const Bessel01r b = bessel01_real(x);
  return {cxd(b.j0, 0.0), cxd(b.j1, 0.0), cxd(b.y0, 0.0), cxd(b.y1, 0.0)};
}

// the Taylor panels at complex z, 0 < Re z < BP_PANELS, |Im z| <= BP_STRIP.
// A polynomial with real coefficients at complex d takes two real FMAs per
// coefficient: b_m = c_m + 2 Re d b_{m+1} - |d|^2 b_{m+2}, p(d) = c_0 - |d|^2 b_2 + d b_1.
static __device__ __noinline__ Bessel01d bessel01_panel(cxd z) {
  const double two_over_pi = 0.63661977236758134308;
  const int n = (int)z.re;
  const double dr = z.re - ((double)n + 0.5), di = z.im;
  const double u = 2.0 * dr, v = -(dr * dr + di * di);
  const double2* c = reinterpret_cast<const double2*>(g_bessel_panels.c[n]);
  // value series (coefficients c_m) and derivative series (m c_m, one degree less)
  double a1 = 0.0, a2 = 0.0, b1 = 0.0, b2 = 0.0, e1 = 0.0, e2 = 0.0, f1 = 0.0, f2 = 0.0;
#pragma unroll
  for (int m = BP_CPLX - 1; m >= 1; --m) {
    const double2 k = __ldg(c + m);
    const double a = fma(u, a1, fma(v, a2, k.x)), b = fma(u, b1, fma(v, b2, k.y));
    a2 = a1;
    a1 = a;
    b2 = b1;
    b1 = b;
    if (m >= 2) {
      const double e = fma(u, e1, fma(v, e2, (double)m * k.x)), f = fma(u, f1, fma(v, f2, (double)m * k.y));
      e2 = e1;
      e1 = e;
      f2 = f1;
      f1 = f;
    }
  }
  const double2 k0 = __ldg(c), k1 = __ldg(c + 1);
  const cxd j0(fma(dr, a1, fma(v, a2, k0.x)), di * a1), g0(fma(dr, b1, fma(v, b2, k0.y)), di * b1);
  const cxd jp(fma(dr, e1, fma(v, e2, k1.x)), di * e1), gp(fma(dr, f1, fma(v, f2, k1.y)), di * f1);
  Bessel01d r;
  r.j0 = j0;
  r.j1 = -jp;
  if (n < BP_G) {
    const double az = hypot(z.re, z.im);
    if (az < BP_SMALL) r.j1 = j1_small(z, -0.25 * (z * z));
    const cxd l = two_over_pi * cxd(log(az), atan2(z.im, z.re));
    r.y0 = g0 + l * j0;
    r.y1 = l * r.j1 - two_over_pi * (j0 * cinv(z)) - gp;
  } else {
    r.y0 = g0;
    r.y1 = -gp;
  }
  return r;
}

// p(t), real coefficients c[0..N-1] at complex t (see bessel01_panel)
template <int N>
__device__ __forceinline__ cxd real_poly(const double* c, double u, double v, cxd t) {
  double b1 = c[N - 1], b2 = 0.0;
#pragma unroll
  for (int m = N - 2; m >= 1; --m) {
    const double b = m == N - 2 ? fma(u, b1, c[m]) : fma(u, b1, fma(v, b2, c[m]));
    b2 = b1;
    b1 = b;
  }
  return {fma(t.re, b1, fma(v, b2, c[0])), t.im * b1};
}

// the asymptotic expansion with NP + NQ terms, Re z > 0: 17 terms from |z| = 32, 9 from 128
template <int NP, int NQ>
static __device__ __noinline__ Bessel01d bessel01_hankel(cxd z) {
  constexpr HankelCoef h = hankel_coef();
  const double n2 = z.re * z.re + z.im * z.im, in2 = 1.0 / n2;
  const cxd w(z.re * in2, -z.im * in2);
  const cxd t(w.re * w.re - w.im * w.im, 2.0 * w.re * w.im);
  const double u = 2.0 * t.re, v = -(t.re * t.re + t.im * t.im);
  const cxd P0 = real_poly<NP>(h.p0, u, v, t), P1 = real_poly<NP>(h.p1, u, v, t);
  const cxd Q0 = w * real_poly<NQ>(h.q0, u, v, t), Q1 = w * real_poly<NQ>(h.q1, u, v, t);
  // sqrt(2 / (pi z)) = sqrt(2/pi) sqrt(w); the phase's 1/sqrt(2) is folded in
  const double t2 = 0.5 * (sqrt(in2) + w.re), it = rsqrt(t2);
  const double f = 0.56418958354775628695;
  const cxd pref(f * (t2 * it), f * (0.5 * w.im * it));
  double s, c;
  sincos(z.re, &s, &c);
  const double ca = c + s, sa = s - c, y = z.im;
  double ch, sh;
  if (fabs(y) < 0.5) {
    const double q = y * y;
    sh = y * fma(q, fma(q, fma(q, fma(q, fma(q, fma(q, 1.0 / 6227020800.0, 1.0 / 39916800.0), 1.0 / 362880.0), 1.0 / 5040.0), 1.0 / 120.0), 1.0 / 6.0), 1.0);
    ch = fma(q, fma(q, fma(q, fma(q, fma(q, fma(q, fma(q, 1.0 / 87178291200.0, 1.0 / 479001600.0), 1.0 / 3628800.0), 1.0 / 40320.0), 1.0 / 720.0), 1.0 / 24.0), 0.5), 1.0);
  } else {
    const double e = exp(y), ie = 1.0 / e;
    ch = 0.5 * (e + ie);
    sh = 0.5 * (e - ie);
  }
  const cxd cw = pref * cxd(ca * ch, -sa * sh), sw = pref * cxd(sa * ch, ca * sh);
  Bessel01d r;
  r.j0 = P0 * cw - Q0 * sw;
  r.y0 = P0 * sw + Q0 * cw;
  r.j1 = P1 * sw + Q1 * cw;
  r.y1 = Q1 * sw - P1 * cw;
  return r;
}

// The ranges: the panels wherever they reach (cheaper than the asymptotic sum
// by a sincos and a square root), the fixed sums where their last term is
// below 1e-17, the general routines for what is left. NaN and infinite
// arguments fail every comparison and reach the general sum.
__device__ __forceinline__ Bessel01d bessel01(cxd z) {
  if (z.re > 0.0 && z.re < (double)BP_PANELS) {
    if (z.im == 0.0) return bessel01_real_c(z.re);
    if (fabs(z.im) <= BP_STRIP) return bessel01_panel(z);
  }
  const double n2 = z.re * z.re + z.im * z.im;
  if (z.re > 0.0 && n2 >= 1024.0 && n2 < 1e280 && fabs(z.im) < 300.0)
    return n2 >= 16384.0 ? bessel01_hankel<5, 4>(z) : bessel01_hankel<9, 8>(z);
  return (hypot(z.re, z.im) < 14.5) ? bessel01_miller(z) : bessel01_asym(z);
}

// ---------------------------------------------------------------------------
// FP32 asymptotic evaluation with FP64 phase reduction (mixed form).
// ---------------------------------------------------------------------------
struct Bessel01f {
  cxf j0, j1, y0, y1;
  __device__ __forceinline__ cxf h0() const { return j0 + cmul_i(y0); }
  __device__ __forceinline__ cxf h1() const { return j1 + cmul_i(y1); }
};

__device__ __forceinline__ Bessel01f bessel01_asym_f32(cxd z64) {
  // phase: x - 2*pi*round(x/(2*pi)) in FP64 (2*pi split in two parts)
  const double x = z64.re;
  const double q = rint(x * 0.15915494309189533577);
  const double xr = fma(-q, 6.2831853071795862320, x) - q * 2.4492935982947064e-16;
  const float xf = (float)xr;
  const cxf z((float)z64.re, (float)z64.im);
  const cxf w = cinv(z);
  const float aw = sqrtf(w.re * w.re + w.im * w.im);
  cxf wk(1.f, 0.f);
  float rk = 1.f, a0 = 1.f, a1 = 1.f, prev = 1e30f;
  cxf P0(0, 0), Q0(0, 0), P1(0, 0), Q1(0, 0);
#pragma unroll 1
  for (int k = 0; k < 16; ++k) {
    float t = fmaxf(fabsf(a0), fabsf(a1)) * rk;
    if (t > prev) break;
    float sg = ((k >> 1) & 1) ? -1.f : 1.f;
    if ((k & 1) == 0) { P0 += (sg * a0) * wk; P1 += (sg * a1) * wk; }
    else              { Q0 += (sg * a0) * wk; Q1 += (sg * a1) * wk; }
    if (t < 3e-9f) break;
    prev = t;
    wk = wk * w;
    rk *= aw;
    float m = (float)(2 * k + 1);
    float d = 8.f * (float)(k + 1);
    a0 *= (-m * m) / d;
    a1 *= (4.f - m * m) / d;
  }
  // sqrt(2/(pi z)) = sqrt(2/pi) / sqrt(z)
  const float mz = sqrtf(z.re * z.re + z.im * z.im);
  float t = sqrtf(0.5f * (mz + fabsf(z.re)));
  cxf sz = (z.re >= 0.f) ? cxf(t, 0.5f * z.im / t) : cxf(0.5f * fabsf(z.im) / t, copysignf(t, z.im));
  cxf pref = 0.797884560802865f * cinv(sz);
  float s, c;
  sincosf(xf, &s, &c);
  const float r2 = 0.70710678118654752f;
  float ca = (c + s) * r2, sa = (s - c) * r2;
  float ch = coshf(z.im), sh = sinhf(z.im);
  cxf cw(ca * ch, -sa * sh), sw(sa * ch, ca * sh);
  Bessel01f r;
  r.j0 = pref * (P0 * cw - Q0 * sw);
  r.y0 = pref * (P0 * sw + Q0 * cw);
  r.j1 = pref * (P1 * sw + Q1 * cw);
  r.y1 = pref * (Q1 * sw - P1 * cw);
  return r;
}

}  // namespace qbg
