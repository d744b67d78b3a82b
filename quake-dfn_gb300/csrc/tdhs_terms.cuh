// Strains of the angular dislocations of a triangle (Nikkhoo & Walter 2015):
// AngDisStrain and AngDisStrainFSC (scripts/Functions_TDstressHS.jl:577-651,
// :654-1034), with their divisions written as products with a few reciprocals
// and their common subexpressions taken out by computer algebra -- term by term,
// nothing expanded, so that the differences that carry the cancellation stay as
// they are.  The formulas in their published form are in the oracle's tdhs.cpp,
// which the tests compare with.
//
// The stiffness is bound by the FP64 pipe, so what counts is the number of FP64
// operations.  As published, an evaluation has hundreds of divisions of eight or
// more operations each (a pair, six evaluations of either kind: 43,500 FP64
// operations); here it takes ~150 (full space) and ~1,000 (free-surface
// correction), three or four divisions and a square root included.
//
// The stresses are differences of large terms, so the formulas' own rounding
// error is 1e-9 of Kn over a near-field block (113-bit arithmetic as the value),
// as published and here alike (6.46e-9 and 6.45e-9); the two differ by 2e-11.
// Over far blocks (18 x 18 triangles, 0.6 to 8 km off, geometric mean of the
// 2-norm of the error and of the difference) 1.5e-11 and 8e-12 at dips of 70
// degrees, 4e-10 and 1.3e-10 at 85: a side near the vertical multiplies either by
// up to cot^2 of its angle to it, 1.6e-7 and 3e-8 at 89.67 degrees.
#pragma once
#include "qdfn_internal.h"

namespace qdfn {
namespace tdhs {

#ifdef __CUDA_ARCH__
#define QDFN_TD __device__ __forceinline__
#else
#define QDFN_TD inline __host__ __device__
#endif

// Strains (xx, yy, zz, xy, xz, yz) of an angular dislocation in a full space
// with slip (0, by, bz), times 8 pi (1 - nu); sinA, cosA: of its angle,
// M2 = 2 - 2 nu.
QDFN_TD void ang_strain(double x, double y, double z, double sinA, double cosA, double by, double bz, double nu,
                        double M2, double e[6]) {
    const double eta = y * cosA - z * sinA, zeta = y * sinA + z * cosA;
    const double r = sqrt(x * x + y * y + z * z);
    const double ir = 1.0 / r, iW = 1.0 / (zeta - r), iz = 1.0 / (r - z);
    const double C = (r * cosA - z) * (iW * ir), S = (r * sinA - y) * (iW * ir);
    const double s0 = ir * ir;
    const double s1 = x * x;
    const double s2 = s0 * s1;
    const double s3 = (-3.0 + M2);
    const double s4 = fma(-iW, ir * s1, s2 + s3);
    const double s5 = bz * sinA;
    const double s6 = iz * iz;
    const double s7 = cosA * iW;
    const double s8 = iW * ir;
    const double s9 = ir * ir * ir;
    const double s10 = y * y;
    const double s11 = s10 * s9;
    const double s12 = fma(-iW, s11, fma(S, S, s8));
    const double s13 = ir * iz;
    const double s14 = M2 * ir;
    const double s15 = s14 * ((iz + s7));
    const double s16 = M2 * s8;
    const double s17 = fma(-iW, s9 * z * z, fma(C, C, s8));
    const double s18 = s9 * z;
    const double s19 = S * nu;
    const double s20 = s1 * s8;
    const double s21 = S * s20;
    const double s22 = s1 * s9;
    const double s23 = iW * y;
    const double s24 = 2.0 * cosA;
    const double s25 = 2.0 * y;
    const double s26 = iz * y;
    const double s27 = s14 * (fma(eta, iW, s26));
    const double s28 = C * nu;
    const double s29 = C * s20;
    const double s30 = s1 * s18;
    const double s31 = 2.0 * sinA;
    const double s32 = s18 * y;
    const double s33 = s0 * z;
    const double s34 = cosA * y;
    const double s35 = fma(sinA, z, s34);
    const double s36 = iW * iW;
    e[0] = -ir * x * (fma(iW, s4 * s5, by * (fma(-ir, s1 * s6, fma(-s4, s7, fma(-iz, s3, -iz * s2))))));
    e[1] = x * (fma(s12, s5, by * (fma(s0, s10 * s6, fma(-cosA, s12, fma(iz, s11, s15 - s13))))));
    e[2] = x * (fma(bz, sinA * ((s17 - s16)), -by * (fma(cosA, s17, s18))));
    e[3] = fma(0.5, by * (fma(-nu, s13 * s25, fma(s22, s25 * s7, fma(s2, s25 * s6, fma(2.0, s22 * s26, fma(s21, s24,
        fma(s19, s24, -s27))))))), -s5 * (fma(s22, s23, s19 + s21)));
    e[4] = fma(-0.5, bz * (fma(s31, (fma(iW, s30, s28 + s29)), s27)), by * (fma(s30, s7, fma(ir, nu, fma(cosA, s29,
        fma(cosA, s28, -s22))))));
    e[5] = 0.5 * x * (fma(-by, (fma(-ir, s24 * s35 * s36, fma(2.0, s33 * s34 * s36, fma(s31, s36 * cosA * cosA,
        fma(-2.0, s32 * s7, fma(s25, s9, s16 * sinA)))))), bz * (fma(iW, s31 * (fma(-s35, s8, fma(s7, sinA, fma(s23,
        s33, -s32)))), s15))));
}

// Free-surface correction strains of an angular dislocation in a half-space
// times 4 pi (1 - nu); sinB, cosB, cotB, icosB = 1 / cosB: of its angle,
// N1 = 1 - 2 nu, M2 = 2 - 2 nu.
QDFN_TD void ang_strain_fsc(double y1, double y2, double y3, double sinB, double cosB, double cotB, double icosB,
                            double b1, double b2, double b3, double nu, double N1, double M2, double a, double v[6]) {
    const double y3b = y3 + 2 * a;
    const double z1b = y1 * cosB + y3b * sinB, z3b = -y1 * sinB + y3b * cosB;
    const double rb = sqrt(y1 * y1 + y2 * y2 + y3b * y3b);
    const double irb = 1.0 / rb, iW6 = 1.0 / (rb + y3b), iW7 = 1.0 / (rb + z3b);
    const double W8 = y3 + a;
    // sums that cancel, without fused operations and W3 with a division, as in
    // the published form: their rounding is most of the result's
    const double W1 = rb * cosB + y3b, RS = rb * sinB - y1, UB = y1 * irb - sinB;
    const double W2 = cosB + a * irb, W3 = cosB + y3b / rb, CY = cosB * y3b * irb + 1, SY = irb * sinB * y1 - 1;
    const double t0 = iW7 * iW7;
    const double t1 = W2 * t0;
    const double t2 = cosB * t1;
    const double t3 = UB * t2;
    const double t4 = iW6 * y1;
    const double t5 = irb * irb * irb;
    const double t6 = a * t5;
    const double t7 = t4 * t6;
    const double t8 = cosB * iW7;
    const double t9 = t6 * y1;
    const double t10 = t8 * t9;
    const double t11 = a * irb;
    const double t12 = (1.0 + t11);
    const double t13 = iW6 * iW6;
    const double t14 = irb * y1;
    const double t15 = t13 * t14;
    const double t16 = irb * irb;
    const double t17 = a * t16;
    const double t18 = (iW6 + t17);
    const double t19 = t16 * y1;
    const double t20 = t18 * t19;
    const double t21 = 2.0 * t6;
    const double t22 = (t13 + t21);
    const double t23 = t14 * t22;
    const double t24 = W1 * iW7;
    const double t25 = t17 * y3b;
    const double t26 = fma(W2, t24, t25);
    const double t27 = UB * t0;
    const double t28 = cosB * t27;
    const double t29 = t19 * t8;
    const double t30 = W1 * t0;
    const double t31 = W2 * t30;
    const double t32 = W2 * t8;
    const double t33 = irb * irb * irb * irb;
    const double t34 = a * t33;
    const double t35 = t34 * y3b;
    const double t36 = 2.0 * t35;
    const double t37 = t36 * y1;
    const double t38 = fma(-t14, t32, fma(t24, t9, fma(UB, t31, t37)));
    const double t39 = t38 * t8;
    const double t40 = W8 * irb;
    const double t41 = N1 * cotB;
    const double t42 = cosB * t41;
    const double t43 = UB * t1;
    const double t44 = t41 * y1;
    const double t45 = t44 * t6;
    const double t46 = (t8 - iW6);
    const double t47 = cotB * cotB;
    const double t48 = (1.0 + N1);
    const double t49 = t47 * t48;
    const double t50 = N1 * irb;
    const double t51 = t49 * t50;
    const double t52 = t46 * t51;
    const double t53 = -t11;
    const double t54 = cotB * ((N1 + t53));
    const double t55 = (nu + t11);
    const double t56 = iW6 * t55;
    const double t57 = t56 * y1;
    const double t58 = (t54 - t57);
    const double t59 = N1 * t15;
    const double t60 = cotB * t6;
    const double t61 = t60 * y1;
    const double t62 = y1 * y1;
    const double t63 = t6 * t62;
    const double t64 = iW6 * t63;
    const double t65 = irb * t62;
    const double t66 = t13 * t55;
    const double t67 = N1 * iW6;
    const double t68 = t67 * (fma(t65, t66, t61 + t64 - t56));
    const double t69 = 3.0 * t34;
    const double t70 = cotB * y1;
    const double t71 = t69 * t70;
    const double t72 = -N1;
    const double t73 = (t12 + t72);
    const double t74 = iW6 * t73;
    const double t75 = t74 * y1;
    const double t76 = -t41;
    const double t77 = t17 * y1;
    const double t78 = (t76 + t77);
    const double t79 = (t75 + t78);
    const double t80 = t16 * t79;
    const double t81 = cotB * t25;
    const double t82 = cosB * t48;
    const double t83 = cotB * (fma(N1, cosB, t53));
    const double t84 = fma(W1, t83, RS * t82);
    const double t85 = fma(-iW7, t84, t81);
    const double t86 = -t85;
    const double t87 = -iW6 * t73;
    const double t88 = t13 * t73;
    const double t89 = t62 * t88;
    const double t90 = -t17;
    const double t91 = fma(2.0, t34 * t62, t90);
    const double t92 = t0 * t84;
    const double t93 = cosB * t83;
    const double t94 = b1 * y2;
    const double t95 = cosB * z1b;
    const double t96 = icosB * t11;
    const double t97 = t41 * (fma(RS, t96, -t95));
    const double t98 = cosB * cosB;
    const double t99 = icosB * y1;
    const double t100 = t6 * t99;
    const double t101 = iW7 * t41;
    const double t102 = (1.0 + t49);
    const double t103 = t102 * t8;
    const double t104 = (nu + t49);
    const double t105 = irb * t4;
    const double t106 = cotB * t11;
    const double t107 = -a;
    const double t108 = fma(nu, y3b, t107);
    const double t109 = fma(t56, t62, fma(t106, y1, t108 - t44));
    const double t110 = t60 * t62;
    const double t111 = y1 * y1 * y1;
    const double t112 = irb * t111;
    const double t113 = iW6 * t6;
    const double t114 = fma(t111, t113, t41);
    const double t115 = 3.0 * t62;
    const double t116 = a * cotB * irb * irb * irb * irb * irb;
    const double t117 = -t115 * t116;
    const double t118 = cosB * sinB;
    const double t119 = -t118;
    const double t120 = t6 * y3b;
    const double t121 = t120 * t99;
    const double t122 = -t82;
    const double t123 = (1.0 + t96);
    const double t124 = t123 * t24;
    const double t125 = (t122 + t124);
    const double t126 = -t125;
    const double t127 = RS * irb;
    const double t128 = t126 * t127;
    const double t129 = cotB * ((t119 + t121 + t128));
    const double t130 = (-1.0 + N1);
    const double t131 = (a + t44);
    const double t132 = fma(-irb, t131, t65 * t74);
    const double t133 = (t130 + t132 + t63);
    const double t134 = -t13 * t133;
    const double t135 = t16 * t74;
    const double t136 = iW6 * irb;
    const double t137 = icosB * t25;
    const double t138 = cosB * t123;
    const double t139 = RS * iW7;
    const double t140 = cotB * iW7;
    const double t141 = irb * t140;
    const double t142 = iW7 * sinB;
    const double t143 = t1 * z1b;
    const double t144 = iW7 * z1b;
    const double t145 = t17 * t4;
    const double t146 = t13 * y1;
    const double t147 = -cosB;
    const double t148 = (t11 + t147);
    const double t149 = (1.0 + t25);
    const double t150 = irb * z1b;
    const double t151 = t149 * t150;
    const double t152 = W1 * z1b;
    const double t153 = y2 * y2;
    const double t154 = fma(-cosB, sinB * t153, t11 * t152);
    const double t155 = -t154;
    const double t156 = iW7 * t155;
    const double t157 = t0 * (fma(-sinB, t148, fma(-irb, t156, t151)));
    const double t158 = t16 * z1b;
    const double t159 = t149 * t158;
    const double t160 = 2.0 * t118;
    const double t161 = b3 * y2;
    const double t162 = t144 * t6;
    const double t163 = t8 * ((N1 + t49));
    const double t164 = -nu;
    const double t165 = (t164 + t49);
    const double t166 = iW6 * t165;
    const double t167 = fma(t54, y1, fma(t153, t56, t108));
    const double t168 = t13 * t50;
    const double t169 = t153 * t6;
    const double t170 = iW6 * t169;
    const double t171 = -t170;
    const double t172 = irb * t153;
    const double t173 = (t107 + t44);
    const double t174 = fma(t172, t74, fma(irb, t173, t130 + t169));
    const double t175 = t13 * t174;
    const double t176 = fma(-t153, t98, t106 * t152);
    const double t177 = iW7 * t176;
    const double t178 = t41 * z1b;
    const double t179 = fma(a, cosB, t178);
    const double t180 = t60 * y3b;
    const double t181 = fma(-irb, t179, fma(t180, z1b, t98));
    const double t182 = fma(irb, t177, t181);
    const double t183 = t0 * t182;
    const double t184 = t16 * t173;
    const double t185 = t153 * t69;
    const double t186 = fma(t172, t88, t170);
    const double t187 = cotB * z1b;
    const double t188 = 3.0 * t35;
    const double t189 = irb * t0;
    const double t190 = cotB * t17;
    const double t191 = t153 * t189;
    const double t192 = t123 * t41;
    const double t193 = (t4 - t144);
    const double t194 = t193 * t51;
    const double t195 = t58 * t67;
    const double t196 = t153 * t168 * t58;
    const double t197 = fma(t146, t55, t145 + t190);
    const double t198 = N1 * t136 * t153 * t197;
    const double t199 = 2.0 * nu;
    const double t200 = t199 * t4;
    const double t201 = (iW6 + irb);
    const double t202 = t11 * t201;
    const double t203 = fma(t202, y1, t200 + t76);
    const double t204 = iW6 * t203;
    const double t205 = t153 * t16;
    const double t206 = t13 * t172;
    const double t207 = (t125 + t137);
    const double t208 = t140 * t207;
    const double t209 = nu * t13;
    const double t210 = 2.0 * t209;
    const double t211 = (t13 + t16);
    const double t212 = cotB * t207;
    const double t213 = t21 * y3b;
    const double t214 = icosB * t17;
    const double t215 = t123 * t30;
    const double t216 = irb * t48;
    const double t217 = W2 * iW7;
    const double t218 = W3 * t48;
    const double t219 = (-1.0 + nu);
    const double t220 = t213 * t219;
    const double t221 = (1.0 + t26);
    const double t222 = irb * t221;
    const double t223 = t16 * y3b;
    const double t224 = t120 * t24;
    const double t225 = y3b * y3b;
    const double t226 = 2.0 * t225;
    const double t227 = t226 * t34;
    const double t228 = fma(-CY, t217, fma(W3, t31, t224 + t227 + t90));
    const double t229 = iW6 * t199;
    const double t230 = (t17 + t229);
    const double t231 = -irb * t230;
    const double t232 = (t26 + t72);
    const double t233 = irb * t8;
    const double t234 = W3 * t2;
    const double t235 = irb * t41;
    const double t236 = t120 * t8;
    const double t237 = irb * y3b;
    const double t238 = (1.0 + t237);
    const double t239 = t238 * t88;
    const double t240 = t113 * y3b;
    const double t241 = (t239 + t240);
    const double t242 = t210 * t238;
    const double t243 = -t232;
    const double t244 = W3 * t0;
    const double t245 = cosB * t244;
    const double t246 = t223 * t8;
    const double t247 = t228 * t8;
    const double t248 = W2 * t142;
    const double t249 = t248 * t48;
    const double t250 = (t200 + t78);
    const double t251 = W3 * t8;
    const double t252 = iW6 * t238;
    const double t253 = t41 * t48;
    const double t254 = (t122 + t24);
    const double t255 = cotB * t254;
    const double t256 = W1 * irb;
    const double t257 = -sinB;
    const double t258 = fma(t158, y3b, fma(t144, t256, t257));
    const double t259 = fma(t255, t256, fma(t11, t258, t119));
    const double t260 = 2.0 * t14;
    const double t261 = t5 * y3b;
    const double t262 = cosB * t237;
    const double t263 = cotB * t24;
    const double t264 = W1 * t223;
    const double t265 = sinB * t237;
    const double t266 = t30 * z1b;
    const double t267 = iW7 * irb;
    const double t268 = UB * t143;
    const double t269 = t144 * t9;
    const double t270 = -t32;
    const double t271 = fma(iW6, t12, t270);
    const double t272 = W2 * t191;
    const double t273 = t169 * t8;
    const double t274 = t18 * t5;
    const double t275 = -t233 * t26;
    const double t276 = t16 * t22;
    const double t277 = t153 * t5;
    const double t278 = t277 * t8;
    const double t279 = t0 * t205;
    const double t280 = cosB * t279;
    const double t281 = fma(t17, t24, t213 + t270 + t31);
    const double t282 = t205 * t8;
    const double t283 = t281 * t282;
    const double t284 = fma(-sinB, t148, fma(t154, t267, t151));
    const double t285 = t14 * t95;
    const double t286 = fma(-t152, t19, fma(W1, cosB, t285));
    const double t287 = iW7 * icosB;
    const double t288 = -t58;
    const double t289 = -t203;
    const double t290 = fma(t210, t65, -t229);
    const double t291 = iW6 * t17;
    const double t292 = b2 * y2;
    const double t293 = t169 * t4;
    const double t294 = t153 * t74;
    const double t295 = t14 * t88;
    const double t296 = iW6 * t79;
    const double t297 = fma(-t136, t79, t233 * t85);
    const double t298 = irb * t18;
    const double t299 = t1 * t48;
    const double t300 = t142 * t48;
    const double t301 = t216 * t46;
    const double t302 = t13 * t238;
    const double t303 = t12 * t302;
    const double t304 = sinB * t221;
    const double t305 = t142 * t221;
    const double t306 = 3.0 * t35;
    const double t307 = cotB * t306;
    const double t308 = (t209 + t6);
    const double t309 = t260 * t308;
    const double t310 = t7 * y3b;
    const double t311 = t302 * t55;
    const double t312 = fma(t311, y1, t180 + t310);
    const double t313 = N1 * t302;
    const double t314 = W3 * t1;
    const double t315 = (-1.0 + t199);
    const double t316 = icosB * t120;
    const double t317 = fma(a, icosB * t5 * y1 * y3b, fma(-t125, t127, -t118));
    const double t318 = t61 * y3b;
    const double t319 = t64 * y3b;
    const double t320 = 3.0 * t116 * y1 * y3b;
    const double t321 = 3.0 * t225 * t34;
    const double t322 = cosB * t14;
    const double t323 = W1 * t19;
    const double t324 = t261 * y1;
    const double t325 = fma(W1, t16 * y3b * z1b, fma(-W1, sinB, -CY * z1b));
    const double t326 = t180 * t315;
    const double t327 = -cotB * t254;
    const double t328 = t256 * t327;
    const double t329 = -t11 * t258;
    const double t330 = t170 * y3b;
    const double t331 = -t176;
    v[0] = fma(b3, y2 * (fma(-t40, (fma(t26, t29, fma(t26, t28, t39 - t20 - t23))), N1 * (fma(-t12, t15, t10 + t3 -
        t7)))), fma(-t94, (fma(t58, t59, fma(t45, t8, fma(t42, t43, fma(t40, (fma(-t8, (fma(-UB, t92, fma(iW7,
        (fma(t14, t93, fma(W1, t61, SY * t82))), cotB * t37))), fma(-iW6, (fma(-irb, t89, -t64 - t87 - t91)), fma(t4,
        t80, fma(t29, t86, fma(t28, t86, fma(t15, t79, t71))))))), -t52 - t68))))), -b2 * (fma(t67, (fma(t112, t66,
        fma(-2.0, t57, t110 + t114 - t106))), fma(t27, t97, fma(t109, t59, fma(t101, (fma(-SY, t96, fma(RS, t100,
        t98))), fma(W8, (fma(-t141, (fma(-icosB, t115 * t35, fma(-RS, t126 * t19, fma(t139, (fma(-t138, t14, fma(W1,
        t100, UB * t124))), fma(SY, t126, t137))))), fma(-t136, (fma(-t131, t19, fma(t112, t88, fma(t111, t69,
        fma(t111, t135, fma(-2.0, t77, fma(-2.0, t75, t114))))))), fma(t134, t14, fma(t129, t27, t117 + t60))))), N1
        * (fma(-t104, t105, UB * t103))))))))));
    v[1] = fma(-irb, t161 * (fma(W8, (fma(iW7, (fma(irb, t0 * t155, fma(iW7, t155 * t16, fma(a, sinB * t16, fma(-t36,
        z1b, fma(-iW7, (fma(-t17, t95, fma(t152, t6, t160))), -t159)))))), t20 + t23 - t157)), N1 * (fma(-t12, t146,
        fma(t144, t17, t142 + t143 - t145))))), fma(t94, (fma(t1, t150 * t41, fma(-t67, (fma(-t172, t66, fma(2.0,
        t56, t171 + t61))), fma(-t50, ((t163 - t166)), fma(-t40, (fma(-iW7, (fma(-t187, t188, fma(-t176, t189,
        fma(-t16, t177, fma(-iW7, (fma(-t190, t95, fma(t152, t60, 2.0 * t98))), t16 * t179))))), fma(iW6, (fma(t135,
        t153, fma(-2.0, t74, fma(-2.0, t17, t184 + t185 + t186)))), t175 + t183 - t71))), fma(t167, t168, t162 *
        t41)))))), b2 * (fma(icosB, t101 * t169, fma(-t101, t123, fma(t40, (fma(-t141, t153 * (fma(-t123, t8,
        fma(t214, t24, fma(icosB, t213, t215)))), fma(t105, t153 * (fma(t17, t201, fma(t11, t211, t210))), fma(-t205,
        t208, fma(-t191, t212, fma(t204, t205, fma(t203, t206, fma(cotB, t185, t208 - t190 - t204)))))))), fma(t191,
        t192, t196 - t194 - t195 - t198)))))));
    v[2] = fma(-t142, t161 * (fma(t40, (fma(W3, iW7 * t221, fma(t221, t223, t228))), fma(t217, t218, t216 - t220 -
        t222))), fma(-t94, (fma(t48, (fma(t142, t235, t241 - t234 - t236)), fma(t40, (fma(t243, t246, fma(t243, t245,
        fma(t223, t230, t242 + t36 - t247)))), fma(t232, t233, t231)))), b2 * (fma(t239, t48 * y1, fma(-t220, t4,
        fma(-t143, t218, fma(-irb, t250, fma(t253, ((t251 - t252)), fma(t144, t220, fma(iW7, t259, fma(W8,
        (fma(-t244, t259, fma(t267, (fma(-t255, t264, fma(-t25, t258, fma(t263, (fma(-W3, t24, 1.0 + t262)), fma(t11,
        (fma(-t226, t5 * z1b, fma(-t144, t264, fma(-W3, t266, fma(W1, t142, fma(CY, t144, t150 + t265)))))), CY *
        t255))))), fma(t260, (fma(t209, t238, t35)), t250 * t261)))), t249)))))))))));
    v[3] = fma(-0.5, t292 * (fma(t197, t4 * t50, fma(t101, t214 * ((t127 + t257)), fma(-t287, t45, fma(-t192, t27,
        fma(t50, (fma(-iW6, t104, t103)), fma(t40, (fma(t16, t289 * t4, fma(-6.0, t34 * t70, fma(-t141, (fma(t139,
        (fma(W1, t214, t124 - t138)), fma(sinB, t126, fma(-3.0, t121, -t128)))), fma(-t140, (fma(cosB, iW7 * irb *
        t123 * y1, fma(-t36, t99, fma(-t100, t24, -UB * t215)))), fma(-t136, (fma(t291, t62, fma(3.0, t63, t132 +
        t89))), fma(-iW6, (fma(t17, t211 * t62, fma(t201, t63, t290 - t202))), fma(t212, t27, fma(t19, t208, fma(t15,
        t289, fma(t0, t129, t134))))))))))), fma(t288, t59, fma(t189, t97, fma(t109, t168, t52 + t68)))))))))),
        fma(0.5, b3 * (fma(-W8, (fma(-t27, t284, fma(-t153, t276, fma(-t153, t274, fma(t276, t62, fma(t274, t62,
        fma(t267, (fma(a, sinB * t16 * y1, fma(a, iW7 * irb * t286, fma(-t149, t19 * z1b, fma(-iW7, t154 * t19,
        fma(-t37, z1b, fma(-t154, t27, cosB * t149))))))), fma(t26, t280, fma(t26, t278, t275 + t283))))))))),
        fma(-N1, (fma(-t12, t13 * t65, fma(UB, t142, t268 + t269 + t271 - t64))), N1 * (fma(-t12, t206, fma(cosB,
        t272, t171 + t271 + t273)))))), 0.5 * b1 * (fma(-t67, (fma(-t14, t153 * t66, t110 + t54 - t293)), fma(-t273,
        t41, fma(-t272, t42, fma(-W8, (fma(t205, t4 * ((t21 + t291 + t88)), fma(t13, t153 * t80, fma(3.0, t116 *
        t153, fma(-t282, (fma(iW7, (fma(t118, t48, fma(W1, t190, t93))), fma(2.0, t180, -t92))), fma(-t280, t85,
        fma(-t278, t85, fma(-t267, (fma(a, cotB * iW7 * irb * t286, fma(a, cosB * cotB * t16 * y3b, fma(-t188, t70 *
        z1b, fma(t16, t179 * y1, fma(-t177, t19, fma(-t176, t27, -t42))))))), fma(t277, t296, fma(t14, t175,
        fma(t136, (fma(t19, t294, fma(t185, y1, fma(t184, y1, fma(t153, t295, t293 + t76))))), fma(UB, t183, t117 +
        t297)))))))))))), fma(-N1, (fma(-t105, t165, UB * t163)), fma(t178, t43, fma(t167, t59, fma(t162, t44, t194 +
        t195 + t198 - t196)))))))))));
    v[4] = fma(0.5, b1 * y2 * (fma(a, cosB * cotB * iW7 * t315 * t5 * y3b, fma(N1, iW7 * irb * sinB * t47 * t48,
        fma(a, cotB * t5, fma(N1, iW6 * t312, fma(-t48, (fma(t235, t46, t295 + t7 - t10 - t3)), fma(-t40, (fma(-t246,
        t85, fma(-t245, t85, fma(-t232, t29, fma(-t232, t28, fma(t8, (fma(-iW7, (fma(-t160, t219 * t237, fma(W1,
        t180, CY * t83))), fma(-cotB, t227, fma(W3, t92, t190)))), fma(t4, ((t241 + t36)), fma(t302, t79, fma(t223,
        t296, fma(t19, t230, t307 + t309 - t39)))))))))), fma(-t314, t42, fma(-t313, t58, -t297))))))))), fma(-0.5,
        t161 * (fma(UB, sinB * t299, fma(-t40, (fma(2.0, a * t33 * y3b, fma(t16, t18 * y3b, fma(-t27, t304,
        fma(-t246, t26, fma(-t245, t26, fma(-t19, t305, fma(-t142, t38, fma(t13, t238, -t247))))))))), fma(-N1,
        ((t234 + t236 - t240 - t303)), fma(t300, t9, t275 + t298 + t301))))), -0.5 * b2 * (fma(-t48, t64, fma(-t253,
        (fma(UB, t8, -t105)), fma(-t217, t82, fma(-t216, t89, fma(-t140, t317, fma(-W8, (fma(-cotB, t244 * t317,
        fma(t250, t5 * y1, fma(-t267, (fma(-t255, t322, fma(t263, (fma(UB, t24, -t322)), fma(t258, t77, fma(t255,
        t323, t11 * (fma(2.0, t324 * z1b, fma(-iW7, t285, fma(-W1, t8, fma(t144, t323, fma(UB, t266,
        -t262))))))))))), fma(-t259, t27, fma(t141, (fma(RS, t125 * t223, fma(-t321, t99, fma(-t125, t265, fma(t139,
        (fma(-CY, t123, fma(W3, t124, W1 * t316))), icosB * t77))))), fma(t136, (fma(t223, t62 * t74, fma(-t131,
        t223, fma(t306, t62, fma(t239, t62, t319))))), fma(t133, t302, fma(irb, ((t290 + t91)), t320))))))))),
        fma(t67, (fma(t311, t62, t164 + t318 + t319)), fma(t48, t74, fma(t269, t48, fma(t268, t48, fma(t244, t97,
        fma(t109, t313, fma(t101, (fma(-sinB, t137, fma(RS, t316, t118))), fma(iW6, t133, fma(N1, (fma(-t104, t252,
        t102 * t251)), t61))))))))))))))))));
    v[5] = fma(-0.5, t292 * (fma(-t216, t88 * y1, fma(-t48, t7, fma(-t301, t41, fma(-t192, t244, fma(-irb, t208,
        fma(t40, (fma(iW6, t223 * t289, fma(-t4, (fma(t120, t201, fma(t11, ((t261 + t302)), t242))), fma(-t16, t250,
        fma(-t140, (fma(a, icosB * t16, fma(CY, iW7 * t123, fma(-icosB, t227, fma(-icosB, t224, -W3 * t215))))),
        fma(-t0, ((t118 + t328 + t329)), fma(t289, t302, fma(t267, (fma(t11, z1b * (fma(irb, t24, fma(2.0, t223, t30
        - t8))), fma(t263, ((t147 + t24)), fma(cosB, t327, -t328 - t329)))), fma(t212, t244, fma(t208, t223, -t307 -
        t309)))))))))), fma(t312, t67, fma(t288, t313, fma(t287, t326, fma(t162, t48, fma(t150, t299, fma(t142, t51,
        fma(irb, t204, t60)))))))))))))), fma(-0.5, b3 * (fma(sinB, t1 * t153 * t216, fma(-t298, y1, fma(t193, t216,
        fma(t169, t300, fma(iW7, t284, fma(W8, (fma(t142, t205 * t281, fma(-t142, t222, fma(-W3, t157, fma(t279,
        t304, fma(t277, t305, fma(t267, (fma(-iW7, t11 * t325, fma(t17, z1b * (fma(-t16, t226, 1.0)), fma(t156, t16 *
        y3b, fma(-t159, y3b, fma(t155, t244, fma(sinB, t25, sinB * t149))))))), fma(t18, t324, t14 * ((t302 +
        t36)))))))))), fma(N1, (fma(-t303, y1, fma(t120, t144, fma(W3, t143, fma(W3, t142, -t248 - t310))))),
        -t249)))))))), -0.5 * b1 * (fma(-t48, (fma(a, cosB * iW7 * t153 * t5, fma(W2, cosB * irb * t0 * t153,
        fma(-t193, t235, -t186 - t32 - t87)))), fma(-t178, t314, fma(-t167, t313, fma(-iW7, t182, fma(-iW6, t174,
        fma(t67, (fma(-t153, t311, nu + t318 - t330)), fma(t248, t41, fma(t144, t326, fma(W8, (fma(2.0, t205 * t308,
        fma(-t267, (fma(-iW7, t106 * t325, fma(t16, t179 * y3b, fma(iW7, t223 * t331, fma(-t187, t321, fma(-sinB,
        t41, fma(t244, t331, fma(t190, z1b, sinB * t81)))))))), fma(-t233, t243, fma(t244, (fma(-t267, t331, t181)),
        fma(t243, t280, fma(t243, t278, fma(t230, t277, fma(t175, t238, fma(t136, (fma(t223, t294, fma(t184, y3b,
        fma(t153, t306, fma(t153, t239, t330))))), t231 - t283 - t320)))))))))), fma(N1, (fma(-t166, t238, W3 *
        t163)), t61)))))))))))));
}

}  // namespace tdhs
}  // namespace qdfn
